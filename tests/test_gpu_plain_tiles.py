"""The plain X-engine at the edges of its tiles: station counts around multiples of
the 6-station tile and the 3-station sub-block, frame counts around the pair of
frames a step takes and the runs of frames summed apart, both accumulators.

Tolerance: the plain path's bar against the float64 oracle (1e-5), far above the
few 1e-7 that FP32 sums of this length leave; a wrong or missing product is off by
order 1/frames of an auto-correlation or more.
"""

from __future__ import annotations

import numpy as np
import pytest

from abi_driver import drive_rows

pytestmark = pytest.mark.gpu

CASES = [(1, 512, 1), (3, 512, 2), (4, 1024, 33), (6, 512, 300), (7, 2048, 17), (9, 1024, 64),
         (10, 512, 31), (12, 2048, 257), (13, 512, 5), (22, 512, 40), (25, 1024, 3),
         (31, 512, 16), (97, 512, 9)]


@pytest.mark.parametrize("acc64", [False, True], ids=["fp32rows", "fp64rows"])
@pytest.mark.parametrize("n,nf,frames", CASES)
def test_tile_edges_match_the_oracle(pkg, cuda, oracle, n, nf, frames, acc64):
    torch = cuda
    rng = np.random.default_rng(1000 * n + frames)
    x = rng.integers(-60, 61, size=(n, frames, 2 * nf)).astype(np.int8)
    eng = pkg.FxEngine(n, nf, max_frames=frames, xmode=0)
    try:
        if acc64:
            eng.set_accumulator(pkg.abi.CORRX_ACC_FP64)
        acc = eng.new_acc()
        xs = torch.from_numpy(x).cuda()
        eng.accumulate(xs, frames, acc)
        torch.cuda.synchronize()
        eng.check()
        once = acc.cpu().numpy()
        eng.accumulate(xs, frames, acc)   # adds to what is there
        torch.cuda.synchronize()
        twice = acc.cpu().numpy()
    finally:
        eng.close()
    ref = oracle.correlate(x)
    assert oracle.rel_rms(once, ref) < 1e-5
    assert oracle.normalized_max_err(once, ref, n) < 1e-5
    assert np.array_equal(twice, once + once)


def test_rows_do_not_depend_on_timing(pkg, cuda):
    """The same frames give the same bits, with parts of the frames summed by several
    warps (n_freq 512) and by one."""
    torch = cuda
    rng = np.random.default_rng(5)
    for n, nf, frames in [(8, 512, 256), (24, 4096, 64)]:
        x = torch.from_numpy(rng.integers(-60, 61, size=(n, frames, 2 * nf)).astype(np.int8)).cuda()
        eng = pkg.FxEngine(n, nf, max_frames=frames, xmode=0)
        rows = []
        for _ in range(4):
            acc = eng.new_acc()
            eng.accumulate(x, frames, acc)
            rows.append(acc)
        torch.cuda.synchronize()
        eng.check()
        eng.close()
        assert all(torch.equal(rows[0], r) for r in rows[1:])


def test_few_tiles_of_long_rows(pkg, cuda, oracle):
    """18 stations, n_freq 32768 over eight devices by baseline range: the last one
    computes one tile, which as many channel tiles side by side as there are warps
    would not fit in shared memory. The rows are one device's, bit for bit."""
    n, nf, frames = 18, 32768, 8
    x = np.random.default_rng(18).integers(-60, 61, size=(1, n, frames, 2 * nf)).astype(np.int8)
    one = drive_rows(pkg, x, frames, frames)
    pkg.set_device_map([0] * 8)
    try:
        split = drive_rows(pkg, x, frames, frames, devices=list(range(8)), split_mode=0)
    finally:
        pkg.set_device_map(None)
    assert oracle.normalized_max_err(one, oracle.correlate_rows(x, frames), n) < 1e-5
    assert split.tobytes() == one.tobytes()


@pytest.mark.parametrize("acc64", [False, True], ids=["fp32rows", "fp64rows"])
@pytest.mark.parametrize("n,nf,frames", [(n, 1024, f) for n in (3, 7, 24) for f in (1, 9, 33, 257)] +
                         [(7, 32768, 9)])   # 32768: the frames are not summed in parts
def test_odd_frame_counts_in_narrow_tiles(pkg, cuda, n, nf, frames, acc64):
    """Spectra tiles narrower than the 16 channels of a warp, in launches whose last pair
    of frames has only one: the layout moves data and changes no sum, so the rows are those
    of contiguous spectra bit for bit."""
    torch = cuda
    rng = np.random.default_rng(100 * n + frames)
    x = torch.from_numpy(rng.integers(-60, 61, size=(n, frames, 2 * nf)).astype(np.int8)).cuda()
    eng = pkg.FxEngine(n, nf, max_frames=frames, xmode=0)
    rows = {}
    try:
        if acc64:
            eng.set_accumulator(pkg.abi.CORRX_ACC_FP64)
        for ytile in (nf, 2, 4, 8):
            eng.set_tiles(ytile)
            rows[ytile] = eng.new_acc()
            eng.accumulate(x, frames, rows[ytile])
        torch.cuda.synchronize()
        eng.check()
    finally:
        eng.close()
    assert rows[nf].abs().max() > 0
    for ytile in (2, 4, 8):
        assert torch.equal(rows[ytile], rows[nf]), ytile

"""The F-engine of n_freq 4096 .. 16384 (frames in groups of a CTA's warps): few frames
and ragged counts, frames missing so that the groups get out of step, lost packets.

Tolerance: the plain path's bar against the float64 oracle (1e-5); a misplaced or
stale point shows at order 1.
"""

from __future__ import annotations

import numpy as np
import pytest

from abi_driver import drive_rows

pytestmark = pytest.mark.gpu

# stations x frames of 1 and 3 leave groups without a frame; 500 and 1201 are a few
# frames per group on every SM, and one more
SHAPES = [(1, 1), (3, 1), (1, 500), (1, 1201)]


@pytest.mark.parametrize("nf", [4096, 6144, 8192, 10240, 12288, 14336, 16384])
@pytest.mark.parametrize("n,frames", SHAPES)
def test_ragged_counts_and_missing_frames(pkg, cuda, oracle, nf, n, frames):
    torch = cuda
    rng = np.random.default_rng(nf + frames)
    x = rng.integers(-128, 128, size=(n, frames, 2 * nf), dtype=np.int16).astype(np.int8)
    masks = [None]
    if frames > 1:   # every third frame only; a run missing; all but the last missing
        f = np.arange(frames)
        masks += [f % 3 == 0, (f < 100) | (f > 400), f == frames - 1]
    eng = pkg.FxEngine(n, nf, max_frames=frames, xmode=0)
    try:
        xs = torch.from_numpy(x).cuda()
        for keep in masks:
            present = None if keep is None else np.broadcast_to(keep, (n, frames))
            ms = None
            if present is not None:
                ms = torch.from_numpy(np.packbits(present.astype(np.uint8), axis=1,
                                                  bitorder="little")).cuda()
            acc = eng.new_acc()
            eng.accumulate(xs, frames, acc, mask=ms)
            torch.cuda.synchronize()
            eng.check()
            ref = oracle.correlate(x, present)
            assert oracle.rel_rms(acc.cpu().numpy(), ref) < 1e-5
    finally:
        eng.close()


@pytest.mark.parametrize("nf", [18432, 20480, 22528, 24576, 26624, 28672, 30720, 32768])
@pytest.mark.parametrize("n,frames", [(1, 1), (1, 331)])   # 331: two or three a CTA
def test_split_frames_missing(pkg, cuda, oracle, nf, n, frames):
    """Above 16384 (two transforms a frame): the next frame is regrouped during the one
    before, with frames missing in between."""
    test_ragged_counts_and_missing_frames(pkg, cuda, oracle, nf, n, frames)


@pytest.mark.parametrize("nf", [4096, 6144, 10240, 16384])
def test_every_single_packet(pkg, cuda, oracle, nf):
    """Frame f keeps only packet f mod the frame's packets."""
    torch = cuda
    packets = 2 * nf // 1024
    frames = packets + 1
    rng = np.random.default_rng(nf)
    x = rng.integers(-100, 101, size=(1, frames, 2 * nf)).astype(np.int8)
    words = np.array([[1 << (f % packets) for f in range(frames)]], dtype=np.uint32)
    kept = np.zeros_like(x)
    for f in range(frames):
        p = f % packets
        kept[0, f, p * 1024:(p + 1) * 1024] = x[0, f, p * 1024:(p + 1) * 1024]
    eng = pkg.FxEngine(1, nf, max_frames=frames, xmode=0)
    try:
        acc = eng.new_acc()
        eng.accumulate(torch.from_numpy(x).cuda(), frames, acc,
                       packets=torch.from_numpy(words.view(np.int32)).cuda())
        torch.cuda.synchronize()
        eng.check()
    finally:
        eng.close()
    assert oracle.rel_rms(acc.cpu().numpy(), oracle.correlate(kept)) < 1e-5


# Enough transforms for several frames to a CTA, each in its own group of warps: frames x
# stations from 6144 on at n_freq 4096, from 1536 on at 6144 and 8192; one station and
# several, whole rounds and ragged ones.
GROUPED = [(4096, 1, 6144), (4096, 7, 901), (6144, 1, 1536), (6144, 7, 221), (8192, 1, 1537),
           (8192, 5, 331)]


@pytest.mark.parametrize("nf,n,frames", GROUPED)
def test_groups_with_packets_missing(pkg, cuda, oracle, nf, n, frames):
    """Of station s, frame f keeps packet (f + s) mod the frame's packets alone; every
    fifth frame all of them, every seventh none."""
    torch = cuda
    packets = 2 * nf // 1024
    rng = np.random.default_rng(nf + frames + n)
    x = rng.integers(-100, 101, size=(n, frames, 2 * nf)).astype(np.int8)
    f, s = np.arange(frames)[None, :], np.arange(n)[:, None]
    words = np.uint32(1) << ((f + s) % packets).astype(np.uint32)
    words[:, ::5] = (1 << packets) - 1
    words[:, ::7] = 0
    eng = pkg.FxEngine(n, nf, max_frames=frames, xmode=0)
    try:
        acc = eng.new_acc()
        eng.accumulate(torch.from_numpy(x).cuda(), frames, acc,
                       packets=torch.from_numpy(words.view(np.int32)).cuda())
        torch.cuda.synchronize()
        eng.check()
    finally:
        eng.close()
    ref = oracle.correlate(oracle.zero_lost_packets(x, words))
    assert oracle.rel_rms(acc.cpu().numpy(), ref) < 1e-5


@pytest.mark.parametrize("xmode,ytile", [(0, 2), (0, 64), (1, 8), (2, 4)])
@pytest.mark.parametrize("nf,n,frames", GROUPED)
def test_groups_in_channel_tiles(pkg, cuda, oracle, nf, n, frames, xmode, ytile):
    """Frames missing; spectra in channel tiles give the rows of contiguous spectra bit for
    bit, and the plain ones are the oracle's."""
    torch = cuda
    rng = np.random.default_rng(nf + frames + n)
    x = rng.integers(-100, 101, size=(n, frames, 2 * nf)).astype(np.int8)
    keep = rng.random((n, frames)) > 0.3
    xs = torch.from_numpy(x).cuda()
    mask = torch.from_numpy(np.packbits(keep.astype(np.uint8), axis=1, bitorder="little")).cuda()
    eng = pkg.FxEngine(n, nf, max_frames=frames, xmode=xmode)
    rows = []
    try:
        for tiles in [(nf, 8, 16), (ytile, ytile, 16)]:
            eng.set_tiles(*tiles)
            rows.append(eng.new_acc())
            eng.accumulate(xs, frames, rows[-1], mask=mask)
        torch.cuda.synchronize()
        eng.check()
    finally:
        eng.close()
    assert torch.equal(rows[0], rows[1])
    if ytile == 2:
        assert oracle.rel_rms(rows[0].cpu().numpy(), oracle.correlate(x, keep)) < 1e-5


@pytest.mark.parametrize("nf,frames", [(4096, 256), (8192, 64)])
def test_groups_without_a_frame(pkg, cuda, oracle, nf, frames):
    """24 stations over eight devices by baseline range: each device has too few of the
    run's frames for all of its groups, and takes the kernel that one device takes. The
    rows are one device's, bit for bit."""
    x = np.random.default_rng(nf).integers(-60, 61, size=(1, 24, frames, 2 * nf)).astype(np.int8)
    one = drive_rows(pkg, x, frames, frames, chunk_frames=frames)
    pkg.set_device_map([0] * 8)
    try:
        split = drive_rows(pkg, x, frames, frames, chunk_frames=frames, devices=list(range(8)),
                           split_mode=0)
    finally:
        pkg.set_device_map(None)
    assert oracle.normalized_max_err(one, oracle.correlate_rows(x, frames), 24) < 1e-5
    assert split.tobytes() == one.tobytes()

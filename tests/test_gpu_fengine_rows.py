"""The F-engine of n_freq 4096 .. 16384 (frames in groups of a CTA's warps): few frames
and ragged counts, frames missing so that the groups get out of step, lost packets.

Tolerance: the plain path's bar against the float64 oracle (1e-5); a misplaced or
stale point shows at order 1.
"""

from __future__ import annotations

import numpy as np
import pytest

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


# Launches long enough for several frames to a CTA, each in its own group of warps:
# n_freq 4096 from 256 frames on, 6144 and 8192 from 64. One station leaves groups without
# a frame (256 and 64 frames are fewer than the GPU's groups), three go round several times.
GROUPED = [(4096, 256), (4096, 301), (6144, 64), (6144, 101), (8192, 64), (8192, 203)]


@pytest.mark.parametrize("n", [1, 3])
@pytest.mark.parametrize("nf,frames", GROUPED)
def test_groups_with_packets_missing(pkg, cuda, oracle, nf, frames, n):
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
@pytest.mark.parametrize("n", [1, 3])
@pytest.mark.parametrize("nf,frames", GROUPED)
def test_groups_in_channel_tiles(pkg, cuda, nf, frames, n, xmode, ytile):
    """Spectra in channel tiles, frames missing: the rows of contiguous spectra bit for bit
    (those against the oracle: test_ragged_counts_and_missing_frames)."""
    torch = cuda
    rng = np.random.default_rng(nf + frames + n)
    x = torch.from_numpy(rng.integers(-100, 101, size=(n, frames, 2 * nf)).astype(np.int8)).cuda()
    keep = rng.random((n, frames)) > 0.3
    mask = torch.from_numpy(np.packbits(keep.astype(np.uint8), axis=1, bitorder="little")).cuda()
    eng = pkg.FxEngine(n, nf, max_frames=frames, xmode=xmode)
    rows = []
    try:
        for tiles in [(nf, 8, 16), (ytile, ytile, 16)]:
            eng.set_tiles(*tiles)
            rows.append(eng.new_acc())
            eng.accumulate(x, frames, rows[-1], mask=mask)
        torch.cuda.synchronize()
        eng.check()
    finally:
        eng.close()
    assert rows[0].abs().max() > 0
    assert torch.equal(rows[0], rows[1])

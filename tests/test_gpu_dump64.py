"""corrx_dump of complex128 rows: the double quotient rounded once to float.

Values of every size: ordinary sums, zeros, values around and past the range the
FP32 arithmetic takes, subnormal and overflowing results, infinities, NaN. Tolerance:
the product is formed to 2^-46, so a result may differ from the correctly rounded one
only by one unit in the last place, and only where the quotient is within 2^-21 units
of a tie: none expected in a few thousand values, one in 10^6 allowed.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames", [1, 3, 301, 1024, 4095, 1 << 40])
def test_dump_rounds_once(pkg, cuda, frames):
    torch = cuda
    n, nf = 3, 1024
    rng = np.random.default_rng(frames % 1000)
    v = rng.standard_normal((6, nf, 2)) * np.exp2(rng.uniform(-30, 60, size=(6, nf, 2)))
    special = [0.0, -0.0, 1.0, -1.0, 2.0 ** -63, 2.0 ** -63 * (1 - 2.0 ** -53), 2.0 ** 65,
               2.0 ** 65 * (1 - 2.0 ** -53), 1e-40, -1e-45, 1e-320, 1e38, 3.5e38, -1e300,
               np.inf, -np.inf, np.nan, 1 + 2.0 ** -24, 1 + 2.0 ** -24 + 2.0 ** -52,
               1 + 3 * 2.0 ** -24, 1 + 2.0 ** -24 - 2.0 ** -52]
    flat = v.reshape(-1)
    flat[:len(special)] = special
    flat[-len(special):] = special
    eng = pkg.FxEngine(n, nf, max_frames=1, xmode=0)
    try:
        eng.set_accumulator(pkg.abi.CORRX_ACC_FP64)
        acc = torch.view_as_complex(torch.from_numpy(v).cuda().contiguous())
        out = eng.dump(acc, frames)
        torch.cuda.synchronize()
        got = torch.view_as_real(out).cpu().numpy().reshape(-1)
    finally:
        eng.close()
    with np.errstate(over="ignore", under="ignore", invalid="ignore"):
        want = (flat * (1.0 / frames)).astype(np.float32)
    special_at = np.r_[0:len(special), flat.size - len(special):flat.size]
    np.testing.assert_array_equal(got[special_at].view(np.uint32) * (1 - np.isnan(want[special_at])),
                                  want[special_at].view(np.uint32) * (1 - np.isnan(want[special_at])))
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = np.isfinite(want)
    off = got[ok].view(np.int32).astype(np.int64) - want[ok].view(np.int32).astype(np.int64)
    assert np.abs(off).max() <= 1 and np.count_nonzero(off) <= max(1, flat.size // 10 ** 6)
    assert np.array_equal(got[~ok & ~np.isnan(want)], want[~ok & ~np.isnan(want)])


@pytest.mark.parametrize("frames", [1, 3, 7, 301, 1024, 4095, 1000003, 1 << 40, (1 << 40) + 1])
def test_dump_near_ties(pkg, cuda, frames):
    """Quotients at and within a few last places (of the double) of a tie between two
    floats, where the 24 and 23 bits of the FP32 arithmetic do not decide: the correctly
    rounded float of the double product, without exception."""
    torch = cuda
    n, nf = 3, 4096
    s = 1.0 / frames
    rng = np.random.default_rng(frames % 1000)
    shape = (6, nf, 2)
    tie = 2 * rng.integers(1 << 23, 1 << 24, size=shape).astype(np.float64) + 1
    tie *= np.exp2(rng.integers(-24, 0, size=shape)) * rng.choice([-1.0, 1.0], size=shape)
    v = tie / s
    steps = rng.integers(-300, 301, size=shape)
    steps[rng.random(shape) < 0.6] %= 4
    v = (v.view(np.int64) + steps).view(np.float64)
    v = np.where(np.abs(v) < 2.0 ** 65, v, 1.0)
    eng = pkg.FxEngine(n, nf, max_frames=1, xmode=0)
    try:
        eng.set_accumulator(pkg.abi.CORRX_ACC_FP64)
        out = eng.dump(torch.view_as_complex(torch.from_numpy(v).cuda().contiguous()), frames)
        torch.cuda.synchronize()
        got = torch.view_as_real(out).cpu().numpy()
    finally:
        eng.close()
    want = (v * s).astype(np.float32)
    assert np.count_nonzero(got.view(np.uint32) != want.view(np.uint32)) == 0

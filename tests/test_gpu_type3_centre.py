"""The FP32 type-3 kernels against FP64 data through the same gridding, where
the gridding's pre- and post-compensation are near 1: values and compared
frequencies in the middle of extents that single ones at the ends set (those
points carry no value).  Without the compensations' dynamic range only FP32
rounding is left.

Tolerance: weights (an exponential of an exact argument, 2 units of 2^-24), sums
of a cell's points (a few units), the FFT (18 radix-2 stages' worth in
quadrature, three times that for a side with a large prime), sums of a
footprint's taps (two units): under 20 units in quadrature; 64 are allowed."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _middle(rng, n, lo, hi):
    """n values in the middle 30 percent of [lo, hi], after lo and hi themselves."""
    return np.concatenate([[lo, hi], (lo + hi) / 2 + (hi - lo) * rng.uniform(-0.15, 0.15, n)])


@pytest.mark.parametrize("eps,M,N,scale", [
    (0.5, 300, 200, 1.0), (1e-4, 1000, 777, 3.0), (1e-6, 33, 65, 1.0), (1e-6, 20000, 30000, 0.02),
    (1e-6, 50, 60, 8.0),  # far fewer than tiles
    (1e-6, 100000, 50000, 1.0), (1e-9, 5000, 4000, 1.0), (1e-13, 500, 300, 1.0),
])
def test_f32_matches_f64(eps, M, N, scale):
    from miscellaneous_gb300.nufft3 import NUFFT_2D
    rng = np.random.default_rng(M + N)
    x, y = scale * _middle(rng, M, -40, 25), scale * _middle(rng, M, -18, 20)
    s, t = _middle(rng, N, -3, 4), _middle(rng, N, -2.5, 2.5)
    f = torch.tensor((rng.standard_normal(M + 2) + 1j * rng.standard_normal(M + 2)).astype(np.complex64))
    f[:2] = 0
    want = NUFFT_2D(x, y, s, t, f.to(torch.complex128), eps)[2:]
    got = NUFFT_2D(x, y, s, t, f, eps)[2:]
    assert float((got.to(torch.complex128) - want).norm() / want.norm()) < 64 * 2.0 ** -24

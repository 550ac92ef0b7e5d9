"""The FP32 type-3 kernels (dense products over tile patches) against FP64
data through the same gridding, which runs other kernels: patch edges that
fill their register tiles and that do not, ragged batches, single points and
frequencies, more than one work item a tile.

Tolerance: FP32 rounding, 2^-24, times the dynamic range of the gridding, the
pre-compensation exp(b pi^2 / 4) of each dimension at the extents' edge (b =
(msp - 2) / 4 pi; 2 * 10^3 at eps 1e-6, 4 * 10^5 at 1e-13), with a factor of 4;
at least 1e-5, the bound FP32 data are held to against exact sums."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps,M,N,scale", [
    (0.5, 300, 200, 1.0),       # the narrowest footprint
    (1e-2, 2, 1, 1.0),          # one batch of two points, one frequency
    (1e-4, 1000, 777, 3.0),
    (1e-6, 33, 65, 1.0),        # just over one batch each
    (1e-6, 20000, 30000, 0.02),  # all in a few tiles: several items a tile
    (1e-13, 500, 300, 1.0),     # the widest patches
])
def test_f32_matches_f64(eps, M, N, scale):
    from miscellaneous_gb300.nufft3 import NUFFT_2D
    rng = np.random.default_rng(M + N)
    x, y = scale * rng.uniform(-40, 25, M), scale * rng.normal(0, 6, M)
    s, t = rng.uniform(-3, 4, N), rng.uniform(-2.5, 2.5, N)
    f = torch.tensor((rng.standard_normal(M) + 1j * rng.standard_normal(M)).astype(np.complex64))
    want = NUFFT_2D(x, y, s, t, f.to(torch.complex128), eps)
    got = NUFFT_2D(x, y, s, t, f, eps)
    assert got.dtype == torch.complex64
    msp = 2 + 2 * 2.2 ** 2 * -math.log(eps / 76) / (math.pi * (2.2 ** 2 - 2))
    bound = max(1e-5, 4 * 2.0 ** -24 * math.exp((msp - 2) / (4 * math.pi) * math.pi ** 2 / 2))
    assert float((got.to(torch.complex128) - want).norm() / want.norm()) < bound

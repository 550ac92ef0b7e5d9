"""Binning in one launch (up to 2^17 points, up to 2048 tiles) against the separate
passes, which plans with a chunk above the spread's item size keep: the same
cells in the same order, a permutation, the same transforms.

Tolerance of the transforms: the same records in another order within a cell,
so sums of M_cell terms in another order: 1e-6 relative in FP32, 1e-13 in FP64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _points(M, seed, dtype, width=1.0):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return [width * (torch.rand(M, generator=g, device="cuda", dtype=dtype) - 0.5) for _ in range(2)]


def _cells(x, N, n):
    v = np.rint(x.double().cpu().numpy() * (2.0 * N))
    return np.mod(v, n).astype(np.int64)


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("N1,N2,M,width,coords", [
    (10, 14, 1, 1.0, torch.float64),
    (32, 32, 31, 1.0, torch.float32),
    (64, 64, 4097, 0.02, torch.float32),      # a few cells hold all points
    (250, 378, 65537, 1.0, torch.float32),    # reduction in FP64, cut last tiles
    (256, 256, 131072, 1.0, torch.float64),   # the most points
    (256, 256, 131073, 1.0, torch.float32),   # separate passes
    (512, 256, 70000, 0.3, torch.float32),    # 2048 tiles
    (528, 256, 70000, 0.3, torch.float32),    # separate passes
])
def test_same_as_separate_passes(precision, N1, N2, M, width, coords):
    from miscellaneous_gb300.nfft import Plan
    x1, x2 = _points(M, 7, coords, width)
    ctype = torch.complex64 if precision == "f32" else torch.complex128
    F = torch.randn(N1, N2, device="cuda", dtype=ctype)
    f = torch.randn(M, device="cuda", dtype=ctype)
    res = []
    for tuning in ({}, {"chunk": 4096}):
        with Plan(N1, N2, precision=precision) as p:
            p.set_tuning(**tuning)
            got = []
            for y1, y2, kw in ((x1, x2, {}), (x2, x1, {"sync": False}), (x1, x2, {"sync": False})):
                p.set_points(y1, y2, **kw)
                perm = p.permutation().cpu().numpy()
                assert np.array_equal(np.sort(perm), np.arange(M))
                got.append((_cells(y1, N1, 2 * N1)[perm], _cells(y2, N2, 2 * N2)[perm], p.forward(F), p.adjoint(f)))
            out = p.bin_and_forward(x1, x2, F)
            p.synchronize()
            got.append((out,))
            res.append(got)
    tol = 1e-6 if precision == "f32" else 1e-13
    for a, b in zip(*res):
        if len(a) == 4:
            assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
        for u, v in zip(a[-2:] if len(a) == 4 else a, b[-2:] if len(b) == 4 else b):
            assert float((u - v).norm() / v.norm()) < tol


@pytest.mark.parametrize("sync", [True, False])
def test_nonfinite_is_reported_and_forgotten(sync):
    from miscellaneous_gb300 import _lib
    from miscellaneous_gb300.nfft import Plan
    x1, x2 = _points(3000, 3, torch.float32)
    bad = x1.clone()
    bad[2999] = float("nan")
    F = torch.randn(64, 64, device="cuda", dtype=torch.complex64)
    with Plan(64, 64) as p:
        with pytest.raises(_lib.NFFT2DError):
            p.set_points(bad, x2, sync=sync)
            p.synchronize()
        p.set_points(x1, x2, sync=sync)
        out = p.forward(F)
        p.synchronize()
        assert bool(torch.isfinite(out.abs()).all())

"""The fused FFT passes for sides of small prime factors (the default where the
grid is no power of two a side) against FP64 plans and against cuFFT (fft_mode
0): every factor, repeated factors, sides at the shortest and longest it takes,
long and narrow grids, and sizes next to the rule's lines that keep cuFFT.

Tolerance: the FFT's FP32 rounding (at most 24 radix-2 stages' worth at 2^-24,
adding in quadrature; a radix-13 butterfly is 12 additions deep at most, that of
a larger prime, at most 67, half as many terms) and
that of tables and weights stays under 1e-6 relative for w 6; cuFFT's FP32 error
adds to it in the comparison with fft_mode 0."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(N1, N2, x1, x2, F, f, precision="f32", **tuning):
    from miscellaneous_gb300.nfft import Plan
    c = torch.complex64 if precision == "f32" else torch.complex128
    r = torch.float32 if precision == "f32" else torch.float64
    with Plan(N1, N2, precision=precision) as p:
        if tuning:
            p.set_tuning(**tuning)
        p.set_points(x1.to(r), x2.to(r))
        out = p.forward(F.to(c)), p.adjoint(f.to(c)), p.bin_and_forward(x1.to(r), x2.to(r), F.to(c))
        p.synchronize()
        return p.info()["fft_mode"], out


def _rel(a, b):
    return float((a.to(torch.complex128) - b.to(torch.complex128)).norm() / b.norm())


@pytest.mark.parametrize("N1,N2,mode", [
    (32, 36, 2), (36, 32, 2), (50, 50, 2), (44, 52, 2), (98, 162, 2), (242, 338, 2), (250, 378, 2),
    (1458, 34 + 2, 2), (40, 1250, 2), (2000, 66, 2), (66, 2048, 2), (1024, 50, 2), (686, 700, 2),
    (1100, 1300, 2), (2000, 2000, 2),
    (34, 36, 2), (38, 46, 2), (106, 134, 2), (244, 248, 2), (510, 512, 2), (58, 1360, 2),  # one prime from 17 to 67
    (1536, 1536, 1), (1050, 1024, 1), (1230, 1230, 1), (250, 382, 0), (142, 50, 0), (782, 800, 0), (30, 50, 0),
])
def test_mixed_fft(N1, N2, mode):
    g = torch.Generator(device="cuda")
    g.manual_seed(N1 * 4099 + N2)
    M = 3001
    x1, x2 = [torch.rand(M, generator=g, device="cuda") - 0.5 for _ in range(2)]
    F = torch.randn(N1, N2, generator=g, device="cuda", dtype=torch.complex64)
    f = torch.randn(M, generator=g, device="cuda", dtype=torch.complex64)
    got_mode, got = _run(N1, N2, x1, x2, F, f)
    assert got_mode == mode
    _, exact = _run(N1, N2, x1, x2, F, f, precision="f64")
    _, lib = _run(N1, N2, x1, x2, F, f, fft_mode=0)
    for a, e, b in zip(got, exact, lib):
        assert _rel(a, e) < 1e-6
        assert _rel(a, b) < 2e-6


def test_grid_is_reused_across_directions_and_non_finite_data():
    """A transform reads nothing of what another left in the grid."""
    from miscellaneous_gb300.nfft import Plan
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    x1, x2 = [torch.rand(2000, generator=g, device="cuda") - 0.5 for _ in range(2)]
    F = torch.randn(100, 90, generator=g, device="cuda", dtype=torch.complex64)
    f = torch.randn(2000, generator=g, device="cuda", dtype=torch.complex64)
    with Plan(100, 90) as p:
        p.set_points(x1, x2)
        a, b = p.forward(F), p.adjoint(f)
        p.adjoint(torch.full_like(f, float("nan")))
        p.forward(torch.full_like(F, float("inf")))
        c, d = p.forward(F), p.adjoint(f)
        p.synchronize()
    assert torch.equal(a, c) and _rel(d, b) < 1e-6

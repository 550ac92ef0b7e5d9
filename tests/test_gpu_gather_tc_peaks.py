"""The tensor-core gather on grids with one strong peak, whose neighbouring
cells differ by many powers of two, and at points that meet the peak only with
the tails of their windows: compared with the FP32 gather of the same plan
sizes (gather_variant tiled), both against FP64 plans, by size of the result.

Tolerance: what the split operands leave out is at most 2^-26 of the largest
cell a tap, and the peak's cells are a few taps; the sums differ in rounding,
10 percent of the FP32 gather's own error."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _taper(N, beta):
    n = torch.arange(N, device="cuda", dtype=torch.float64) - N / 2
    z = beta * torch.sqrt(torch.clamp(1 - (2 * n / N) ** 2, min=0))
    return torch.special.i0(z) / math.exp(beta)


def _run(N, K, x, F, precision="f32", **tuning):
    from miscellaneous_gb300.nfft import Plan
    with Plan(N, N, K=K, precision=precision) as p:
        p.set_tuning(**tuning)
        p.set_points(*x)
        out = p.forward(F)
        p.synchronize()
        return p.paths()["gather"], out


@pytest.mark.parametrize("K", [6, 7, 8])
@pytest.mark.parametrize("beta", [6.0, 12.0])
def test_peak_and_tails(K, beta):
    N, M = 512, 1 << 20
    g = torch.Generator(device="cuda")
    g.manual_seed(K)
    x = [torch.rand(M, generator=g, device="cuda") - 0.5 for _ in range(2)]
    for v in x:  # half of the points within 12 cells of the peak
        v[: M // 2] *= 24 / (2 * N)
    t = _taper(N, beta)
    F = (t[:, None] * t[None]).to(torch.complex64)
    path, tc = _run(N, K, x, F)
    assert path == 2
    path, ref = _run(N, K, x, F, gather_variant=1)
    assert path == 0
    _, want = _run(N, K, [v.double() for v in x], F.to(torch.complex128), precision="f64")
    size, top = want.abs(), float(want.abs().max())
    e_tc, e_ref = (tc - want).abs(), (ref - want).abs()
    for d in range(7):
        at = (size <= top * 10.0 ** -d) & (size > top * 10.0 ** -(d + 1))
        assert int(at.sum()) > 1000
        rms = [float(e[at].square().mean().sqrt()) for e in (e_tc, e_ref)]
        assert rms[0] < 1.1 * rms[1] + 2.0 ** -26 * top, (d, rms)

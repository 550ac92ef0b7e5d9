"""Kernels that may start while the one before them ends: back-to-back calls on
fresh data give what the same calls give with a wait after each, captured calls
what direct ones give.

Tolerance: the spread adds patches in any order, 1e-6 relative in FP32 (the
forward sums in a fixed one)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a - b).norm() / b.norm())


@pytest.mark.parametrize("N1,N2,M", [(256, 256, 9000), (250, 378, 200000), (512, 512, 300000), (100, 90, 140000)])
def test_back_to_back_and_captured(N1, N2, M):
    from miscellaneous_gb300.nfft import Plan
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    rounds = 12
    x = [[torch.rand(M, generator=g, device="cuda") - 0.5 for _ in range(2)] for _ in range(rounds)]
    F = [torch.randn(N1, N2, generator=g, device="cuda", dtype=torch.complex64) for _ in range(rounds)]
    f = [torch.randn(M, generator=g, device="cuda", dtype=torch.complex64) for _ in range(rounds)]
    with Plan(N1, N2) as p:
        want = []
        for i in range(rounds):
            p.set_points(*x[i])
            a = p.forward(F[i])
            torch.cuda.synchronize()
            b = p.adjoint(f[i])
            torch.cuda.synchronize()
            want.append((a, b))
        got = []
        for i in range(rounds):  # nothing waits between these
            p.set_points(*x[i], sync=False)
            got.append((p.forward(F[i] * 1), p.adjoint(f[i] * 1)))
        p.synchronize()
        for (a, b), (c, d) in zip(got, want):
            assert _rel(a, c) < 1e-6 and _rel(b, d) < 1e-6
        s = torch.cuda.Stream()
        p.set_stream(s)
        out, Out = torch.empty_like(f[0]), torch.empty_like(F[0])
        Fin, fin = F[0].clone(), f[0].clone()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            p.forward(Fin, out=out)
            p.adjoint(fin, out=Out)
        last = want[rounds - 1]
        Fin.copy_(F[rounds - 1])
        fin.copy_(f[rounds - 1])
        for _ in range(5):
            graph.replay()
        torch.cuda.synchronize()
        assert _rel(out, last[0]) < 1e-6 and _rel(Out, last[1]) < 1e-6

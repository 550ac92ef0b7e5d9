"""Whole transforms in one launch (small FP32 plans) against FP64 plans of the
same window on the same points: every window width, square and rectangular
grids up to the largest it takes, point counts at its edges, points in one
tile, the options that reach it, capture and two streams.

Tolerance: FP32 rounding of the FFTs (at most 16 radix-2 stages at 2^-24 each,
adding in quadrature), tables and weights stays under 1e-6 relative; the FP64
plan of the same width has the same window error."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(N1, N2, M, seed, width=1.0):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = [width * (torch.rand(M, generator=g, device="cuda") - 0.5) for _ in range(2)]
    F = torch.randn(N1, N2, generator=g, device="cuda", dtype=torch.complex64)
    f = torch.randn(M, generator=g, device="cuda", dtype=torch.complex64)
    return x[0], x[1], F, f


def _exact(N1, N2, K, x1, x2, F, f):
    from miscellaneous_gb300.nfft import Plan
    with Plan(N1, N2, K=K, precision="f64") as p:
        p.set_points(x1.double(), x2.double())
        out = p.forward(F.to(torch.complex128)), p.adjoint(f.to(torch.complex128))
        p.synchronize()
    return out


def _rel(a, b):
    return float((a.to(torch.complex128) - b).norm() / b.norm())


@pytest.mark.parametrize("K", range(2, 9))
@pytest.mark.parametrize("N1,N2,M,width", [
    (32, 32, 1, 1.0), (32, 64, 33, 1.0), (64, 32, 1000, 1.0), (64, 64, 4097, 1.0), (64, 64, 16384, 0.1),
    (32, 256, 8191, 1.0), (256, 32, 8192, 1.0), (64, 64, 8192, 1.0), (128, 128, 4096, 1.0), (64, 64, 32768, 1.0),
    (64, 64, 8193, 1.0), (64, 64, 32769, 1.0), (128, 128, 4097, 0.3),  # next to the rule's lines
])
def test_matches_f64(K, N1, N2, M, width):
    from miscellaneous_gb300.nfft import Plan
    x1, x2, F, f = _inputs(N1, N2, M, seed=K, width=width)
    want, Want = _exact(N1, N2, K, x1, x2, F, f)
    with Plan(N1, N2, K=K) as p:
        p.set_points(x1, x2)
        for _ in range(3):  # the barrier's words are back at zero after each
            out, Out = p.forward(F), p.adjoint(f)
        p.set_tuning(io_order="binned")
        perm = p.permutation().long()
        binned, Binned = p.forward(F), p.adjoint(f[perm])
        p.set_tuning(io_order="caller", compensated=0)
        p.set_points(x1, x2, sync=False)  # work items counted on the device only
        late, Late = p.forward(F), p.adjoint(f)
        p.synchronize()
    for a in (out, late):
        assert _rel(a, want) < 1e-6
    assert _rel(binned, want[perm]) < 1e-6
    for a in (Out, Binned, Late):
        assert _rel(a, Want) < 1e-6


def test_one_launch_and_separate_kernels_agree():
    """bin_and_forward, captured calls and a second stream's plan give what the
    separate kernels (fft_mode 2) give."""
    from miscellaneous_gb300.nfft import Plan
    x1, x2, F, f = _inputs(64, 64, 4096, seed=5)
    with Plan(64, 64) as p:
        p.set_tuning(fft_mode=2)
        p.set_points(x1, x2)
        want, Want = p.forward(F).to(torch.complex128), p.adjoint(f).to(torch.complex128)
    with Plan(64, 64) as p, Plan(64, 64, stream=torch.cuda.Stream()) as q:
        assert _rel(p.bin_and_forward(x1, x2, F), want) < 1e-6
        q.set_points(x1, x2)
        p.set_points(x1, x2)
        torch.cuda.synchronize()
        out, Out, other = torch.empty_like(f), torch.empty_like(F), torch.empty_like(f)
        for _ in range(50):
            p.adjoint(f, out=Out)
            q.forward(F, out=other)
            p.forward(F, out=out)
        torch.cuda.synchronize()
        for a, b in ((out, want), (Out, Want), (other, want)):
            assert _rel(a, b) < 1e-6
        s = torch.cuda.Stream()
        p.set_stream(s)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            p.forward(F, out=out)
            p.adjoint(f, out=Out)
        out.zero_(), Out.zero_()
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
        assert _rel(out, want) < 1e-6 and _rel(Out, Want) < 1e-6

"""The gather of bin_and_forward reads the binning's records and work items,
which the kernels just before it on its stream write: behind a backlog on that
stream, on points the plan has not met, and in a captured call whose points
change between replays, it gives what set_points and forward give.  Both
gathers that may begin early in other calls, on sets binned by the separate
passes.

Tolerance: one gather, the same records in the same cells; a record's place
within its cell may change, not its own sum: equal bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _points(M, seed, width):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return [width * (torch.rand(M, generator=g, device="cuda") - 0.5) for _ in range(2)]


def _want(N, M, variant, sets, F):
    from miscellaneous_gb300.nfft import Plan
    out = []
    with Plan(N, N) as p:
        p.set_tuning(gather_variant=variant)
        for x in sets:
            p.set_points(*x)
            out.append(p.forward(F))
            p.synchronize()
    return out


@pytest.mark.parametrize("variant", [1, 2])  # tiled, direct
@pytest.mark.parametrize("N,M", [(64, 70000), (512, 200001), (250, 131073)])
def test_behind_a_backlog_on_new_points(N, M, variant):
    from miscellaneous_gb300.nfft import Plan
    sets = [_points(M, s, w) for s, w in ((1, 1.0), (2, 0.05), (3, 0.6), (4, 1.0))]
    F = torch.randn(N, N, device="cuda", dtype=torch.complex64)
    want = _want(N, M, variant, sets, F)
    big = torch.empty(1 << 27, device="cuda")
    s = torch.cuda.Stream()
    with Plan(N, N, stream=s) as p:
        p.set_tuning(gather_variant=variant)
        p.set_points(*sets[3])
        torch.cuda.synchronize()
        for _ in range(3):
            got = []
            with torch.cuda.stream(s):
                for _ in range(4):
                    big.fill_(1.0)  # the host runs ahead of the stream from here
                for x in sets:
                    got.append(p.bin_and_forward(*x, F))
            p.synchronize()
            for a, b in zip(got, want):
                assert torch.equal(a, b)


@pytest.mark.parametrize("variant", [1, 2])
@pytest.mark.parametrize("N,M", [(64, 70000), (512, 200001), (250, 131073)])
def test_captured(N, M, variant):
    from miscellaneous_gb300.nfft import Plan
    sets = [_points(M, s, w) for s, w in ((1, 1.0), (2, 0.05), (3, 0.6))]
    F = torch.randn(N, N, device="cuda", dtype=torch.complex64)
    want = _want(N, M, variant, sets, F)
    s = torch.cuda.Stream()
    x, out = [v.clone() for v in sets[0]], torch.empty(M, device="cuda", dtype=torch.complex64)
    with Plan(N, N, stream=s) as p:
        p.set_tuning(gather_variant=variant)
        p.bin_and_forward(*sets[1], F, out=out)  # the plan's buffers are there before the capture
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            p.bin_and_forward(*x, F, out=out)
        for k in (0, 1, 2, 1, 0):
            for v, w in zip(x, sets[k]):
                v.copy_(w)
            out.zero_()
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(out, want[k])
        p.synchronize()

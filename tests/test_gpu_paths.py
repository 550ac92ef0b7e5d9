"""Which kernels a plan's calls run, on both sides of every line of the rules:
the tests of a kernel reach it, those next to a line do not.  Their results
are held by the tests of each kernel at the same sizes, but for the longest
grids of the one-launch transforms, which are compared with FP64 plans here.

Tolerance there: FP32 rounding of the FFTs (15 radix-2 stages' worth at 2^-24
each, adding in quadrature), tables and weights stays under 1e-6 relative; the
FP64 plan of the same width has the same window error."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _x(M):
    return [torch.rand(M, device="cuda") - 0.5 for _ in range(2)]


def _paths(N1, N2, M, tuning=None, bin_and_forward=False, **kw):
    from miscellaneous_gb300.nfft import Plan
    with Plan(N1, N2, **kw) as p:
        p.set_tuning(**(tuning or {}))
        assert p.paths()["binning"] == 0
        if bin_and_forward:
            p.bin_and_forward(*_x(M), torch.zeros(N1, N2, device="cuda", dtype=p.cdtype))
        else:
            p.set_points(*_x(M))
        d = p.paths()
        p.synchronize()
        return d


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("N1,N2,M,tuning,want", [
    (10, 14, 1, {}, 2), (256, 256, 1 << 17, {}, 2), (256, 256, (1 << 17) + 1, {}, 1),
    (512, 256, 70000, {}, 2), (528, 256, 70000, {}, 1),  # 2048 tiles, 2112
    (64, 64, 4096, {"chunk": 512}, 2), (64, 64, 4096, {"chunk": 513}, 1),
])
def test_binning(N1, N2, M, tuning, want, precision):
    assert _paths(N1, N2, M, tuning, precision=precision)["binning"] == want


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("M,want", [(1 << 16, 2), ((1 << 16) + 1, 1)])
def test_binning_without_a_wait(M, want, precision):
    from miscellaneous_gb300.nfft import Plan
    with Plan(64, 64, precision=precision) as p:
        p.set_points(*_x(M), sync=False)
        assert p.paths()["binning"] == want
        p.synchronize()


@pytest.mark.parametrize("M,precision,want", [(1 << 16, "f32", 2), ((1 << 16) + 1, "f32", 1), (1000, "f64", 1)])
def test_binning_beside_the_forward(M, precision, want):
    assert _paths(64, 64, M, bin_and_forward=True, precision=precision)["binning"] == want


@pytest.mark.parametrize("K", range(2, 9))
@pytest.mark.parametrize("N1,N2,M,forward,adjoint", [
    (32, 32, 1, 1, 1), (64, 64, 1 << 13, 1, 1), (64, 64, (1 << 13) + 1, 0, 1), (64, 64, 1 << 15, 0, 1),
    (64, 64, (1 << 15) + 1, 0, 0), (32, 256, 4096, 0, 1), (32, 256, 4097, 0, 0), (128, 128, 4096, 0, 1),
    (128, 128, 4097, 0, 0), (128, 256, 1000, 0, 0), (32, 36, 1000, 0, 0),
])
def test_one_launch_transforms(K, N1, N2, M, forward, adjoint):
    d = _paths(N1, N2, M, K=K)
    assert (d["forward"], d["adjoint"]) == (forward, adjoint)


@pytest.mark.parametrize("K", [2, 6, 7])
@pytest.mark.parametrize("N1,N2,M", [(32, 256, 4096), (256, 32, 4000), (32, 128, 1 << 13), (128, 32, 77)])
def test_one_launch_on_long_grids(K, N1, N2, M):
    from miscellaneous_gb300.nfft import Plan
    x = _x(M)
    F = torch.randn(N1, N2, device="cuda", dtype=torch.complex64)
    f = torch.randn(M, device="cuda", dtype=torch.complex64)
    with Plan(N1, N2, K=K, precision="f64") as p:
        p.set_points(*[v.double() for v in x])
        want, Want = p.forward(F.to(torch.complex128)), p.adjoint(f.to(torch.complex128))
    with Plan(N1, N2, K=K) as p:
        p.set_points(*x)
        assert p.paths()["adjoint"] == 1 and p.paths()["forward"] == int(4 * N1 * N2 <= 128 * 128)
        out, Out = p.forward(F), p.adjoint(f)
        p.synchronize()
    assert float((out.to(torch.complex128) - want).norm() / want.norm()) < 1e-6
    assert float((Out.to(torch.complex128) - Want).norm() / Want.norm()) < 1e-6


@pytest.mark.parametrize("tuning", [{"gather_variant": 1}, {"spread_variant": 2}, {"fft_mode": 2}, {"chunk": 513}, {"tile": 8}])
def test_tuned_plans_run_their_stages(tuning):
    d = _paths(64, 64, 1000, tuning)
    assert (d["forward"], d["adjoint"]) == (0, 0)


def test_timed_plans_run_their_stages():
    from miscellaneous_gb300.nfft import Plan
    with Plan(64, 64) as p:
        p.set_points(*_x(1000))
        p.enable_timing(True)
        assert (p.paths()["forward"], p.paths()["adjoint"]) == (0, 0)
        p.enable_timing(False)
        assert (p.paths()["forward"], p.paths()["adjoint"]) == (1, 1)


@pytest.mark.parametrize("N,M,K,tuning,want", [
    (512, 1 << 19, 6, {}, 2), (512, (1 << 19) - 1, 6, {}, 1), (1024, 1 << 21, 6, {}, 2),   # 128 points a tile
    (1024, (1 << 21) - 1, 6, {}, 1), (1024, 786432, 7, {}, 2), (1024, 786431, 8, {}, 1),     # 48 points a tile
    (512, 1 << 20, 5, {}, 1), (512, 1 << 20, 8, {"gather_variant": 1}, 0), (256, 1 << 18, 6, {}, 1),
    (256, (1 << 17) - 1, 6, {}, 0), (128, 32768, 6, {}, 1), (128, 32767, 6, {}, 0),          # tiled below 128 a tile
])
def test_gather(N, M, K, tuning, want):
    assert _paths(N, N, M, tuning, K=K)["gather"] == want

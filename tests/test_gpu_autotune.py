"""The tuner on a plan whose automatic choice is the fastest: it keeps it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_small_plans_keep_the_one_launch_transforms(tmp_path):
    from miscellaneous_gb300 import autotune
    from miscellaneous_gb300.nfft import Plan
    N, M, path = 64, 4096, str(tmp_path / "tune.json")
    x = [torch.rand(M, device="cuda") - 0.5 for _ in range(2)]
    F = torch.randn(N, N, device="cuda", dtype=torch.complex64)
    f = torch.randn(M, device="cuda", dtype=torch.complex64)
    with Plan(N, N) as p:
        p.set_points(*x)
        want = p.forward(F)
        for cached in (False, True):
            got = autotune.tune(p, *x, F, f, path=path)
            assert got["cached"] is cached and got["ms"] > 0
            assert p.paths() == {"binning": 2, "forward": 1, "adjoint": 1, "gather": 0}
            assert torch.equal(p.forward(F), want)
            p.synchronize()

"""The far-field step's two binnings -- one launch that scales the coordinates
as it reads them, and scaled copies binned per transform where the cell
counters exceed shared memory -- and the filter in the crop, against the
unfiltered step, the general batch calls and what they refuse.

The same FP32 product of coordinate and factor and of field and weight on every
path, so only the spread's order of additions differs: 1e-6 relative."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N1,N2", [(32, 48), (88, 88), (160, 130)])  # the last: counters above 200 KB
@pytest.mark.parametrize("M", [1, 777])
def test_far_field_against_general_calls(N1, N2, M):
    from miscellaneous_gb300.nfft import Batch
    g = torch.Generator(device="cuda")
    g.manual_seed(N1 + M)
    rnd = lambda *s: torch.rand(*s, generator=g, device="cuda")  # noqa: E731
    X, Y = [list(rnd(3, M) * 7 - 3) for _ in range(2)]
    E = list(torch.randn(3, M, generator=g, device="cuda", dtype=torch.complex64))
    filt, sx, sy = rnd(N1 * N2), 1.2345, 0.7071
    with Batch([(N1, N2)] * 3) as b:
        got = b.far_field(X, Y, E, sx, sy, filt)
        plain = b.far_field(X, Y, E, sx, sy)
        b.synchronize()
        c = torch.tensor([sx, sy], dtype=torch.float32, device="cuda")
        b.set_points([x * c[0] for x in X], [y * c[1] for y in Y], units="grid")
        want = b.spread_ref(E)
        b.synchronize()
        for a, p, w in zip(got, plain, want):
            assert float((p - w).norm() / w.norm()) < 1e-6
            assert float((a - filt * w).norm() / (filt * w).norm()) < 1e-6
        from miscellaneous_gb300 import _lib
        bad = X[1].clone()
        bad[M - 1] = float("inf")
        with pytest.raises(_lib.NFFT2DError):
            b.far_field([X[0], bad, X[2]], Y, E, sx, sy, filt)
        again = b.far_field(X, Y, E, sx, sy, filt)
        b.synchronize()
        for a, w in zip(again, want):
            assert float((a - filt * w).norm() / (filt * w).norm()) < 1e-6


def test_lists_are_checked_tensor_by_tensor():
    from miscellaneous_gb300.nfft import Batch
    X = [torch.zeros(8, device="cuda") for _ in range(2)]
    E = [torch.zeros(8, device="cuda", dtype=torch.complex64) for _ in range(2)]
    with Batch([(32, 32)] * 2) as b:
        b.far_field([torch.nn.Parameter(x) for x in X], X, E, 1.0, 1.0)
        for bad, err in ((X[0].cpu(), TypeError), (X[0].double(), TypeError), (X[0][:7], ValueError),
                         (torch.zeros(16, device="cuda")[::2], ValueError), (None, TypeError)):
            with pytest.raises(err):
                b.far_field(X, [X[0], bad], E, 1.0, 1.0)

"""A grid barrier of the one-launch binning or transforms that is given up on
(by a plan's own self-test switch: no wait, no stalled GPU) is reported, leaves
points that later calls read in bounds, and leaves the barrier ready for the
next launch, whatever the host calls in between.

Tolerance: the spread adds in any order, 1e-6 relative in FP32; the forward
sums in a fixed one."""
import pytest
import torch

pytestmark = pytest.mark.gpu

N, M = 64, 4096


def _data(precision):
    g = torch.Generator(device="cuda")
    g.manual_seed(8)
    c = torch.complex64 if precision == "f32" else torch.complex128
    x = [torch.rand(M, generator=g, device="cuda") - 0.5 for _ in range(2)]
    far = [torch.rand(3 * M, generator=g, device="cuda") - 0.5 for _ in range(2)]
    return x, far, torch.randn(N, N, generator=g, device="cuda", dtype=c), torch.randn(M, generator=g, device="cuda", dtype=c)


def _reference(precision, x, F, f):
    from miscellaneous_gb300.nfft import Plan
    with Plan(N, N, precision=precision) as p:
        p.set_points(*x)
        out = p.forward(F), p.adjoint(f)
        p.synchronize()
    return out


def _good(p, x, F, f, want, **kw):
    p.set_points(*x, **kw)
    a, b = p.forward(F), p.adjoint(f)
    p.synchronize()
    assert torch.equal(a, want[0])
    assert float((b - want[1]).norm() / want[1].norm()) < 1e-6


def _give_up(p, barrier):
    from miscellaneous_gb300 import _lib
    assert _lib.load().nfft2d_plan_selftest_barrier(p.handle, barrier) == 0


def _expect(status, call):
    from miscellaneous_gb300 import _lib
    with pytest.raises(_lib.NFFT2DError) as e:
        call()
    assert e.value.status == getattr(_lib, status)


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("barrier", [1, 2, 3])
def test_binning(barrier, precision):
    from miscellaneous_gb300.nfft import Plan
    x, far, F, f = _data(precision)
    want = _reference(precision, x, F, f)
    with Plan(N, N, precision=precision) as p:
        p.set_points(*far)  # records of points that the next set does not have
        for _ in range(2):
            _give_up(p, barrier)
            _expect("ERR_DEVICE_TIMEOUT", lambda: p.set_points(*x))
            _expect("ERR_NO_POINTS", lambda: p.forward(F))
            _give_up(p, 0)
            _good(p, x, F, f, want)  # straight after: the barrier's words are zero
        for direct in (False, True):  # every gather and spread reads those points in bounds
            p.set_points(*far)
            _give_up(p, barrier)
            p.set_points(*x, sync=False)
            _give_up(p, 0)
            if precision == "f32":
                p.set_tuning(gather_variant=2 if direct else 1, spread_variant=2 if direct else 1)
            p.forward(F), p.adjoint(f)
            _expect("ERR_DEVICE_TIMEOUT", p.synchronize)
            _expect("ERR_NO_POINTS", lambda: p.forward(F))
            p.synchronize()  # reported once
            p.set_tuning(gather_variant=0, spread_variant=0)
            _good(p, x, F, f, want, sync=False)


@pytest.mark.parametrize("adjoint,barrier", [(False, 1), (False, 2), (True, 1), (True, 2), (True, 3)])
def test_transforms(adjoint, barrier):
    from miscellaneous_gb300.nfft import Plan
    x, _, F, f = _data("f32")
    want = _reference("f32", x, F, f)
    with Plan(N, N) as p:
        p.set_points(*x)
        for read in (True, False):  # the status is read, or cleared unread by the next binning
            _give_up(p, barrier)
            p.adjoint(f) if adjoint else p.forward(F)
            _give_up(p, 0)
            if read:
                _expect("ERR_DEVICE_TIMEOUT", p.synchronize)
                a = p.forward(F)  # the points are as they were
                p.synchronize()
                assert torch.equal(a, want[0])
            _good(p, x, F, f, want)

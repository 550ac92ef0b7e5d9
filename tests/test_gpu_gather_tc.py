"""The tensor-core gather (dense sets, w >= 6) against FP64 plans on the same
points: grids whose last tiles are cut, grids smaller than a patch, odd and
even windows, work items that leave ragged batches, both tile sizes it takes.

Tolerance: FP32 rounding of the two-dimensional FFT (at most 22 radix-2 stages
at 2^-24 each, adding in quadrature) and of tables and weights stays under
1e-6 relative; the FP64 plan's own error is 5e-12 at w 6 and less above."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

M0 = 1 << 19  # the fewest points it is chosen for


def _inputs(N1, N2, M, seed, spread=None):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = [torch.rand(M, generator=g, device="cuda", dtype=torch.float32) - 0.5 for _ in range(2)]
    if spread:
        x = [torch.remainder(spread * torch.randn(M, generator=g, device="cuda") + 0.5, 1.0) - 0.5 for _ in range(2)]
    F = torch.randn(N1, N2, generator=g, device="cuda", dtype=torch.complex64)
    return x[0], x[1], F


def _exact(N1, N2, K, x1, x2, F):
    from miscellaneous_gb300.nfft import Plan
    with Plan(N1, N2, K=K, precision="f64") as p:
        p.set_points(x1.double(), x2.double())
        out = p.forward(F.to(torch.complex128))
        p.synchronize()
    return out


def _rel(a, b):
    return float((a.to(torch.complex128) - b).norm() / b.norm())


@pytest.mark.parametrize("K", [6, 7, 8])
@pytest.mark.parametrize("N1,N2,M,spread,tuning", [
    (250, 378, M0 + 77, None, {}),                       # cut last tiles, odd point count
    (10, 14, M0, None, {}),                              # a grid smaller than a patch
    (256, 256, M0 + 1, 0.05, {"chunk": 100}),            # dense tiles, ragged batches
    (256, 256, M0 + 1, 0.05, {"chunk": 100000}),         # items of many batches
    (128, 256, M0, None, {"tile": 8, "compensated": 0}),
])
def test_matches_f64(K, N1, N2, M, spread, tuning):
    from miscellaneous_gb300.nfft import Plan
    x1, x2, F = _inputs(N1, N2, M, seed=K, spread=spread)
    with Plan(N1, N2, K=K) as p:
        p.set_tuning(gather_variant=2, **tuning)
        p.set_points(x1, x2)
        out = p.forward(F)
        p.synchronize()
        p.set_tuning(io_order="binned")
        binned = p.forward(F)
        perm = p.permutation().long()
        p.set_tuning(io_order="caller")
        p.set_points(x1, x2, sync=False)  # work items counted on the device only
        late = p.forward(F)
        p.synchronize()
    want = _exact(N1, N2, K, x1, x2, F)
    assert _rel(out, want) < 1e-6
    assert _rel(late, want) < 1e-6
    assert _rel(binned, want[perm]) < 1e-6


def test_values_over_the_exponent_range():
    """The split operands need no scaling: results follow F by powers of two."""
    from miscellaneous_gb300.nfft import Plan
    x1, x2, F = _inputs(128, 128, M0, seed=3)
    with Plan(128, 128) as p:
        p.set_points(x1, x2)
        out = p.forward(F)
        for e in (-60, 60):
            got = p.forward(F * 2.0 ** e)
            p.synchronize()
            assert _rel(got * 2.0 ** -e, out.to(torch.complex128)) < 1e-7


def test_batch_mixes_both_gathers():
    from miscellaneous_gb300.nfft import Batch
    sizes, Ms = [(128, 128), (64, 96), (250, 130), (32, 32)], [M0 + 5, 3000, M0, 0]
    ins = [_inputs(a, b, m, seed=i) for i, ((a, b), m) in enumerate(zip(sizes, Ms))]
    with Batch(sizes, K=[6, 6, 8, 6]) as b:
        b.set_points([i[0] for i in ins], [i[1] for i in ins])
        outs = b.forward([i[2] for i in ins])
        b.synchronize()
    for (a, c), K, i, out in zip(sizes, [6, 6, 8, 6], ins, outs):
        if out.numel():
            assert _rel(out, _exact(a, c, K, *i)) < 1e-6

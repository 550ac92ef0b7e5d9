"""FP64 plans evaluate the window by polynomials: against the restated
algorithm's closed form at the ends of sigma's range, the narrowest, an odd
and the widest window, with points on cells (t = 0) and half-way between them
(t = 1/2, where the polynomials end).

Tolerance: the closed form and the fits agree to 1e-14 of the window's peak,
and the deapodization amplifies rounding by the window transform's range over
the band, in each dimension (2 * 10^3 at sigma 1.25 and K = 8; closed-form taps
differ from the restatement by 1.2e-11 there): 2^-52 times its square, at least
1e-13."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma", [1.25, 4.0])
@pytest.mark.parametrize("K", [2, 5, 8])
def test_f64_window(orc, sigma, K):
    from miscellaneous_gb300.nfft import Plan
    N1, N2, M = 32, 48, 400
    rng = np.random.default_rng(K)
    x1, x2 = rng.uniform(-N1 / 2, N1 / 2, M), rng.uniform(-N2 / 2, N2 / 2, M)
    x1[:100] = np.rint(x1[:100] * 2 * sigma) / (2 * sigma) * (1 - 1e-15)
    x2[50:150] = np.rint(x2[50:150] * 2 * sigma) / (2 * sigma) * (1 - 1e-15)
    F = rng.standard_normal((N1, N2)) + 1j * rng.standard_normal((N1, N2))
    f = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    dev = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
    with Plan(N1, N2, sigma=sigma, K=K, precision="f64") as p:
        p.set_points(dev(x1), dev(x2), units="grid")
        fwd = p.forward(dev(F)).cpu().numpy()
        ref = p.spread_ref(dev(f)).cpu().numpy()
        p.synchronize()
    alpha = (2 - 1 / sigma) * np.pi - 0.01
    span = np.i0(K * alpha) / np.i0(K * np.sqrt(alpha ** 2 - (np.pi / sigma) ** 2))
    bound = max(1e-13, 2.0 ** -52 * span ** 2)
    assert orc.rel_l2(fwd, orc.nfft1_2d(F, x1, x2, c=sigma, K=K)) < bound
    assert orc.rel_l2(ref, orc.nfft2_2d(f, x1, x2, N1, N2, c=sigma, K=K)) < bound

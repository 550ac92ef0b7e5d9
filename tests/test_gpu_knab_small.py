"""The FP32 regridder on small rasters whose oversampled grid is a power of two a
side, where plain plans need no cuFFT plan and the regridder does: against the
CPU oracle's restatement, and again on the same regridder.

Tolerance: the FP32 path's bound against the FP64 oracle, 1e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(64, 64, 40, 50), (128, 64, 90, 45), (64, 256, 33, 200)])
def test_power_of_two_grids(dev, orc, shape):
    import torch

    from miscellaneous_gb300 import knab
    Nrows, Ncols, len1, len2 = shape
    rng = np.random.default_rng(9)
    rho_in, cos_in = 100.0 + 0.3 * np.arange(Ncols), -0.1 + 0.01 * np.arange(Nrows)
    rho_out, cos_out = np.meshgrid(np.linspace(rho_in[3], rho_in[-4], len2), np.linspace(cos_in[3], cos_in[-4], len1))
    B1, B2 = 0.45 / 0.3, 0.4 / 0.01
    r = knab.Regridder(rho_in, cos_in, B1, B2, precision="f32")
    r.set_points(torch.tensor(rho_out, device=dev), torch.tensor(cos_out, device=dev))
    info = r.info()
    assert info["N1"] & (info["N1"] - 1) == 0 and info["N2"] & (info["N2"] - 1) == 0
    for _ in range(2):
        data = rng.standard_normal((Nrows, Ncols)) + 1j * rng.standard_normal((Nrows, Ncols))
        ref, _ = orc.knab_nfft2d(0.0, rho_in, cos_in, data, rho_out, cos_out, B1, B2)
        out = r(torch.tensor(data, dtype=torch.complex64, device=dev), 0.0)
        r.synchronize()
        out = out.cpu().numpy()
        assert np.linalg.norm(out.ravel() - np.asarray(ref).ravel()) / np.linalg.norm(ref) < 1e-5
    r.close()

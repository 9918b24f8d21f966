"""The sample filter's flux sums and scaling in pairs of floats: planes of very different magnitude, of
both signs with nine tenths of the flux cancelled, and one with a NaN, which stays in its plane.
Against the FP64 oracle at the filter's bound (1e-6): an output adds 2 x 85 products whose weights sum to
one, so its rounding is a few 2^-24 of the values; the scale's is that over the root of the voxels, ten
times that where a tenth of the flux is left."""
import numpy as np
import pytest

from mesolf_gb300 import synth
from oracle import mesolf_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["magnitudes", "signs", "nan"])
@pytest.mark.parametrize("lenslets", [(7, 6), (23, 11)])
def test_flux(cuda, kind, lenslets):
    import torch
    from mesolf_gb300 import PhaseSpacePSF, RLSolver
    from mesolf_gb300.api import _fortran
    Z = 5
    w = synth.small_config(lenslets=lenslets, K0=61, Z=Z)
    H, Ht = w.psf()
    shape = w.image_shape
    X = np.random.default_rng(5).uniform(0.5, 1.5, shape + (Z,))
    if kind == "magnitudes":
        X *= np.array([1e-30, 1e-12, 1.0, 1e12, 1e30])
    elif kind == "signs":
        X -= 0.9 * X.mean(axis=(0, 1))
    X = X.astype(np.float32)
    if kind == "nan":
        X[3, 5, 1] = np.nan
    s = RLSolver(PhaseSpacePSF(H, Ht), shape)
    got = s.sample_filter(_fortran(torch.as_tensor(np.ascontiguousarray(X)).cuda())[0]).cpu().numpy().astype(np.float64)
    ref = R.sample_filter(X.astype(np.float64), R.nip_filter_bank(*shape, Z, 15))
    for z in range(Z):
        if kind == "nan" and z == 1:
            assert np.isnan(got[:, :, z]).all()
        else:
            assert np.linalg.norm(got[:, :, z] - ref[:, :, z]) <= 1e-6 * np.linalg.norm(ref[:, :, z]), z

"""The sample filter's flux sums at the top of the floats' range: a thread's sum of a few voxels is beyond
it, the FP64 sum is not; planes of both signs, and one with an infinity, which stays in its plane.  Against the
FP64 oracle at the filter's bound (1e-6: 2 x 85 products whose weights sum to one, and a scale of the root of
the voxels less)."""
import numpy as np
import pytest

from mesolf_gb300 import synth
from oracle import mesolf_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lenslets", [(7, 6), (23, 11), (11, 30)])
def test_flux_of_large_planes(cuda, lenslets):
    import torch
    from mesolf_gb300 import PhaseSpacePSF, RLSolver
    from mesolf_gb300.api import _fortran
    Z = 5
    w = synth.small_config(lenslets=lenslets, K0=61, Z=Z)
    H, Ht = w.psf()
    shape = w.image_shape
    X = np.random.default_rng(3).uniform(0.5, 1.5, shape + (Z,))
    X[:, :, 3] -= 0.9 * X[:, :, 3].mean()
    X = (X * np.array([1e37, 2e38, 1.0, 5e37, 1.0])).astype(np.float32)
    X[4, 2, 4] = np.inf
    s = RLSolver(PhaseSpacePSF(H, Ht), shape)
    got = s.sample_filter(_fortran(torch.as_tensor(np.ascontiguousarray(X)).cuda())[0]).cpu().numpy().astype(np.float64)
    ref = R.sample_filter(np.where(np.isinf(X), 0, X).astype(np.float64), R.nip_filter_bank(*shape, Z, 15))
    for z in range(4):
        assert np.linalg.norm(got[:, :, z] - ref[:, :, z]) <= 1e-6 * np.linalg.norm(ref[:, :, z]), z
    assert not np.isfinite(got[:, :, 4]).any()

"""The view kernel's two tiles (2 x 4 outputs per thread for small patches, 4 x 8 else) against
the FP64 oracle for every tap count, with sides that are and are not multiples of either tile, on
both sides of the line between them, and for patches whose smaller tile count just reaches 256.
Tolerance 1e-5, the bound of test_gpu_parity.py for these entry points."""
import numpy as np
import pytest

from mesolf_gb300 import synth
from oracle import mesolf_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lenslets,K0,Z", [
    ((8, 9), 61, 2), ((13, 7), 91, 3), ((9, 10), 121, 2), ((10, 11), 151, 2), ((11, 13), 181, 2),
    ((13, 14), 211, 2), ((15, 16), 231, 2), ((17, 18), 255, 1),
    ((64, 32), 61, 1),     # 16 x 16 small tiles: 256
    ((68, 32), 61, 1),     # 17 x 16: the large tile
    ((33, 31), 61, 14),    # 126 K threads of the large tile: the large tile
    ((33, 31), 61, 13),    # 117 K: the small one
])
def test_tiles_match_oracle(cuda, lenslets, K0, Z):
    import torch
    from mesolf_gb300 import PhaseSpacePSF, RLSolver
    from mesolf_gb300.api import _fortran

    def dev(x):
        return _fortran(torch.as_tensor(np.ascontiguousarray(x.astype(np.float32))).cuda())[0]

    def rel(a, b):
        return np.linalg.norm(a.cpu().numpy().astype(np.float64) - b) / np.linalg.norm(b)

    w = synth.small_config(lenslets=lenslets, K0=K0, Z=Z)
    H, Ht = w.psf()
    rng = np.random.default_rng(K0 + Z)
    Xr, Xc = w.image_shape
    X, LF = rng.uniform(0.5, 1.5, (Xr, Xc, Z)), rng.uniform(50.0, 150.0, (Xr, Xc))
    Hps, Htc = R.gen_phasespace_psf(*R.normalize_psf(H, Ht))
    psf = PhaseSpacePSF(H, Ht)
    s = RLSolver(psf, (Xr, Xc))
    u, v = 2, 12
    X32, LF32 = X.astype(np.float32).astype(np.float64), LF.astype(np.float32).astype(np.float64)
    proj = rng.random(lenslets).astype(np.float32)
    assert rel(s.forward_view(dev(X), u, v), R.forward_ps(Hps[:, :, u, v, :], X32, 15)) <= 1e-5
    assert rel(s.backward_view(dev(proj), u, v),
               R.backward_ps(Htc[:, :, u, v, :], proj.astype(np.float64), u, v, 15)) <= 1e-5
    got = s.view_step(dev(LF), dev(X), u, v, 0.3)
    assert rel(got, R.rl_view_step(X32, LF32, Hps, Htc, u, v, 0.3, 15)) <= 1e-5
    s.close()
    psf.close()

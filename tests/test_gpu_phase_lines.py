"""The volume's layout kernels and the filter's line passes at their edges: lines that are no multiple
of four in number or length, one lenslet on a side, and an image side of more lenslets than a block
takes at once.  Against the FP64 oracle.  Projections: a sum of at most T^2 Z N^2 non-negative FP32
products in several short chains, within 1e-5 (the bound of the other projection tests); the filter:
1e-6 (the bound of the other filter test); the tensor-core projector: 1e-5 (its own tests' bound)."""
import numpy as np
import pytest

from mesolf_gb300 import synth
from oracle import mesolf_ref as R

pytestmark = pytest.mark.gpu


def dev(x):
    import torch
    from mesolf_gb300.api import _fortran
    return _fortran(torch.as_tensor(np.ascontiguousarray(x.astype(np.float32))).cuda())[0]


def rel(a, b):
    a = a.detach().cpu().numpy().astype(np.float64)
    assert a.shape == b.shape
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("lenslets,Z", [((1, 1), 1), ((5, 3), 2), ((3, 9), 3), ((33, 7), 2), ((110, 1), 3)])
def test_projections_and_filter(cuda, lenslets, Z):
    from mesolf_gb300 import PhaseSpacePSF, RLSolver
    w = synth.small_config(lenslets=lenslets, K0=61, Z=Z)
    H, Ht = w.psf()
    shape = w.image_shape
    rng = np.random.default_rng(Z + lenslets[0])
    vol = (0.5 + rng.random(shape + (Z,))).astype(np.float32)
    proj = (0.5 + rng.random(lenslets)).astype(np.float32)
    Hps, Htc = R.gen_phasespace_psf(*R.normalize_psf(H, Ht))
    s = RLSolver(PhaseSpacePSF(H, Ht), shape)
    for u, v in ((7, 7), (2, 12)):
        assert rel(s.forward_view(dev(vol), u, v), R.forward_ps(Hps[:, :, u, v, :], vol.astype(np.float64), 15)) <= 1e-5
        assert rel(s.backward_view(dev(proj), u, v),
                   R.backward_ps(Htc[:, :, u, v, :], proj.astype(np.float64), u, v, 15)) <= 1e-5
    assert rel(s.sample_filter(dev(vol)), R.sample_filter(vol.astype(np.float64), R.nip_filter_bank(*shape, Z, 15))) <= 1e-6


def test_side_of_several_blocks(cuda):
    from mesolf_gb300 import mex_lfm_convolution_vec
    rng = np.random.default_rng(3)
    bm = rng.random((3100, 31, 2)).astype(np.float32)
    K = rng.random((7, 7, 15, 15)).astype(np.float32)
    assert rel(mex_lfm_convolution_vec(dev(bm), dev(K), method="tensor"), R.lfm_conv_vec(bm, K)) <= 1e-5

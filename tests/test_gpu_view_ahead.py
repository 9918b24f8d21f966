"""The view kernels with the next channel requested ahead: one channel per slot and many, a last round
in which only some slots have a channel, both tiles, forward kernels with two X planes and (a patch
too large for them) with one.  Against the FP64 oracle; an output is a sum of non-negative FP32
products in chains of at most T^2 terms, within 1e-5 (the bound of the other projection tests)."""
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


@pytest.mark.parametrize("lenslets,K0,Z", [
    ((6, 5), 61, 1),       # fewer channels than slots
    ((31, 17), 121, 7),    # several slots per CTA, a partial last round
    ((24, 26), 181, 5),
    ((67, 66), 61, 3),     # two slots
    ((40, 61), 231, 2),    # the widest taps
    ((110, 62), 61, 2),    # one slot, shared memory for one X plane
])
def test_forward_and_step(cuda, lenslets, K0, Z):
    from mesolf_gb300 import PhaseSpacePSF, RLSolver
    w = synth.small_config(lenslets=lenslets, K0=K0, Z=Z)
    H, Ht = w.psf()
    shape = w.image_shape
    rng = np.random.default_rng(K0 + Z)
    vol = (0.5 + rng.random(shape + (Z,))).astype(np.float32)
    lf = (0.5 + rng.random(shape)).astype(np.float32)
    Hps, Htc = R.gen_phasespace_psf(*R.normalize_psf(H, Ht))
    s = RLSolver(PhaseSpacePSF(H, Ht), shape)
    for u, v in ((7, 7), (3, 10)):
        assert rel(s.forward_view(dev(vol), u, v), R.forward_ps(Hps[:, :, u, v, :], vol.astype(np.float64), 15)) <= 1e-5
    ref = R.rl_view_step(vol.astype(np.float64), lf.astype(np.float64), Hps, Htc, 4, 8, 0.2, 15)
    assert rel(s.view_step(dev(lf), dev(vol), 4, 8, 0.2), ref) <= 1e-5

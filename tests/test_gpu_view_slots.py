"""Forward partial sums of the view kernel where a CTA holds several channel slots: a last CTA
that is not full, slots with one and with several channels, and the two-slot form that leaves
the sum to the reduction kernel.  Tolerance: every term is non-negative and an output's
additions are at most ~80 deep (T*T taps, the channels of a slot, the slots, the planes), so
80 * 2^-24 = 4.8e-6 bounds the relative error."""
import numpy as np
import pytest

from mesolf_gb300 import synth
from oracle import mesolf_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lenslets,K0,Z", [
    ((32, 24), 61, 1),    # 24 tiles: 8 slots, 225 channels, one slot used in the last CTA
    ((9, 3), 61, 23),     # 2 tiles: 32 slots, more channels than one round of the grid
    ((41, 33), 91, 6),    # 54 tiles: 3 slots
    ((64, 36), 61, 3),    # 72 tiles: 2 slots, added by the reduction
])
def test_forward_view_over_slots(cuda, lenslets, K0, Z):
    import torch
    from mesolf_gb300 import PhaseSpacePSF, RLSolver
    from mesolf_gb300.api import _fortran
    w = synth.small_config(lenslets=lenslets, K0=K0, Z=Z)
    H, Ht = w.psf()
    vol = np.random.default_rng(Z).random(w.image_shape + (Z,)).astype(np.float32)
    Hps, _ = R.gen_phasespace_psf(*R.normalize_psf(H, Ht))
    psf = PhaseSpacePSF(H, Ht)
    s = RLSolver(psf, w.image_shape)
    for u, v in [(7, 7), (1, 12)]:
        hx = s.forward_view(_fortran(torch.as_tensor(vol).cuda())[0], u, v).cpu().numpy()
        ref = R.forward_ps(Hps[:, :, u, v, :], vol.astype(np.float64), 15)
        assert np.linalg.norm(hx - ref) / np.linalg.norm(ref) <= 4.8e-6, (u, v)
    s.close()
    psf.close()

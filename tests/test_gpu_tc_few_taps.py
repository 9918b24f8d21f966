"""col2im below nine taps a row (T 3, 5 and 7: splits over the warps, two or four of them at once) and the
general form above: one split, fewer and more splits than a pass over them, patches narrower than the taps.
One forward view in bf16x3 against the FP64 oracle at test_gpu_tc.py's bound for a step (1e-5)."""
import numpy as np
import pytest

from mesolf_gb300 import synth
from oracle import mesolf_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lenslets,K0,Z", [
    ((11, 11), 61, 21),   # T 3: more splits than the five groups of four
    ((6, 7), 61, 1),      # T 3: two channel tiles
    ((64, 70), 61, 2),    # T 3: many positions, few splits
    ((2, 40), 91, 9),     # T 5: rows narrower than the taps
    ((23, 9), 91, 11),    # T 5
    ((9, 5), 121, 8),     # T 7
    ((45, 31), 121, 5),   # T 7
    ((14, 13), 151, 4),   # T 9: the general form
])
def test_forward_view_of_few_taps(cuda, lenslets, K0, Z):
    import torch
    from mesolf_gb300 import PhaseSpacePSF, RLSolver
    from mesolf_gb300.api import _fortran
    w = synth.small_config(lenslets=lenslets, K0=K0, Z=Z)
    H, Ht = w.psf()
    Hps, _ = R.gen_phasespace_psf(*R.normalize_psf(H, Ht))
    vol = np.random.default_rng(K0 + Z).uniform(0.5, 1.5, w.image_shape + (Z,)).astype(np.float32)
    psf = PhaseSpacePSF(H, Ht)
    s = RLSolver(psf, w.image_shape)
    d = _fortran(torch.as_tensor(vol).cuda())[0]
    for u, v in [(7, 7), (0, 13)]:
        hx = s.forward_view(d, u, v, precision="bf16x3").cpu().numpy()
        ref = R.forward_ps(Hps[:, :, u, v, :], vol.astype(np.float64), 15)
        assert np.linalg.norm(hx - ref) / np.linalg.norm(ref) <= 1e-5, (u, v)
    s.close()
    psf.close()

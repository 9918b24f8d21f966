"""Every forward partial plane that the reduction adds has been written: the partials are filled with
NaN before each call.  Odd channel counts whose last CTA of two slots has one channel, one slot, and
three and more slots that a CTA adds itself.  The launch shape is asserted, so that a case which no
longer reaches its form fails.  Tolerances: as for the forward partial sums (at most ~80 additions of
non-negative terms, 80 * 2^-24 = 4.8e-6), and test_gpu_parity.py's 1e-5 for a view step."""
import ctypes

import numpy as np
import pytest

from mesolf_gb300 import synth
from oracle import mesolf_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lenslets,K0,Z,tile,slots,ctas", [
    ((64, 36), 61, 3, (4, 8), 2, 338),     # 675 channels, the second slot of the last CTA without one
    ((48, 48), 61, 5, (4, 8), 2, 563),     # 1125 channels
    ((67, 67), 61, 1, (4, 8), 2, 113),     # 225 channels, two slots of 160 threads
    ((24, 24), 61, 7, (2, 4), 2, 788),     # 1575 channels, the small tile
    ((71, 71), 61, 3, (4, 8), 1, None),    # one slot
    ((11, 11), 61, 21, (2, 4), 10, 473),   # the last CTA has five of ten slots
    ((41, 33), 91, 24, (4, 8), 3, None),   # three slots: a CTA adds its own
    ((30, 31), 91, 40, (4, 8), 6, None),
])
def test_no_plane_is_read_unwritten(cuda, lenslets, K0, Z, tile, slots, ctas):
    import torch
    from mesolf_gb300 import PhaseSpacePSF, RLSolver, _lib
    from mesolf_gb300.api import _fortran
    lib = _lib.load()
    w = synth.small_config(lenslets=lenslets, K0=K0, Z=Z)
    H, Ht = w.psf()
    psf = PhaseSpacePSF(H, Ht)
    s = RLSolver(psf, w.image_shape)
    plan = (ctypes.c_int64 * 5)()

    def poison():
        torch.cuda.synchronize()
        assert lib.mlf_probe_view_plan(s._h, plan, 1, None) == 0
        torch.cuda.synchronize()

    poison()
    assert (plan[0], plan[1]) == tile
    nch = 225 * Z
    assert plan[2] == slots
    if ctas is not None:  # the grid holds all channels at once
        assert plan[3] == ctas == -(-nch // plan[2])
    assert plan[4] <= nch

    rng = np.random.default_rng(Z)
    vol = rng.uniform(0.5, 1.5, w.image_shape + (Z,)).astype(np.float32)
    dvol = _fortran(torch.as_tensor(vol).cuda())[0]
    Hn, Hnt = R.normalize_psf(H, Ht)
    Hps, Hpst = R.gen_phasespace_psf(Hn, Hnt)
    for u, v in [(7, 7), (1, 12)]:
        poison()
        hx = s.forward_view(dvol, u, v).cpu().numpy()
        ref = R.forward_ps(Hps[:, :, u, v, :], vol.astype(np.float64), 15)
        assert np.linalg.norm(hx - ref) / np.linalg.norm(ref) <= 4.8e-6, (u, v)
    poison()
    assert torch.isfinite(s.forward_project(dvol)).all()
    LF = rng.uniform(50.0, 150.0, w.image_shape).astype(np.float32)
    lf = _fortran(torch.as_tensor(LF).cuda())[0]
    poison()
    got = s.view_step(lf, dvol.clone(), 7, 7, 0.7).cpu().numpy()
    ref = R.rl_view_step(vol.astype(np.float64), LF.astype(np.float64), Hps, Hpst, 7, 7, 0.7, 15)
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) <= 1e-5
    # a solve's first view is projected by the forward kernel, the others inside the view steps: the
    # same with partials of other contents (each kernel's sums are deterministic)
    poison()
    one = s.run(lf, 1, precision="fp32", want_stats=False)
    again = s.run(lf, 1, precision="fp32", want_stats=False)
    assert torch.equal(one, again)
    s.close()
    psf.close()

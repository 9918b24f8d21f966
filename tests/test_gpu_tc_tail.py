"""Full forward projections of many patches on the tensor cores, where the patches of a nearly empty
last wave are projected for several views per launch (counts for 152 SMs): one tile per patch, several,
a patch boundary that is not a wave's, a last launch of fewer views, and counts that leave no such
wave.  Through the MEX projector against the FP64 oracle at its own tests' bound (1e-5)."""
import numpy as np
import pytest

from oracle import mesolf_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,n,kw", [
    (20, 17, 160, 9),     # 160 tiles: 8 left over
    (16, 31, 305, 4),     # two waves and one tile
    (190, 190, 79, 7),    # two tiles per patch: 158, six left over
    (270, 255, 52, 16),   # three tiles per patch: 156, cut at 150
    (30, 33, 152, 5),     # whole waves
    (45, 16, 300, 5),     # a last wave that is nearly full
])
def test_forward_of_many_patches(cuda, W, H, n, kw):
    import torch
    from mesolf_gb300 import mex_lfm_convolution_vec
    from mesolf_gb300.api import _fortran
    rng = np.random.default_rng(W + n)
    bm = rng.random((W, H, n)).astype(np.float32)
    K = rng.random((kw, kw, 15, 15)).astype(np.float32)
    d = [_fortran(torch.as_tensor(x).cuda())[0] for x in (bm, K)]
    out = mex_lfm_convolution_vec(*d, method="tensor").cpu().numpy().astype(np.float64)
    pick = sorted({0, 1, n // 2, n - 9, n - 2, n - 1})
    for i in pick:
        ref = R.lfm_conv_vec(bm[:, :, i:i + 1], K)[:, :, 0]
        assert np.linalg.norm(out[:, :, i] - ref) <= 1e-5 * np.linalg.norm(ref), i
    same = mex_lfm_convolution_vec(d[0], d[1], method="direct").cpu().numpy().astype(np.float64)
    assert np.linalg.norm(out - same) <= 1e-5 * np.linalg.norm(same)

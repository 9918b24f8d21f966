"""The direct MEX kernel on narrow images, whose CTAs have warps that only stage (8 or 4 warps for 32
lanes, 4 for 64): a stack of slices equals the slices one by one bit for bit (an output's additions do not
depend on the launch shape), and the FP64 oracle at the bound of the other tests of this entry point."""
import numpy as np
import pytest

from oracle import mesolf_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,n,kw", [(31, 31, 30, 21), (31, 31, 60, 15), (62, 62, 40, 15), (90, 47, 23, 4), (14, 200, 9, 33),
                                      (46, 16, 11, 16), (39, 100, 17, 120)])
def test_stack_equals_slices(cuda, W, H, n, kw):
    import torch
    from mesolf_gb300 import mex_lfm_convolution_vec
    from mesolf_gb300.api import _fortran
    rng = np.random.default_rng(W + kw)
    bm = rng.random((W, H, n)).astype(np.float32)
    K = rng.random((kw, kw, 15, 15)).astype(np.float32)
    dK = _fortran(torch.as_tensor(K).cuda())[0]

    def run(x):
        return mex_lfm_convolution_vec(_fortran(torch.as_tensor(np.ascontiguousarray(x)).cuda())[0], dK,
                                       method="direct").cpu().numpy()

    out = run(bm)
    for k in (0, n // 2, n - 1):
        assert np.array_equal(out[:, :, k], run(bm[:, :, k:k + 1])[:, :, 0]), k
    ref = R.lfm_conv_vec(bm[:, :, :1], K)
    assert np.linalg.norm(out[:, :, :1] - ref) <= 1e-5 * np.linalg.norm(ref)

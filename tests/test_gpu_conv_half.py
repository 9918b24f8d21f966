"""The direct MEX kernel's half segments: kernel widths around the 16 columns of a trip and its tail,
outputs that end inside the first and the second half, even widths, a width of one, and the value
that a pixel outside an output's window must not have on it (an infinity), for both halves.  Against the
FP64 oracle; an output is one FMA chain of kw^2 non-negative terms, so kw^2 * 2^-24 bounds its relative
error, and 1e-5 (the bound of the other tests of this entry point) covers what these widths reach."""
import numpy as np
import pytest

from oracle import mesolf_ref as R

pytestmark = pytest.mark.gpu


def run(bm, K):
    import torch
    from mesolf_gb300 import mex_lfm_convolution_vec
    from mesolf_gb300.api import _fortran
    d = [_fortran(torch.as_tensor(x).cuda())[0] for x in (bm, K)]
    return mex_lfm_convolution_vec(*d, method="direct").cpu().numpy()


@pytest.mark.parametrize("W,H,n,kw", [(31, 17, 2, 1), (38, 16, 1, 2), (23, 30, 2, 15), (24, 31, 1, 16), (53, 20, 1, 17),
                                      (60, 18, 3, 31), (52, 33, 1, 32), (97, 15, 1, 33), (7, 40, 2, 47), (8, 9, 5, 3),
                                      (495, 16, 1, 19)])
def test_widths_and_ends(cuda, W, H, n, kw):
    rng = np.random.default_rng(W + kw)
    bm = rng.random((W, H, n)).astype(np.float32)
    K = rng.random((kw, kw, 15, 15)).astype(np.float32)
    out, ref = run(bm, K), R.lfm_conv_vec(bm, K)
    assert out.shape == (W, H, n)
    assert np.linalg.norm(out - ref) <= 1e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("x", [0, 14, 22, 23, 44])
def test_infinite_pixel_stays_in_its_windows(cuda, x):
    W, H, kw = 45, 31, 7
    rng = np.random.default_rng(x)
    bm = rng.random((W, H, 1)).astype(np.float32)
    K = (0.5 + rng.random((kw, kw, 15, 15))).astype(np.float32)
    bm[x, 12, 0] = np.inf
    out = run(bm, K)[:, :, 0]
    i, j = np.mgrid[0:W, 0:H]
    hit = (np.abs(i - x) <= kw // 2) & (np.abs(j - 12) <= kw // 2)
    assert np.isposinf(out[hit]).all() and np.isfinite(out[~hit]).all()

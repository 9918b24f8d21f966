"""Edges of the direct MEX kernel's lane mapping: images narrower than a segment with many groups
per warp, two groups of segments along x, a last warp that is not full, one slice and many, rows
off the image above and below for most kernel rows, even kernel widths, and the widest kernel on a
narrow image.  Against the FP64 oracle; every product is non-negative and an output is one FMA
chain of kw^2 terms, so kw^2 * 2^-24 bounds its relative error and 1e-5 (the bound of the other
tests of this entry point) is below that for these widths; the expected error grows with its root."""
import numpy as np
import pytest

from oracle import mesolf_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,n,kw", [
    (7, 11, 3, 5),        # half a segment, fewer rows than phases
    (14, 46, 37, 4),      # 37 slices: groups of many slices in a warp
    (16, 31, 2, 31),      # two segments, the second of one pixel
    (481, 17, 1, 7),      # 33 segments: two groups along x
    (700, 40, 3, 16),     # 47 segments, even width
    (46, 3, 1, 41),       # a kernel much taller than the image
    (9, 20, 1, 341),      # the widest kernel, narrow
    (150, 120, 24, 9),    # two rows per thread
])
def test_conv_lanes_match_oracle(cuda, W, H, n, kw):
    import torch
    from mesolf_gb300 import mex_lfm_convolution_vec
    from mesolf_gb300.api import _fortran
    rng = np.random.default_rng(W + 3 * H + kw)
    bm = rng.random((W, H, n)).astype(np.float32)
    K = rng.random((kw, kw, 15, 15)).astype(np.float32)
    dev = [_fortran(torch.as_tensor(x).cuda())[0] for x in (bm, K)]
    out = mex_lfm_convolution_vec(*dev, method="direct").cpu().numpy()
    ref = R.lfm_conv_vec(bm, K)
    assert out.shape == (W, H, n)
    assert np.linalg.norm(out - ref) / np.linalg.norm(ref) <= 1e-5

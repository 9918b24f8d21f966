"""Edges of the row-walking rectification kernel: row blocks and 16-column tiles that are not
full, stages of fewer than four frames, pitches that repeat raw columns (< 1 px) or skip them
(> 1 px), frames on and off the 16-byte grid, 16- and 32-bit frames; and the division by the
movie's maximum, which must be the correctly rounded quotient of the undivided movie.
Tolerance of the interpolation: three roundings of values of at most the peak (and of the FP32
weights), so 4 * 2^-24 = 2.4e-7 of the peak per pixel."""
import numpy as np
import pytest

from mesolf_gb300 import rectify as RC
from oracle import mesolf_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,n,dx,dtype", [
    ((64, 61), 1, 15.27, "u16"),     # one frame, narrower than a tile of columns twice
    ((128, 100), 3, 15.27, "u16"),   # 128 rows: last block of rows partly idle
    ((200, 130), 6, 9.1, "u16"),     # pitch 0.61: raw columns repeated
    ((211, 173), 5, 22.4, "u16"),    # pitch 1.49, odd frame size (alignment changes per frame)
    ((120, 90), 4, 15.27, "f32"),
    ((143, 77), 7, 17.9, "f32"),
    ((300, 290), 2, 61.0, "u16"),    # pitch 4.07: tile too large for shared memory, gathered
])
def test_rows_match_oracle_and_divide_exactly(cuda, shape, n, dx, dtype):
    import torch
    rng = np.random.default_rng(shape[0] + n)
    fr = rng.integers(0, 4000, shape + (n,)).astype(np.uint16)
    if dtype == "f32":
        fr = fr.astype(np.float32) * np.float32(0.37)
    yc, xc = shape[0] / 2 + 0.3, shape[1] / 2 - 0.4
    size = RC.rectified_size(shape, xc, yc, 15, dx)
    info = {"size": size, "raw_cut": [[1, shape[0]], [1, shape[1]]], "raw_cut_xCenter": xc, "raw_cut_yCenter": yc}
    SI = {"Nnum": 15, "frames_dx": dx}
    plain = RC.image_load_module_aug(info, SI, fr, normalize=False)
    div = RC.image_load_module_aug(info, SI, fr)
    ref = R.image_load(fr, info, SI)              # divided by its maximum
    assert plain.shape == (size[0] * size[1], n)
    assert np.abs(plain - ref * plain.max()).max() <= 2.4e-7 * 2 * np.abs(plain).max()
    np.testing.assert_array_equal(div, plain / plain.max())

"""The maximum of the rectified movie when most of it is never interpolated for it: the largest output
in the first, a middle or the last frame and tile; where it is extrapolated outside the raw cut;
constant movies (every raw value equals the largest output); negative values; NaN and infinite pixels.
The divided movie must be the undivided one over its maximum, to the bit."""
import numpy as np
import pytest

from mesolf_gb300 import rectify as RC

pytestmark = pytest.mark.gpu


def movie(kind, shape, n, rng):
    y, x = np.mgrid[0:shape[0], 0:shape[1]]
    fr = rng.integers(100, 3000, shape + (n,)).astype(np.uint16)
    if kind.startswith("peak"):
        f = {"peak_first": 0, "peak_mid": n // 2, "peak_last": n - 1}[kind]
        r = {"peak_first": 3, "peak_mid": shape[0] // 2, "peak_last": shape[0] - 4}[kind]
        fr[r:r + 2, r % shape[1]:r % shape[1] + 2, f] = 60000
    elif kind == "border":   # rises towards every side: the largest output is extrapolated
        d = np.maximum(np.abs(y - shape[0] / 2) / shape[0], np.abs(x - shape[1] / 2) / shape[1])
        fr = np.repeat((100 + 8000 * d)[:, :, None], n, 2).astype(np.uint16)
    elif kind == "constant":
        fr[:] = 777
    elif kind == "zero_frames":
        fr[:, :, :-1] = 0
    elif kind == "negative":
        fr = -1.0 - fr.astype(np.float32)
    elif kind == "nan":
        fr = fr.astype(np.float32)
        fr[10, 20, 0], fr[40:50, 30:60, 2] = np.nan, np.nan
    elif kind == "inf":
        fr = fr.astype(np.float32)
        fr[33, 44, 1] = -np.inf
    elif kind == "huge":
        fr = fr.astype(np.float32) * np.float32(1e35)
        fr[20, 20, 3] = -3e38
    return fr


@pytest.mark.parametrize("kind", ["random", "peak_first", "peak_mid", "peak_last", "border", "constant", "zero_frames",
                                  "negative", "nan", "inf", "huge"])
@pytest.mark.parametrize("shape,n", [((181, 140), 9), ((64, 330), 40)])
def test_divided_by_the_maximum(cuda, kind, shape, n):
    fr = movie(kind, shape, n, np.random.default_rng(n))
    yc, xc, dx = shape[0] / 2 + 0.3, shape[1] / 2 - 0.4, 15.27
    size = RC.rectified_size(shape, xc, yc, 15, dx)
    info = {"size": size, "raw_cut": [[1, shape[0]], [1, shape[1]]], "raw_cut_xCenter": xc, "raw_cut_yCenter": yc}
    SI = {"Nnum": 15, "frames_dx": dx}
    plain = RC.image_load_module_aug(info, SI, fr, normalize=False)
    div = RC.image_load_module_aug(info, SI, fr)
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(div, plain / np.nanmax(plain))

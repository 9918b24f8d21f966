"""Short movies on both sides of the line between the one-pass power iteration and the two passes: 20 to 130
frames, few and many pixel blocks per cluster, both modes.  Against the FP64 oracle with the bounds of
test_gpu_summary.py (1e-4 for the image, 1e-5 for the backgrounds)."""
import numpy as np
import pytest

from oracle import mesolf_ref as R
from mesolf_gb300 import synth

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


@pytest.mark.parametrize("P,T", [(29184, 40), (29185, 40), (60003, 127), (60000, 128), (50000, 96), (1000, 20)])
@pytest.mark.parametrize("mode", ["pixelwise", "global"])
def test_short_movies(cuda, P, T, mode):
    from mesolf_gb300.api import summary_image
    Y = synth.sensor_movie(P, T, seed=P + T)
    img, s, t = summary_image(Y, mode, 3, window_1=min(100, T // 2), window_2=5)
    ri, rs, rt = R.summary_image(Y, mode, 3, min(100, T // 2), 5, 3)
    assert rel(s, rs) <= 1e-5 and rel(t, rt) <= 1e-5
    assert rel(img, ri) <= 1e-4

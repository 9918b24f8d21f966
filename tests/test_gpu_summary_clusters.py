"""One-pass power iterations of the summary image in clusters of five CTAs, at the fewest and the most frames of
them and on both sides, few and many pixel blocks, frames off the 16-byte grid.  Against the FP64 oracle with
the bounds of test_gpu_summary.py (1e-4 for the image, 1e-5 for the backgrounds)."""
import numpy as np
import pytest

from oracle import mesolf_ref as R
from mesolf_gb300 import synth

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


@pytest.mark.parametrize("P,T", [(131, 1024), (4100, 1025), (963, 1280), (20001, 1100), (64, 1281), (2051, 600)])
def test_cluster_sizes(cuda, P, T):
    from mesolf_gb300.api import summary_image
    Y = synth.sensor_movie(P, T, seed=P + T)
    img, s, t = summary_image(Y, "pixelwise", 3)
    ri, rs, rt = R.summary_image(Y, "pixelwise", 3)
    assert rel(s, rs) <= 1e-5 and rel(t, rt) <= 1e-5
    assert rel(img, ri) <= 1e-4

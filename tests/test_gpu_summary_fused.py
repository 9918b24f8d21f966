"""Edges of the one-pass power iteration of the summary image: clusters of 1, 2, 4 and 8 CTAs, CTAs
with fewer frames than the others, blocks of pixels that are not full, every alignment of a frame,
very short movies, and movies that keep the two-pass kernels (more than 2048 frames, off the
16-byte grid).  Image and backgrounds against the FP64 oracle with the bounds of
test_gpu_summary.py (1e-4 and 1e-5)."""
import numpy as np
import pytest

from oracle import mesolf_ref as R
from mesolf_gb300 import synth

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


@pytest.mark.parametrize("P,T,it", [
    (64, 130, 2),      # one block, one CTA per cluster
    (65, 256, 3),      # a second block of one pixel; the most frames of a single CTA
    (1027, 257, 3),    # two CTAs; P = 3 mod 4
    (2050, 520, 3),    # four CTAs
    (126, 1025, 2),    # eight CTAs, the last with fewer frames
    (40000, 515, 2),   # more blocks than clusters
    (4098, 2048, 2),   # the most frames
    (333, 2049, 2),    # two passes
    (301, 3, 2),       # three frames: a stage smaller than the final sums
    (5, 20, 3),        # fewer pixels than a vector and a half
])
def test_summary_edges(cuda, P, T, it):
    from mesolf_gb300.api import summary_image
    Y = synth.sensor_movie(P, T, seed=3 * P + T)
    img, s, t = summary_image(Y, "pixelwise", it)
    ri, rs, rt = R.summary_image(Y, "pixelwise", it)
    assert rel(s, rs) <= 1e-5 and rel(t, rt) <= 1e-5
    if np.isfinite(ri).all():
        assert rel(img, ri) <= 1e-4
    else:  # every window covers the whole series: a zero image, 0/0 as in MATLAB
        assert np.isnan(img).all()


def test_movie_off_the_16_byte_grid(cuda):
    """A device movie that starts 4 bytes into an allocation takes the two-pass kernels."""
    import torch
    from mesolf_gb300.api import summary_image
    P, T = 501, 200
    Y = synth.sensor_movie(P, T, seed=5)
    d = torch.empty(P * T + 1, device="cuda")[1:].view(T, P)
    d.copy_(torch.as_tensor(np.ascontiguousarray(Y.T)))
    ri, rs, rt = R.summary_image(Y, "pixelwise", 3, 100, 20, 3)
    img, s, t = (x.cpu().numpy() for x in summary_image(d.T, "pixelwise", 3))
    assert rel(img, ri) <= 1e-4 and rel(s, rs) <= 1e-5 and rel(t, rt) <= 1e-5

"""A frame whose column sum is infinite: the temporal background after one iteration is 0 for the other
frames and NaN for that one (a finite sum over an infinite norm, and infinity over infinity)."""
import numpy as np
import pytest

from mesolf_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,T", [(40000, 30), (301, 200)])
def test_infinite_pixel_in_one_frame(cuda, P, T):
    from mesolf_gb300.api import summary_image
    Y = synth.sensor_movie(P, T, seed=1)
    Y[P // 2, 17] = np.inf
    _, _, t = summary_image(Y, "pixelwise", 1)
    assert np.isnan(t[17])
    assert (np.delete(t, 17) == 0).all()

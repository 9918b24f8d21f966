"""More than 1048560 single output frames are refused on every pitch whose tiles of 128 x 4 outputs fit the
staged kernel, whichever kernel would take them."""
import pytest

from mesolf_gb300 import _lib
from mesolf_gb300 import rectify as RC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dx,dtype", [(15.27, "u16"), (18.0, "f32")])
def test_too_many_frames_are_refused(cuda, dx, dtype):
    import torch
    shape, n = (22, 21), 1048561
    fr = torch.ones((n, shape[1], shape[0]), device=cuda, dtype=torch.uint16 if dtype == "u16" else torch.float32)
    yc, xc = shape[0] / 2 + 0.3, shape[1] / 2 - 0.4
    info = {"size": RC.rectified_size(shape, xc, yc, 15, dx), "raw_cut": [[1, shape[0]], [1, shape[1]]],
            "raw_cut_xCenter": xc, "raw_cut_yCenter": yc}
    with pytest.raises(_lib.MesoLFError) as e:
        RC.image_load_module_aug(info, {"Nnum": 15, "frames_dx": dx}, fr.permute(2, 1, 0))
    assert e.value.code == _lib.MLF_ERR_UNSUPPORTED

"""The direct MEX projector's launch plans (host arithmetic): what a CTA's threads read of its dynamic
shared memory, columns that are loaded ahead and not used among it, stays inside what the launch
asks for, for both variants at every kernel width."""
import ctypes

import pytest

from mesolf_gb300 import _lib

SMS, SMEM_CTA, SMEM_SM = 152, 232448, 233472
ROWS = {0: 1, 1: 2}   # rows per thread
TAPS = {0: 8, 1: 16}  # floats per kernel column of the staged taps


def conv_plan(lib, W, H, n, kw, variant):
    p = (ctypes.c_int64 * 10)()
    rc = lib.mlf_probe_conv_plan(W, H, n, kw, SMS, SMEM_CTA, SMEM_SM, variant, p)
    return list(p) if rc == _lib.MLF_OK else None


def last_read(variant, kwp, SX, pitch, gstride, groups):
    """Highest float read, in buffer 1: of the rows, the last segment of the last row of the last group;
    of the taps, the column after the last."""
    t = TAPS[variant]
    ahead = 16 if variant == 0 else 15  # inputs held per row and thread
    row = 2 * t * kwp + groups * gstride + (groups - 1) * gstride + (ROWS[variant] - 1) * pitch
    tap = t * kwp + t * (kwp + (1 if variant == 0 else 0)) + t - 1
    return max(row + 15 * (SX - 1) + kwp - 1 + ahead, tap)


@pytest.mark.parametrize("variant", [0, 1])
def test_reads_stay_inside_shared_memory(lib, variant):
    for W in (1, 14, 15, 16, 31, 120, 253, 376, 390, 481, 990):
        for H, n in ((1, 1), (15, 1), (40, 2), (198, 4), (376, 20)):
            for kw in range(1, 342):
                p = conv_plan(lib, W, H, n, kw, variant)
                if p is None:
                    continue  # one variant alone need not fit
                v, warps, smem, kwp, SX, pitch, gstride, groups, lanes, cta_lanes = p
                assert v == variant and 1 <= warps <= 12 and smem <= SMEM_CTA
                assert 1 <= cta_lanes <= 32 * warps and groups * SX + SX > min(cta_lanes, lanes)
                assert 4 * (last_read(v, kwp, SX, pitch, gstride, groups) + 1) <= smem, (W, H, n, kw)


def test_every_call_has_a_plan(lib):
    # widths up to the projector's limit, images narrower than a segment and wider than a group
    for W, H, n in ((1, 1, 1), (7, 3000, 1), (15, 16, 4000), (16, 16, 1), (500, 3, 9), (4000, 4000, 1)):
        for kw in (1, 2, 30, 135, 136, 340, 341):
            assert conv_plan(lib, W, H, n, kw, -1), (W, H, n, kw)


def test_narrow_images_get_staging_warps(lib):
    # at most six segments a row and room on the SMs: one warp of lanes, the others stage only
    assert conv_plan(lib, 31, 31, 60, 15, -1)[1::8] == [4, 32]
    assert conv_plan(lib, 31, 31, 30, 21, -1)[1::8] == [8, 32]
    for W, H, n, kw in ((253, 198, 4, 136), (100, 100, 60, 15), (40, 35, 2, 21)):
        p = conv_plan(lib, W, H, n, kw, -1)
        assert p[9] == 32 * p[1]

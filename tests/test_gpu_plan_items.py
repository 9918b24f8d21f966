"""The item tables of the fused view step are part of a work set's device bytes, and of the plan that
bounds them: the bytes grow with the first bf16x2 solve, after one whose view steps need no tables has
allocated everything else."""
import numpy as np
import pytest

from mesolf_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tune", ["0", "1"])
def test_item_tables_are_counted(cuda, monkeypatch, tune):
    import torch
    from mesolf_gb300 import BatchSolver, PhaseSpacePSF
    monkeypatch.setenv("MLF_TUNE", tune)
    H, Ht = synth.make_psf(61, 15, np.arange(7) - 3, seed=1)
    psf = PhaseSpacePSF(H, Ht)
    geo = [((40, 31), (0, 7)), ((12, 60), (2, 3)), ((6, 6), (6, 1))]
    shapes, planes = [(a * 15, b * 15) for (a, b), _ in geo], [p for _, p in geo]
    b = BatchSolver(psf, shapes, planes)
    lfs = [torch.rand((xc, xr), device="cuda").t() + 1 for xr, xc in shapes]
    b.run(lfs, 1, precision="bf16x3")
    before = b.device_bytes
    b.run(lfs, 1, precision="bf16x2")
    tables = b.device_bytes - before
    # one entry per position tile at least: 10 + 6 + 1 tiles
    assert 4 * 17 <= tables < 1 << 20
    assert b.device_bytes <= BatchSolver.plan_bytes(psf, shapes, planes)
    b.close()
    psf.close()

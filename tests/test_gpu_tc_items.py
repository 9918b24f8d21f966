"""Balance of the fused tensor-core view step over uneven patches: the split counts and the item
table must not change what is computed.  A batch of patches with few and many planes (splits of a
patch's own planes, patches with fewer channel tiles than splits, more CTAs than items and more
items than CTAs) against single FP32 solves; tolerance: the bf16x2 solve bound of test_gpu_tc.py
(1e-3)."""
import numpy as np
import pytest

from mesolf_gb300 import synth

pytestmark = pytest.mark.gpu

GEO = [
    [((5, 6), (0, 1)), ((9, 12), (0, 7)), ((6, 5), (6, 1))],                   # one-plane patches at both ends
    [((31, 28), (2, 3)), ((12, 40), (0, 7)), ((33, 30), (1, 5)), ((6, 6), (3, 2))],
]


@pytest.mark.parametrize("geo", GEO)
@pytest.mark.parametrize("tune", ["0", "1"])
def test_uneven_batch_matches_fp32(cuda, monkeypatch, geo, tune):
    import torch
    from mesolf_gb300 import BatchSolver, PhaseSpacePSF, RLSolver
    from mesolf_gb300.api import _fortran
    monkeypatch.setenv("MLF_TUNE", tune)
    H, Ht = synth.make_psf(61, 15, np.arange(7) - 3, seed=2)
    psf = PhaseSpacePSF(H, Ht)
    rng = np.random.default_rng(len(geo))
    shapes = [(a * 15, b * 15) for (a, b), _ in geo]
    lfs = [_fortran(torch.as_tensor(rng.uniform(50, 150, s).astype(np.float32)).cuda())[0] for s in shapes]
    b = BatchSolver(psf, shapes, [p for _, p in geo])
    outs = b.run(lfs, 2, precision="bf16x2")
    for k, (z0, nz) in enumerate(p for _, p in geo):
        sub = PhaseSpacePSF(np.asfortranarray(H[..., z0:z0 + nz]), np.asfortranarray(Ht[..., z0:z0 + nz]))
        s = RLSolver(sub, shapes[k])
        ref = s.run(lfs[k], 2).cpu().numpy().astype(np.float64)
        got = outs[k].cpu().numpy()
        assert np.linalg.norm(got - ref) / np.linalg.norm(ref) <= 1e-3, k
        s.close()
        sub.close()
    b.close()
    psf.close()

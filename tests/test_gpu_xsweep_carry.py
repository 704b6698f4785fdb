"""The face that the FP64 x sweeps hand from one tile to the next through shared
memory: boxes with enough lines to fill the GPU and lines of several tiles,
walked 16 tiles at a time, against one tile per block (which hands on nothing),
bitwise and over repeated evaluations."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [160, 259])
@pytest.mark.parametrize("scheme", ["weno5js", "weno5z", "weno7js"])
def test_carried_faces_equal_formed_ones(nx, scheme, monkeypatch):
    import torch
    import nuc3d_b200 as nb
    desc = nb.BoxDesc(nx, 96, 64, mach=0.3, reynolds=300.0, scheme=(nb.SCHEMES[scheme],) * 3)
    q = [torch.from_numpy(a).cuda() for a in nb.hit_field(desc, seed=5, k_peak=3.0, mach_t=0.2)]
    want = None
    for run, tile in ((1, 32), (4, 64)):  # 1 tile per block, 16 tiles
        monkeypatch.setenv("NUC3D_SWEEP_RUN", str(run))
        monkeypatch.setenv("NUC3D_SWEEP_TILE", str(tile))
        with nb.Solver(desc) as s:
            s.set_state(q)
            for _ in range(20):
                out = [torch.empty_like(q[0]) for _ in range(5)]
                s.rhs(out)
                got = torch.stack(out)
                want = got if want is None else want
                assert torch.isfinite(got).all() and torch.equal(got, want)

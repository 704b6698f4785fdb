"""The FP64 WENO5 y and z sweeps' marching kernel at the sizes where its
bookkeeping can go wrong: lines of one chunk or less, partial last chunks and
phases, groups of 32 lines cut by row ends and by the box's end, every chunk
length, against the oracle's right-hand side at the FP64 parity bar."""

import numpy as np
import pytest

from helpers import desc_from_box, max_rel_l2

pytestmark = pytest.mark.gpu

# (run, tile) environment pins of the five chunk lengths 8, 16, 32, 64, 128
PINS = [(1, 32), (2, 32), (4, 32), (2, 64), (4, 64)]


@pytest.mark.parametrize("shape", [(8, 8, 8), (9, 10, 11), (33, 13, 9), (8, 130, 31), (31, 9, 137)])
@pytest.mark.parametrize("scheme", ["WENO5JS", "WENO5Z"])
@pytest.mark.parametrize("riemann", [0, 2])
def test_march_chunks_match_oracle(shape, scheme, riemann, monkeypatch):
    import torch
    import oracle_ctypes as oc
    import nuc3d_b200 as nb
    nx, ny, nz = shape
    box = oc.Box(nx, ny, nz, scheme=(getattr(oc, scheme),) * 3, mach=0.3, reynolds=700.0,
                 riemann=riemann)
    rng = np.random.default_rng(11)
    q = [np.ascontiguousarray(a * (1 + 0.02 * rng.standard_normal(a.shape)))
         for a in oc.Oracle().tgv(box)]
    want, _ = oc.Oracle().rhs(box, q)
    first = None
    for run, tile in PINS:
        monkeypatch.setenv("NUC3D_SWEEP_RUN", str(run))
        monkeypatch.setenv("NUC3D_SWEEP_TILE", str(tile))
        with nb.Solver(desc_from_box(box)) as s:
            s.set_state(q)
            out = [torch.empty(nz, ny, nx, dtype=torch.float64, device="cuda") for _ in range(5)]
            s.rhs(out)
            got = [o.cpu().numpy() for o in out]
        assert max_rel_l2(got, want) < 1e-12
        first = got if first is None else first
        assert all(np.array_equal(a, b) for a, b in zip(got, first))

"""The FP64 CRWENO5 y and z sweeps by marching elimination on their longest lines (up
to the 512 cells that boxes admit) at equal spacings, where the oracle's steps stay
finite: right-hand side and steps at the FP64 parity bar."""

import numpy as np
import pytest

from helpers import desc_from_box, max_rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(9, 512, 8), (8, 9, 512), (33, 8, 259), (10, 301, 9)])
@pytest.mark.parametrize("riemann", [0, 2])
def test_long_lines_match_oracle(shape, riemann):
    import torch
    import oracle_ctypes as oc
    import nuc3d_b200 as nb
    nx, ny, nz = shape
    box = oc.Box(nx, ny, nz, lx=0.2 * nx, ly=0.2 * ny, lz=0.2 * nz, scheme=(oc.CRWENO5,) * 3,
                 mach=0.3, reynolds=700.0, riemann=riemann)
    rng = np.random.default_rng(13)
    q = [np.ascontiguousarray(a * (1 + 0.02 * rng.standard_normal(a.shape)))
         for a in oc.Oracle().tgv(oc.Box(nx, ny, nz, mach=0.3))]
    with nb.Solver(desc_from_box(box)) as s:
        s.set_state(q)
        out = [torch.empty(nz, ny, nx, dtype=torch.float64, device="cuda") for _ in range(5)]
        s.rhs(out)
        want, _ = oc.Oracle().rhs(box, q)
        assert max_rel_l2([o.cpu().numpy() for o in out], want) < 1e-12
        want, _, _ = oc.Oracle().run_steps(box, 0.3, 2, list(q))
        assert all(np.isfinite(a).all() for a in want)
        s.step(2, 0.3)
        assert max_rel_l2(s.get_state(), want) < 1e-12

"""The 2.5-D stencil kernels at the short pencil depths that small boxes run:
boxes thinner and flatter than a tile, depths that do and do not divide the
planes, both stencil reaches.  Every depth computes every cell alike, so the
states after a step are bitwise those of the 32-plane pencils."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(8, 8, 8), (33, 9, 11), (40, 17, 13)])
@pytest.mark.parametrize("vis", ["cd6", "cd8"])
@pytest.mark.parametrize("precision", [0, 1])
def test_short_pencils_equal_long_ones(shape, vis, precision, monkeypatch):
    import nuc3d_b200 as nb
    nx, ny, nz = shape
    desc = nb.BoxDesc(nx, ny, nz, mach=0.3, reynolds=300.0, precision=precision,
                      vis_scheme=(nb.VIS_SCHEMES[vis],) * 3)
    rng = np.random.default_rng(3)
    q = nb.hit_field(desc, seed=2, k_peak=2.0, mach_t=0.2)
    q = [np.ascontiguousarray(a * (1 + 0.02 * rng.standard_normal(a.shape))) for a in q]
    want = None
    for depth in (32, 8, 4, 2):
        monkeypatch.setenv("NUC3D_PENCIL_DEPTH", str(depth))
        with nb.Solver(desc) as s:
            s.set_state(q)
            s.step(1, 0.5)
            got = s.get_state()
            assert s.tuning()["pencil_depth"][0] == depth
        want = got if want is None else want
        assert all(np.isfinite(a).all() and np.array_equal(a, b) for a, b in zip(got, want))

"""Boxes much longer along one axis than a launch grid's y extent (65535 blocks)
could cover: a periodic box that repeats a short one computes, cell for cell, the
short one's values, bitwise (power-of-two repeats leave the spacings exact)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis,long", [("z", 1 << 20), ("x", 1 << 21)])
def test_long_box_repeats_short_one(axis, long):
    import torch
    import nuc3d_b200 as nb
    d = "xyz".index(axis)
    n = [8, 8, 8]
    n[d] = 16
    box = dict(mach=0.3, reynolds=300.0, scheme=(nb.WENO5JS,) * 3)
    short = nb.BoxDesc(*n, **box)
    rng = np.random.default_rng(17)
    q = [np.ascontiguousarray(a * (1 + 0.02 * rng.standard_normal(a.shape)))
         for a in nb.hit_field(short, seed=4, k_peak=2.0, mach_t=0.2)]
    with nb.Solver(short) as s:
        s.set_state(q)
        s.step(2, 0.5)
        want = [torch.from_numpy(a).cuda() for a in s.get_state()]
    reps = long // n[d]
    n[d] = long
    lengths = [2 * np.pi] * 3
    lengths[d] *= reps
    dims = [1, 1, 1]
    dims[2 - d] = reps
    with nb.Solver(nb.BoxDesc(*n, lx=lengths[0], ly=lengths[1], lz=lengths[2], **box)) as s:
        s.set_state([torch.from_numpy(a).cuda().repeat(dims) for a in q])
        s.step(2, 0.5)
        got = [torch.empty(*n[::-1], dtype=torch.float64, device="cuda") for _ in range(5)]
        s.get_state(got)
        for g, w in zip(got, want):
            assert torch.equal(g, w.repeat(dims))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("axis", ["x", "y", "z"])
def test_one_long_box_in_a_batch_of_small_ones(axis, precision):
    """Launches of a batch cover each box's own extents, not the longest's: states
    equal those of the boxes alone."""
    import nuc3d_b200 as nb
    long = [9, 10, 12]
    long["xyz".index(axis)] = 1100
    # (the reference's dt leaves z out, so the spacings are alike)
    descs = [nb.BoxDesc(*n, lx=0.2 * n[0], ly=0.2 * n[1], lz=0.2 * n[2], mach=0.3,
                        reynolds=300.0, precision=precision, scheme=(s,) * 3)
             for s in (nb.WENO5JS, nb.WENO5Z, nb.WENO7JS) for n in ((16, 12, 9), long, (8, 33, 10))]

    def state(d, seed):
        rng = np.random.default_rng(seed)
        return [np.ascontiguousarray(a * (1 + 0.02 * rng.standard_normal(a.shape)))
                for a in nb.hit_field(d, seed=2, k_peak=2.0, mach_t=0.2)]
    states = [state(d, k) for k, d in enumerate(descs)]
    alone = []
    for d, q in zip(descs, states):
        with nb.Solver(d) as s:
            s.set_state(q)
            s.step(2, 0.3)
            alone.append(s.get_state())
    with nb.Batch(precision) as b:
        ids = [b.add(d) for d in descs]
        for i, q in zip(ids, states):
            b.set_state(i, q)
            b.set_cfl(i, 0.3)
        b.step(2)
        for i, a in zip(ids, alone):
            assert all(np.isfinite(x).all() and np.array_equal(x, y)
                       for x, y in zip(b.get_state(i), a))

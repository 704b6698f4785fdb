"""The tuned shapes of the FP64 sweeps follow the size of what is stepped: what small
boxes were tuned to does not stay for a large box that joins them, and a size met
before takes its stored choice."""

import pytest

pytestmark = pytest.mark.gpu


def test_chunks_are_chosen_again_for_a_large_box():
    import nuc3d_b200 as nb
    with nb.Batch(nb.FP64) as b:
        small = b.add(nb.BoxDesc(16, 16, 16, mach=0.3))
        b.init_state(small, "tgv")
        b.step(1)
        first = {k: v for k, v in b.tuning().items() if k.startswith("weno5js")}
        assert set(first) == {"weno5js_x", "weno5js_y", "weno5js_z"}
        large = b.add(nb.BoxDesc(192, 192, 192, mach=0.3))
        b.init_state(large, "tgv")
        b.step(1)
        for name, (choice, times) in b.tuning().items():
            if name in first:
                # 36864 lines: the shortest chunk is not among what such a box times
                assert times[choice] > 0.0 and times["32x32" if name[-1] == "x" else "8x8"] == 0.0
        b.remove(large)
        b.step(1)
        for name, (choice, _) in b.tuning().items():
            if name in first:
                assert choice == first[name][0]

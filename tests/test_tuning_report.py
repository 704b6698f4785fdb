"""The Python report of the autotuner's choices: a pencil depth that was not timed (0
from the library) is left out, so that it cannot pass for the fastest."""

import ctypes as C


def test_untimed_depths_are_left_out():
    import nuc3d_b200 as nb

    def sweeps(_h, rl, ms):
        return nb.OK

    def pencil(_h, depth, ms):
        depth._obj.value = 4
        C.memmove(ms, (C.c_double * 3)(0.25, 0.125, 0.0), 24)
        return nb.OK
    assert nb._tuning(sweeps, None, pencil) == {"pencil_depth": (4, {32: 0.25, 16: 0.125})}

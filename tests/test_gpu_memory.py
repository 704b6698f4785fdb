"""Device memory that the solvers of a process keep: bounded for all of them together,
given back with the last, and shared safely by threads that create and destroy
solvers at once."""

import gc
import threading

import pytest

pytestmark = pytest.mark.gpu


def _used():
    import torch
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def test_idle_memory_is_bounded_over_all_solvers_and_given_back():
    import torch
    import nuc3d_b200 as nb
    desc = nb.BoxDesc(128, 128, 128, mach=0.3)

    def solver():
        s = nb.Solver(desc)
        s.init_state("tgv")
        s.step(1, 0.5)
        s.spectra()  # 130 MB of scratch, freed again
        return s
    solver().close()  # modules, cuFFT
    gc.collect()
    torch.cuda.empty_cache()
    base = _used()
    solvers = [solver() for _ in range(5)]
    boxes = 5 * desc.device_bytes()
    # 256 MB kept, and the plans, graphs and the pool's granularity: 24 MB a solver
    assert _used() - base - boxes <= (256 + 5 * 24) << 20
    for s in solvers:
        s.close()
    assert _used() - base <= 64 << 20


def test_solvers_come_and_go_in_threads():
    import torch
    import nuc3d_b200 as nb
    errors = []

    def work(k):
        try:
            stream = torch.cuda.Stream()
            for n in range(12):
                desc = nb.BoxDesc(16 + 8 * ((k + n) % 4), 24, 32, mach=0.3)
                with nb.Solver(desc, stream=stream) as s:
                    s.init_state("tgv")
                    s.step(2, 0.5)
                    s.spectra()
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(e)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]

"""Entry points whose launch needs a per-kernel shared-memory limit, called by two
host threads with very different needs at once: no call may lower the limit
under the other's launch, and results are those of one thread alone."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _both(work, jobs, rounds):
    """work(job) by one thread per job, `rounds` times each; the first errors."""
    errors = []

    def loop(job):
        try:
            for _ in range(rounds):
                work(job)
        except Exception as e:  # noqa: BLE001 - reported by the caller
            errors.append(e)

    threads = [threading.Thread(target=loop, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


@pytest.mark.parametrize("scheme", ["crweno5", "hccs", "hccs77"])
def test_reconstruct_of_short_and_long_lines(scheme):
    import torch
    import nuc3d_b200 as nb
    s = nb.SCHEMES[scheme]
    h = nb.SCHEME_HALO[s]
    jobs = []
    for nx, lines in ((4096, 8), (48, 64)):
        g = torch.Generator(device="cuda").manual_seed(nx)
        f = 1 + 0.3 * torch.rand(1, lines, nx, generator=g, device="cuda", dtype=torch.float64)
        job = dict(f=f, hl=f[..., -h:].contiguous(), hr=f[..., :h].contiguous(),
                   out=torch.empty(1, lines, nx + 1, device="cuda", dtype=torch.float64),
                   stream=torch.cuda.Stream())
        torch.cuda.synchronize()
        jobs.append(job)

    def work(j):
        nb.reconstruct(s, 1, nb.QUIRKS_REFERENCE, j["f"], j["hl"], j["hr"], j["out"],
                       stream=j["stream"])
        j["stream"].synchronize()
    for j in jobs:
        work(j)
        j["want"] = j["out"].clone()
    torch.cuda.synchronize()
    _both(work, jobs, 5000)
    for j in jobs:
        assert torch.equal(j["out"], j["want"])


def test_spectra_of_small_and_large_boxes():
    import nuc3d_b200 as nb
    jobs = []
    for n in (176, 208):  # both above the 48 KB that need no limit
        desc = nb.BoxDesc(n, n, n, mach=0.3)
        s = nb.Solver(desc)
        s.set_state(nb.hit_field(desc, seed=1, k_peak=3.0, mach_t=0.2))
        jobs.append(dict(solver=s, want=s.spectra()))

    def work(j):
        assert np.array_equal(j["solver"].spectra(), j["want"])
    _both(work, jobs, 200)
    for j in jobs:
        j["solver"].close()

"""The line-solve schemes' reconstruction operator over the line lengths and
counts its dispatch turns on: the shortest lines (one or two lanes hold rows),
lengths around the warp's 32-lane partition, the longest line (one warp per
block), and short lines in numbers that go to the thread-per-line kernel,
against the oracle at the FP64 parity bar."""

import numpy as np
import pytest

from helpers import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", ["crweno5", "hccs", "hccs77"])
@pytest.mark.parametrize("up", [1, -1])
@pytest.mark.parametrize("nx,lines", [(9, 5), (15, 3), (31, 9), (47, 17), (48, 8), (69, 7),
                                      (133, 9), (512, 3), (4096, 2), (47, 16385), (48, 16385)])
def test_reconstruct_lines_match_oracle(scheme, up, nx, lines):
    import torch
    import nuc3d_b200 as nb
    from oracle_ctypes import QUIRKS_REFERENCE, Oracle
    sch = nb.SCHEMES[scheme]
    h = nb.SCHEME_HALO[sch]
    rng = np.random.default_rng(nx + lines)
    x = np.linspace(0.0, 6.0 * np.pi, nx + 2 * h)
    f = np.sin(x + rng.uniform(0, 6, (1, lines, 1))) + 0.05 * rng.standard_normal((1, lines, nx + 2 * h))
    parts = [np.ascontiguousarray(p) for p in (f[..., h:-h], f[..., :h], f[..., -h:])]
    want = Oracle().reconstruct_field(sch, up, QUIRKS_REFERENCE, *parts)
    dev = [torch.from_numpy(p).cuda() for p in parts]
    out = torch.full((1, lines, nx + 1), float("nan"), dtype=torch.float64, device="cuda")
    nb.reconstruct(sch, up, QUIRKS_REFERENCE, *dev, out)
    assert rel_l2(out.cpu().numpy(), want) < 1e-12

"""Shell spectra over the sizes their launch turns on: odd and even extents, box
sizes on both sides of the batched transforms, the same solver asked twice and
two boxes of different sizes asked in turn (the transform plan follows the
size), against numpy's transforms binned mode by mode."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shell(k):
    f = np.floor(k)
    return np.where(k - f - 0.5 <= 0, f, f + 1).astype(int)


def _want(desc, q):
    nx, ny, nz = desc.nx, desc.ny, desc.nz
    kmax = min(nx, ny, nz) // 2
    u = [q[i] / q[0] for i in (1, 2, 3)]
    F = [np.fft.fftn(f) / f.size for f in u]
    k = [np.where(np.arange(n) >= n / 2, np.arange(n) - n, np.arange(n)).astype(float)
         for n in (nz, ny, nx)]
    mag = np.sqrt(k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2)
    mag = np.where(mag < 1e-6, 1.0, mag)
    on = mag < kmax
    kin = np.bincount(_shell(mag[on]), 0.5 * sum(np.abs(f) ** 2 for f in F)[on], kmax + 1)[:kmax]
    i = [np.arange(n).astype(float) for n in (nz, ny, nx)]
    k0 = np.sqrt(i[0][:, None, None] ** 2 + i[1][None, :, None] ** 2 + i[2][None, None, :] ** 2)
    on = k0 < kmax
    den = (np.abs(np.fft.fftn(q[0]) / q[0].size) ** 2)
    return kin, np.bincount(_shell(k0[on]), den[on], kmax + 1)[:kmax]


@pytest.mark.parametrize("shapes", [[(9, 12, 15), (16, 9, 33)], [(64, 64, 64), (65, 64, 66)],
                                    [(97, 70, 45)]])
def test_spectra_match_numpy(shapes):
    import nuc3d_b200 as nb
    with nb.Batch(nb.FP64) as b:
        boxes = []
        for nx, ny, nz in shapes:
            d = nb.BoxDesc(nx, ny, nz, mach=1.0)
            rng = np.random.default_rng(nx)
            q = [np.ascontiguousarray(a + 0.01 * rng.standard_normal(a.shape))
                 for a in nb.hit_field(d, seed=nx, k_peak=2.0, mach_t=0.3)]
            i = b.add(d)
            b.set_state(i, q)
            boxes.append((i, d, q))
        for i, d, q in boxes * 2:
            s = dict(zip(nb.SPECTRA_NAMES, b.spectra(i)))
            kin, den = _want(d, q)
            # both sides FP64: rounding of the transforms
            assert np.linalg.norm(s["kin"] - kin) <= 1e-12 * np.linalg.norm(kin)
            assert np.linalg.norm(s["den"] - den) <= 1e-12 * np.linalg.norm(den)
            assert np.linalg.norm(s["kinc"] + s["kins"] - kin) <= 1e-12 * np.linalg.norm(kin)

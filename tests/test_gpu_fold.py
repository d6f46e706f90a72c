"""The folded correlation's half lengths (jerk_fold.cu) against the defining
circular correlation in float64, through JerkPlan.volume with a caller's own
kernel rows: rows of every support, so that every window and every way a row
is folded occurs, and rows without a support (random values at every
frequency), which only the whole half length holds."""

import numpy as np
import pytest

from prestozl_b200 import jerk

pytestmark = pytest.mark.gpu


def _rows(rng, N, hs):
    """One row per support h: taps on [-2h, 2h), none (h = 0): any values."""
    out = np.zeros((len(hs), N), dtype=np.complex64)
    for i, h in enumerate(hs):
        if h == 0:
            k = rng.standard_normal((N, 2))
            out[i] = ((k[:, 0] + 1j * k[:, 1]) / np.sqrt(2.0)).astype(np.complex64)
            continue
        t = np.arange(-2 * h, 2 * h)
        k = np.zeros(N, dtype=np.complex128)
        k[t % N] = (rng.standard_normal(4 * h) + 1j * rng.standard_normal(4 * h)) / np.sqrt(8.0 * h)
        out[i] = np.fft.fft(k).astype(np.complex64)
    return out


def _plan(N, hw, uselen, rows, bins, batch):
    o = jerk.Obs()
    o.numbins, o.lobin, o.highestbin = bins, 0, bins - 1
    o.rlo, o.zlo, o.wlo = float(hw + 3), -(len(rows) - 1), 0
    o.corr_uselen, o.numz, o.numw, o.numharmstages = uselen, len(rows), 0, 1
    o.numindep[0], o.powcut[0] = bins, 1e30
    sub = dict(numharm=1, harmnum=1, zmax=len(rows) - 1, wmax=0, numz=len(rows), numw=1,
               fftlen=N, halfwidth=hw, kern=rows[None])
    return jerk.JerkPlan(o, [sub], batch=batch)


@pytest.mark.parametrize("N,hw,short", [(512, 30, 0), (768, 40, 2), (1024, 60, 100), (1280, 70, 0),
                                        (2048, 100, 6), (2048, 40, 900), (4096, 200, 0),
                                        (4096, 64, 1500)])
def test_windows_match_the_circular_correlation(N, hw, short):
    rng = np.random.default_rng(N + hw)
    M = N // 2
    uselen = N - 4 * hw - short  # short: good bins that do not fill the length
    hs = sorted({1, 2, 7, hw // 2, hw - 1, hw, min(hw + 9, N // 4), N // 4})
    # supports at the edges of every half length's window
    for L in (256, 384, 512, 640, 768, 1024, 1280, 1536, 1792):
        for d in (-1, 0, 1):
            h = (L - uselen // 2) // 2 + d
            if 0 < h <= hw:
                hs.append(h)
    hs = hs + [0] * (3 if (len(hs) + 3) % 2 else 2)  # odd row count: zmax even
    rows = _rows(rng, N, hs)
    bins = 3 * M
    spec = (rng.standard_normal((bins, 2)) @ np.array([1.0, 1j])).astype(np.complex64)
    plan = _plan(N, hw, uselen, rows, bins, batch=2)
    for rstep in (0, plan.num_rsteps - 1):
        vol, rlo = plan.volume(spec, rstep, 0)
        lo = rlo - hw
        d = np.zeros(M, dtype=np.complex128)
        have = spec[lo:lo + M]
        d[:len(have)] = have
        p = d.real ** 2 + d.imag ** 2
        d /= np.sqrt(np.sort(p)[(M - 1) // 2] / np.log(2.0))
        X = np.tile(np.fft.fft(d), 2)
        y = np.fft.ifft(X * np.conj(rows.astype(np.complex128)), axis=1)[:, 2 * hw:2 * hw + uselen]
        want = y.real ** 2 + y.imag ** 2
        # the volumes' bound everywhere in these tests: 1e-5 of max(power, 1)
        assert vol.shape == (1, len(hs), uselen)
        assert np.all(np.abs(vol[0] - want) <= 1e-5 * np.maximum(want, 1.0))
    plan.close()

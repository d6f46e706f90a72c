"""Plans on a resident bank fold its rows by the supports generated rows have,
plans on rows of the caller's own by measured ones: the same volumes, bit for bit,
from the same rows -- generated, generated but for one row, and any."""

import ctypes as C

import numpy as np
import pytest

from prestozl_b200 import jerk

pytestmark = pytest.mark.gpu


def _bank(subs):
    bank = jerk.DeviceBank(subs)
    n = sum(s["numw"] * s["numz"] * s["fftlen"] for s in subs)
    rows = np.empty(n, dtype=np.complex64)
    jerk._check(jerk.lib().jerk_copy_to_host(rows.ctypes.data_as(C.c_void_p), bank.ptr, 8 * n))
    bank.close()
    return rows


@pytest.mark.parametrize("change", ["none", "one", "narrow", "all"])
@pytest.mark.parametrize("zmax,wmax,numharm", [(20, 60, 8), (100, 0, 16), (200, 300, 2),
                                               (300, 100, 1), (6, 20, 32)])
def test_same_volumes_by_either_way_of_folding(zmax, wmax, numharm, change):
    torch = pytest.importorskip("torch")
    N = 1 << 18
    rng = np.random.default_rng(zmax)
    spec = (rng.standard_normal((N // 2, 2)) @ np.array([1.0, 1j])).astype(np.complex64)
    obs, fftlen, _ = jerk.obs_from_params(N // 2, N, 64e-6, zmax, wmax, numharm, 3.0,
                                          wmax_given=wmax > 0)
    subs = jerk.subharm_sizes(obs, fftlen)
    rows = _bank(subs)
    if change == "all":
        rows = (rng.standard_normal((len(rows), 2)) @ np.array([1.0, 1j])).astype(np.complex64)
    off = 0
    for s in subs:
        n = s["numw"] * s["numz"]
        mine = rows[off:off + n * s["fftlen"]].reshape(n, s["fftlen"])
        off += mine.size
        if s is subs[-1] and change == "one":  # the narrowest response, now without a support
            mine[n // 2] = np.exp(2j * np.pi * rng.uniform(size=s["fftlen"])).astype(np.complex64)
        if s is subs[0] and change == "narrow":  # ... and the widest, now one of four taps
            mine[0] = np.fft.fft(np.r_[1.0, 0.5, np.zeros(s["fftlen"] - 4), 0.25, 0.5])
        s["kern"] = mine.reshape(s["numw"], s["numz"], s["fftlen"]).copy()
    dev = torch.from_numpy(rows.view(np.float32)).cuda()
    own = jerk.JerkPlan(obs, subs, batch=2)
    plan = jerk.JerkPlan(obs, subs, batch=2, device_bank=dev.data_ptr())
    for k in (0, plan.num_rsteps - 1):
        for i in range(len(subs)):
            a, b = own.volume(spec, k, i), plan.volume(spec, k, i)
            assert a[1] == b[1] and np.array_equal(a[0].view(np.uint32), b[0].view(np.uint32))
    own.close()
    plan.close()

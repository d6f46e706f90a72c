"""The harmonic sum's ring of row copies (the default form on large volumes)
against the gather form (harm_mode 1): the same adds in the same order, so the
same hits bit for bit -- at every stage count, one and several w rows, one and
several r tiles, z rows that do not divide, a short last batch, and thresholds
low enough that a CTA's hits overflow its shared-memory list."""

import numpy as np
import pytest

from prestozl_b200 import jerk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zmax,wmax,numharm,batch,rsteps,sigma", [
    (100, 100, 1, 13, 20, -9.0), (150, 100, 2, 9, 14, -9.0), (102, 60, 4, 16, 23, -9.0),
    (50, 140, 8, 16, 17, -9.0), (64, 0, 8, 64, 70, -9.0), (100, 0, 16, 24, 31, -9.0),
    (90, 40, 16, 11, 12, -9.0), (260, 120, 4, 5, 6, -9.0), (50, 140, 8, 16, 17, -12.0)])
def test_ring_equals_gathers(zmax, wmax, numharm, batch, rsteps, sigma):
    torch = pytest.importorskip("torch")
    N = 1 << 21
    g = torch.Generator(device="cuda")
    g.manual_seed(zmax + numharm)
    spec = torch.view_as_complex(torch.randn((N // 2, 2), generator=g, device="cuda"))
    spec[40_000::3001] *= 12.0
    obs, fftlen, _ = jerk.obs_from_params(N // 2, N, 64e-6, zmax, wmax, numharm, 3.0,
                                          wmax_given=wmax > 0)
    for i in range(obs.numharmstages):  # cutoffs by powers: noise crosses them
        obs.powcut[i] = (11.0 if sigma > -10 else 8.0) + 3.0 * (1 << i) ** 0.75
    subs = jerk.subharm_sizes(obs, fftlen)
    bank = jerk.DeviceBank(subs)
    got = []
    for mode in (0, 1):
        plan = jerk.JerkPlan(obs, subs, batch=batch, device_bank=bank.ptr.value, harm_mode=mode)
        got.append(plan.search(spec, 3, rsteps, want_hits=True)[1:])
        plan.close()
    bank.close()
    assert len(got[1][0]) > 0
    assert np.array_equal(got[0][0], got[1][0])
    assert np.array_equal(got[0][1].view(np.uint32), got[1][1].view(np.uint32))

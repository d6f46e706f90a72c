"""Overlapped launches of a batch: plain passes, passes replayed from a graph and
passes with events between all launches (each then waits for the one before)
give the same hits, bit for bit, also when repeated -- with row sets launched by
themselves, merged, and both, and a short last batch."""

import numpy as np
import pytest

from prestozl_b200 import jerk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zmax,wmax,numharm,batch,rsteps", [
    (20, 60, 8, 8, 27), (100, 0, 16, 32, 70), (50, 140, 8, 32, 65), (150, 200, 4, 16, 20),
    (260, 300, 1, 4, 9)])
def test_overlapped_launches_equal_serial(zmax, wmax, numharm, batch, rsteps):
    torch = pytest.importorskip("torch")
    N = 1 << 21
    g = torch.Generator(device="cuda")
    g.manual_seed(zmax + numharm)
    spec = torch.view_as_complex(torch.randn((N // 2, 2), generator=g, device="cuda"))
    spec[40_000::3001] *= 12.0
    obs, fftlen, _ = jerk.obs_from_params(N // 2, N, 64e-6, zmax, wmax, numharm, 3.0,
                                          wmax_given=wmax > 0)
    for i in range(obs.numharmstages):
        obs.powcut[i] = 11.0 + 3.0 * (1 << i) ** 0.75
    subs = jerk.subharm_sizes(obs, fftlen)
    bank = jerk.DeviceBank(subs)
    want = None
    for profile, graph in ((True, False), (False, False), (False, True)):
        plan = jerk.JerkPlan(obs, subs, batch=batch, device_bank=bank.ptr.value, use_graph=graph)
        plan.set_profiling(profile)
        for _ in range(1 if profile else 4):
            got = plan.search(spec, 3, rsteps, want_hits=True)[1:]
            if want is None:
                want = got
                assert len(want[0]) > 0
            assert np.array_equal(got[0], want[0])
            assert np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
        plan.close()
    bank.close()


def test_series_back_to_back_equal_alone():
    """Series of several lengths whitened and zapped one right after the other:
    each as with the device idle before every call."""
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    series = [torch.randn(n, generator=g, device="cuda") for n in (32768, 98304, 786432, 32768)]
    lo = np.array([0.2, 0.5, 0.5001]) * 16384

    def one(ts, idle):
        if idle:
            torch.cuda.synchronize()
        out = jerk.spectrum_from_timeseries(ts)
        if idle:
            torch.cuda.synchronize()
        return jerk.zap_birdies(out, ts.numel(), lo, lo + 3.0)

    alone = [one(ts, True).clone() for ts in series]
    torch.cuda.synchronize()
    for _ in range(5):
        got = [one(ts, False) for ts in series]
        for a, b in zip(alone, got):
            assert torch.equal(torch.view_as_real(a).view(torch.int32),
                               torch.view_as_real(b).view(torch.int32))


def test_polishing_in_sequence_equals_fresh():
    """Candidates of one, few and many harmonics, with and without w, polished
    one after another by one polisher: each as by a polisher of its own, from a
    spectrum on the device and on the host."""
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda")
    g.manual_seed(9)
    spec = torch.view_as_complex(torch.randn((1 << 20, 2), generator=g, device="cuda"))
    host = spec.cpu().numpy()
    cands = [(1, 40000.25, 3.0, 0.0), (16, 30123.5, 9.5, -14.0), (4, 90000.0, -40.0, 60.0),
             (8, 20011.75, 0.0, 0.0), (16, 30123.5, 9.5, -14.0)]
    shared = jerk.Polisher()
    for numharm, r, z, w in cands:
        fresh = jerk.Polisher()
        want = fresh.optimize(host, numharm, r, z, w)
        fresh.close()
        for src in (spec, host):
            got = shared.optimize(src, numharm, r, z, w)
            assert tuple(got[0]) == tuple(want[0])
            assert np.array_equal(np.asarray(got[1]["pow"]), np.asarray(want[1]["pow"]))
            assert np.array_equal(np.asarray(got[2]), np.asarray(want[2]))
    shared.close()

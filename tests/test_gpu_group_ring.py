"""Waves whose harmonic sums take the ring of row copies, several plans merged in
one launch: each plan's raw hits equal, bit for bit, those of the plan searched
alone and those of the gather form -- for plans of unequal size, short last
batches, and beside one whose volumes are large enough for a launch of its own."""

import numpy as np
import pytest

from prestozl_b200 import jerk

pytestmark = pytest.mark.gpu

RING, OWN = 48e6, 1e9  # volume bytes of a batch: the ring from, its own launch from


def _rstep_bytes(obs, subs):
    rows = [(s["numw"] * s["numz"], int(obs.corr_uselen * s["harmnum"] / s["numharm"]))
            for s in subs]
    return 4.0 * sum(n * (r + 7) for n, r in rows)


# (zmax, wmax, batch, rsteps) of each plan
@pytest.mark.parametrize("numharm,plans", [
    (8, [(50, 160, 9, 31), (64, 100, 20, 45), (60, 60, 8, 46)]),
    (8, [(50, 160, 9, 31), (100, 200, 28, 33), (60, 60, 8, 46)]),
    (16, [(90, 40, 6, 16), (50, 100, 16, 39), (80, 60, 10, 24)]),
    (2, [(100, 100, 20, 46), (64, 140, 33, 73)]),
    (1, [(150, 140, 20, 47), (120, 140, 24, 62)])])
def test_merged_ring_equals_each_plan_alone(numharm, plans):
    torch = pytest.importorskip("torch")
    N = 1 << 20
    stream = torch.cuda.Stream()
    group, alone, banks, large = [], [], [], 0
    for i, (zmax, wmax, batch, rsteps) in enumerate(plans):
        g = torch.Generator(device="cuda")
        g.manual_seed(31 + i)
        spec = torch.view_as_complex(torch.randn((N // 2, 2), generator=g, device="cuda"))
        spec[40_000::3001] *= 12.0
        obs, fftlen, _ = jerk.obs_from_params(N // 2, N, 64e-6, zmax, wmax, numharm, 3.0,
                                              wmax_given=True)
        for k in range(obs.numharmstages):
            obs.powcut[k] = 11.0 + 3.0 * (1 << k) ** 0.75
        subs = jerk.subharm_sizes(obs, fftlen)
        per = _rstep_bytes(obs, subs)
        assert 1.02 * RING <= per * (rsteps % batch) and rsteps > batch
        assert per * batch <= 0.98 * OWN or per * batch >= 1.02 * OWN
        large += per * batch >= OWN
        bank = jerk.DeviceBank(subs)
        torch.cuda.synchronize()
        gather = jerk.JerkPlan(obs, subs, batch=batch, device_bank=bank.ptr.value, harm_mode=1)
        want = gather.search(spec, 1, rsteps, want_hits=True)[1:]
        gather.close()
        p = jerk.JerkPlan(obs, subs, batch=batch, stream=stream.cuda_stream,
                          device_bank=bank.ptr.value)
        assert 1 + rsteps <= p.num_rsteps
        got = p.search(spec, 1, rsteps, want_hits=True)[1:]
        assert len(want[0]) > 0
        assert np.array_equal(got[0], want[0])
        assert np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
        group.append((p, spec, rsteps))
        alone.append(want)
        banks.append(bank)
    assert len(plans) - large >= 2  # merged with one another
    for p, spec, rsteps in group:
        p.begin(spec, 1, rsteps)
    while jerk.group_advance([p for p, _, _ in group], ahead=2):
        pass
    for (p, _, _), want in zip(group, alone):
        got = p.collect(want_hits=True)[1:]
        assert np.array_equal(got[0], want[0])
        assert np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
    for p, _, _ in group:
        p.close()
    for b in banks:
        b.close()

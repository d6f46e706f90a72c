"""A volume asked of a plan whose search is in flight: the volume of an idle plan,
and a pass whose hits are, bit for bit, those of a pass left alone."""

import numpy as np
import pytest

from prestozl_b200 import jerk

pytestmark = pytest.mark.gpu


def _problem(torch, batch, max_hits=0, graph=False):
    N = 1 << 20
    g = torch.Generator(device="cuda")
    g.manual_seed(21)
    spec = torch.view_as_complex(torch.randn((N // 2, 2), generator=g, device="cuda"))
    spec[40_000::3001] *= 12.0
    obs, fftlen, _ = jerk.obs_from_params(N // 2, N, 64e-6, 20, 60, 8, 3.0, wmax_given=True)
    for i in range(obs.numharmstages):
        obs.powcut[i] = 11.0 + 3.0 * (1 << i) ** 0.75
    subs = jerk.subharm_sizes(obs, fftlen)
    bank = jerk.DeviceBank(subs)
    return spec, jerk.JerkPlan(obs, subs, batch=batch, max_hits=max_hits, use_graph=graph,
                               device_bank=bank.ptr.value), bank


def _same_hits(got, want):
    assert np.array_equal(got[0], want[0])
    assert np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))


@pytest.mark.parametrize("waves", [1, 2, 5])
def test_volume_between_waves_leaves_the_pass_alone(waves):
    """The spectrum is on the device; volumes of rsteps before and after the
    batches in flight, after an odd and an even number of batches."""
    torch = pytest.importorskip("torch")
    spec, plan, bank = _problem(torch, batch=4)
    rsteps = 4 * 9 + 3
    want = plan.search(spec, 2, rsteps, want_hits=True)[1:]
    assert len(want[0]) > 0
    ks = (0, 40, plan.num_rsteps - 1)
    alone = [plan.volume(spec, k, sub) for k in ks for sub in (0, 3)]
    plan.begin(spec, 2, rsteps)
    assert jerk.group_advance([plan], ahead=waves) == 1
    got = [plan.volume(spec, k, sub) for k in ks for sub in (0, 3)]
    _same_hits(plan.collect(want_hits=True)[1:], want)
    for (v, r), (v0, r0) in zip(got, alone):
        assert r == r0 and np.array_equal(v.view(np.uint32), v0.view(np.uint32))
    plan.close()
    bank.close()


@pytest.mark.parametrize("graph,host", [(False, True), (True, False), (True, True)])
def test_volume_of_another_spectrum_leaves_a_staged_pass_alone(graph, host):
    """The pass reads its spectrum from the plan's own copy (host memory, or a plan
    that replays graphs); the volume is of another spectrum, and the pass is also
    run again from that copy (more hits than the buffer holds)."""
    torch = pytest.importorskip("torch")
    spec, plan, bank = _problem(torch, batch=4, max_hits=64, graph=graph)
    other = torch.flip(spec, (0,))
    if host:
        spec, other = spec.cpu().numpy(), other.cpu().numpy()
    ref_spec, ref, ref_bank = _problem(torch, batch=4)
    want = ref.search(ref_spec, 2, 39, want_hits=True)[1:]
    v0 = ref.volume(torch.flip(ref_spec, (0,)), 20, 1)
    plan.begin(spec, 2, 39)
    assert jerk.group_advance([plan], ahead=2) == 1
    v = plan.volume(other, 20, 1)
    assert v[1] == v0[1] and np.array_equal(v[0].view(np.uint32), v0[0].view(np.uint32))
    _same_hits(plan.collect(want_hits=True)[1:], want)
    assert len(want[0]) > 64
    for p in (plan, bank, ref, ref_bank):
        p.close()

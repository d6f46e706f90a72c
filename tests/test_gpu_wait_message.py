"""A bounded wait that gives up is reported as the step it belongs to."""

import pytest

from prestozl_b200 import jerk, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("probe,step", [(True, "correlation"), (2, "harmonic sum")])
def test_timed_out_copy_names_its_step(probe, step):
    spec, N, dt = synth.small_spectrum()
    obs, fftlen, _ = jerk.obs_from_params(len(spec), N, dt, 20, 60, 8, 2.0)
    subs = jerk.subharm_sizes(obs, fftlen)
    bank = jerk.DeviceBank(subs)
    plan = jerk.JerkPlan(obs, subs, batch=4, device_bank=bank.ptr.value)
    plan.set_wait_probe(probe)
    with pytest.raises(jerk.JerkError) as ei:
        plan.search(spec, 100, 4)
    assert ei.value.code == jerk.JERK_ECUDA
    assert str(ei.value).split(": ")[1].startswith(step) and "timed out" in str(ei.value)
    plan.set_wait_probe(False)
    plan.search(spec, 100, 4)
    plan.close()
    bank.close()

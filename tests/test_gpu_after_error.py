"""A CUDA error that a call has reported is not reported again by the next."""

import ctypes as C

import pytest

from prestozl_b200 import jerk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["realfft", "deredden", "downsample", "search"])
def test_calls_after_an_allocation_that_did_not_fit(call):
    torch = pytest.importorskip("torch")
    N = 1 << 18
    ts = torch.randn(N, device="cuda")
    spec = jerk.realfft(ts)
    obs, fftlen, _ = jerk.obs_from_params(N // 2, N, 64e-6, 20, 0, 4, 3.0)
    subs = jerk.subharm_sizes(obs, fftlen)
    bank = jerk.DeviceBank(subs)
    plan = jerk.JerkPlan(obs, subs, batch=4, device_bank=bank.ptr.value)
    p = C.c_void_p()
    assert jerk.lib().jerk_device_alloc(1 << 50, C.byref(p)) == jerk.JERK_ECUDA
    assert "out of memory" in jerk.lib().jerk_last_error().decode()
    if call == "realfft":
        jerk.realfft(ts)
    elif call == "deredden":
        jerk.deredden(spec)
    elif call == "downsample":
        jerk.downsample_subbands(ts.reshape(-1, 32), 2)
    else:
        plan.search(spec, 0, 4)
    torch.cuda.synchronize()
    plan.close()
    bank.close()

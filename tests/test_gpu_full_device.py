"""A plan made while there was room, used when the device has none left: what a
search still has to allocate takes the place of the plan's optional buffers, and
the hits are those of a device with room."""

import ctypes as C

import numpy as np
import pytest

from prestozl_b200 import jerk

pytestmark = pytest.mark.gpu


def _fill(torch, need, filled):
    """Takes device memory until less than `need` bytes are left."""
    size = torch.cuda.mem_get_info()[0]
    while size >= 1 << 20 and torch.cuda.mem_get_info()[0] >= need:
        p = C.c_void_p()
        if (torch.cuda.mem_get_info()[0] - size >= need // 4 and
                jerk.lib().jerk_device_alloc(size, C.byref(p)) == jerk.JERK_OK):
            filled.append(p)
        else:
            size //= 2
    assert torch.cuda.mem_get_info()[0] < need


@pytest.mark.parametrize("graph", [False, True])
def test_host_spectrum_is_staged_on_a_full_device(graph):
    torch = pytest.importorskip("torch")
    N, batch = 1 << 21, 256
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    spec = torch.view_as_complex(torch.randn((N // 2, 2), generator=g, device="cuda"))
    spec[40_000::3001] *= 12.0
    host = spec.cpu().numpy()
    obs, fftlen, _ = jerk.obs_from_params(N // 2, N, 64e-6, 20, 0, 16, 3.0)
    for i in range(obs.numharmstages):
        obs.powcut[i] = 11.0 + 3.0 * (1 << i) ** 0.75
    subs = jerk.subharm_sizes(obs, fftlen)
    bank = jerk.DeviceBank(subs)
    ref = jerk.JerkPlan(obs, subs, batch=batch, device_bank=bank.ptr.value)
    want = ref.search(spec, want_hits=True)[1:]  # (and every kernel is loaded)
    assert len(want[0]) > 0
    plan = jerk.JerkPlan(obs, subs, batch=batch, device_bank=bank.ptr.value, use_graph=graph)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    need = 8 * (N // 2)
    filled = []
    try:
        _fill(torch, need, filled)
        got = plan.search(host, want_hits=True)[1:]
    finally:
        for p in filled:
            jerk.lib().jerk_device_free(p)
    again = plan.search(host, want_hits=True)[1:]
    for h in (got, again):
        assert np.array_equal(h[0], want[0])
        assert np.array_equal(h[1].view(np.uint32), want[1].view(np.uint32))
    for p in (plan, ref, bank):
        p.close()

"""A plan made while there was room, used when the device has none left: what a
search still has to allocate takes the place of the plan's optional buffers, and
the hits are those of a device with room."""

import numpy as np
import pytest

from prestozl_b200 import jerk

pytestmark = pytest.mark.gpu


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
    need = 8 * (N // 2)
    # all but half a spectrum, a piece at a time
    filled, piece = [], torch.cuda.mem_get_info()[0] // 2
    while piece >= 1 << 20:
        if torch.cuda.mem_get_info()[0] - piece < need // 2:
            piece //= 2
            continue
        try:
            filled.append(torch.empty(piece, dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            piece //= 2
    try:
        assert torch.cuda.mem_get_info()[0] < need
        got = plan.search(host, want_hits=True)[1:]
    finally:
        del filled
        torch.cuda.empty_cache()
    again = plan.search(host, want_hits=True)[1:]
    for h in (got, again):
        assert np.array_equal(h[0], want[0])
        assert np.array_equal(h[1].view(np.uint32), want[1].view(np.uint32))
    for p in (plan, ref, bank):
        p.close()

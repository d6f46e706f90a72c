"""The whitening's scratch: one word per 6 bins, rounded to 256 bytes, as callers
that allocate it once have sized it, and nothing outside it is written."""

import numpy as np
import pytest

from oracle import bindings as ob
from prestozl_b200 import jerk
from tests import helpers as H

SIZES = [8, 18, 19, 35, 36, 200, 401, 5003, 70001, 1 << 20]


def _size(n):
    return (4 * (n // 6 + 2) + 255) // 256 * 256


def test_scratch_is_one_word_per_six_bins():
    for n in SIZES + [1 << 24, (1 << 31) - 1]:
        assert jerk.lib().jerk_deredden_scratch_bytes(n) == _size(n)


@pytest.mark.gpu
@pytest.mark.parametrize("n", SIZES)
def test_whitening_stays_inside_its_scratch(n):
    torch = pytest.importorskip("torch")
    H.ensure_oracle()
    a = np.random.default_rng(n).standard_normal((n, 2)).astype(np.float32)
    spec = np.ascontiguousarray(a).view(np.complex64)[:, 0]
    d = torch.from_numpy(spec.copy()).cuda()
    guard = 4096
    buf = torch.full((guard + _size(n) + guard,), 0x5a, dtype=torch.uint8, device="cuda")
    rc = jerk.lib().jerk_deredden(d.data_ptr(), n, buf.data_ptr() + guard, _size(n),
                                  torch.cuda.current_stream().cuda_stream or None)
    assert rc == jerk.JERK_OK
    torch.cuda.synchronize()
    assert bool((buf[:guard] == 0x5a).all()) and bool((buf[-guard:] == 0x5a).all())
    assert np.array_equal(d.cpu().numpy().view(np.uint32), ob.deredden(spec).view(np.uint32))

"""Dedispersion's tilings and window staging at their edges: subband counts
around the quads, pairs and chunks of 32 that are staged together, block
lengths around the tiles, offset tables whose rows lie together, apart and at
both ends, and blocks off 16-byte alignment.  Bar: bit-exact (the sums' order is
the oracle's)."""

import numpy as np
import pytest

from oracle import bindings as ob
from prestozl_b200 import build, jerk
from tests import helpers as H

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def built():
    build.build()
    H.ensure_oracle()


def _offsets(kind, numdms, nsub, worklen, rng):
    d, s = np.arange(numdms)[:, None], np.arange(nsub)[None, :]
    if kind == "together":
        off = (d * (nsub - 1 - s)) // 8
    elif kind == "steep":  # neighbouring rows further apart than a tile
        off = (nsub - 1 - s) * 300 + d
    elif kind == "jagged":  # every other row at the far end
        off = (s % 2) * worklen - (s % 2) * d
    else:
        off = rng.integers(0, worklen + 1, (numdms, nsub))
    return np.clip(off, 0, worklen).astype(np.int32)


@pytest.mark.parametrize("kind", ["together", "steep", "jagged", "random"])
@pytest.mark.parametrize("worklen,nsub,numdms,shift", [
    (255, 4, 3, 0), (513, 12, 65, 0), (1025, 33, 17, 0), (700, 31, 64, 0), (640, 36, 9, 1),
    (3000, 51, 40, 0), (2048, 100, 33, 0), (129, 7, 130, 3), (4097, 64, 70, 0), (64, 2, 1, 0)])
def test_tiles_and_staging_bit_exact(kind, worklen, nsub, numdms, shift):
    rng = np.random.default_rng(worklen + nsub)
    cur, last = (rng.standard_normal((2, worklen, nsub)) * 20 + 100).astype(np.float32)
    off = _offsets(kind, numdms, nsub, worklen, rng)

    def device(x):  # shift words off the allocation's alignment
        buf = torch.empty(x.size + shift, dtype=torch.float32, device="cuda")
        v = buf[shift:].view(worklen, nsub)
        v.copy_(torch.from_numpy(x))
        return v

    dd = jerk.Dedisperser(worklen, nsub, off)
    got = dd(device(cur), device(last)).cpu().numpy()
    dd.close()
    want = ob.dedisp_subbands(cur, last, off)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))

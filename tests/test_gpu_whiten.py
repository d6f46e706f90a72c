"""Whitening and zapping at the inputs where their selections can go wrong,
bit-exact against the oracle: medians of blocks with ties, zeros and powers
over many octaves; birdies that overlap or lie within each other's windows,
in any order, and more of them than one launch takes."""

import numpy as np
import pytest

from oracle import bindings as ob
from prestozl_b200 import jerk
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _spec(rng, kind, n):
    a = rng.standard_normal((n, 2))
    if kind == "ties":
        a = rng.integers(-2, 3, (n, 2)).astype(float)
        a[:, 0] += 4.0
    elif kind == "octaves":
        a *= 2.0 ** rng.integers(-30, 31, (n, 1))
    elif kind == "one value":
        a[:] = 3.0
    elif kind == "spikes":
        a[rng.integers(0, n, n // 9)] *= 1e6
    return (a[:, 0] + 1j * a[:, 1]).astype(np.complex64)


@pytest.mark.parametrize("kind", ["noise", "ties", "octaves", "one value", "spikes"])
@pytest.mark.parametrize("n", [8, 13, 14, 200, 5003, 70001])
def test_whitening_selects_the_same_medians(n, kind):
    torch = pytest.importorskip("torch")
    H.ensure_oracle()
    spec = _spec(np.random.default_rng(n), kind, n)
    d = torch.from_numpy(spec.copy()).cuda()
    jerk.deredden(d)
    assert np.array_equal(d.cpu().numpy().view(np.uint32), ob.deredden(spec).view(np.uint32))


@pytest.mark.parametrize("n,spread", [(1, 1.0), (40, 1.0), (300, 0.02), (150, 0.2), (280, 1.0)])
def test_zapping_keeps_the_list_order(n, spread):
    torch = pytest.importorskip("torch")
    H.ensure_oracle()
    bins = 1 << 17
    rng = np.random.default_rng(n)
    spec = _spec(rng, "noise", bins)
    lo = 500.0 + rng.uniform(0, spread * (bins - 2000), n)
    hi = lo + rng.uniform(0.5, 40.0, n)
    d = torch.from_numpy(spec.copy()).cuda()
    jerk.zap_birdies(d, 2 * bins, lo, hi)
    want = ob.zap_list(spec, 2 * bins, lo, hi)
    assert np.array_equal(d.cpu().numpy().view(np.uint32),
                          np.asarray(want, dtype=np.complex64).view(np.uint32))

"""The block median of the data preparation, through jerk_volume_static with
one all-ones kernel (a single tap): the even good bins are then the
normalised powers of the chunk."""

import numpy as np
import pytest

from prestozl_b200 import jerk

pytestmark = pytest.mark.gpu


def _chunk(rng, kind, M):
    if kind == "noise":
        a = rng.standard_normal((M, 2))
    elif kind == "spread":  # powers over forty octaves
        a = rng.standard_normal((M, 2)) * 2.0 ** rng.integers(-20, 21, (M, 1))
    elif kind == "ties":    # few distinct powers, many of them equal
        a = np.repeat(rng.integers(1, 5, (M, 1)).astype(float), 2, axis=1)
    else:                   # neighbours one float apart around the median
        base = np.float32(1.5).view(np.uint32)
        bits = base + rng.permutation(M).astype(np.uint32)
        a = np.stack([np.sqrt(bits.view(np.float32).astype(np.float64)), np.zeros(M)], axis=1)
    return (a[:, 0] + 1j * a[:, 1]).astype(np.complex64)


@pytest.mark.parametrize("kind", ["noise", "spread", "ties", "close"])
@pytest.mark.parametrize("fftlen", [128, 192, 768, 1280, 2048, 4096, 7680])
def test_block_median(fftlen, kind):
    torch = pytest.importorskip("torch")
    M, hw = fftlen // 2, 8
    rng = np.random.default_rng(fftlen + len(kind))
    spec = _chunk(rng, kind, M)
    uselen = fftlen - 4 * hw
    sp = torch.from_numpy(spec).cuda()
    kern = torch.ones(fftlen, dtype=torch.complex64, device="cuda")
    vol = torch.zeros(uselen, dtype=torch.float32, device="cuda")
    sub = dict(numharm=1, harmnum=1, numz=1, numw=1, fftlen=fftlen, halfwidth=hw)
    numrs, rlo = jerk.volume_static(sp.data_ptr(), M, 0, sub, kern.data_ptr(), float(hw), uselen,
                                    0.0, vol.data_ptr(),
                                    torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert (numrs, rlo) == (uselen, hw)
    # the powers as float32 operations, and the element a sort puts at (M-1)/2
    pw = spec.real * spec.real + spec.imag * spec.imag
    norm = np.float64(np.sort(pw)[(M - 1) // 2]) / np.log(2.0)
    want = pw[hw:hw + uselen // 2].astype(np.float64) / norm
    got = vol.cpu().numpy()[0::2].astype(np.float64)
    # FP32 transforms: rounding scales with the chunk's largest amplitude
    # (|y| error about 5e-7 of it, twice that times |y| in the power)
    amax = np.sqrt(pw.max() / norm)
    tol = 2 * 1e-6 * amax * np.sqrt(want) + (1e-6 * amax) ** 2 + 1e-6 * want
    assert np.all(np.abs(got - want) <= tol)

"""Plain passes of 64 and 128 points compute in FP32 with FP32 factors and
round to FP16 twice, once between the two phases and once at the end: their
error is that of these roundings and no more.  The same two phases in FP64
with the two roundings give it; FP32 rounding adds less than a thousandth of
it in energy and tips some roundings that are nearly ties, which leaves the
error as it is, so one in a hundred is allowed.  Factors rounded to FP16
inside a radix-16 step (errors up to 1.5e-4 of a product) add several."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)
pytestmark = pytest.mark.gpu

import mcfft_b200 as mc  # noqa: E402
from tests.gpu_util import rand_complex, rounded, run  # noqa: E402


def _f16(z):
    return z.real.astype(np.float16).astype(np.float64) + 1j * z.imag.astype(np.float16).astype(np.float64)


def _pass(x, r1, sign):
    """The last axis: r1-point DFTs, twiddles, r2-point DFTs; scaled by 1/r1
    and 1/r2, an FP16 rounding after each."""
    n = x.shape[-1]
    r2 = n // r1

    def dft(r):
        k = np.arange(r)
        return np.exp(sign * 2j * np.pi * np.outer(k, k) / r) / r

    a = x.reshape(x.shape[:-1] + (r1, r2))                    # n = n1 r2 + v
    a = np.einsum("kn,...nv->...kv", dft(r1), a)
    a = _f16(a * np.exp(sign * 2j * np.pi * np.outer(np.arange(r1), np.arange(r2)) / n))
    a = _f16(np.einsum("mv,...kv->...km", dft(r2), a))        # X[k1 + r1 k2]
    return np.swapaxes(a, -1, -2).reshape(x.shape)


@pytest.mark.parametrize("direction", [mc.FORWARD, mc.INVERSE])
@pytest.mark.parametrize("shape,batch", [((64,), 300), ((128,), 300), ((128,), 70000), ((64, 64), 3), ((128, 64), 5)])
def test_two_roundings_per_pass(shape, batch, direction, monkeypatch):
    monkeypatch.setenv("MCFFT_AUTOTUNE", "0")
    kinds = min(batch, 100)
    x = rand_complex((kinds,) + shape, seed=sum(shape))
    full = np.concatenate([x] * (batch // kinds))
    with mc.Plan(shape, full.shape[0]) as p:
        y, _ = run(p, full, True, direction=direction)
    y = y.reshape(full.shape)[:kinds]
    ref = _pass(rounded(x, True), 8, direction)               # rows: 8 x 8, 8 x 16
    if len(shape) == 2:                                       # columns: 8 x 8, 16 x 8
        ref = np.swapaxes(_pass(np.swapaxes(ref, 1, 2), 8 if shape[0] == 64 else 16, direction), 1, 2)
    axes = tuple(range(1, len(shape) + 1))
    z = rounded(x, True)
    exact = np.fft.fftn(z, axes=axes) / np.prod(shape) if direction == mc.FORWARD else np.fft.ifftn(z, axes=axes)
    got, allowed = np.linalg.norm(y - exact), np.linalg.norm(ref - exact)
    assert got < 1.01 * allowed, got / allowed

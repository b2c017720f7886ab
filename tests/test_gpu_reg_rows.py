"""Register passes: in-place execs of single-pass plans on every kernel that
serves them, transforms that hold infinities or NaNs beside others of the same
tile, and the inverse of the column passes."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)
pytestmark = pytest.mark.gpu

import mcfft_b200 as mc  # noqa: E402
from oracle import oracle  # noqa: E402
from tests.gpu_util import compare, rand_complex, rounded, run, to_device  # noqa: E402

FORMS = {"plain": (mc.PREC_FP16, 0, True, 1e-3), "split": (mc.PREC_SPLIT, 0, False, 2e-6),
         "split16": (mc.PREC_SPLIT, mc.FLAG_INPUT_F16, True, 2e-6)}


def _words(t):
    return t.view(torch.int32)


def _exec(plan, x, y, direction=mc.FORWARD):
    plan.exec_ptr(x.data_ptr(), y.data_ptr(), direction, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    plan.check_status()


@pytest.mark.parametrize("form,n,batch", [
    # without TMA; 4096-point tiles; full tiles
    ("plain", 64, 1), ("plain", 512, 9001), ("plain", 4096, 5), ("plain", 4096, 3001), ("plain", 256, 50001),
    ("plain", 2048, 9), ("split", 64, 1), ("split", 512, 3001), ("split", 512, 9001), ("split", 1024, 20001),
    ("split", 4096, 5), ("split", 4096, 1501)])
@pytest.mark.parametrize("direction", [mc.FORWARD, mc.INVERSE])
def test_in_place(form, n, batch, direction):
    prec, flags, f16, _ = FORMS[form]
    x = to_device(rand_complex((batch, n), seed=n + batch), f16)
    y = torch.empty_like(x)
    with mc.Plan((n,), batch, prec, flags) as p:
        assert p.info().num_passes == 1
        _exec(p, x, y, direction)
        _exec(p, x, x, direction)
    assert torch.equal(_words(x), _words(y))


@pytest.mark.parametrize("form,shape,batch", [
    (f, s, b) for f in FORMS for s, b in [((64,), 1000), ((512,), 37), ((1024,), 11000), ((4096,), 9),
                                          ((1 << 14,), 5), ((1 << 18,), 3), ((128, 64), 7), ((64, 64, 64), 3)]
] + [("plain", (2048,), 17)])
def test_one_transform_not_finite(form, shape, batch):
    """An infinity and a NaN in two transforms: theirs are not finite, every
    other transform is bit for bit what it is without them."""
    prec, flags, f16, _ = FORMS[form]
    n = int(np.prod(shape))
    x = rand_complex((batch, n), seed=batch)
    clean = to_device(x, f16)
    x[batch // 2, n // 3] = complex(np.inf, 0.0)
    x[batch - 1, n - 1] = complex(0.0, np.nan)
    bad = to_device(x, f16)
    odt = torch.complex64 if prec == mc.PREC_SPLIT else torch.complex32
    y0, y1 = (torch.empty(batch * n, dtype=odt, device="cuda") for _ in range(2))
    with mc.Plan(shape, batch, prec, flags) as p:
        _exec(p, clean, y0)
        _exec(p, bad, y1)
    w0, w1 = _words(y0).reshape(batch, -1), _words(y1).reshape(batch, -1)
    same = (w0 == w1).all(dim=1)
    expect = torch.ones(batch, dtype=torch.bool, device="cuda")
    expect[batch // 2] = expect[batch - 1] = False
    assert torch.equal(same, expect)
    for b in (batch // 2, batch - 1):
        assert not torch.isfinite(torch.view_as_real(y1.reshape(batch, n)[b]).float()).all()


def test_one_transform_not_finite_uneven():
    shapes = [(256,)] * 70 + [(512,)] * 33 + [(4096,)] * 5 + [(1 << 14,)] * 3 + [(128, 256)] * 2
    size = [int(np.prod(s)) for s in shapes]
    at = np.concatenate([[0], np.cumsum(size)])
    x = rand_complex((int(at[-1]),), seed=3)
    clean = to_device(x, True)
    hit = [5, 80, 104, 109, 111]
    for i in hit:
        x[at[i] + 1] = complex(np.nan, np.inf)
    bad = to_device(x, True)
    y0, y1 = torch.empty_like(clean), torch.empty_like(clean)
    with mc.Plan(descs=[(s, 1, int(a), int(a)) for s, a in zip(shapes, at)]) as p:
        assert p.info().launches == 1
        _exec(p, clean, y0)
        _exec(p, bad, y1)
    for i, s in enumerate(size):
        a, b = _words(y0)[at[i]:at[i] + s], _words(y1)[at[i]:at[i] + s]
        assert torch.equal(a, b) == (i not in hit), (i, shapes[i])


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("shape,batch", [((64, 32), 3), ((128, 16), 5), ((256, 32), 9), ((512, 16), 3),
                                         ((1024, 64), 15), ((64, 128, 32), 7), ((256, 64, 16), 11)])
def test_columns_inverse(shape, batch, form):
    prec, flags, f16, tol = FORMS[form]
    x = rand_complex((batch,) + shape, seed=batch)
    with mc.Plan(shape, batch, prec, flags) as p:
        y, sl = run(p, x, f16, direction=mc.INVERSE)
    ref = oracle.fftnd(rounded(x, f16), list(shape), sign=+1) * 2.0 ** sl
    assert compare(y, ref)[0] < tol

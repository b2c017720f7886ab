"""Register pass kernels on the GPU: every length they hold in each form and
direction, with enough tiles that every CTA reuses its buffers many times
(both groups of the split form), a ragged last tile, passes with fewer columns
than a tile, and four-step pairs over many transforms.  A sample of the
transforms is compared with the FP64 oracle; bounds as in test_gpu_parity."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)
pytestmark = pytest.mark.gpu

import mcfft_b200 as mc  # noqa: E402
from oracle import oracle  # noqa: E402
from tests.gpu_util import compare, from_device, rounded, to_device  # noqa: E402

FORMS = {"plain": (mc.PREC_FP16, 0, True, 1e-3), "split": (mc.PREC_SPLIT, 0, False, 2e-6),
         "split16": (mc.PREC_SPLIT, mc.FLAG_INPUT_F16, True, 2e-6)}


def _check(shape, batch, form, direction):
    prec, flags, f16, tol = FORMS[form]
    n = int(np.prod(shape))
    rng = np.random.default_rng(n + batch)
    # a few distinct transforms, repeated over the batch
    kinds = min(batch, 5)
    x = rng.uniform(-1, 1, (kinds, n)) + 1j * rng.uniform(-1, 1, (kinds, n))
    xd = to_device(x, f16).reshape(kinds, n)
    pick = torch.arange(batch, device="cuda") % kinds
    if f16:
        xs = torch.view_as_real(xd)[pick].contiguous()
        xs = torch.view_as_complex(xs)
    else:
        xs = xd[pick].contiguous()
    odt = torch.complex64 if prec == mc.PREC_SPLIT else torch.complex32
    out = torch.empty(batch * n, dtype=odt, device="cuda")
    out.view(torch.uint8).fill_(0xFF)
    with mc.Plan(shape, batch, prec, flags) as p:
        p.exec_ptr(xs.data_ptr(), out.data_ptr(), direction, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        p.check_status()
        scale = 2.0 ** p.info().scale_log2
    # every transform equals the first one of its kind, bit for bit
    words = out.view(torch.int32).reshape(batch, -1)
    for k in range(kinds):
        same = (words[k::kinds] == words[k]).all()
        assert bool(same), f"transforms of one input differ (kind {k})"
    xr = rounded(x, f16).reshape((kinds,) + tuple(shape))
    if direction == mc.FORWARD:
        ref = oracle.fftnd(xr, list(shape)) * scale
    else:
        ref = np.conj(oracle.fftnd(np.conj(xr), list(shape))) * scale
    y = from_device(out[:kinds * n])
    rel, mx = compare(y, ref)
    assert rel < tol, (rel, mx)


@pytest.mark.parametrize("direction", [mc.FORWARD, mc.INVERSE])
@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("n", [64, 128, 256, 512, 1024])
def test_rows(n, form, direction):
    _check((n,), (10 << 20) // n + 3, form, direction)


@pytest.mark.parametrize("direction", [mc.FORWARD, mc.INVERSE])
@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("n,batch", [(64, 1), (64, 40001), (128, 70), (256, 17), (256, 12345), (512, 9001),
                                     (1024, 3), (1024, 2000), (4096, 1), (4096, 5), (4096, 1501)])
def test_few_rows(n, batch, form, direction):
    """4096-point tiles: from one transform up to several tiles per CTA."""
    _check((n,), batch, form, direction)


@pytest.mark.parametrize("direction", [mc.FORWARD, mc.INVERSE])
@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("n,batch", [(1 << 14, 301), (1 << 17, 61), (1 << 18, 30), (1 << 20, 9)])
def test_four_step(n, batch, form, direction):
    _check((n,), batch, form, direction)


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("shape,batch", [((64, 32), 3), ((128, 16), 5), ((256, 32), 9), ((512, 16), 3),
                                         ((1024, 64), 150), ((64, 128, 32), 7), ((256, 64, 16), 11)])
def test_columns(shape, batch, form):
    _check(shape, batch, form, mc.FORWARD)


@pytest.mark.parametrize("direction", [mc.FORWARD, mc.INVERSE])
@pytest.mark.parametrize("shape,batch", [((2048,), 1), ((2048,), 8), ((2048,), 5001), ((64, 2048), 9),
                                         ((2048, 128), 5)])
def test_rows_2048(shape, batch, direction):
    _check(shape, batch, "plain", direction)


# every variant of the one-launch kernel: 1D lengths of one pass and of two,
# 2D and 3D shapes; counts that leave ragged tiles
UNEVEN = [((64,), 1), ((128,), 300), ((256,), 67), ((512,), 33), ((1024,), 17), ((2048,), 9), ((4096,), 5),
          ((1 << 13,), 3), ((1 << 14,), 3), ((1 << 15,), 2), ((1 << 17,), 2), ((1 << 18,), 1), ((1 << 20,), 1),
          ((1 << 19,), 1), ((64, 2048), 3), ((64, 64), 3), ((128, 1024), 2), ((512, 256), 2), ((1024, 512), 1), ((64, 64, 128), 1)]


def _uneven(shapes, order, direction, execs=3):
    """One descriptor per transform; inputs packed in the given order, outputs
    in the opposite one.  Returns the results transform by transform."""
    items = [s for s, c in shapes for _ in range(c)]
    rng = np.random.default_rng(11)
    if order == "mixed":
        rng.shuffle(items)
    size = [int(np.prod(s)) for s in items]
    io = np.concatenate([[0], np.cumsum(size)])
    oo = [int(io[-1] - e) for e in io[1:]] if order == "mixed" else io[:-1]
    descs = [(s, 1, int(a), int(b)) for s, a, b in zip(items, io, oo)]
    total = int(io[-1])
    x = rng.uniform(-1, 1, total) + 1j * rng.uniform(-1, 1, total)
    xd = to_device(x, True)
    out = torch.empty(total, dtype=torch.complex32, device="cuda")
    with mc.Plan(descs=descs, precision=mc.PREC_FP16) as p:
        if order == "packed" or min(size) >= 256:
            assert p.info().launches == 1
        for _ in range(execs):  # the counters of one exec are the next one's
            out.view(torch.uint8).fill_(0xFF)
            p.exec_ptr(xd.data_ptr(), out.data_ptr(), direction, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        p.check_status()
    return descs, rounded(x, True), from_device(out)


@pytest.mark.parametrize("direction", [mc.FORWARD, mc.INVERSE])
@pytest.mark.parametrize("order", ["packed", "mixed"])
@pytest.mark.parametrize("shapes", [UNEVEN, [s for s in UNEVEN if s[0] not in ((64,), (128,), (64, 64))],
                                    [((256,), 65), ((512,), 1)]])
def test_uneven_one_launch(shapes, order, direction):
    """Against the oracle: the packed batch, transforms at unrelated offsets
    (with 64 or 128 points among them: other kernels), and a batch whose
    tables all stay in shared memory."""
    descs, xr, y = _uneven(shapes, order, direction)
    worst = 0.0
    for shape, _, io, oo in descs:
        n = int(np.prod(shape))
        v = xr[io:io + n].reshape((1,) + tuple(shape))
        ref = oracle.fftnd(v, list(shape)) if direction == mc.FORWARD else \
            np.conj(oracle.fftnd(np.conj(v), list(shape)))
        rel, _ = compare(y[oo:oo + n], ref / n)
        worst = max(worst, rel)
    assert worst < 1e-3, worst

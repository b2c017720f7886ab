"""Which kernels a plan runs: switches and rules that choose between kernel
families, seen in the plan's information rather than in its results."""
import math

import pytest

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)
pytestmark = pytest.mark.gpu

import mcfft_b200 as mc  # noqa: E402
from oracle import oracle  # noqa: E402
from tests.gpu_util import compare, rand_complex, rounded, run  # noqa: E402

PLAIN_TOL, SPLIT_TOL = 1e-3, 2e-6


@pytest.mark.parametrize("points", [8192, 16384])
@pytest.mark.parametrize("shape,batch", [((32,), 512), ((64,), 256), ((128,), 128), ((256,), 67),
                                         ((512,), 32), ((1024,), 16), ((2048,), 8), ((2048,), 5),
                                         ((4096,), 8), ((4096,), 3), ((1 << 20,), 1),
                                         ((512, 512), 1), ((64, 64, 64), 1)])
def test_tile_points_switch(shape, batch, points, monkeypatch):
    """MCFFT_TILE_POINTS names the tile size of every pass that has a layout
    for it; with 8192 plain passes run on the 8K-point tiles, which the
    plan-time tuner may choose on its own."""
    monkeypatch.setenv("MCFFT_TILE_POINTS", str(points))
    monkeypatch.setenv("MCFFT_AUTOTUNE", "0")
    x = rand_complex((batch,) + shape, seed=batch)
    with mc.Plan(shape, batch, mc.PREC_FP16) as p:
        # 32-point rows have an 8K layout only
        assert p.info().tile_points == (8192 if shape == (32,) else points)
        y, sl = run(p, x, True)
    ref = oracle.fftnd(rounded(x, True), shape) * 2.0 ** sl
    assert compare(y, ref)[0] < PLAIN_TOL


@pytest.mark.parametrize("n,batch", [(256, 67), (4096, 5)])
def test_tile_points_switch_split(n, batch, monkeypatch):
    monkeypatch.setenv("MCFFT_TILE_POINTS", "8192")
    x = rand_complex((batch, n), seed=batch)
    with mc.Plan((n,), batch, mc.PREC_SPLIT) as p:
        assert p.info().tile_points == 8192
        y, _ = run(p, x, False)
    assert compare(y, oracle.fft1d(rounded(x, False)))[0] < SPLIT_TOL


def _route(capfd, monkeypatch, make):
    """The plan's line and its passes' lines as MCFFT_DEBUG_PLAN prints them."""
    monkeypatch.setenv("MCFFT_DEBUG_PLAN", "1")
    capfd.readouterr()
    with make():
        pass
    lines = capfd.readouterr().err.splitlines()
    plan = [ln for ln in lines if ln.startswith("[mcfft] plan: ")]
    passes = [ln.split(": ", 1)[1] for ln in lines if ln.startswith("[mcfft] pass ")]
    assert len(plan) == 1, lines
    return plan[0].split("passes, ", 1)[1], passes


@pytest.mark.parametrize("shape,batch,prec,expect", [
    # few rows: 4096-point tiles without TMA; more: with TMA; many: full tiles
    ((1024,), 8, mc.PREC_FP16, ["L=1024, register, 4096-point tiles, no TMA"]),
    ((4096,), 256, mc.PREC_FP16, ["L=4096, register, 4096-point tiles, no TMA"]),
    ((4096,), 4000, mc.PREC_FP16, ["L=4096, register, 4096-point tiles"]),
    ((1024,), 16384, mc.PREC_FP16, ["L=1024, register, 16384-point tiles"]),
    ((64,), 3, mc.PREC_SPLIT, ["L=64, register, 4096-point tiles, no TMA"]),
    ((4096,), 1000, mc.PREC_SPLIT, ["L=4096, register, 4096-point tiles"]),
    ((1024,), 16384, mc.PREC_SPLIT, ["L=1024, register, 8192-point tiles"]),
    ((2048,), 5001, mc.PREC_FP16, ["L=2048, register, 16384-point tiles"]),
    ((1024, 1024), 16, mc.PREC_FP16, ["L=1024, register, 16384-point tiles"] * 2),
    ((1 << 18,), 30, mc.PREC_SPLIT, ["L=512, register, 8192-point tiles"] * 2),
    # lengths without a register routine
    ((32,), 512, mc.PREC_FP16, ["L=32, tcgen05, 8192-point tiles"]),
    ((8192,), 8, mc.PREC_FP16, ["L=8192, tcgen05, 16384-point tiles"]),
    ((2048,), 8, mc.PREC_SPLIT, ["L=2048, tcgen05, 8192-point tiles"])])
def test_pass_kernels(shape, batch, prec, expect, capfd, monkeypatch):
    monkeypatch.setenv("MCFFT_AUTOTUNE", "0")
    how, passes = _route(capfd, monkeypatch, lambda: mc.Plan(shape, batch, prec))
    assert how == "pass by pass"
    assert passes == expect


def _descs(shapes, mixed):
    """One descriptor per transform, back to back; mixed: outputs in the
    opposite order."""
    items = [s for s, c in shapes for _ in range(c)]
    size = [math.prod(s) for s in items]
    total, at, descs = sum(size), 0, []
    for s, n in zip(items, size):
        descs.append((s, 1, at, total - at - n if mixed else at))
        at += n
    return descs


ALL = [((64,), 1), ((128,), 300), ((256,), 67), ((512,), 33), ((1024,), 17), ((2048,), 9), ((4096,), 5),
       ((1 << 13,), 3), ((1 << 14,), 3), ((1 << 15,), 2), ((1 << 17,), 2), ((1 << 18,), 1), ((1 << 20,), 1),
       ((1 << 19,), 1), ((64, 2048), 3), ((64, 64), 3), ((128, 1024), 2), ((512, 256), 2), ((1024, 512), 1),
       ((64, 64, 128), 1)]
LONG = [s for s in ALL if s[0] not in ((64,), (128,), (64, 64))]


@pytest.mark.parametrize("shapes,mixed,prec,expect", [
    (ALL, False, mc.PREC_FP16, "register passes, tables reloaded"),
    (LONG, False, mc.PREC_FP16, "register passes, tables reloaded"),
    (LONG, True, mc.PREC_FP16, "register passes, tables reloaded"),
    ([((256,), 65), ((512,), 1)], False, mc.PREC_FP16, "register passes, tables resident"),
    ([((256,), 65), ((512,), 1)], True, mc.PREC_FP16, "register passes, tables resident"),
    # the batch of the timeout test
    ([((256,), 3), ((4096,), 2), ((1 << 16,), 1), ((128, 256), 1)], False, mc.PREC_FP16,
     "register passes, tables reloaded"),
    # no routine: 1D lengths of 64 and 128 points at unrelated offsets, a side
    # of 32, rows of 2048 as a second pass, the split form
    ([((128,), 3), ((256,), 3)], True, mc.PREC_FP16, "batch kernel"),
    ([((256,), 3), ((32, 256), 1)], False, mc.PREC_FP16, "batch kernel"),
    ([((256,), 3), ((1 << 21,), 1)], False, mc.PREC_FP16, "batch kernel"),
    ([((256,), 3), ((512,), 1)], False, mc.PREC_SPLIT, "batch kernel")])
def test_uneven_kernels(shapes, mixed, prec, expect, capfd, monkeypatch):
    """The lists of the uneven parity tests among them, which cannot tell the
    two one-launch kernels apart."""
    monkeypatch.setenv("MCFFT_AUTOTUNE", "0")
    how, passes = _route(capfd, monkeypatch, lambda: mc.Plan(descs=_descs(shapes, mixed), precision=prec))
    assert how == "one launch, " + expect
    family = "register" if "register" in expect else "tcgen05"
    assert all(family in p for p in passes), passes


@pytest.mark.parametrize("make", [
    lambda: mc.Plan((1024,), 8),
    lambda: mc.Plan((256, 256), 3),
    lambda: mc.Plan((1024,), 8, mc.PREC_SPLIT),
    lambda: mc.Plan(descs=_descs([((256,), 3), ((512,), 2)], False)),
    lambda: mc.Plan(descs=_descs([((128,), 3), ((256,), 3)], True)),
    lambda: mc.Plan(descs=_descs([((256,), 3), ((32, 256), 1)], False)),
    lambda: mc.Plan(descs=_descs([((256,), 3), ((1 << 21,), 1)], False)),
    lambda: mc.Plan(descs=_descs([((64, 64, 64 << i), 1) for i in range(7)]
                                 + [((64, 128, 64 << i), 1) for i in range(7)]
                                 + [((64 << i, 64), 1) for i in range(5)], False))],
    ids=["1d", "2d", "split", "uneven", "uneven_mixed_128", "uneven_side_32", "uneven_2p21", "uneven_52_passes"])
def test_plan_built_once(make, capfd, monkeypatch):
    """The choice between the one-launch kernels is made before anything is
    built."""
    monkeypatch.setenv("MCFFT_AUTOTUNE", "0")
    monkeypatch.setenv("MCFFT_DEBUG_PLAN", "1")
    capfd.readouterr()
    with make():
        pass
    assert capfd.readouterr().err.count("[mcfft] begin plan") == 1


@pytest.fixture
def no_records():
    mc.wisdom_forget()
    yield
    mc.wisdom_forget()


@pytest.mark.parametrize("shape,batch", [((1024, 1024), 16), ((1 << 20,), 4)])
def test_records_of_other_kernels(shape, batch, no_records):
    """The passes of a plan bound for the batch kernel (a side of 32) are
    tcgen05 tiles; what its tuner records says nothing about a plan of the
    same passes on register kernels, which is tuned by itself."""
    with mc.Plan(shape, batch) as p:
        alone = p.info().timed_passes
    mc.wisdom_forget()
    n = math.prod(shape) * batch
    with mc.Plan(descs=[(shape, batch, 0, 0), ((32, 256), 1, n, n)]) as p:
        assert p.info().timed_passes > 0
    with mc.Plan(shape, batch) as p:
        assert p.info().timed_passes == alone > 0
    with mc.Plan(shape, batch) as p:
        assert p.info().timed_passes == 0


def test_records_of_older_kernels(no_records, tmp_path, capfd, monkeypatch):
    """Records written before they named the kernels: read, but no plan
    follows them (here they ask for 8K-point tiles and another split)."""
    path = tmp_path / "w.txt"
    with mc.Plan((1 << 20,), 64) as p:
        alone = p.info().timed_passes
    mc.wisdom_export(str(path))
    old = []
    for ln in path.read_text().splitlines()[1:]:
        name, sms, key, _ = ln.split("\t")
        old.append("\t".join([name, sms, key.split(" g")[0], "9" if key.startswith("fourstep") else "8192"]))
    assert len(old) >= 3
    path.write_text("\n".join(["mcfft-wisdom 1"] + old) + "\n")
    mc.wisdom_forget()
    mc.wisdom_import(str(path))
    monkeypatch.setenv("MCFFT_DEBUG_PLAN", "1")
    with mc.Plan((1 << 20,), 64) as p:
        assert p.info().timed_passes == alone
    assert "pass 0: L=1024, register, 16384-point tiles" in capfd.readouterr().err
    mc.wisdom_export(str(path))  # kept beside the new ones
    assert set(old) <= set(path.read_text().splitlines())

"""Which kernels a plan runs: switches and rules that choose between kernel
families, seen in the plan's information rather than in its results."""
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

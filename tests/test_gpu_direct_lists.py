"""Direct lists (Rasterizer::draw*List): skipped primitives compacted in order by the counting
launch's last block -- around the 1,024 primitives of a block, many blocks, all or none
skipped -- against the oracle; a primitive queue the caller made too small is reported."""
import numpy as np
import pytest

from softwarerenderer_gb300 import scenes
from softwarerenderer_gb300.abi import DrawMode, PS, RASTER_VERTEX_FLOATS, RasterMode, VS

from .parity import describe, diff, oracle_render

pytestmark = pytest.mark.gpu


def _scene(n, mode, skip, seed=0):
    rng = np.random.default_rng([n, int(mode), seed])
    per = {DrawMode.Point: 1, DrawMode.Line: 2, DrawMode.Triangle: 3}[mode]
    nv = max(4, n * per // 2)
    w, h = 71, 53
    rv = np.zeros((nv, RASTER_VERTEX_FLOATS), np.float32)
    rv[:, 0:2] = rng.random((nv, 2)) * np.array([w, h])
    rv[:, 2] = rng.integers(0, 16, nv) / 16.0
    rv[:, 3] = 0.5 + rng.random(nv)
    rv[:, 20:23] = rng.random((nv, 3))
    idx = rng.integers(0, nv, (n, per)).astype(np.int32)
    if mode != DrawMode.Point:  # short primitives: neighbours of the first vertex
        idx[:, 1:] = (idx[:, :1] + rng.integers(1, 4, (n, per - 1))) % nv
    idx[rng.random(n) < skip, 0] = -1
    return scenes.Scene(name=f"list{n}", vs=VS.POS_RGB, ps=PS.VCOLOR, width=w, height=h, draw_mode=mode,
                        raster=RasterMode.Block, scissor=(0, 0, w, h), indices=idx.reshape(-1), raster_vertices=rv)


@pytest.mark.parametrize("mode", [DrawMode.Point, DrawMode.Line, DrawMode.Triangle])
@pytest.mark.parametrize("n", [1, 4, 1023, 1024, 1025, 3000])
@pytest.mark.parametrize("skip", [0.0, 0.4, 1.0])
def test_skips_keep_order(gpu_lib, port, mode, n, skip):
    from softwarerenderer_gb300.device import DeviceScene, DeviceTarget
    sc = _scene(n, mode, skip)
    ref, rst = oracle_render(port, sc)
    ds = DeviceScene(sc)
    for _ in range(2):  # the block counter is ready again
        tg = DeviceTarget(sc)
        st = ds.draw(tg)
        got = tg.to_host()
        assert not diff(ref, got), [describe(ref, got, k) for k in diff(ref, got)]
        assert st["fragments"] == rst["fragments"]


def test_many_blocks(gpu_lib, port):
    from softwarerenderer_gb300.device import DeviceScene, DeviceTarget
    sc = _scene(1_400_000, DrawMode.Point, 0.5)  # more blocks than the launch has CTAs
    ref, _ = oracle_render(port, sc)
    tg = DeviceTarget(sc)
    DeviceScene(sc).draw(tg)
    got = tg.to_host()
    assert not diff(ref, got), [describe(ref, got, k) for k in diff(ref, got)]


def test_undersized_primitive_queue_is_reported(gpu_lib, port):
    from softwarerenderer_gb300 import _lib
    from softwarerenderer_gb300.device import DeviceScene, DeviceTarget
    sc = _scene(3000, DrawMode.Triangle, 0.1)
    ds = DeviceScene(sc)
    ds.rast.ctx.set_queue_capacity(50, 0)
    tg = DeviceTarget(sc)
    before = tg.to_host()
    ds.draw(tg, sync=False)
    rc, st = ds.rast.ctx.finish()
    assert rc == _lib.SWR_EOVERFLOW and st["fragments"] == 0
    assert not diff(before, tg.to_host())
    ds.draw(tg)
    assert not diff(oracle_render(port, sc)[0], tg.to_host())

"""Queues of more than 32M ids, whose segments' id ranges do not fit the sort's bitmap: cells gone
through in windows of it (one and several, dense and sparse) or ranked, lines and triangles, bit
for bit against the oracle."""
import numpy as np
import pytest

from softwarerenderer_gb300 import scenes
from softwarerenderer_gb300.abi import DrawMode, PS, RASTER_VERTEX_FLOATS, VS

from .parity import diff, oracle_render

pytestmark = pytest.mark.gpu


def _check(port, sc, primitives=0, bin_entries=0):
    from softwarerenderer_gb300.device import DeviceScene, DeviceTarget
    ds, tg = DeviceScene(sc), DeviceTarget(sc)
    ds.rast.ctx.set_queue_capacity(primitives, bin_entries)
    st = ds.draw(tg)
    ref, rst = oracle_render(port, sc)
    assert not diff(ref, tg.to_host()) and st["fragments"] == rst["fragments"]


def _lines(n, width, height, length, seed):
    rng = np.random.default_rng(seed)
    rv = np.zeros((2 * n, RASTER_VERTEX_FLOATS), np.float32)
    rv[0::2, 0:2] = rng.random((n, 2)) * [width, height]
    rv[1::2, 0:2] = rv[0::2, 0:2] + (rng.random((n, 2)) - 0.5) * 2 * length
    rv[:, 2] = rng.integers(0, 64, 2 * n) / 64.0
    rv[:, 3] = 0.5 + rng.random(2 * n)
    rv[:, 20:23] = rng.random((2 * n, 3))
    return scenes.Scene(name="lines", vs=VS.POS_RGB, ps=PS.VCOLOR, width=width, height=height,
                        draw_mode=DrawMode.Line, scissor=(0, 0, width, height),
                        indices=np.arange(2 * n, dtype=np.int32), raster_vertices=rv)


@pytest.mark.parametrize("queue", [(1 << 25) - 5, (1 << 25) + 1, 1 << 26])  # both sides of the fit
@pytest.mark.parametrize("n,width,height,length", [
    (45000, 16, 16, 12),     # one tile: 300,000 fragments in a cell, windows of 131,072 ids
    (60000, 640, 360, 40),   # 1M fragments over 920 tiles: hundreds to thousands of ids a cell
    (20000, 640, 360, 8),    # some 90 ids over 90,000: below the chunk, left to the raster
    (26000, 640, 360, 40),   # around the line between ranks and windows
])
def test_lines(gpu_lib, port, queue, n, width, height, length):
    _check(port, _lines(n, width, height, length, n), bin_entries=queue)


@pytest.mark.parametrize("queue", [(1 << 25) - 5, (1 << 25) + 1])
@pytest.mark.parametrize("n", [600, 5000, 200000])
def test_triangles(gpu_lib, port, queue, n):
    _check(port, scenes.stack_scene(4, n), primitives=queue)

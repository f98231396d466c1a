"""Draws of up to 1,024 triangles at the edges of the box windows: tiles that none, one or all of
several windows' boxes hit, the overwriting shaders' list of the primitives that do (from 128 on)
and its rows, against the oracle and the general path."""
import dataclasses

import pytest

from softwarerenderer_gb300 import scenes
from softwarerenderer_gb300.abi import PS, RasterMode, VS

from .parity import describe, diff, oracle_render

pytestmark = pytest.mark.gpu


def _check(port, sc, graph=False):
    from softwarerenderer_gb300.device import DeviceScene, DeviceTarget
    ref, rst = oracle_render(port, sc)
    stats = []
    for general in (False, True):
        ds, tg = DeviceScene(sc), DeviceTarget(sc)
        if general:
            ds.rast.ctx.set_queue_capacity(0, 1 << 22)
            ds.rast.ctx.set_tile_slicing(0)
        ds.rast.ctx.set_graph_mode(graph)
        st = ds.draw(tg)
        got = tg.to_host()
        assert not diff(ref, got), [describe(ref, got, k) for k in diff(ref, got)]
        stats.append([st[k] for k in ("fragments", "primitives", "bin_pairs", "flags", "passes")])
    assert stats[0] == stats[1] and stats[0][0] == rst["fragments"]


@pytest.mark.parametrize("raster", [RasterMode.Span, RasterMode.Block, RasterMode.Adaptive])
@pytest.mark.parametrize("ps", [PS.VCOLOR, PS.VCOLOR_AFFINE])
@pytest.mark.parametrize("n", [127, 128, 129, 256, 257, 769, 1024])
@pytest.mark.parametrize("width,height", [(48, 40), (700, 500), (3000, 60)])
def test_windows(gpu_lib, port, raster, ps, n, width, height):
    sc = scenes.stack_scene(n, n, ps=ps, raster=raster, width=width, height=height)
    if ps == PS.VCOLOR_AFFINE:
        sc = dataclasses.replace(sc, vs=VS.POS_RGB_AFFINE)
    _check(port, sc)


@pytest.mark.parametrize("ps", [PS.VCOLOR, PS.VCOLOR_AFFINE])
@pytest.mark.parametrize("first", [0, 255, 256, 1023])
def test_one_tile_of_many(gpu_lib, port, ps, first):
    """A thousand triangles in one corner and one elsewhere, in a window of its own."""
    sc = scenes.stack_scene(6, 1024, ps=ps, width=48, height=40)
    pos = sc.attribs[0][0]
    pos[:, 0:2] = (pos[:, 0:2] + 1.0) * 0.05 - 1.0
    pos[3 * first:3 * first + 3, 0:2] = [(0.5, 0.5), (0.9, 0.6), (0.6, 0.9)]
    sc = dataclasses.replace(sc, width=1000, height=600, viewport=(0, 0, 1000, 600), scissor=(0, 0, 1000, 600),
                             vs=VS.POS_RGB_AFFINE if ps == PS.VCOLOR_AFFINE else sc.vs)
    _check(port, sc)


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("n", [511, 512, 513, 1024])  # one and two half batches of geometry
def test_clipped_half_batches(gpu_lib, port, graph, n):
    sc = scenes.soup_scene(n, width=300, height=200, seed=n)
    _check(port, sc, graph)

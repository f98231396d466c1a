"""Overwriting shaders in Block and Adaptive mode: tiles of up to 32 primitives (coverage masks, each
pixel's largest id) and of more (rows and blocks scattered), at the lines between them, partial tiles
at the target's edges, 16- and 32-pixel tiles, slices of a few primitives, Span and Block draws
into one target, and targets of so many tiles that none is sliced; against the oracle."""
import dataclasses

import pytest

from softwarerenderer_gb300 import scenes
from softwarerenderer_gb300.abi import PS, RasterMode, VS

from .parity import describe, diff, oracle_render

pytestmark = pytest.mark.gpu

MODES = [RasterMode.Block, RasterMode.Adaptive, RasterMode.Span]


def _scene(seed, n, raster, width, height):
    sc = scenes.stack_scene(seed, n, ps=PS.VCOLOR_AFFINE, raster=raster, width=width, height=height)
    return dataclasses.replace(sc, vs=VS.POS_RGB_AFFINE)


def _check(port, sc, tile=16):
    from softwarerenderer_gb300.device import DeviceScene, DeviceTarget
    ref, rst = oracle_render(port, sc)
    ds, tg = DeviceScene(sc, tile=tile), DeviceTarget(sc)
    ds.rast.ctx.set_queue_capacity(0, 1 << 20)  # (bins, for few triangles too)
    for _ in range(2):
        tg.clear()
        st = ds.draw(tg)
        got = tg.to_host()
        assert not diff(ref, got), [describe(ref, got, k) for k in diff(ref, got)]
        assert st["fragments"] == rst["fragments"] == st["passes"]


@pytest.mark.parametrize("tile", [16, 32])
@pytest.mark.parametrize("raster", MODES)
@pytest.mark.parametrize("n", [1, 15, 16, 31, 32, 33, 127, 128, 129])
@pytest.mark.parametrize("width,height", [(16, 16), (13, 21), (150, 70)])
def test_entries_of_a_tile(gpu_lib, port, tile, raster, n, width, height):
    _check(port, _scene(n, n, raster, width, height), tile)


@pytest.mark.parametrize("tile", [16, 32])
@pytest.mark.parametrize("raster", MODES)
@pytest.mark.parametrize("n", [513, 600, 1023, 1025])  # one tile in 32 slices of 16 to 33
def test_slices_of_a_few(gpu_lib, port, tile, raster, n):
    _check(port, _scene(n, n, raster, 16, 16), tile)


@pytest.mark.parametrize("raster", MODES)
@pytest.mark.parametrize("width,height,n", [(640, 976, 3000), (641, 976, 3000), (1300, 1000, 40000), (400, 300, 40000)])
def test_many_tiles(gpu_lib, port, raster, width, height, n):
    """2,440 tiles and more are rasterized whole (2,432 is the line), fewer in slices."""
    _check(port, _scene(7, n, raster, width, height))


@pytest.mark.parametrize("n", [10, 40, 900])
def test_modes_in_one_target(gpu_lib, port, n):
    """Span, Block and Adaptive draws of one batch into the same target."""
    from softwarerenderer_gb300.batch import BatchRenderer
    from softwarerenderer_gb300.device import DeviceTarget
    scs = [_scene(k, n, MODES[k % 3], 60, 44) for k in range(4)]
    ref = scenes.Target(scs[0])
    for sc in scs:
        port.draw(sc, ref)
    tg = DeviceTarget(scs[0])
    br = BatchRenderer(scs, targets=[tg] * len(scs))
    br.clear()
    br.draw()
    assert not diff(ref.arrays(), tg.to_host())

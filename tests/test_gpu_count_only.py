"""Primitives that cannot show behind depths already written are only counted (shaders with
the depth cull): dense piles and soups in every raster mode and tile size, from a far and a
near clear depth, with and without per-pixel counts, whole tiles and heavy-tile runs, against
the oracle; the statistics do not depend on whether the target records counts."""
import pytest

from softwarerenderer_gb300 import scenes
from softwarerenderer_gb300.abi import PS, RasterMode

from .parity import describe, diff

pytestmark = pytest.mark.gpu


def _check(port, sc, tile, clear_depth, slicing=-1):
    from softwarerenderer_gb300.device import DeviceScene, DeviceTarget
    t = scenes.Target(sc, clear_depth=clear_depth)
    rst = port.draw(sc, t)
    ref = t.arrays()
    passes = set()
    for aux in (True, False):
        ds = DeviceScene(sc, tile=tile)
        if slicing != -1:
            ds.rast.ctx.set_tile_slicing(slicing)
        tg = DeviceTarget(sc, aux=aux, clear_depth=clear_depth)
        st = ds.draw(tg)
        got = tg.to_host()
        want = {k: ref[k] for k in got}
        assert not diff(want, got), (aux, [describe(want, got, k) for k in diff(want, got)])
        assert st["fragments"] == rst["fragments"]
        passes.add(st["passes"])
    assert len(passes) == 1


@pytest.mark.parametrize("raster", [RasterMode.Span, RasterMode.Block, RasterMode.Adaptive])
@pytest.mark.parametrize("tile", [8, 16, 32])
@pytest.mark.parametrize("clear_depth", [float("inf"), 0.6])
def test_piles(gpu_lib, port, raster, tile, clear_depth):
    for n, w, h in ((2400, 48, 40), (6000, 61, 37)):
        _check(port, scenes.stack_scene(n, n, raster=raster, width=w, height=h), tile, clear_depth)


@pytest.mark.parametrize("raster", [RasterMode.Span, RasterMode.Block, RasterMode.Adaptive])
@pytest.mark.parametrize("tile", [16, 32])
def test_soups(gpu_lib, port, raster, tile):
    """Slanted triangles clipped at both planes, spans starting left of the tile and the target."""
    _check(port, scenes.soup_scene(1 << 13, width=203, height=151, seed=21, raster=raster), tile, float("inf"))
    sc = scenes.soup_scene(1 << 13, width=203, height=151, seed=22, raster=raster)
    sc.scissor = (-40, -3, 190, 140)
    _check(port, sc, tile, 0.9)


@pytest.mark.parametrize("ps", [PS.VCOLOR, PS.TEX_NEAREST])
def test_heavy_tile_runs(gpu_lib, port, ps):
    _check(port, scenes.stack_scene(5, 3000, ps=ps), 16, float("inf"), slicing=1)

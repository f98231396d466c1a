"""Overwrite shaders (no depth test): bins in any order, largest covering id per pixel, one
shaded fragment per pixel.  Against the oracle at the edges of the work split (32 and 128
entries per tile), of the slicing (512), in every raster mode and tile size, with and without
the per-pixel counts, on the general path and on the small draws' one."""
import numpy as np
import pytest

from softwarerenderer_gb300 import scenes
from softwarerenderer_gb300.abi import PS, RasterMode, VS

from .parity import describe, diff, oracle_render

pytestmark = pytest.mark.gpu


def _scene(n, raster, width=48, height=40, seed=0):
    sc = scenes.stack_scene(seed, n, raster=raster, width=width, height=height)
    sc.vs, sc.ps = VS.POS_RGB_AFFINE, PS.VCOLOR_AFFINE
    return sc


def _draw(sc, tile=16, aux=True, general=False, draws=1):
    from softwarerenderer_gb300.device import DeviceScene, DeviceTarget
    ds = DeviceScene(sc, tile=tile)
    if general:
        ds.rast.ctx.set_queue_capacity(0, 1 << 22)
    for _ in range(draws):
        tg = DeviceTarget(sc, aux=aux)
        st = ds.draw(tg)
    return tg.to_host(), st


@pytest.mark.parametrize("raster", [RasterMode.Span, RasterMode.Block, RasterMode.Adaptive])
@pytest.mark.parametrize("n", [1, 31, 32, 127, 128, 300, 512, 513, 1025, 5000])
@pytest.mark.parametrize("tile", [16, 32])
def test_piles(gpu_lib, port, n, raster, tile):
    sc = _scene(n, raster, seed=n)
    ref, rst = oracle_render(port, sc)
    for aux in (True, False):
        for general in (True, False):
            got, st = _draw(sc, tile, aux, general)
            want = ref if aux else {k: ref[k] for k in got}
            assert not diff(want, got), (aux, general, [describe(want, got, k) for k in diff(want, got)])
            assert st["fragments"] == st["passes"] == rst["fragments"]


def test_wide_tall_target_and_repeated_draws(gpu_lib, port):
    """Odd sizes; the winners and counters of sliced tiles are ready again for the next draw."""
    sc = scenes.benchmark_scene(4096)
    sc.width, sc.height = 333, 217
    sc.viewport = sc.scissor = (0, 0, 333, 217)
    ref, _ = oracle_render(port, sc)
    for draws in (1, 3):
        got, _ = _draw(sc, draws=draws)
        assert not diff(ref, got), [describe(ref, got, k) for k in diff(ref, got)]


def test_two_draws_into_one_target(gpu_lib, port):
    """A batch whose items share a target: the later item's primitives win."""
    from softwarerenderer_gb300.batch import BatchRenderer
    from softwarerenderer_gb300.device import DeviceTarget
    scs = [_scene(700, RasterMode.Adaptive, seed=s) for s in (1, 2)]
    tg = DeviceTarget(scs[0])
    br = BatchRenderer(scs, graph=False, targets=[tg, tg])
    br.draw()
    t = scenes.Target(scs[0])
    for sc in scs:
        port.draw(sc, t)
    want, got = t.arrays(), tg.to_host()
    assert not diff(want, got), [describe(want, got, k) for k in diff(want, got)]


@pytest.mark.parametrize("raster", [RasterMode.Span, RasterMode.Block, RasterMode.Adaptive])
@pytest.mark.parametrize("tile", [16, 32])
@pytest.mark.parametrize("scissor", [None, (5, 3, 171, 120), (-40, -3, 190, 140)])
def test_halves_told_by_their_end_rows(gpu_lib, port, raster, tile, scissor):
    """Bins of 128 entries and more (several classified batches): triangles that miss a tile's
    columns, cover all of them or cut them, thin slanted ones, scissors cutting both sides."""
    for sc in (scenes.benchmark_scene(6000), scenes.soup_scene(1 << 13, seed=23), scenes.soup_scene(3000, seed=24)):
        sc.width, sc.height, sc.raster = 203, 151, raster
        sc.viewport = (0, 0, 203, 151)
        sc.scissor = scissor or sc.viewport
        sc.vs, sc.ps = VS.POS_RGB_AFFINE, PS.VCOLOR_AFFINE
        ref, rst = oracle_render(port, sc)
        for aux in (True, False):
            got, st = _draw(sc, tile, aux)
            want = ref if aux else {k: ref[k] for k in got}
            assert not diff(want, got), (aux, [describe(want, got, k) for k in diff(want, got)])
            assert st["fragments"] == st["passes"] == rst["fragments"]

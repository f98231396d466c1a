"""Draws of at most 1,024 triangles (no bins: every tile's CTA picks its primitives from
their tile boxes, geometry in one CTA) against the oracle, and the general path on the same
scenes (a caller-sized bin queue keeps it): edges of the rule and of the 256-box windows,
clipping, every shader, graph replay, direct lists, statistics alike on both paths."""
import numpy as np
import pytest

from softwarerenderer_gb300 import scenes
from softwarerenderer_gb300.abi import DrawMode, PS, RasterMode

from .parity import describe, diff, oracle_render

pytestmark = pytest.mark.gpu

STATS = ("fragments", "primitives", "bin_pairs", "clip_polygons", "flags", "passes")


def _draw(sc, general=False, graph=False, draws=1):
    from softwarerenderer_gb300.device import DeviceScene, DeviceTarget
    ds = DeviceScene(sc)
    if general:
        ds.rast.ctx.set_queue_capacity(0, 1 << 22)
        ds.rast.ctx.set_tile_slicing(0)  # heavy-tile runs would count depth-test passes per run
    if graph:
        ds.rast.ctx.set_graph_mode(True)
    for _ in range(draws):
        tg = DeviceTarget(sc)
        st = ds.draw(tg)
    return tg.to_host(), st


def _check(port, sc, graph=False, draws=1, stats=STATS):
    ref, rst = oracle_render(port, sc)
    got, st = _draw(sc, graph=graph, draws=draws)
    assert not diff(ref, got), [describe(ref, got, k) for k in diff(ref, got)]
    assert st["fragments"] == rst["fragments"]
    gen, gst = _draw(sc, general=True, graph=graph, draws=draws)
    assert not diff(ref, gen), [describe(ref, gen, k) for k in diff(ref, gen)]
    assert {k: st[k] for k in stats} == {k: gst[k] for k in stats}


@pytest.mark.parametrize("seed", range(48))
def test_random_triangles_on_both_paths(gpu_lib, port, seed):
    _check(port, scenes.random_scene(seed, draw_mode=DrawMode.Triangle))


@pytest.mark.parametrize("n", [1, 255, 256, 257, 513, 1023, 1024, 1025])
@pytest.mark.parametrize("raster", [RasterMode.Span, RasterMode.Block, RasterMode.Adaptive])
def test_piles_at_the_edges_of_the_rule(gpu_lib, port, n, raster):
    """All n triangles over a few tiles (several windows and chunks per tile)."""
    _check(port, scenes.stack_scene(n, n, ps=PS.VCOLOR, raster=raster))


@pytest.mark.parametrize("ps", [PS.LAMBERT, PS.LAMBERT_TEX, PS.TEX_NEAREST])
def test_piles_of_every_depth_shader(gpu_lib, port, ps):
    _check(port, scenes.stack_scene(3, 900, ps=ps))


@pytest.mark.parametrize("n_prims", [120, 1024])
def test_clipped_fans(gpu_lib, port, n_prims):
    for seed in (7, 8, 11):
        _check(port, scenes.random_scene(seed, direct=False, draw_mode=DrawMode.Triangle, n_prims=n_prims))


def test_box_and_derivative_shaders(gpu_lib, port):
    for f in range(3):
        _check(port, scenes.box_scene(f))
        _check(port, scenes.deriv_scene(f))


@pytest.mark.parametrize("draws", [1, 3])
def test_graph_replay(gpu_lib, port, draws):
    _check(port, scenes.cube_scene(5), graph=True, draws=draws, stats=STATS[1:5])


@pytest.mark.parametrize("width", [4080, 4081])
def test_widest_target(gpu_lib, port, width):
    sc = scenes.sphere_scene(1, level=2, width=width, height=48)
    _check(port, sc)


def test_overflow_is_reported_and_recovers(gpu_lib, port):
    from softwarerenderer_gb300 import _lib
    from softwarerenderer_gb300.device import DeviceScene, DeviceTarget
    sc = scenes.sphere_scene(1, level=3, width=200, height=100)
    sc.indices = sc.indices[:3 * 1000]
    ds = DeviceScene(sc)
    ds.rast.ctx.set_queue_capacity(10, 0)
    tg = DeviceTarget(sc)
    before = tg.to_host()
    ds.draw(tg, sync=False)
    rc, st = ds.rast.ctx.finish()
    assert rc == _lib.SWR_EOVERFLOW and st["fragments"] == 0
    assert not diff(before, tg.to_host())
    ds.draw(tg)
    assert not diff(oracle_render(port, sc)[0], tg.to_host())


def test_bad_index_is_reported(gpu_lib):
    from softwarerenderer_gb300 import _lib
    from softwarerenderer_gb300.device import DeviceScene, DeviceTarget
    sc = scenes.cube_scene(0)
    sc.indices = np.array(sc.indices)
    sc.indices[7] = 24
    ds = DeviceScene(sc)
    with pytest.raises(_lib.SwrError) as e:
        ds.draw(DeviceTarget(sc))
    assert e.value.code == _lib.SWR_EINDEX

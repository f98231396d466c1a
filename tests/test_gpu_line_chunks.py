"""Points and lines where the tile raster's chunks of 256 fragments change form: tiles of 255 to 257
fragments, cells of more than a chunk (sorted ahead, rasterized in runs, resumed at their ends
inside a chunk of whole cells) and of exactly one, fragments of a line far enough apart to fall in
cells of their own; against the oracle."""
import numpy as np
import pytest

from softwarerenderer_gb300 import scenes
from softwarerenderer_gb300.abi import DrawMode, PS, RASTER_VERTEX_FLOATS, VS

from .parity import describe, diff, gpu_render, oracle_render

pytestmark = pytest.mark.gpu


def _scene(mode, n, x0, x1, y0, y1, width, height, seed):
    rng = np.random.default_rng(seed)
    per = 1 if mode == DrawMode.Point else 2
    rv = np.zeros((per * n, RASTER_VERTEX_FLOATS), np.float32)
    rv[:, 0] = x0 + (x1 - x0) * rng.random(per * n)
    rv[:, 1] = y0 + (y1 - y0) * rng.random(per * n)
    rv[:, 2] = rng.integers(0, 16, per * n) / 16.0
    rv[:, 3] = 0.5 + rng.random(per * n)
    rv[:, 20:23] = rng.random((per * n, 3))
    return scenes.Scene(name="chunks", vs=VS.POS_RGB, ps=PS.VCOLOR, width=width, height=height, draw_mode=mode,
                        scissor=(0, 0, width, height), indices=np.arange(per * n, dtype=np.int32), raster_vertices=rv)


def _check(port, sc):
    ref, rst = oracle_render(port, sc)
    got, gst = gpu_render(sc)
    assert not diff(ref, got), [describe(ref, got, k) for k in diff(ref, got)]
    assert gst["fragments"] == rst["fragments"]


@pytest.mark.parametrize("n", [255, 256, 257, 8192, 8193, 8700, 40001])  # (8,193: cells of 512, 256 before)
def test_points_of_one_tile(gpu_lib, port, n):
    _check(port, _scene(DrawMode.Point, n, 16, 32, 0, 16, 50, 37, n))


@pytest.mark.parametrize("n", [8193, 30000])
def test_points_of_two_tiles(gpu_lib, port, n):
    """Most in one tile, few in the next: large and small cells of both."""
    sc = _scene(DrawMode.Point, n, 0, 16, 0, 16, 50, 37, n)
    sc.raster_vertices[n // 2:n // 2 + 300, 0] += 16.0
    _check(port, sc)


@pytest.mark.parametrize("n", [30, 300, 9000])
def test_lines_of_one_tile(gpu_lib, port, n):
    _check(port, _scene(DrawMode.Line, n, 16, 31.9, 16, 31.9, 50, 37, n))


@pytest.mark.parametrize("n", [1, 33, 2500])
def test_lines_of_many_steps(gpu_lib, port, n):
    """Few lines of many fragments: fewer than 32 of them a warp, down to one."""
    _check(port, _scene(DrawMode.Line, n, -500, 3000, -400, 900, 1300, 500, n))


@pytest.mark.parametrize("mode,n", [(DrawMode.Point, 4096), (DrawMode.Point, 4097), (DrawMode.Point, 9001),
                                    (DrawMode.Line, 600), (DrawMode.Line, 4000)])
def test_heavy_tiles(gpu_lib, port, mode, n):
    """Tiles of around and above 4,096 fragments, rasterized by four CTAs of four rows each: one
    whole tile, one at the target's right and lower edges, all fragments in one row and one pixel."""
    _check(port, _scene(mode, n, 0, 16, 0, 16, 50, 37, n))
    _check(port, _scene(mode, n, 46, 50, 33, 37, 50, 37, n))
    _check(port, _scene(mode, n, 0, 16, 7.1, 7.9, 50, 37, n))
    _check(port, _scene(mode, n, 5.1, 5.9, 9.1, 9.9, 50, 37, n))


@pytest.mark.parametrize("mode,n", [(DrawMode.Point, 1000000), (DrawMode.Line, 20000)])
def test_more_heavy_tiles_than_slots(gpu_lib, port, mode, n):
    _check(port, _scene(mode, n, 0, 200, 0, 200, 200, 200, n))

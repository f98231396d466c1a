"""Points and lines binned by tile: bit for bit against the oracle where the path changes
form -- one primitive, tiles at and around the 512 fragments a tile's CTA orders itself,
cells above the 64 entries sorted by bitmap, chunks of 256 fragments with a remainder, lines
crossing many tiles, and the direct lists with skipped primitives."""
import numpy as np
import pytest

from softwarerenderer_gb300 import scenes
from softwarerenderer_gb300.abi import DrawMode, PS, RASTER_VERTEX_FLOATS, VS

from .parity import describe, diff, gpu_render, oracle_render

pytestmark = pytest.mark.gpu


def _check(port, sc, tile=16):
    ref, rst = oracle_render(port, sc)
    got, gst = gpu_render(sc, tile=tile)
    assert not diff(ref, got), [describe(ref, got, k) for k in diff(ref, got)]
    assert gst["fragments"] == rst["fragments"]


@pytest.mark.parametrize("mode", [DrawMode.Line, DrawMode.Point])
@pytest.mark.parametrize("n", [1, 257, 5000, 40000])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_random_scenes_of_many_sizes(gpu_lib, port, mode, n, seed):
    _check(port, scenes.random_scene(9000 + seed, draw_mode=mode, n_prims=n))


@pytest.mark.parametrize("tile", [16, 32])
@pytest.mark.parametrize("n", [511, 512, 513, 2600])
def test_one_tile_of_points(gpu_lib, port, n, tile):
    """All points in one 16 x 16 tile, depths tying often, some lists skipping entries."""
    rng = np.random.default_rng(n)
    rv = np.zeros((n, RASTER_VERTEX_FLOATS), np.float32)
    rv[:, 0:2] = 16.0 * rng.random((n, 2)) + 16.0
    rv[:, 2] = rng.integers(0, 8, n) / 8.0
    rv[:, 3] = 0.5 + rng.random(n)
    rv[:, 20:23] = rng.random((n, 3))
    idx = rng.permutation(n).astype(np.int32)
    idx[::97] = -1
    _check(port, scenes.Scene(name=f"tile{n}", vs=VS.POS_RGB, ps=PS.VCOLOR, width=50, height=37,
                              draw_mode=DrawMode.Point, scissor=(0, 0, 50, 37), indices=idx, raster_vertices=rv), tile)


def test_long_lines(gpu_lib, port):
    """Lines across a 1000 x 300 target and past its edges: up to thousands of steps each."""
    rng = np.random.default_rng(5)
    n = 60
    rv = np.zeros((2 * n, RASTER_VERTEX_FLOATS), np.float32)
    rv[:, 0:2] = rng.random((2 * n, 2)) * np.array([3000, 500]) - np.array([1000, 100])
    rv[:, 2] = rng.random(2 * n)
    rv[:, 3] = 0.5 + rng.random(2 * n)
    rv[:, 20:23] = rng.random((2 * n, 3))
    _check(port, scenes.Scene(name="long", vs=VS.POS_RGB, ps=PS.VCOLOR, width=1000, height=300,
                              draw_mode=DrawMode.Line, scissor=(3, 5, 990, 290),
                              indices=np.arange(2 * n, dtype=np.int32), raster_vertices=rv))

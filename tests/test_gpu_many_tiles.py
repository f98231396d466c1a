"""Batches of more than 65,536 tiles, whose raster CTAs take a second tile each when more than
half of the tiles hold primitives: both sides of the line, mostly empty and full targets,
depth-tested shaders and raster modes, against the oracle."""
import pytest

from softwarerenderer_gb300 import scenes
from softwarerenderer_gb300.abi import PS, RasterMode

from .parity import diff, oracle_render

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("raster", [RasterMode.Span, RasterMode.Block, RasterMode.Adaptive])
@pytest.mark.parametrize("kind", ["soup", PS.VCOLOR, PS.LAMBERT, PS.LAMBERT_TEX])
@pytest.mark.parametrize("draws", [16, 17])  # of 4,096 tiles
@pytest.mark.parametrize("n", [300, 20000])
def test_batch(gpu_lib, port, raster, kind, draws, n):
    from softwarerenderer_gb300.batch import BatchRenderer
    if kind == "soup":
        make = lambda k: scenes.soup_scene(n // 4, width=1024, height=1024, seed=k, raster=raster)
    else:
        make = lambda k: scenes.stack_scene(k, n, ps=kind, raster=raster, width=1024, height=1024)
    scs = [make(k) for k in range(draws)]
    br = BatchRenderer(scs, aux=True)
    for _ in range(2):
        br.clear()
        br.draw()
    for k in (0, draws // 2, draws - 1):
        ref, _ = oracle_render(port, scs[k])
        assert not diff(ref, br.targets[k].to_host()), k

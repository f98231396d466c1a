"""The Lambert shader above 65,536 tiles with its heavy-tile runs off (by default their CTAs keep the
launch of one tile a CTA): two tiles a CTA, one target and many, against the oracle."""
import pytest

from softwarerenderer_gb300 import scenes
from softwarerenderer_gb300.abi import PS, RasterMode

from .parity import diff, gpu_render, oracle_render

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("raster", [RasterMode.Span, RasterMode.Block])
@pytest.mark.parametrize("n", [300, 20000])
def test_lambert_batch(gpu_lib, port, raster, n):
    from softwarerenderer_gb300.batch import BatchRenderer
    scs = [scenes.stack_scene(k, n, ps=PS.LAMBERT, raster=raster, width=1024, height=1024) for k in range(17)]
    br = BatchRenderer(scs, aux=True)
    br.ctx.set_tile_slicing(0)
    for _ in range(2):
        br.clear()
        br.draw()
    for k in (0, 8, 16):
        assert not diff(oracle_render(port, scs[k])[0], br.targets[k].to_host()), k


@pytest.mark.parametrize("ps", [PS.LAMBERT, PS.VCOLOR])
@pytest.mark.parametrize("width,height", [(4096, 4096), (4097, 4096)])  # 65,536 tiles and 65,792
def test_one_target(gpu_lib, port, ps, width, height):
    sc = scenes.stack_scene(9, 30000, ps=ps, width=width, height=height)
    got, st = gpu_render(sc, slicing=0)
    ref, rst = oracle_render(port, sc)
    assert not diff(ref, got) and st["fragments"] == rst["fragments"]

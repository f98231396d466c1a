"""Draws whose bin entries sum to 2^32 or more: 66,000 triangles over all 65,536 tiles of a
4096 x 4096 target (30,408,704 when read in 32 bits, which a queue would hold).  Such a draw is
reported, the target and the queue stay as they are, and the context draws on."""
import numpy as np
import pytest

from softwarerenderer_gb300 import _lib, scenes
from softwarerenderer_gb300.abi import DrawMode, PS, RASTER_VERTEX_FLOATS, RasterMode, VS

from .parity import diff, oracle_render

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ps", [PS.VCOLOR, PS.VCOLOR_AFFINE])
def test_entries_past_32_bits_are_refused(gpu_lib, port, ps):
    from softwarerenderer_gb300.device import DeviceScene, DeviceTarget
    side, n = 4096, 66000
    rv = np.zeros((3, RASTER_VERTEX_FLOATS), np.float32)
    rv[:, 0:2] = [(0, 0), (2 * side, 0), (0, 2 * side)]
    rv[:, 3] = 1.0
    sc = scenes.Scene(name="full", vs=VS.POS_RGB, ps=ps, width=side, height=side, draw_mode=DrawMode.Triangle,
                      raster=RasterMode.Block, scissor=(0, 0, side, side),
                      indices=np.tile(np.arange(3, dtype=np.int32), n), raster_vertices=rv)
    ds, tg = DeviceScene(sc), DeviceTarget(sc, aux=False)
    tg.clear()
    queue = None
    for _ in range(3):
        ds.draw(tg, sync=False)
        rc, st = ds.rast.ctx.finish()
        assert rc == _lib.SWR_ENOMEM and st["fragments"] == 0 and st["bin_pairs"] == 2 ** 32 - 1
        assert queue in (None, ds.rast.ctx.queue_capacity())  # a larger queue would not help
        queue = ds.rast.ctx.queue_capacity()
    assert not bool(tg.color.any()) and bool((tg.depth == float("inf")).all())
    with pytest.raises(_lib.SwrError) as e:
        ds.draw(tg)
    assert e.value.code == _lib.SWR_ENOMEM
    small = scenes.stack_scene(2, 3000, width=200, height=90)
    tg = DeviceTarget(small)
    DeviceScene(small, ds.rast.ctx).draw(tg)
    assert not diff(oracle_render(port, small)[0], tg.to_host())

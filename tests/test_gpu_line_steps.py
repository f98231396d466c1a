"""Line lists whose DDA steps sum to 2^32 or more: screen-space lines are not clipped, so a few
endpoints far outside the target are enough.  Such a draw asks for more fragments than any queue
holds, however the sum reads in 32 bits: it is reported, the target and the queue stay as they
are, and the context draws on."""
import numpy as np
import pytest

from softwarerenderer_gb300 import _lib, scenes
from softwarerenderer_gb300.abi import DrawMode, PS, RASTER_VERTEX_FLOATS, VS

from .parity import diff, oracle_render

pytestmark = pytest.mark.gpu

BIG = 2 ** 31 - 1  # steps of a line from 0 to 2^31 and beyond: truncation saturates


def _scene(lengths):
    rng = np.random.default_rng(len(lengths))
    n = len(lengths)
    rv = np.zeros((2 * n, RASTER_VERTEX_FLOATS), np.float32)
    rv[1::2, 0] = [3.0e9 if s == BIG else s for s in lengths]
    rv[:, 1] = np.repeat(rng.integers(0, 40, n), 2)
    rv[:, 2] = rng.random(2 * n)
    rv[:, 3] = 1.0
    rv[:, 20:23] = rng.random((2 * n, 3))
    return scenes.Scene(name="steps", vs=VS.POS_RGB, ps=PS.VCOLOR, width=64, height=40, draw_mode=DrawMode.Line,
                        scissor=(0, 0, 64, 40), indices=np.arange(2 * n, dtype=np.int32), raster_vertices=rv)


@pytest.mark.parametrize("lengths", [
    [BIG, BIG, 1],                          # 2^32 - 1
    [BIG, BIG, 2],                          # 2^32: reads 0
    [BIG] * 2 + [50] * 100,                 # reads 4998
    [BIG] + [40] * 200 + [BIG] + [40] * 7,  # the long ones in different warps
    [BIG] * 64 + [30] * 3000,               # a warp of its own wraps, several times
])
def test_steps_past_32_bits_are_refused(gpu_lib, port, lengths):
    from softwarerenderer_gb300.device import DeviceScene, DeviceTarget
    assert sum(lengths) >= 2 ** 32 - 1
    sc = _scene(lengths)
    ds = DeviceScene(sc)
    small = _scene([40] * 50)
    ok = DeviceScene(small, ds.rast.ctx)
    ok.draw(DeviceTarget(small))
    held, queue = ds.rast.ctx.memory_used(), None
    tg = DeviceTarget(sc)
    before = tg.to_host()
    for _ in range(3):
        ds.draw(tg, sync=False)
        rc, st = ds.rast.ctx.finish()
        assert rc == _lib.SWR_ENOMEM and st["fragments"] == 0
        assert queue in (None, ds.rast.ctx.queue_capacity())  # a larger queue would not help
        queue = ds.rast.ctx.queue_capacity()
    assert ds.rast.ctx.memory_used() < held + (64 << 20)
    assert not diff(before, tg.to_host())
    with pytest.raises(_lib.SwrError) as e:
        ds.draw(tg)
    assert e.value.code == _lib.SWR_ENOMEM
    tg = DeviceTarget(small)
    ok.draw(tg)
    assert not diff(oracle_render(port, small)[0], tg.to_host())

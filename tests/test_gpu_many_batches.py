"""Draws of very many triangles: above 2,048 batches of 1,024 the counting launch's last block
computes the batch bases that the emitting blocks otherwise sum for themselves.  Both sides of
the line, one draw and many draws, against the grid-barrier front end, which always sums."""
import numpy as np
import pytest

from softwarerenderer_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2048 * 1024, 2048 * 1024 + 1, 2049 * 1024 + 512, 2050 * 1024 - 3])
def test_single_draw(gpu_lib, n):
    from softwarerenderer_gb300.device import DeviceScene, DeviceTarget
    sc = scenes.soup_scene(n, width=96, height=64, seed=3)
    out = []
    for persistent in (False, True):
        ds = DeviceScene(sc)
        ds.rast.ctx.set_persistent_geometry(persistent)
        tg = DeviceTarget(sc)
        st = ds.draw(tg)
        out.append((tg.to_host(), [st[k] for k in ("primitives", "fragments", "clip_polygons", "bin_pairs", "flags")]))
    assert out[0][1] == out[1][1]
    for k in out[0][0]:
        assert np.array_equal(out[0][0][k], out[1][0][k]), k


def test_draws_of_a_batch(gpu_lib):
    """Small and empty-ended draws around a large one: per-draw primitive numbers (winner)."""
    from softwarerenderer_gb300.batch import BatchRenderer
    scs = [scenes.soup_scene(n, width=96, height=64, seed=n) for n in (1, 1025, 2048 * 1024, 7, 5000)]
    out = []
    for persistent in (False, True):
        br = BatchRenderer(scs, aux=True)
        br.ctx.set_persistent_geometry(persistent)
        br.clear()
        st = br.draw()
        out.append(([t.to_host() for t in br.targets], int(st["fragments"]), int(st["primitives"])))
    assert out[0][1:] == out[1][1:]
    for a, b in zip(out[0][0], out[1][0]):
        for k in a:
            assert np.array_equal(a[k], b[k]), k

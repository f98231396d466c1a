"""Graph replay after one of the context's buffers has moved.  The buffers grow at sizes of their
own: of the sizes below the last but one makes only the batches' bases move (3,752 batches of
1,024 where room for 3,751 was left), and the graph captured for the size before it must not be
replayed over the old ones."""
import numpy as np
import pytest

from softwarerenderer_gb300 import scenes
from softwarerenderer_gb300.abi import DrawMode

pytestmark = pytest.mark.gpu

SIZES = (3072000, 3841000, 3841000, 3841100, 3841000, 3841000, 3841100)


def test_replay_over_moved_buffers(gpu_lib):
    from softwarerenderer_gb300.device import DeviceScene, DeviceTarget
    sc = scenes.soup_scene(max(SIZES), width=96, height=64, seed=5)
    graph, plain = DeviceScene(sc), DeviceScene(sc)
    graph.rast.ctx.set_graph_mode(True)
    expected = {}
    for n in SIZES:
        out = []
        for ds in (graph, plain) if n not in expected else (graph,):
            tg = DeviceTarget(sc)
            ds.bind(tg)
            st = ds.vp.drawElements(DrawMode.Triangle, 3 * n, ds.indices)
            out.append((tg.to_host(), [st[k] for k in ("primitives", "fragments", "clip_polygons", "bin_pairs", "flags")]))
        expected.setdefault(n, out[-1])
        assert out[0][1] == expected[n][1]
        for k, a in out[0][0].items():
            assert np.array_equal(a, expected[n][0][k]), (n, k)

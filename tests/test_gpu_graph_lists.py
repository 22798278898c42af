"""Graph frames with long command lists, of one canvas and of several: the composite's tail launch
belongs to frames of several canvases, in a captured graph as in an eager run. Pixels against the
oracle's, bit for bit."""
import numpy as np
import pytest

import blend2d_gb300 as bg
import oracle_lib
from blend2d_gb300 import scenes

pytestmark = pytest.mark.gpu

SIZES = [(40, 37, 700), (33, 6, 500), (90, 64, 40)]


def _streams(seed):
    return [scenes.random_mix(seed=seed + i, width=w, height=h, count=n).to_bytes() for i, (w, h, n) in enumerate(SIZES)]


def _polygons(seed):
    return scenes.polygons(seed, 64, 48, 600).to_bytes()


def _runtime(graph):
    rt = bg.Runtime(0)
    cfg = rt.launch_config()
    cfg.graph_frames = graph
    rt.set_launch_config(cfg)
    return rt


def _render(rt, streams):
    targets = [np.zeros(bg.stream_size(s)[::-1], dtype=np.uint32) for s in streams]
    rt.render_batch(streams, targets)
    return targets


@pytest.mark.parametrize("canvases", [1, 3])
def test_a_graph_holds_the_eager_launches(canvases):
    with _runtime(0) as rt:
        _render(rt, [_polygons(5 + i) for i in range(canvases)])
        eager = rt.stats().kernel_launches
    with _runtime(1) as rt:
        for k in range(3):
            streams = [_polygons(5 + 3 * k + i) for i in range(canvases)]
            for stream, target in zip(streams, _render(rt, streams)):
                assert np.array_equal(target, oracle_lib.render(stream))
        assert rt.stats().graph_frames == 2
        assert rt.stats().kernel_launches == eager + 1      # frame_gate_kernel


@pytest.mark.parametrize("first", [1, 3])
def test_frames_of_one_and_of_several_canvases_in_turn(first):
    with _runtime(1) as rt:
        for k in range(8):
            streams = _streams(700 + 10 * k)[: first if k % 2 == 0 else 4 - first]
            for stream, target in zip(streams, _render(rt, streams)):
                assert np.array_equal(target, oracle_lib.render(stream)), k
        assert rt.stats().graph_frames > 0

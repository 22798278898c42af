"""A frame replayed as a graph between graph frames: the replay captures the kept frame's pipeline on its
own arrays, the next graph frame's arrays go by capacities. Pixels against the oracle's, bit for bit."""
import numpy as np
import pytest

import blend2d_gb300 as bg
import oracle_lib
from blend2d_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("larger_first", [False, True])
def test_replays_between_graph_frames(larger_first):
    streams = [scenes.random_mix(seed=40 + i, width=131, height=77, count=30).to_bytes() for i in range(5)]
    with bg.Runtime(0) as rt:
        if larger_first:                         # arenas larger than any later frame's capacities
            bg.render_stream(rt, scenes.random_mix(seed=9, width=600, height=500, count=900).to_bytes())
        cfg = rt.launch_config()
        cfg.graph_frames = 1
        rt.set_launch_config(cfg)
        for stream in streams:
            assert np.array_equal(bg.render_stream(rt, stream), oracle_lib.render(stream))
            rt.replay(True)
            rt.synchronize()
        assert rt.stats().graph_frames > 0

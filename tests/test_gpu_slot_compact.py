"""Masks and work items handed out to the slots with segments: many commands of one slot (more than 32 in a
warp's 128 slots, so commands are searched for), of a few, and of whole rows of slots with few segments,
mixed, on canvases of one and of several tiles. Pixels against the oracle's, bit for bit."""
import numpy as np
import pytest

import blend2d_gb300 as bg
import oracle_lib
from blend2d_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mix", ["tiny", "wide", "both"])
@pytest.mark.parametrize("size", [(31, 4), (65, 33), (700, 260)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_slots_of_every_density(size, mix):
    w, h = size
    rng = np.random.Generator(np.random.PCG64(w * 7 + h))
    sw = scenes.StreamWriter(w, h)
    for i in range(900 if mix != "wide" else 120):
        sw.comp_op(scenes.SRC_COPY if rng.random() < 0.3 else scenes.SRC_OVER)
        sw.solid(int(rng.integers(0, 2**32, dtype=np.uint64)))
        if mix == "wide" or (mix == "both" and rng.random() < 0.1):
            p = rng.uniform(-0.2, 1.2, (4, 2)) * np.array([w, h])
        else:
            p = rng.uniform(0.0, 1.0, 2) * np.array([w, h]) + rng.uniform(-2.0, 2.0, (3, 2))
        sw.fill_polygon(p)
    stream = sw.to_bytes()
    with bg.Runtime(0) as rt:
        assert np.array_equal(bg.render_stream(rt, stream), oracle_lib.render(stream))

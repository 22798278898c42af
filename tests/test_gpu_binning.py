"""Binning (strip rows of segments, slot layout) at the sizes where its units change: canvases wider
than a warp's share of the slots, rows of one tile column, runs of commands without slots between
commands with them, segments across the whole canvas. Pixels against the oracle's, bit for bit."""
import numpy as np
import pytest

import blend2d_gb300 as bg
import oracle_lib
from blend2d_gb300 import scenes

pytestmark = pytest.mark.gpu

# width, height, polygons, box fills after each polygon
SHAPES = [(1, 1, 3, 0), (31, 200, 40, 1), (33, 5, 40, 2), (127, 127, 200, 33), (1024, 64, 60, 70), (4095, 13, 30, 0),
          (4097, 37, 30, 5), (9001, 9, 25, 0), (40, 6000, 25, 0), (2100, 1100, 20, 0)]


def _scene(w, h, n, boxes, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    sw = scenes.StreamWriter(w, h)
    sw.solid(0xFF102030)
    sw.fill_all()
    for i in range(n):
        sw.fill_rule(int(rng.integers(0, 2)))
        sw.solid(int(rng.integers(0, 2**32, dtype=np.uint64)))
        size = np.array([w, h]) * (1.0 if i % 3 else 0.1) + 1.0
        org = rng.uniform(-0.05, 0.95, 2) * np.array([w, h]) * (0.0 if i % 3 else 1.0)
        xy = rng.uniform(-0.1, 1.1, (int(rng.integers(3, 9)), 2)) * size + org
        if i % 5 == 0:
            xy = np.round(xy)                      # whole pixels: vertices on tile and strip edges
        sw.fill_polygon(xy)
        for k in range(boxes):
            sw.fill_rect_i(int(rng.integers(0, w)), int(rng.integers(0, h)), 1 + k % 3, 2)
    return sw.to_bytes()


@pytest.mark.parametrize("shape", SHAPES, ids=[f"{s[0]}x{s[1]}" for s in SHAPES])
def test_binning_matches_the_oracle(shape):
    streams = [_scene(*shape, seed=k) for k in range(2)]
    with bg.Runtime(0) as rt:
        for stream in streams:
            assert np.array_equal(bg.render_stream(rt, stream), oracle_lib.render(stream))
        if shape[0] * shape[1] < 200_000:          # both at once: slots of several canvases side by side
            targets = [np.zeros((shape[1], shape[0]), dtype=np.uint32) for _ in streams]
            rt.render_batch(streams, targets)
            for stream, target in zip(streams, targets):
                assert np.array_equal(target, oracle_lib.render(stream))

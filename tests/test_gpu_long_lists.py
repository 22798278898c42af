"""Batches whose few strips have long command lists, which the composite leaves to its tail launch: small
canvases with many commands of every kind beside sparse ones, in the three target formats, at several
list-row heights. Pixels against the oracle's, bit for bit."""
import numpy as np
import pytest

import blend2d_gb300 as bg
import oracle_lib
from blend2d_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [32, 4])
@pytest.mark.parametrize("fmt", [scenes.FORMAT_PRGB32, scenes.FORMAT_XRGB32, scenes.FORMAT_A8], ids=["prgb", "xrgb", "a8"])
def test_tail_rows_match_the_oracle(fmt, rows):
    sizes = [(40, 37, 700), (33, 6, 500), (1, 1, 300), (90, 64, 40), (31, 33, 66)]
    streams = [scenes.random_mix(seed=300 + i, width=w, height=h, count=n, dither=i % 2 == 0, format=fmt).to_bytes()
               for i, (w, h, n) in enumerate(sizes)]
    dtype = np.uint8 if fmt == scenes.FORMAT_A8 else np.uint32
    targets = [np.zeros((h, w), dtype=dtype) for w, h, _ in sizes]
    with bg.Runtime(0) as rt:
        cfg = rt.launch_config()
        cfg.list_rows = rows
        rt.set_launch_config(cfg)
        for _ in range(2):
            rt.render_batch(streams, targets)
            for stream, target in zip(streams, targets):
                assert np.array_equal(target, oracle_lib.render(stream))

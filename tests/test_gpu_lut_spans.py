"""Gradient tables written span by span: spans of no, one, two and a few entries, spans that begin on the
entry the one before ends on, around multiples of 32, tables that end in a trailing fill, opaque and not,
in every builder. Pixels against the oracle's, bit for bit."""
import numpy as np
import pytest

import blend2d_gb300 as bg
import oracle_lib
from blend2d_gb300 import scenes

pytestmark = pytest.mark.gpu


def _stops(kind, opaque, rng):
    size = 1024.0
    entries = {"one": [0.4], "two": [0.0, 1.0], "late": [0.31, 0.32], "short": [0.0, 0.2 / size, 1.1 / size, 2.3 / size, 5.0 / size, 31.0 / size,
               32.0 / size, 33.5 / size, 63.9 / size, 64.0 / size, 0.5, 0.5, 0.5 + 0.6 / size, 1.0],
               "ends": [0.0, 0.0, 0.25, 0.25, 0.25, 0.999], "dense": np.sort(rng.uniform(0.0, 0.08, 40)).tolist()}[kind]
    cols = rng.integers(0, 2**64, len(entries), dtype=np.uint64)
    if opaque:
        cols |= np.uint64(0xFFFF000000000000)
    return [(float(o), int(c)) for o, c in zip(entries, cols)]


@pytest.mark.parametrize("variant,dither", [("default", False), ("avx2", False), ("scalar", False), ("default", True)])
def test_spans_give_the_same_tables(variant, dither):
    rng = np.random.Generator(np.random.PCG64(4100 + dither))
    kinds = ["one", "two", "late", "short", "ends", "dense"]
    w, band = 1100, 3                                         # wider than a table: every entry shows
    sw = scenes.StreamWriter(w, band * 2 * len(kinds))
    if dither:
        sw.hint(scenes.HINT_GRADIENT_QUALITY, scenes.GRADIENT_DITHER)
    for i, kind in enumerate(kinds):
        for opaque in (0, 1):
            sw.gradient(scenes.LINEAR, [0.0, 0.0, float(w), 0.0], i % 3, _stops(kind, opaque, rng))
            sw.fill_rect_i(0, band * (2 * i + opaque), w, band)
    stream = sw.to_bytes()
    with bg.Runtime(0, {"default": bg.LUT_SSE2, "avx2": bg.LUT_AVX2, "scalar": bg.LUT_SCALAR}[variant]) as rt:
        assert np.array_equal(bg.render_stream(rt, stream), oracle_lib.render(stream, variant))

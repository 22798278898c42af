"""Occlusion before the masks are rasterized: opaque SrcCopy paths, aligned and fractional boxes and A8
masks over earlier fills, on canvases whose last tiles and strips are cut, at every list-row height, and
in the three target formats. Pixels against the oracle's, bit for bit, and against rendering with the
occlusion off."""
import numpy as np
import pytest

import blend2d_gb300 as bg
import oracle_lib
from blend2d_gb300 import scenes

pytestmark = pytest.mark.gpu


def _scene(seed, w, h, fmt):
    rng = np.random.Generator(np.random.PCG64(seed))
    sw = scenes.StreamWriter(w, h, fmt)
    sw.solid(0xFF304050)
    sw.fill_all()
    for i in range(160):
        sw.comp_op(scenes.SRC_COPY if rng.random() < 0.6 else scenes.SRC_OVER)
        sw.fill_alpha(1.0 if rng.random() < 0.8 else float(rng.uniform(0.2, 0.99)))
        sw.fill_rule(int(rng.integers(0, 2)))
        if rng.random() < 0.7:
            sw.solid(int(rng.integers(0, 2**32, dtype=np.uint64)))
        else:
            p = rng.uniform(0, max(w, h), 4)
            sw.gradient(scenes.LINEAR, p.tolist(), int(rng.integers(0, 3)), [(0.0, 0xFFFF000000000000), (1.0, 0x8000FFFF00000000)])
        k = int(rng.integers(0, 5))
        x0, y0 = rng.uniform(-0.4 * w, 0.7 * w), rng.uniform(-0.4 * h, 0.7 * h)
        x1, y1 = x0 + rng.uniform(0.2, 1.2) * w, y0 + rng.uniform(0.2, 1.2) * h
        if k == 0:
            sw.fill_box_d(x0, y0, x1, y1)
        elif k == 1:
            sw.fill_rect_i(int(x0), int(y0), int(x1 - x0) + 1, int(y1 - y0) + 1)
        elif k == 2:
            mask = np.full((int(rng.integers(1, 60)), int(rng.integers(1, 60))), 255, dtype=np.uint8)
            mask[:, : int(rng.integers(0, mask.shape[1]))] = int(rng.integers(0, 256))
            sw.fill_mask_i(int(x0), int(y0), mask)
        else:
            if k == 3:                                        # edges on the tile grid: slots covered to their sides
                x0, y0, x1, y1 = (np.round(np.array([x0, y0, x1, y1]) / 32.0) * 32.0).tolist()
            sw.fill_polygon(np.array([[x0, y0], [x1, y0], [x1 + (k - 3) * 20.0, y1], [x0, y1]]))
    return sw.to_bytes()


@pytest.mark.parametrize("fmt", [scenes.FORMAT_PRGB32, scenes.FORMAT_XRGB32, scenes.FORMAT_A8], ids=["prgb", "xrgb", "a8"])
@pytest.mark.parametrize("size", [(1, 1), (33, 5), (64, 64), (127, 130), (300, 67)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_occlusion_keeps_pixels(size, fmt):
    stream = _scene(size[0] + 7 * fmt, size[0], size[1], fmt)
    want = oracle_lib.render(stream)
    with bg.Runtime(0) as rt:
        for rows in (32, 16, 8, 4):
            for off in (0, 1):
                cfg = rt.launch_config()
                cfg.list_rows, cfg.no_occlusion_cull = rows, off
                rt.set_launch_config(cfg)
                assert np.array_equal(bg.render_stream(rt, stream), want), (rows, off)

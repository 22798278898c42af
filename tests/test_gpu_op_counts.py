"""Pixel operations counted with the occlusion off: every command of every strip is composited, also
below opaque SrcCopy paths that cover a strip their own segments lie in."""
import numpy as np
import pytest

import blend2d_gb300 as bg
from blend2d_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(64, 64), (33, 7), (130, 70)])
def test_counts_without_occlusion_are_the_whole_work(w, h):
    sw = scenes.StreamWriter(w, h)
    sw.comp_op(scenes.SRC_COPY)
    sw.solid(0xFF102030)
    sw.fill_all()
    n = 9
    for i in range(n):
        sw.solid(0xFF000000 | (i * 0x1C1C1C))
        # edges along the canvas border and over it: segments in slots that the polygons cover
        sw.fill_polygon(np.array([[0.0, 0.0], [float(w), 0.0], [float(w), float(h)], [0.0, float(h)]]))
        sw.fill_polygon(np.array([[0.0, 0.0], [w + 40.0, 0.0], [w + 0.0, h / 2.0], [w + 40.0, h * 1.0], [0.0, h * 1.0]]))
    stream = sw.to_bytes()
    with bg.Runtime(0) as rt:
        culled = bg.render_stream(rt, stream)
        cfg = rt.launch_config()
        cfg.no_occlusion_cull = 1
        rt.set_launch_config(cfg)
        full = bg.render_stream(rt, stream)
        assert np.array_equal(culled, full)
        assert rt.stats().pixel_ops == (2 * n + 1) * w * h
        rt.replay(False)
        rt.synchronize()
        assert rt.stats().pixel_ops == (2 * n + 1) * w * h

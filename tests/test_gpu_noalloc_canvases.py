"""The no-allocation entry point on large canvases, whose per-tile arrays take most of its scratch area, and
with as many curves as it holds."""
import numpy as np
import pytest

import blend2d_gb300 as bg
from blend2d_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(20480, 20480), (24000, 24000), (8192, 49999)])
def test_large_canvas_matches_the_context_path(w, h):
    torch = pytest.importorskip("torch")
    rng = np.random.Generator(np.random.PCG64(w + h))
    sw = scenes.StreamWriter(w, h, scenes.FORMAT_A8)
    sw.solid(0x40000000)
    sw.fill_all()
    for _ in range(12):
        sw.solid(int(rng.integers(1, 256)) << 24)
        sw.fill_polygon(rng.uniform(0.0, 1.0, (4, 2)) * np.array([w, h]) * 0.02 + rng.uniform(0.0, 0.98, 2) * np.array([w, h]))
    stream = sw.to_bytes()
    want = torch.zeros((h, w), dtype=torch.uint8, device="cuda")
    got = torch.zeros((h, w), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    with bg.Runtime(0) as rt:
        bg.render_stream(rt, stream, want)
        rt.render_stream_noalloc(stream, got)
    assert bool(torch.equal(got, want))
    assert int((want != 0x40).sum()) > 0


def test_a_path_that_nearly_fills_the_area():
    """28,400 cubics of one path: their pieces and the lists of them take most of the area."""
    torch = pytest.importorskip("torch")
    n, w, h = 28400, 64, 48
    rng = np.random.Generator(np.random.PCG64(3))
    sw = scenes.StreamWriter(w, h)
    sw.solid(0xFF203040)
    sw.fill_all()
    sw.solid(0x80FF0000)
    walk = np.cumsum(rng.uniform(-0.4, 0.4, (3 * n + 1, 2)), axis=0)
    sw.fill_path([scenes.P_MOVE] + [scenes.P_CUBIC, scenes.P_CUBIC, scenes.P_ON] * n, np.abs((walk + 20.0) % 80.0 - 40.0) + 4.0)
    stream = sw.to_bytes()
    want = torch.zeros((h, w), dtype=torch.int32, device="cuda")
    got = torch.zeros((h, w), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    with bg.Runtime(0) as rt:
        bg.render_stream(rt, stream, want)
        rt.render_stream_noalloc(stream, got)
    assert bool(torch.equal(got, want))

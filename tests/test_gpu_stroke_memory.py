"""Device memory of stroked frames: the arrays of the curves' offsets go by the frame's curves, whatever
frames came before. A frame's bytes are compared with those of the same outlines drawn as paths, which
go through the same pipeline arrays."""
import numpy as np
import pytest

import blend2d_gb300 as bg
import oracle_lib
from blend2d_gb300 import scenes

pytestmark = pytest.mark.gpu

W, H, WIDTH = 320, 200, 3.0


def _polylines(paths, points):
    rng = np.random.Generator(np.random.PCG64(paths))
    return [rng.uniform(0.0, 1.0, (points, 2)) * np.array([W, H]) for _ in range(paths)]


def _curved(paths, curves, extent, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    sw = scenes.StreamWriter(W, H)
    sw.solid(0xFF102030)
    sw.fill_all()
    cmds = [scenes.P_MOVE] + [scenes.P_CUBIC, scenes.P_CUBIC, scenes.P_ON] * curves
    sw.stroke_width(WIDTH)
    for _ in range(paths):
        sw.stroke_solid(int(rng.integers(0, 2**32, dtype=np.uint64)) | 0x80000000)
        sw.stroke_path(cmds, rng.uniform(-extent, extent, (len(cmds), 2)) + np.array([W / 2, H / 2]))
    return sw.to_bytes()


def _frame_bytes(rt, stream):
    pixels = bg.render_stream(rt, stream)
    return pixels, int(rt.memory().last_frame_bytes)


def test_lines_reserve_nothing_for_curves():
    paths, points = 50, 2000
    stroked, filled = scenes.StreamWriter(W, H), scenes.StreamWriter(W, H)
    for sw in (stroked, filled):
        sw.solid(0xFF808080)
        sw.fill_all()
        sw.fill_rule(0)
        sw.solid(0xC0FF8000)
        sw.stroke_solid(0xC0FF8000)
        sw.stroke_width(WIDTH)
    for xy in _polylines(paths, points):
        cmds = np.array([scenes.P_MOVE] + [scenes.P_ON] * (points - 1), dtype=np.uint8)
        stroked.stroke_path(cmds, xy)
        filled.fill_path(*bg.stroke_outline(cmds, xy, width=WIDTH))
    with bg.Runtime(0) as a, bg.Runtime(0) as b:
        got, with_strokes = _frame_bytes(a, stroked.to_bytes())
        want, without = _frame_bytes(b, filled.to_bytes())
    assert np.array_equal(got, want)
    # the input (16 B of coordinates and a command byte per vertex), 48 B per figure and 48 B per
    # parameter set, a dozen arrays at 256-byte boundaries
    assert with_strokes - without <= paths * (17 * points + 48 + 48) + 16 * 256


def test_frames_of_long_curves_leave_later_frames_as_they_were():
    ordinary, long = _curved(300, 6, 60.0, 1), _curved(12, 2, 2.0e5, 2)
    want = oracle_lib.render(ordinary)
    with bg.Runtime(0) as rt:
        pixels, before = _frame_bytes(rt, ordinary)
        assert np.array_equal(pixels, want)
        for _ in range(50):
            bg.render_stream(rt, long)
        pixels, after = _frame_bytes(rt, ordinary)
        assert np.array_equal(pixels, want)
        assert after == before
        rt.release_memory()
        pixels, released = _frame_bytes(rt, ordinary)
        assert np.array_equal(pixels, want)
        assert released == before

"""Stroked curves offset on their own (stroke.cu): long curves whose quads exceed the pool sized for a
first frame (the figures' threads then offset them) and fit the next one's, many frames' sizes in
turn, degenerate commands between curves that leave the stroker's current point behind. Pixels
against the oracle's, bit for bit."""
import numpy as np
import pytest

import blend2d_gb300 as bg
import oracle_lib
from blend2d_gb300 import scenes

pytestmark = pytest.mark.gpu


def _long_curves(seed, extent, count):
    rng = np.random.Generator(np.random.PCG64(seed))
    sw = scenes.StreamWriter(300, 200)
    sw.solid(0xFF000000)
    sw.fill_all()
    for i in range(count):
        sw.stroke_width(float(rng.uniform(1.0, 30.0)))
        sw.stroke_join(i % 5)
        sw.stroke_caps(i % 6, (i + 1) % 6)
        sw.stroke_solid(int(rng.integers(0, 2**32, dtype=np.uint64)) | 0x80000000)
        pts = rng.uniform(-extent, extent, (7, 2)) + np.array([150.0, 100.0])
        cmds = [scenes.P_MOVE] + [scenes.P_CUBIC, scenes.P_CUBIC, scenes.P_ON] * 2
        if i % 2:
            cmds, pts = cmds + [scenes.P_CLOSE], np.vstack([pts, pts[:1]])
        sw.stroke_path(cmds, pts)
    return sw.to_bytes()


def _degenerate_steps(seed, count):
    rng = np.random.Generator(np.random.PCG64(seed))
    sw = scenes.StreamWriter(257, 131)
    sw.solid(0xFF203040)
    sw.fill_all()
    for i in range(count):
        sw.stroke_width(float(rng.uniform(0.5, 20.0)))
        sw.stroke_join(int(rng.integers(0, 5)))
        sw.stroke_caps(int(rng.integers(0, 6)), int(rng.integers(0, 6)))
        sw.stroke_solid(int(rng.integers(0, 2**32, dtype=np.uint64)) | 0x40000000)
        cmds, xy = [scenes.P_MOVE], [rng.uniform(0, 130, 2)]
        for _ in range(int(rng.integers(1, 7))):
            last, k = xy[-1], int(rng.integers(0, 7))
            p = rng.uniform(-20, 200, (3, 2))
            if k == 0:
                cmds.append(scenes.P_ON)
                xy.append(last + 1e-11)                       # too short: the current point stays
            elif k == 1:
                cmds += [scenes.P_QUAD, scenes.P_ON]
                xy += [last, p[0]]                            # control point on the start
            elif k == 2:
                cmds += [scenes.P_QUAD, scenes.P_ON]
                xy += [p[0], p[1]]
            elif k == 3:
                cmds += [scenes.P_CUBIC, scenes.P_CUBIC, scenes.P_ON]
                xy += [last, last, last]                      # a point
            elif k == 4:
                cmds += [scenes.P_CUBIC, scenes.P_CUBIC, scenes.P_ON]
                xy += [last + (p[0] - last) * 0.3, last + (p[0] - last) * 1.7, p[0]]   # straight, with a cusp
            elif k == 5:
                cmds.append(scenes.P_ON)
                xy.append(np.round(p[0]))
            else:
                cmds += [scenes.P_CUBIC, scenes.P_CUBIC, scenes.P_ON]
                xy += list(p)
        if i % 3 == 0:
            cmds.append(scenes.P_CLOSE)
            xy.append(xy[0])
        sw.stroke_path(cmds, np.array(xy))
    return sw.to_bytes()


def test_pool_overflow_and_growth():
    streams = [_long_curves(1, 2.0e5, 12), _long_curves(2, 90.0, 200), _long_curves(3, 2.0e5, 30), _long_curves(4, 3.0e4, 7)]
    cmds = np.array([scenes.P_MOVE] + [scenes.P_CUBIC, scenes.P_CUBIC, scenes.P_ON], dtype=np.uint8)
    xy = np.array([[0.0, 0.0], [2.0e5, 1.0e5], [-1.0e5, 2.0e5], [1.5e5, -2.0e5]])
    assert len(bg.stroke_outline(cmds, xy, width=10.0)[0]) > 4 * 24 + 20   # over 24 quads a curve: 2 chunks a vertex
    with bg.Runtime(0) as rt:
        for stream in streams + streams:
            assert np.array_equal(bg.render_stream(rt, stream), oracle_lib.render(stream))


@pytest.mark.parametrize("seed", [1, 2, 3, 4])
def test_degenerate_commands_between_curves(seed):
    stream = _degenerate_steps(seed, 150)
    with bg.Runtime(0) as rt:
        assert np.array_equal(bg.render_stream(rt, stream), oracle_lib.render(stream))

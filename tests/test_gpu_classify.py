"""Splitting of fill commands into lines and curves by a warp: figures and curves across its 32-vertex
steps, several figures a path, closes and moves anywhere, paths that start without a move, curves cut
off by the path's end, polygons with very large coordinates. Pixels against the oracle's, bit for bit."""
import numpy as np
import pytest

import blend2d_gb300 as bg
import oracle_lib
from blend2d_gb300 import scenes

pytestmark = pytest.mark.gpu


def _path(rng, n):
    """About n vertices of commands, with what a well-formed path has and some of what it has not."""
    cmds = []
    while len(cmds) < n:
        r = rng.random()
        if not cmds or r < 0.08:
            if cmds or rng.random() < 0.9:
                cmds.append(scenes.P_MOVE)
            else:
                cmds.append(scenes.P_ON)                      # no figure yet: skipped
        elif r < 0.35:
            cmds.append(scenes.P_ON)
        elif r < 0.6:
            cmds += [scenes.P_CUBIC, scenes.P_CUBIC, scenes.P_ON]
        elif r < 0.75:
            cmds += [scenes.P_QUAD, scenes.P_ON]
        elif r < 0.85:
            cmds += [scenes.P_CONIC, scenes.P_CONIC, scenes.P_ON]
        elif r < 0.92:
            cmds.append(scenes.P_CLOSE)
        else:
            cmds += [scenes.P_CUBIC, int(rng.integers(0, 6)), int(rng.integers(0, 6))]
    if rng.random() < 0.3:
        cmds = cmds[:n]                                       # the end may cut a curve off
    return cmds


def _scene(seed, sizes):
    rng = np.random.Generator(np.random.PCG64(seed))
    sw = scenes.StreamWriter(200, 120)
    sw.solid(0xFF101820)
    sw.fill_all()
    for n in sizes:
        sw.fill_rule(int(rng.integers(0, 2)))
        sw.solid(int(rng.integers(0, 2**32, dtype=np.uint64)) | 0x30000000)
        cmds = _path(rng, n)
        xy = rng.uniform(-40, 240, (len(cmds), 2))
        sw.fill_path(cmds, xy)
        if rng.random() < 0.3:
            xy = rng.uniform(-20, 220, (int(rng.integers(1, 70)), 2))
            if rng.random() < 0.2:                            # beyond the quick finiteness test, yet finite
                xy[int(rng.integers(0, len(xy))), int(rng.integers(0, 2))] = rng.choice([1e155, -1e160])
            sw.fill_polygon(xy)
    return sw.to_bytes()


@pytest.mark.parametrize("sizes", [[1, 2, 3, 4, 5] * 6, [31, 32, 33, 34] * 8, [63, 64, 65, 66, 97] * 5, [500, 1025]],
                         ids=["short", "one_step", "two_steps", "long"])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_items_match_the_oracle(seed, sizes):
    stream = _scene(seed, sizes)
    with bg.Runtime(0) as rt:
        assert np.array_equal(bg.render_stream(rt, stream), oracle_lib.render(stream))


def test_many_commands():
    rng = np.random.Generator(np.random.PCG64(9))             # enough commands for several a warp
    stream = _scene(5, rng.integers(1, 40, 11000).tolist())
    with bg.Runtime(0) as rt:
        assert np.array_equal(bg.render_stream(rt, stream), oracle_lib.render(stream))

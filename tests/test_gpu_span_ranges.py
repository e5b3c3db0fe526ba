"""The rasterizers' span arithmetic outside its short path.

A span whose 1/depth ends, edge distance or first column lie outside the
ranges in which the reciprocal path is exact is drawn by its lane alone with
true divisions (csrc/kernels.cuh, span_put / z_safe).  Scaling the whole world
by a power of two moves 1/depth across both limits (2^58 and 2^-30 for whole
items) and leaves the screen positions as they are, so the same triangles are
drawn by one path, by the other, or some by each: depth, ids, colour and
shadow maps must equal the oracle's bit for bit at every scale.
"""
import dataclasses

import numpy as np
import pytest

import oracle as O
from axi_visualizer_b200 import scenes as S
from axi_visualizer_b200.ops import SceneRenderer

from test_gpu_edges import assert_same

pytestmark = pytest.mark.gpu


def scaled(sc, view, k):
    s = np.float32(2.0 ** k)
    groups = [dataclasses.replace(g, xyz=g.xyz * s) for g in sc.groups]
    shadows = [dataclasses.replace(c, pos=c.pos * s, scale=float(np.float32(c.scale) / s)) for c in sc.shadows]
    return (dataclasses.replace(sc, groups=groups, shadows=shadows, bias=float(np.float32(sc.bias) * s)),
            dataclasses.replace(view, pos=view.pos * s))


# depths are about 5 to 60 units: 1/depth straddles 2^58 at k = -62, lies above
# it at k = -66, straddles 2^-30 at k = 26 and lies below it at k = 30
@pytest.mark.parametrize("k", [-66, -62, 0, 26, 30])
@pytest.mark.parametrize("pos", [(0, 8, -30), (3, 2, -8)])
def test_world_scales_equal_oracle(k, pos):
    sc, view = scaled(S.scene_small(seed=4, flags=S.MIP), S.default_view(320, 250, pos=pos), k)
    clear = np.float32(65535.0 if k <= 0 else 3e38)      # beyond every depth of the scene
    smaps = []
    for i, c in enumerate(sc.shadows):
        m = O.new_shadow_map(c.dim)
        O.shadow_map(sc, i, m)
        smaps.append(m)
    fr = O.Frame(view.w, view.h)
    fr.db[:] = clear
    O.draw_all(sc, view, fr, [])
    R = SceneRenderer(sc, view.w, view.h)
    R.shadow_pass()
    R.set_view(view)
    R.draw.setFrame(depth=np.full((view.h, view.w), clear, np.float32))
    R.draw.drawAll(R.shaders, shadowIds=[])
    r, g, b, db = [x.copy() for x in R.draw.getFrame()]
    tid, cov = R.draw.getIDs()
    assert cov.mean() > 0.2
    assert_same(fr, smaps, (r, g, b, db, tid, cov, [R.draw.getSHM(i) for i in range(len(sc.shadows))]))

"""vertLight at the edges of its reciprocal path and of its vertex quads.

A light's offset of a length outside [2^-30, 2^30], or a product too small for
the reciprocal's range, takes true divisions (csrc/kernels.cuh, light_at), and a
group's last vertices (3 T is no multiple of 4) go one by one; groups of
several sizes share one launch.  Positions scaled by powers of two, vertices on
top of a light and tiny normals: the light must equal the oracle's bit for bit.
"""
import numpy as np
import pytest

import oracle as O
from axi_visualizer_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [-40, -32, 0, 29, 40])
def test_vert_light_ranges_equal_oracle(k):
    from axi_visualizer_b200.ops import CLDraw
    rng = np.random.default_rng(3)
    s = np.float32(2.0 ** k)
    f = lambda *shape: rng.standard_normal(shape).astype(np.float32)   # noqa: E731
    pp, sp, sd = f(5, 3) * s, f(3, 3) * s, f(3, 3)
    pi, si = np.abs(f(5, 3)), np.abs(f(3, 3))
    d = CLDraw(1, 64, 64, 64, 1)
    d.ambLight = np.float32(0.01)
    tex = [np.zeros(4, np.uint16)] * 3
    groups = []
    for tris in (1, 2, 3, 86, 1001):
        xyz, vn, uv = f(3 * tris, 3) * s, f(3 * tris, 3), np.zeros((3 * tris, 2), np.float32)
        xyz[0] = pp[0]                       # on a light
        vn[1] *= np.float32(1e-25)           # products below the reciprocal's range
        d.addTextureGroup(xyz, uv, vn, *tex)
        groups.append((xyz, vn))
    di, dd = np.asarray(S.LIGHT_INTS, np.float32), np.asarray(S.LIGHT_DIRS, np.float32)
    mask = np.array([1, 1, 0, 1, 1], np.uint8)
    d.vertLight(mask, di, dd, pi, pp, si, sd, sp)
    for tn, (xyz, vn) in enumerate(groups):
        got = d.getVertices(tn)[2]
        want = O.vert_light(xyz, vn, di, dd, 0.01, pi, pp, si, sd, sp) if mask[tn] else np.zeros_like(vn)
        assert np.array_equal(got.view(np.uint32), np.asarray(want, np.float32).view(np.uint32)), f"group {tn}"

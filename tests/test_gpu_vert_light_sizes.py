"""vertLight's launches by size: one vertex a thread for small groups, four for
large ones (from 1,024 vertices an SM), groups of both sizes and more than four
groups in one call, against the oracle bit for bit."""
import numpy as np
import pytest

import oracle as O
from axi_visualizer_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(5,), (60000,), (1, 60001, 33, 2, 700)])
def test_vert_light_sizes_equal_oracle(sizes):
    from axi_visualizer_b200.ops import CLDraw
    rng = np.random.default_rng(4)
    f = lambda *shape: rng.standard_normal(shape).astype(np.float32)   # noqa: E731
    pp, sp, sd, pi, si = f(3, 3), f(2, 3), f(2, 3), np.abs(f(3, 3)), np.abs(f(2, 3))
    di, dd = np.asarray(S.LIGHT_INTS, np.float32), np.asarray(S.LIGHT_DIRS, np.float32)
    d = CLDraw(1, 64, 64, 64, 1)
    d.ambLight = np.float32(0.05)
    groups = []
    for tris in sizes:
        xyz, vn = f(3 * tris, 3), f(3 * tris, 3)
        d.addTextureGroup(xyz, np.zeros((3 * tris, 2), np.float32), vn, *[np.zeros(4, np.uint16)] * 3)
        groups.append((xyz, vn))
    d.vertLight([1] * len(sizes), di, dd, pi, pp, si, sd, sp)
    for tn, (xyz, vn) in enumerate(groups):
        want = O.vert_light(xyz, vn, di, dd, 0.05, pi, pp, si, sd, sp)
        assert np.array_equal(d.getVertices(tn)[2].view(np.uint32), want.view(np.uint32)), f"group {tn}"

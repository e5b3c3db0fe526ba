"""vertLight's two forms at the line between them: one vertex a thread below
2,048 vertices an SM (303,104 on 148 SMs) over all groups of a call, four from
there on, with groups whose sizes are no multiple of four, against the oracle
bit for bit."""
import numpy as np
import pytest

import oracle as O
from axi_visualizer_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(101034,), (101035,), (50500, 50501, 33, 2), (1, 100000, 1000, 2, 33, 1), (40000, 20003) * 2])
def test_vert_light_forms_equal_oracle(sizes):
    from axi_visualizer_b200.ops import CLDraw
    rng = np.random.default_rng(6)
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

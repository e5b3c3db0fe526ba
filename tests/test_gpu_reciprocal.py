"""The rasterizers' reciprocal at the one value where it could be wrong.

recip_rn (csrc/raster.cuh) takes an approximate reciprocal, within one ulp, and
one residual step.  Tried for every mantissa and every such start, the step
rounds correctly except from 0.5 for 1.99999988 (mantissa 0x7fffff), where the
result depends on the approximation the GPU gives.
"""
import numpy as np
import pytest

import kat
import oracle as O
from axi_visualizer_b200 import scenes as S
from axi_visualizer_b200.ops import SceneRenderer

from test_gpu_depth_ratios import BASIS, H, W, bits, finish
from test_gpu_edges import assert_same

pytestmark = pytest.mark.gpu

HALF = np.float32(0.5)
NEXT = np.nextafter(HALF, np.float32(1))            # 0.50000006
TWO_DOWN = np.nextafter(np.float32(2), np.float32(0))   # 1.99999988, mantissa 0x7fffff
BACK = np.float32(1) / NEXT                              # the depth that 1 / (1 / TWO_DOWN) gives


@pytest.mark.parametrize("k", [-20, 0, 12])
def test_reciprocal_of_the_largest_mantissa(k):
    """1 / 1.99999988 lies above the midpoint of 0.5 and 0.50000006.  The value
    is reached as a vertex depth (projection) and as an interpolated 1/depth:
    from 2 at the vertex to 1.99999976 two rows on, the row between holds
    1.99999988, exactly.  Small, tiled and caster triangles, scaled by powers
    of two."""
    s = np.float32(2.0 ** k)
    a, b, d = float(HALF * s), float(NEXT * s), float(TWO_DOWN * s)
    assert np.float32(1) / TWO_DOWN == NEXT
    wedge = lambda x, y, n: [(x, y, a), (x - 5, y + 2, b), (x + n, y + 2, b)]   # noqa: E731
    flat = lambda x, y, n: [(x, y, d), (x + n, y + 1, d), (x, y + n, d)]        # noqa: E731
    pts = [wedge(20.0, 16.0, 30), wedge(20.0, 33.0, 200), flat(40.0, 60.0, 40), flat(100.0, 60.0, 150)]
    rng = np.random.default_rng(5)
    view = kat.view(W, H)
    sc = finish([kat._group([kat.tri(W, H, p) for p in pts], rng)])
    fr = O.Frame(W, H)
    O.clear_depth(fr.db)
    O.draw_all(sc, view, fr, [])
    assert all((fr.db[y] == v * s).any() for y, v in ((17, NEXT), (34, NEXT), (80, BACK)))
    R = SceneRenderer(sc, W, H)
    R.set_view(view)
    R.draw.clearZBuffer()
    R.draw.drawAll(R.shaders, shadowIds=[])
    r, g, bl, db = [x.copy() for x in R.draw.getFrame()]
    tid, cov = R.draw.getIDs()
    assert_same(fr, [], (r, g, bl, db, tid, cov, []))

    cam = S.ShadowCam(256, 1.0, np.zeros(3, np.float32), BASIS)
    sh = finish([kat._group([[(128 - x, 128 - y, z) for x, y, z in p] for p in pts], rng)], [cam])
    want = O.new_shadow_map(256)
    O.shadow_map(sh, 0, want)
    assert (want[17] == NEXT * s).any() and (want[80] == BACK * s).any()
    R = SceneRenderer(sh, 64, 48)
    for mode in (0, 2):
        R.draw.setShadowMode(mode)
        R.draw.clearShadowMap(0)
        R.draw.shadowMap(0, [True], R.shaders, sh.bias)
        assert np.array_equal(bits(R.draw.getSHM(0)), bits(want)), mode

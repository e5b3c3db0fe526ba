"""Triangles and casters whose vertices' depths differ by large factors.

The interpolated 1/depth drifts by up to 2^-24 of the LARGEST vertex value a
row, so where the values of one triangle differ by more than about 2^24 / rows
its walk can end at zero or below: such fragments have negative depths (they
pass the depth test before every positive one) or none.  The rasterizers draw
such items by lane with true divisions (csrc/kernels.cuh, z_safe); frames and
maps must equal the oracle's bit for bit on both sides of that rule, opaque and
alpha-tested, through the handle, the tiled shadow pass and both batch forms.
"""
import numpy as np
import pytest

import kat
import oracle as O
from axi_visualizer_b200 import scenes as S
from axi_visualizer_b200.batch import PERSISTENT, PHASED, Batch, depth, shaded
from axi_visualizer_b200.ops import SceneRenderer

from test_gpu_edges import assert_same

pytestmark = pytest.mark.gpu

W, H = 320, 256
BASIS = np.array([[0, 0, 1], [-1, 0, 0], [0, 1, 0]], np.float32)


def finish(groups, shadows=(), flags=0):
    m = (np.indices((16, 16)).sum(0) % 3 > 0).astype(np.uint8)
    alphas = [(m.reshape(-1), 16)] if flags & S.ALPHA else []
    return S.Scene(groups, alphas, np.asarray(S.LIGHT_INTS[0], np.float32), S.LIGHT_DIRS[0].astype(np.float32), 0.2,
                   list(shadows), bias=0.0)


def bits(a):
    return a.view(np.uint32)


def ratio_view(log_ratio, flags):
    """Small triangles with one vertex at depth 1e-5 and two 2^log_ratio times
    as far, over triangles at depth 0.5."""
    rng = np.random.default_rng(100 + log_ratio)
    far = 1e-5 * 2.0 ** log_ratio
    tris = [kat.tri(W, H, [(100.5, 100.5, 1e-5), (60.5, 134.5, far), (120.5, 159.5, far)])]
    for _ in range(120):
        x, y = rng.uniform(10, W - 100), rng.uniform(10, H - 100)
        p = [(x + rng.uniform(0, 90), y + rng.uniform(0, 90)) for _ in range(3)]
        z = [1e-5, far, far * rng.uniform(0.5, 2)]
        rng.shuffle(z)
        tris.append(kat.tri(W, H, [(a, b, c) for (a, b), c in zip(p, z)]))
    back = [kat.tri(W, H, [(5.5, 60.5, 0.5), (200.5, 60.5, 0.5), (60.5, 230.5, 0.5)]),
            kat.tri(W, H, [(250.5, 10.5, 0.5), (310.5, 60.5, 0.5), (260.5, 70.5, 0.5)])]
    uv = np.random.default_rng(3).uniform(0, 1, (len(tris) * 3, 2))
    return finish([kat._group(tris, rng, flags, uv=uv), kat._group(back, rng)], flags=flags)


@pytest.mark.parametrize("flags", [0, S.ALPHA])
@pytest.mark.parametrize("log_ratio", [14, 17, 20, 24, 28])
def test_view_depth_ratios_equal_oracle(log_ratio, flags):
    sc, view = ratio_view(log_ratio, flags), kat.view(W, H)
    fr = O.Frame(W, H)
    O.clear_depth(fr.db)
    O.draw_all(sc, view, fr, [])
    if log_ratio >= 24:
        assert (fr.db < 0).any()
    R = SceneRenderer(sc, W, H)
    R.set_view(view)
    R.draw.clearZBuffer()
    R.draw.drawAll(R.shaders, shadowIds=[])
    r, g, b, db = [x.copy() for x in R.draw.getFrame()]
    tid, cov = R.draw.getIDs()
    assert_same(fr, [], (r, g, b, db, tid, cov, []))
    gf, ai = [g.flags for g in sc.groups], [g.alpha_index for g in sc.groups]
    B = Batch(R.draw, [shaded(view)])
    for mode in (PERSISTENT, PHASED):
        B.set_mode(mode)
        B.render(gf, ai)
        assert np.array_equal(bits(B.frame(0)[3]), bits(fr.db)), mode
        assert np.array_equal(B.ids(0)[0], fr.tri_id), mode


def ratio_casters(dim, log_ratio, flags, n=40):
    """Overlapping casters of up to the map's whole height: vertices about
    2^log_ratio apart in depth, the near ones just in front of the light.  Each
    comes three times at different distances, so that negative depths, where a
    walk ends there, compete for a texel."""
    rng = np.random.default_rng(log_ratio * 7 + dim)
    tris = []
    for _ in range(n):
        x = rng.uniform(0.1, 0.8) * dim
        pts = [(x + rng.uniform(0, 60), rng.uniform(-0.01, 0.3) * dim), (x + rng.uniform(0, 60), rng.uniform(0.2, 0.9) * dim),
               (x + rng.uniform(0, 60), rng.uniform(0.7, 1.01) * dim)]
        z = [30.0 * 2.0 ** -log_ratio * rng.uniform(1, 2), rng.uniform(1, 30), rng.uniform(10, 30)]
        rng.shuffle(z)
        for far in (1.0, 1.3, 0.8):
            tris.append([(dim // 2 - a, dim // 2 - b, c * far) for (a, b), c in zip(pts, z)])
    uv = rng.uniform(0, 3, (3 * len(tris), 2))
    cam = S.ShadowCam(dim, 1.0, np.zeros(3, np.float32), BASIS)
    return finish([kat._group(tris, rng, flags, uv=uv)], [cam], flags)


@pytest.mark.parametrize("flags", [0, S.ALPHA])
@pytest.mark.parametrize("dim,log_ratio", [(256, 12), (256, 18), (256, 24), (4096, 9), (4096, 15), (4096, 19)])
def test_caster_depth_ratios_equal_oracle(dim, log_ratio, flags):
    sc = ratio_casters(dim, log_ratio, flags)
    want = O.new_shadow_map(dim)
    O.shadow_map(sc, 0, want)
    if (dim, log_ratio) in ((256, 24), (4096, 19)):
        assert (want < 0).any()
    R = SceneRenderer(sc, 64, 48)
    for mode in (0, 1, 2):
        R.draw.setShadowMode(mode)
        R.draw.clearShadowMap(0)
        R.draw.shadowMap(0, [True], R.shaders, sc.bias)
        assert np.array_equal(bits(R.draw.getSHM(0)), bits(want)), mode
    B = Batch(R.draw, [depth(sc.shadows[0], sc.bias)])
    for mode in (PERSISTENT, PHASED):
        B.set_mode(mode)
        B.render([g.flags for g in sc.groups], [g.alpha_index for g in sc.groups])
        assert np.array_equal(bits(B.frame(0)), bits(want)), mode

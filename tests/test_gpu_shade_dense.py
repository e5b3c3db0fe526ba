"""The shade of dense views (from 1.5 drawn triangles a pixel), which sets tiles
with many winners up by (winner, row) pair: views whose tiles hold few, some and
nearly one winner a pixel, every material's fragment core, a height that is no
multiple of the tile, through the handle and both batch forms; the frames equal
the oracle's bit for bit."""
import numpy as np
import pytest

from axi_visualizer_b200 import scenes as S
from axi_visualizer_b200.batch import PERSISTENT, PHASED, Batch, scene_batch_views

from test_gpu_parity import check_frame, render_both
from test_gpu_shade_winners import winners

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("build", [
    lambda: S.scene_small(seed=6, terrain_n=96, spheres=150, flags=S.MIP | S.SHADOW),
    lambda: S.scene_normal(seed=6, terrain_n=96, spheres=150),
    lambda: S.scene_multi(seed=6, terrain_n=96, cell=2.0, spheres=60),
], ids=["mip_shadow_alpha", "normal", "multi"])
@pytest.mark.parametrize("dist,most", [(15.0, 1), (80.0, 33), (250.0, 130)])
def test_dense_views_equal_oracle(build, dist, most):
    sc = build()
    view = S.default_view(96, 75, pos=(0.0, dist * 0.8, -dist))
    assert 2 * sc.ntris >= 3 * view.w * view.h
    fr, smaps, got, R = render_both(sc, view)
    assert winners(got[4]) >= most
    assert check_frame(fr, smaps, got)[0] == 1.0
    views = scene_batch_views(sc, view)
    B = Batch(R.draw, views)
    for mode in (PERSISTENT, PHASED):
        B.set_mode(mode)
        B.render([g.flags for g in sc.groups], [g.alpha_index for g in sc.groups])
        rows = view.h // 4 * 4            # a batch's clear covers whole blocks of four rows (clearzb.c)
        for a, b in zip(B.frame(len(views) - 1), got[:4]):
            assert np.array_equal(a[:rows].view(np.uint8), b[:rows].view(np.uint8)), mode

"""The shade pass on tiles with many winners.

A tile's winners (visible triangle halves) are set up 32 at a time
(csrc/kernels.cuh, shade_tile).  Views of fine meshes from afar give tiles with
one to well over 32 winners, up to one a pixel; the frame must equal the
oracle's bit for bit for every material's fragment core, on a frame whose
height is no multiple of the tile.
"""
import numpy as np
import pytest

from axi_visualizer_b200 import scenes as S

from test_gpu_parity import check_frame, render_both

pytestmark = pytest.mark.gpu


def winners(tid):
    h = tid.shape[0] // 16 * 16
    tiles = tid[:h].reshape(h // 16, 16, -1, 16).transpose(0, 2, 1, 3).reshape(-1, 256)
    return max(len(np.unique(t[t >= 0])) for t in tiles)


@pytest.mark.parametrize("build", [
    lambda: S.scene_small(seed=5, terrain_n=96, spheres=150, flags=S.MIP | S.SHADOW),
    lambda: S.scene_normal(seed=5, terrain_n=96, spheres=150),
    lambda: S.scene_multi(seed=5, terrain_n=96, cell=2.0, spheres=60),
], ids=["mip_shadow_alpha", "normal", "multi"])
@pytest.mark.parametrize("dist,most", [(150.0, 33), (400.0, 65)])
def test_tiles_with_many_winners_equal_oracle(build, dist, most):
    sc = build()
    view = S.default_view(160, 123, pos=(0.0, dist * 0.6, -dist))
    fr, smaps, got, _ = render_both(sc, view)
    assert winners(got[4]) >= most
    assert check_frame(fr, smaps, got)[0] == 1.0

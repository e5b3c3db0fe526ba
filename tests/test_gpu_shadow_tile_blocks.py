"""The tiled shadow pass with several blocks a tile and most of them without
units left: every warp of a block has to work on the block's own tile (csrc/
shadow_tiles.cuh, k_shadow_tiles).  Tall casters over a 2048 map, small slices
of units a block, repeated passes; each map equals the oracle's bit for bit.
"""
import numpy as np
import pytest

import kat
import oracle as O
from axi_visualizer_b200 import scenes as S
from axi_visualizer_b200.ops import SceneRenderer

pytestmark = pytest.mark.gpu

DIM = 2048


@pytest.mark.parametrize("flags", [0, S.ALPHA])
def test_many_blocks_a_tile_equal_oracle(flags):
    rng = np.random.default_rng(31)
    tris = []
    for _ in range(150):
        x = rng.uniform(0.05, 0.9) * DIM
        ys = rng.uniform(-0.01, 1.01, 3) * DIM
        tris.append([(DIM // 2 - x - rng.uniform(0, 60), DIM // 2 - y, rng.uniform(1, 30)) for y in ys])
    m = (np.indices((16, 16)).sum(0) % 3 > 0).astype(np.uint8)
    cam = S.ShadowCam(DIM, 1.0, np.zeros(3, np.float32), np.array([[0, 0, 1], [-1, 0, 0], [0, 1, 0]], np.float32))
    sc = S.Scene([kat._group(tris, rng, flags, uv=rng.uniform(0, 3, (450, 2)))], [(m.reshape(-1), 16)] if flags else [],
                 np.asarray(S.LIGHT_INTS[0], np.float32), S.LIGHT_DIRS[0].astype(np.float32), 0.2, [cam], bias=0.0)
    want = O.new_shadow_map(DIM)
    O.shadow_map(sc, 0, want)
    R = SceneRenderer(sc, 64, 48)
    for rep in range(8):
        for mode, slice_ in ((1, 512), (2, 512), (1, 32), (2, 32)):
            R.draw.setShadowMode(mode, slice_)
            R.draw.clearShadowMap(0)
            R.draw.shadowMap(0, [True], R.shaders, sc.bias)
            assert np.array_equal(R.draw.getSHM(0).view(np.uint32), want.view(np.uint32)), (rep, mode, slice_)

"""Short work queues: fewer items than the GPU has warps, a few casters on maps
of many texels, where the rasterizers claim fewer items at a time.  Frames and
maps equal the oracle's bit for bit."""
import numpy as np
import pytest

import kat
import oracle as O
from axi_visualizer_b200 import scenes as S
from axi_visualizer_b200.ops import SceneRenderer

from test_gpu_depth_ratios import BASIS, bits, finish

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, S.ALPHA])
@pytest.mark.parametrize("dim", [64, 1000, 2048])
@pytest.mark.parametrize("n", [1, 9, 300])
def test_few_casters_equal_oracle(n, dim, flags):
    rng = np.random.default_rng(n + dim)
    tris = [[(dim / 2 - x, dim / 2 - y, z) for x, y, z in zip(*(rng.uniform(-0.02, 1.02, (2, 3)) * dim), rng.uniform(1, 30, 3))]
            for _ in range(n)]
    cam = S.ShadowCam(dim, 1.0, np.zeros(3, np.float32), BASIS)
    sc = finish([kat._group(tris, rng, flags, uv=rng.uniform(0, 3, (3 * n, 2)))], [cam], flags)
    want = O.new_shadow_map(dim)
    O.shadow_map(sc, 0, want)
    R = SceneRenderer(sc, 64, 48)
    R.draw.clearShadowMap(0)
    R.draw.shadowMap(0, [True], R.shaders, sc.bias)
    assert np.array_equal(bits(R.draw.getSHM(0)), bits(want))
    w, h = 320, 192
    view = kat.view(w, h)
    tris = []
    for _ in range(n):
        x, y, s = rng.uniform(0, w), rng.uniform(0, h), rng.choice([9.0, 60.0, 200.0])
        tris.append(kat.tri(w, h, [(x + rng.uniform(-s, s), y + rng.uniform(-s, s), rng.uniform(2, 20)) for _ in range(3)]))
    vs = finish([kat._group(tris, rng, flags, uv=rng.uniform(0, 3, (3 * n, 2)))], [], flags)
    fr = O.Frame(w, h)
    O.clear_depth(fr.db)
    O.draw_all(vs, view, fr, [])
    R = SceneRenderer(vs, w, h)
    R.set_view(view)
    R.draw.clearZBuffer()
    R.draw.drawAll(R.shaders, shadowIds=[])
    assert np.array_equal(bits(R.draw.getFrame()[3]), bits(fr.db)) and np.array_equal(R.draw.getIDs()[0], fr.tri_id)

"""The post effects at the edges of their tiles, against the oracle bit for bit.

The bloom takes 128 columns and 63 x 15 half-resolution tiles a block and its
lower vertical taps end at the half width (frames taller than wide); ssao
walks 16 x 16 tiles with a fixed grid and skips pixels beyond depth 6000; dof
stages a 4-pixel halo; gamma and the 8-bit read-back take 8 and 4 pixels a
thread.  Frames are seeded noise over the whole range of the planes, depths
from near to the clear value.
"""
import numpy as np
import pytest

import oracle as O
from axi_visualizer_b200 import scenes as S

pytestmark = pytest.mark.gpu


def noise_frame(w, h, seed):
    rng = np.random.default_rng(seed)
    fr = O.Frame(w, h)
    for name in ("ro", "go", "bo"):
        a = (65535 * rng.random((h, w)) ** 3).astype(np.uint16)
        a[rng.random((h, w)) < 0.05] = 65535
        setattr(fr, name, a)
    fr.db = rng.uniform(1.5, 60.0, (h, w)).astype(np.float32)
    fr.db[rng.random((h, w)) < 0.15] = 65535.0
    fr.db[rng.random((h, w)) < 0.02] = 6000.0
    return fr


@pytest.mark.parametrize("w,h", [(16, 6), (16, 40), (48, 33), (64, 222), (128, 30), (128, 250), (272, 61), (400, 31),
                                 (1040, 62)])
def test_post_effects_equal_oracle(w, h):
    from axi_visualizer_b200.ops import CLDraw
    view = S.default_view(w, h)
    d = CLDraw(1, 64, w, h, 1)
    d.setScaleCull(view.sscale, view.cax, view.cay)
    rnd = np.random.default_rng(7).random(48).astype(np.float32)

    def same(fr, what):
        r, g, b, _ = d.getFrame()
        assert np.array_equal(r, fr.ro) and np.array_equal(g, fr.go) and np.array_equal(b, fr.bo), what

    for seed in (1, 2):
        fr = noise_frame(w, h, seed)
        d.setFrame(fr.ro, fr.go, fr.bo, fr.db)
        if w >= 16 and h >= 16:
            O.ssao(fr, view.sscale, rnd)
            for f in (3.0, 20.0):
                O.dof(fr, f)
        d.ssao(rnd)
        for f in (3.0, 20.0):
            d.dof(f)
        same(fr, "ssao, dof")
        O.bloom(fr)
        d.blur()
        same(fr, "bloom")
        ex = (0.5, 2.0)[seed - 1]
        packed = d.readFrameRGB8Async(ex)
        rgb = d.waitFrame(packed).copy()
        O.gamma(fr, ex)
        d.gamma(ex)
        same(fr, "gamma")
        assert np.array_equal(rgb, np.stack((fr.ro, fr.go, fr.bo), -1).astype(np.uint8)), "8-bit read-back"

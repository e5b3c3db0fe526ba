"""ssao at the edges of the ranges in which its samples need no checks of their
own, against the oracle bit for bit: depths on both sides of 1.5 and of 4, tables whose
scaled lengths are below, at and beyond 1, scales inside and outside
[1, 2^20], flat and noisy depths, heights that are
no multiple of 16.
"""
import numpy as np
import pytest

import oracle as O
from axi_visualizer_b200 import scenes as S

pytestmark = pytest.mark.gpu


def depths(kind, w, h, rng):
    if kind == "near":                          # both sides of the bound, and values next to it
        return rng.choice(np.array([3.9999998, 4.0, 4.0000005, 1e-3, 0.5, 5.0], np.float32), (h, w))
    if kind == "mixed":                         # both sides of 1.5 within a warp
        return rng.choice(np.array([1.4999999, 1.5, 1.5000001, 1.6, 7.0, 0.2], np.float32), (h, w))
    if kind == "close":                         # at and above 1.5 only
        return rng.choice(np.array([1.5, 1.5000001, 1.75, 2.5], np.float32), (h, w))
    if kind == "flat":
        return np.full((h, w), 9.0, np.float32)
    if kind == "far":
        return rng.choice(np.array([5999.5, 6000.0, 6000.0005, 65535.0], np.float32), (h, w))
    y, x = np.mgrid[:h, :w]
    return (4.0 + 0.02 * x + 0.03 * y + 0.3 * rng.random((h, w))).astype(np.float32)      # surfaces


@pytest.mark.parametrize("kind", ["near", "mixed", "close", "flat", "far", "surface"])
@pytest.mark.parametrize("table", [1.0, 1.1, 3.0])
@pytest.mark.parametrize("scale", [None, 0.75, 1.0, 2.0 ** 20, 2.0 ** 21])
def test_ssao_equals_oracle(kind, table, scale):
    from axi_visualizer_b200.ops import CLDraw
    rng = np.random.default_rng(11)
    rnd = (rng.random(48) * table).astype(np.float32)
    for w, h in ((16, 16), (80, 50), (160, 96)):
        view = S.default_view(w, h)
        ss = view.sscale if scale is None else scale
        d = CLDraw(1, 64, w, h, 1)
        d.setScaleCull(ss, view.cax, view.cay)
        fr = O.Frame(w, h)
        for name in ("ro", "go", "bo"):
            setattr(fr, name, rng.integers(0, 65536, (h, w)).astype(np.uint16))
        fr.db = np.ascontiguousarray(depths(kind, w, h, rng))
        d.setFrame(fr.ro, fr.go, fr.bo, fr.db)
        O.ssao(fr, ss, rnd)
        d.ssao(rnd)
        r, g, b, _ = d.getFrame()
        assert np.array_equal(r, fr.ro) and np.array_equal(g, fr.go) and np.array_equal(b, fr.bo), (w, h)

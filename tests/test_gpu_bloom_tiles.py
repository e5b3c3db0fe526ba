"""The bloom at the edges of its vertical pass's tiles (62 x 31 half-resolution
pixels a block and one more column and row): half widths that end on, before and
past a tile's columns, half heights whose last tile is one row or a whole one;
against the oracle bit for bit."""
import numpy as np
import pytest

import oracle as O

from test_gpu_post_shapes import noise_frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(496, 64), (512, 62), (480, 126), (992, 124), (1008, 128), (64, 66), (16, 186)])
def test_bloom_tile_edges_equal_oracle(w, h):
    from axi_visualizer_b200.ops import CLDraw
    d = CLDraw(1, 64, w, h, 1)
    for seed in (3, 4):
        fr = noise_frame(w, h, seed)
        d.setFrame(fr.ro, fr.go, fr.bo, fr.db)
        O.bloom(fr)
        d.blur()
        r, g, b, _ = d.getFrame()
        assert np.array_equal(r, fr.ro) and np.array_equal(g, fr.go) and np.array_equal(b, fr.bo), seed

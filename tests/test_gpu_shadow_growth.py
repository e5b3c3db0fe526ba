"""shadowMap learns of its map's finished passes before it queues another.

The tile-unit queue of the tiled pass grows after a pass that overflowed it.
Once that pass has finished, the next shadowMap call has to see it, also when
nothing else of the handle is called: the second pass is tiled.
"""
import numpy as np
import pytest

import oracle as O
from axi_visualizer_b200 import scenes as S
from axi_visualizer_b200.ops import SceneRenderer

pytestmark = pytest.mark.gpu


def test_second_pass_has_the_grown_queue(monkeypatch):
    import torch
    monkeypatch.setenv("AXR_SHADOW_UNIT_QUEUE", "7")
    sc = S.scene_small(seed=4)
    want = O.new_shadow_map(sc.shadows[0].dim)
    O.shadow_map(sc, 0, want)
    R = SceneRenderer(sc, 64, 48)
    R.draw.setShadowMode(1)
    for _ in range(2):
        R.draw.clearShadowMap(0)
        R.draw.shadowMap(0, [g.cast for g in sc.groups], R.shaders, sc.bias)
        torch.cuda.synchronize()          # finished, and nothing of the handle called
    overflows, units, capacity, _, _ = R.draw.shadowStats(0).values()
    assert overflows == 1 and units <= capacity
    assert np.array_equal(R.draw.getSHM(0).view(np.uint32), want.view(np.uint32))

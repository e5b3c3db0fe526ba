"""Device allocations that fail, made to fail on the host.

Each case runs in a child process with a shim in front of cudaMalloc that, when
armed, lets a chosen later call ask the runtime for more memory than any GPU
has.  The call that needed the memory reports it, and the handle draws the next
frames exactly.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static int left = -1;
void shim_fail(int after) { left = after; }   /* the call number `after` from now; -1: none */
int cudaMalloc(void **p, size_t n) {
  static int (*real)(void **, size_t);
  if (!real) real = (int (*)(void **, size_t))dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), "cudaMalloc");
  return real(p, left >= 0 && left-- == 0 ? (size_t)1 << 60 : n);
}
"""
COMMON = """
import ctypes, os, sys
sys.path[:0] = sys.argv[1:4]
import numpy as np, pytest
import oracle as O
from axi_visualizer_b200 import scenes as S
from axi_visualizer_b200._lib import AxrError
from axi_visualizer_b200.ops import SceneRenderer
shim = ctypes.CDLL(os.environ["LD_PRELOAD"])
sc = S.scene_small(seed=1, flags=S.MIP | S.SHADOW)
views = [S.default_view(320, 240, pos=p) for p in ((3, 2, -8), (2, 3, -9), (1, 2, -7))]
want = [O.render(sc, v)[0] for v in views]
R = SceneRenderer(sc, 320, 240)

def exact(k):
    db = R.draw.getFrame()[3]
    assert np.array_equal(db.view(np.uint32), want[k].db.view(np.uint32)), k
"""
CASES = {
    # the tile-unit queue cannot grow after an overflow: later frames overflow
    # again and are drawn by the fallback, until it can
    "unit_queue": """
R.frame(views[0])
shim.shim_fail(0)
with pytest.raises(AxrError, match="tile-unit queue"):
    R.draw.sync()
for k in (1, 2):
    R.frame(views[k])
    assert R.draw.lastStats()["n_units"] > 16
    exact(k)
""",
    # the same while a frame is being drawn, which learns of the overflow of the
    # frame before last: it reports that, and is complete all the same
    "unit_queue_mid_frame": """
import torch
slow = torch.cuda.ExternalStream(R.draw.stream_ptr())
with torch.cuda.stream(slow):
    torch.cuda._sleep(200_000_000)    # both frames are still unfinished when the third is drawn
R.frame(views[0])
R.frame(views[1])
R.shadow_pass()
R.set_view(views[2])
R.draw.clearZBuffer()
shim.shim_fail(0)
with pytest.raises(AxrError, match="tile-unit queue"):
    R.draw.drawAll(R.shaders, shadowIds=[0, 1])
exact(2)
R.frame(views[1])
exact(1)
""",
    # a shadow map without its counters does not exist, and can be made later
    "shadow_map": """
from axi_visualizer_b200.batch import Batch, shaded
cam = sc.shadows[0]
flags = [g.flags for g in sc.groups]
B = Batch(R.draw, [shaded(views[0], (-1, -2))])
shim.shim_fail(1)
with pytest.raises(AxrError, match="shadow map 96x96"):
    R.draw.addShadowMap(0, 96, cam.scale, 0.2)
with pytest.raises(AxrError, match="does not exist"):
    R.draw.shadowMap(0, [g.cast for g in sc.groups], R.shaders, sc.bias)
with pytest.raises(AxrError, match="does not exist"):
    B.render(flags)
R.draw.addShadowMap(0, cam.dim, cam.scale, 0.2)
for k in range(3):
    R.frame(views[k])
    exact(k)
B.render(flags, [g.alpha_index for g in sc.groups])
assert np.array_equal(B.frame(0)[3].view(np.uint32), want[0].db.view(np.uint32))
""",
    # the triangle lists cannot grow for another group: it is not added, and the
    # others are drawn as before
    "triangle_lists": """
g = sc.groups[0]
planes = sc.groups[2].tex
shim.shim_fail(5)                     # after the group's five arrays
with pytest.raises(AxrError, match="triangle lists"):
    R.draw.addTextureGroup(np.concatenate([g.xyz] * 40), np.concatenate([g.uv] * 40), np.concatenate([g.vn] * 40), *planes)
for k in range(3):
    R.frame(views[k])
    exact(k)
""",
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_failed_allocation(case, tmp_path):
    src, so = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", str(so), str(src), "-ldl"], check=True)
    root = os.path.dirname(HERE)
    env = dict(os.environ, LD_PRELOAD=str(so), AXR_UNIT_QUEUE="16")
    r = subprocess.run([sys.executable, "-c", COMMON + CASES[case], root, os.path.join(root, "oracle"), HERE], env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]

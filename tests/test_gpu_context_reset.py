"""A program that resets its device between two adjustments (cudaDeviceReset, which ends its own context alone)
gets the same results after it as before: what is kept between calls belongs to a context and is not used in
the next.  In a child process, as the reset ends every handle of the process."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes, os
import numpy as np
from v3dsfmtoolkit_b200 import capi, scenes

os.environ["V3DBA_SCHUR"] = "groups"
capi._lib()
runtime = ctypes.CDLL([l.split()[-1] for l in open("/proc/self/maps") if "libcudart" in l][0])

rng = np.random.default_rng(0)
n = 200000
ptr = (3 * np.arange(n + 1)).astype(np.int32)
tracks = dict(track_ptr=ptr, pos=rng.normal(size=(n, 3)), view=rng.integers(0, 40, 3 * n).astype(np.int32),
              id=np.arange(3 * n, dtype=np.int32), mpos=rng.normal(size=(3 * n, 2)).astype(np.float32))
graph = scenes.rotation_graph(n_views=300, n_pairs=3000, seed=1)
triplets = scenes.triplet_batch(n_triplets=20, min_points=20, max_points=90, seed=3)
scene = scenes.sequence_scene(n_cams=20, n_points=2500, seed=1, mode=0)


def everything():
    out = list(capi.bundle_point_structure(tracks, 2).values())          # 14 MB down: through the slots
    R, r = capi.refine_consistent_rotations(graph.rel, graph.pairs, graph.R0)
    out += [R, r.cost]
    b = capi.Batch(triplets)
    res, _ = b.minimize(max_iterations=4)
    out += [np.array([x.cost for x in res])]
    b.close()
    for precision in (capi.PRECISION_MIXED, capi.PRECISION_FP64):
        h = capi.Handle.from_scene(scene)
        r = h.minimize(max_iterations=4, precision=precision, solver=capi.SOLVER_PCG)
        out += [r.cost, *h.get_params()]
        h.close()
    return out


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


first = everything()
assert same(everything(), first)
for _ in range(3):
    assert runtime.cudaDeviceReset() == 0
    assert same(everything(), first)
    assert same(everything(), first)
print("ok")
"""


def test_same_results_after_a_device_reset():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stderr[-2000:]

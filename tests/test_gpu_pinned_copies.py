"""Large results into pinned memory and large inputs from it go over the bus directly: no threads are started
to copy them, and the values are those of pageable arrays.  In a child process, whose threads are its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import os
import numpy as np, torch
from v3dsfmtoolkit_b200 import capi, scenes

def pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()

def threads():
    return len(os.listdir("/proc/self/task"))

L = capi._lib()
probs = scenes.triplet_batch(n_triplets=64, min_points=20, max_points=40, seed=1)
b = capi.Batch(probs)
b.minimize(max_iterations=1)
b.close()

# more than 32 MB up, 16 MB down
n, per = 700, 1000
one = scenes.triplet_batch(n_triplets=1, min_points=per, max_points=per, seed=2)[0]
flat = capi.concat_problems([one] * n)
up = {k: pinned(v) for k, v in flat.items()}
assert sum(v.nbytes for v in up.values()) > 32 << 20
R, T = np.zeros((3 * n, 3, 3)), np.zeros((3 * n, 3))
X = pinned(np.zeros((n * per, 3)))
before = threads()
b = capi.Batch.from_flat(up)
assert threads() <= before, (threads(), before)
capi.check(L.v3dba_batch_get_all_params(b.h, capi._d(R), capi._d(T), capi._d(X)))
assert X.nbytes > 16 << 20 and threads() <= before, (threads(), before)
assert np.array_equal(X, flat["X"])
r1, _ = b.minimize(max_iterations=2)
b.close()
p = capi.Batch.from_flat(flat)
r2, _ = p.minimize(max_iterations=2)
assert threads() > before     # pageable: the threads are there
assert [x.cost for x in r1] == [x.cost for x in r2]
p.close()
print("ok")
"""


def test_pinned_arrays_are_copied_directly():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stderr[-2000:]

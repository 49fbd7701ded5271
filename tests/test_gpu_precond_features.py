"""Two-hop products of the learned preconditioner's edge features at the edges of the kernel's tiles: lower
lists that end one before, at and one after the five edges of a warp and the forty of a block, graphs with and
without triangles, and lists longer than the row of blocks that is held in shared memory.

The products of a sum are exact to 2^-24 each and n = 6 * (triangles) of them are added in FP32, so an entry
differs from the FP64 sum of the same FP32 blocks by at most n * 2^-24 * sum |A| |B|."""
import numpy as np
import pytest

from v3dsfmtoolkit_b200 import capi

pytestmark = pytest.mark.gpu


def _system(n, keep, seed):
    """Blocks of a diagonally dominant system over the pairs i < l for which keep(i, l)."""
    rng = np.random.default_rng(seed)
    bi, bl, blocks = [], [], []
    for i in range(n):
        for l in range(i, n):
            if i == l or keep(i, l):
                bi.append(i)
                bl.append(l)
                g = rng.normal(size=(6, 6))
                blocks.append(g @ g.T + 12 * np.eye(6) if i == l else g)
    return np.array(bi, np.int32), np.array(bl, np.int32), np.array(blocks)


@pytest.mark.parametrize("n,every", [(2, 1), (3, 1), (6, 1), (7, 1), (12, 12), (40, 1), (41, 1), (42, 1), (60, 3), (258, 2), (259, 1)])
def test_two_hop_products(n, every):
    bi, bl, blocks = _system(n, lambda i, l: (l - i) % every == 0 or l - i == 1, n)
    pset = capi.PrecondSet()
    pset.add_blocks(n, bi, bl, blocks)
    ea, eb, xe, _, _ = pset.features(0)
    F = {(b, a): xe[e, :36].reshape(6, 6).astype(np.float64) for e, (a, b) in enumerate(zip(ea, eb))}
    zero = np.zeros((6, 6))
    M = np.array([[F.get((b, a), zero) for a in range(n)] for b in range(n)]).transpose(0, 2, 1, 3)   # [b, r, a, c]
    M2, A2 = M.reshape(6 * n, 6 * n), np.abs(M).reshape(6 * n, 6 * n)
    for k, (want, size) in enumerate(((M2 @ M2, A2 @ A2), (M2 @ M2.T, A2 @ A2.T))):
        for e, (a, b) in enumerate(zip(ea, eb)):
            w, s = (x[6 * b:6 * b + 6, 6 * a:6 * a + 6] for x in (want, size))
            got = xe[e, 36 * (k + 1):36 * (k + 2)].reshape(6, 6)
            assert np.all(np.abs(got - w) <= 6 * n * 2.0**-24 * s), (k, a, b)
    pset.close()

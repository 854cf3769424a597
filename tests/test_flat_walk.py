"""The walk of scenes whose top table reaches the leaves (flat_step) against
the walk of every level (VE_RAYCAST_FULL_WALK), ray by ray and bit for bit:
every depth that takes it (3..10), its neighbours that do not (2, 11), node
arrays with blocks that start at, straddle and lie past the end of the array,
and rays on the faces, along the axes and with non-finite components.  Whole
numbers: the tolerance is zero.
"""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


def arrays(ve, rng, depth):
    """A tree of random voxels, and the same words with broken blocks."""
    cpu = ve.OctreeCPU(depth)
    n = min(4000, max(4, (1 << (3 * depth)) // 8))
    cpu.insert_many(helpers.random_voxels(rng, depth, n / float(1 << (3 * depth))))
    tree = ve.Octree(depth)
    tree.set(cpu)
    words = tree.words()
    words = words[: max(9, tree.size)]
    yield words
    bad = words.copy()
    internal = np.nonzero(bad[1:] & 1)[0] + 1
    if len(internal):
        pick = rng.choice(internal, max(1, len(internal) // 8), replace=False)
        size = len(bad)
        to = rng.choice([size - 9, size - 3, size - 1, size, size + 1, size + 1000, (1 << 28) - 1], len(pick))
        bad[pick] = (bad[pick] & 15) | (np.maximum(to, 0).astype(np.uint32) << 4)
    yield bad


def rays(rng, depth, n):
    L = float(1 << depth)
    o = rng.uniform(-0.2 * L, 1.2 * L, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    k = n // 8
    o[:k] = rng.integers(0, (1 << depth) + 1, (k, 3))          # lattice points, the faces at 2^D among them
    d[:k] = rng.choice([-1.0, -0.0, 0.0, 1.0], (k, 3))
    d[k:2 * k] *= rng.choice([0.0, -0.0, 1e-40, 1e-30, 1.0], (k, 3)).astype(np.float32)
    o[2 * k:3 * k, :] = rng.uniform(0, L, (k, 3))
    o[np.arange(2 * k, 3 * k), rng.integers(0, 3, k)] = L      # sliding along a face
    d[np.arange(2 * k, 3 * k), rng.integers(0, 3, k)] = 0.0
    odd = np.array([np.nan, np.inf, -np.inf, 0.0, 1e38, -1e38], np.float32)
    d[3 * k:3 * k + 64] = rng.choice(odd, (64, 3))
    o[3 * k + 64:3 * k + 128] = rng.choice(odd, (64, 3))
    return o, d


@pytest.mark.parametrize("depth", [2, 3, 4, 5, 6, 7, 8, 9, 10, 11])
def test_flat_walk_matches_full_walk(ve, depth):
    rng = np.random.default_rng(100 + depth)
    r = ve.Renderer(hash_log2=8)
    try:
        for words in arrays(ve, rng, depth):
            sid = r.upload_scene(words, depth, keep_normals=True)
            for cc in (0, 5, 300):
                o, d = rays(rng, depth, 4001)
                full = r.raycast_batch(sid, o, d, cc, full_walk=True)
                flat = r.raycast_batch(sid, o, d, cc)
                bad = np.nonzero((full != flat).any(1))[0]
                assert bad.size == 0, (depth, cc, o[bad[0]], d[bad[0]], full[bad[0]], flat[bad[0]])
            r.release_scene(sid)
    finally:
        r.close()

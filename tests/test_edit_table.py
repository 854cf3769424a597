"""ve_scene_apply_edits rebuilds the top table only when an edit changes what
the table holds: after every kind of edit — leaf words, child counts, removed
and added blocks, a slot listed twice, no change — rays through the table equal
rays that walk every level, and the clip box equals a fresh upload's.  Exact."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


def edits(rng, words, kind):
    """(slots, new words) of one kind on the current words."""
    w = words[1:]
    leaf = np.nonzero(((w & 1) == 0) & ((w & 0xFE) != 0))[0] + 1
    inner = np.nonzero((w & 1) == 1)[0] + 1
    if kind == "dig":
        s = rng.choice(leaf, min(200, len(leaf) - 8), replace=False)
        return s, np.zeros(len(s), np.uint32)
    if kind == "repaint":
        s = rng.choice(leaf, min(200, len(leaf)), replace=False)
        return s, (rng.integers(1, 128, len(s)) << 1).astype(np.uint32)
    if kind == "counts":
        s = rng.choice(inner, min(50, len(inner)), replace=False)
        return s, (words[s] & ~np.uint32(14)) | (rng.integers(0, 8, len(s)).astype(np.uint32) << 1)
    if kind == "cut":
        s = rng.choice(inner, min(20, len(inner)), replace=False)
        return s, np.zeros(len(s), np.uint32)
    if kind == "move":
        s = rng.choice(inner, min(20, len(inner)), replace=False)
        return s, words[rng.permutation(s)]
    if kind == "twice":  # both entries of a slot are the same word, so that the order does not matter
        s = np.repeat(rng.choice(inner, min(10, len(inner)), replace=False), 2)
        return s, np.zeros(len(s), np.uint32)
    return leaf[:5], words[leaf[:5]]


@pytest.mark.parametrize("depth", [2, 3, 6, 9, 11])
def test_table_follows_edits(ve, depth):
    rng = np.random.default_rng(depth)
    cpu = ve.OctreeCPU(depth)
    cpu.insert_many(helpers.random_voxels(rng, depth, min(1.0, 6000.0 / float(1 << (3 * depth)))))
    tree = ve.Octree(depth)
    tree.set(cpu)
    words = tree.words()[: max(9, tree.size)].copy()
    L = float(1 << depth)
    with ve.Renderer(hash_log2=8) as r:
        sid = r.upload_scene(words, depth, keep_normals=True)
        for kind in ("dig", "none", "counts", "repaint", "cut", "dig", "move", "twice", "repaint"):
            slots, new = edits(rng, words, kind)
            r.apply_edits(sid, slots, new, keep_normals=True)
            words[slots] = new
            assert np.array_equal(r.download_scene(sid), words), kind
            o = rng.uniform(0, L, (3000, 3)).astype(np.float32)
            o[:300, 0] = L
            d = rng.normal(size=(3000, 3)).astype(np.float32)
            assert np.array_equal(r.raycast_batch(sid, o, d, 200), r.raycast_batch(sid, o, d, 200, full_walk=True)), kind
            fresh = r.upload_scene(words, depth, keep_normals=True)
            for a, b in zip(r.clip_box(sid), r.clip_box(fresh)):
                assert np.array_equal(a, b), kind
            r.release_scene(fresh)

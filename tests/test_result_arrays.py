"""Arrays that results come back in (pinned blocks, used again): an array that
is still held keeps its values while later calls run, blocks come back when the
last view of them is dropped, the pool stays within its limit and is empty
after the last renderer."""
import gc
import threading

import numpy as np
import pytest

import helpers


def test_size_classes(ve):
    pool = ve._ResultPool
    for n in [1, 65535, 65536, 65537, 1 << 20, (1 << 20) + 1, 12345678, (1 << 29) - 1]:
        s = pool._size_class(n)
        assert s >= n and s % (64 << 10) == 0 and s <= max(n + n // 8 + 1, 2 * (64 << 10))


def test_small_and_refused_blocks_are_ordinary_arrays(ve, monkeypatch):
    pool = ve._ResultPool()
    assert pool.empty((5, 3), np.float32).flags.owndata
    pool.LIMIT = 0
    a = pool.empty((512, 512), np.uint32)
    assert a.shape == (512, 512) and a.dtype == np.uint32 and not a.any() and pool._held == 0


@pytest.mark.gpu
@pytest.mark.parametrize("n", [8191, 8192, 8193, 100003])
def test_held_results_keep_their_values(ve, n):
    rng = np.random.default_rng(n)
    words, depth, _, _, _ = helpers.small_setup()
    with ve.Renderer(hash_log2=8) as r:
        sid = r.upload_scene(words, depth)
        rays = [(rng.uniform(0, 128, (n, 3)), rng.normal(size=(n, 3))) for _ in range(4)]
        first = [r.raycast_batch(sid, o, d) for o, d in rays]
        copies = [a.copy() for a in first]
        part = first[0][10:20]  # a view keeps its block
        for o, d in rays[::-1]:
            r.raycast_batch(sid, o, d)
        for a, b in zip(first, copies):
            assert np.array_equal(a, b)
        del first, a
        gc.collect()
        for (o, d), b in zip(rays, copies):
            assert np.array_equal(r.raycast_batch(sid, o, d), b)
        assert np.array_equal(part, copies[0][10:20])
        held = ve._results._held
        for o, d in rays * 3:
            r.raycast_batch(sid, o, d)
        assert ve._results._held == held <= ve._results.LIMIT
    assert np.array_equal(part, copies[0][10:20])  # outlives the renderer


@pytest.mark.gpu
def test_pool_is_given_back(ve):
    gc.collect()
    assert ve._results._renderers == 0, "a renderer of another test is still open"

    def work():
        words, depth, mats, cam, fc = helpers.small_setup()
        with ve.Renderer(hash_log2=12) as r:
            r.set_materials(mats)
            sid = r.upload_scene(words, depth)
            for _ in range(4):
                r.render(sid, cam, fc)

    ts = [threading.Thread(target=work) for _ in range(3)]
    for t in ts:
        t.start()
    for t in ts:
        t.join(120)
    gc.collect()
    assert ve._results._held == 0 and not ve._results._free

"""The pool of pinned result arrays, over a library that hands out ordinary
memory (no GPU): a size is pinned when it is asked for again, a free block
serves sizes from half its own up, the blocks longest unused make room at the
limit, and blocks that end anywhere (another thread, a collection inside the
pool) come back."""
import ctypes
import gc
import threading
import types

import numpy as np
import pytest

MB = 1 << 20


@pytest.fixture
def pool(ve, monkeypatch):
    live = {}

    def alloc(size, out):
        buf = ctypes.create_string_buffer(size)
        live[ctypes.addressof(buf)] = buf
        out._obj.value = ctypes.addressof(buf)
        return ve.VE_OK

    def free(p):
        del live[p]  # a block freed twice fails here
        return ve.VE_OK

    lib = types.SimpleNamespace(ve_host_alloc=alloc, ve_host_free=free)
    monkeypatch.setattr(ve, "load_library", lambda: lib)
    monkeypatch.setattr(ve, "_lib", lib)
    p = ve._ResultPool()
    p.live = live
    p.opened()
    return p


def pinned(pool, a):
    return any(q <= a.ctypes.data < q + len(b) for q, b in pool.live.items())


def test_pinned_from_the_second_request(pool):
    a = pool.empty((MB,), np.uint8)
    assert a.flags.owndata and not pool.live and not a.any()
    b = pool.empty((MB,), np.uint8)
    assert pinned(pool, b) and pool._held == MB
    c = pool.empty((2 * MB,), np.uint8)  # another size: its first request
    assert c.flags.owndata
    at = b.ctypes.data
    del b
    assert pool.empty((MB,), np.uint8).ctypes.data == at
    assert len(pool.live) == 1


@pytest.mark.parametrize("n,fits", [(2 * MB, True), (2 * MB - 5, True), (MB, True), (MB - 1, True), (7 * MB // 8, False),
                                    (2 * MB + 1, False), (MB // 2, False)])
def test_a_free_block_serves_sizes_down_to_half_its_own(pool, n, fits):
    pool.empty((2 * MB,), np.uint8)
    pool.empty((2 * MB,), np.uint8)
    assert len(pool.live) == 1 and pool._free
    a = pool.empty((n,), np.uint8)
    assert pinned(pool, a) == fits and a.shape == (n,)


def test_the_longest_unused_block_makes_room(pool):
    pool.LIMIT = 8 * MB
    sizes = [MB, 2 * MB, 4 * MB]
    held = [[pool.empty((s,), np.uint8) for _ in range(2)][1] for s in sizes]
    at = [a.ctypes.data for a in held]
    assert pool._held == 7 * MB
    a = held = None  # given back in order: 1, 2, 4 MB
    for s, p in ((2 * MB, at[1]), (MB, at[0])):  # used again: now the 4 MB block is the oldest
        a = pool.empty((s,), np.uint8)
        assert a.ctypes.data == p
        a = None
    a = [pool.empty((5 * MB,), np.uint8) for _ in range(2)]
    assert pinned(pool, a[1]) and pool._held <= pool.LIMIT
    assert at[2] not in pool.live and at[0] in pool.live and at[1] in pool.live
    assert pool.empty((9 * MB,), np.uint8).flags.owndata and pool.empty((9 * MB,), np.uint8).flags.owndata
    a = None
    pool.closed()
    assert pool._held == 0 and not pool._free and not pool.live


def test_blocks_that_end_inside_the_pool_and_in_threads(ve, pool):
    class Cycle:
        pass

    def leave(n):
        c = Cycle()
        c.me, c.a = c, pool.empty((n,), np.uint8)  # ends in a collection only

    # a collection inside every allocation the pool makes
    alloc = pool_alloc = ve.load_library().ve_host_alloc

    def collecting(size, out):
        gc.collect()
        return pool_alloc(size, out)

    ve.load_library().ve_host_alloc = collecting
    for k in range(40):
        leave(MB + (k % 7) * 200000)
    errors = []

    def work(seed):
        try:
            rng = np.random.default_rng(seed)
            keep = []
            for _ in range(300):
                a = pool.empty((int(rng.integers(60000, 3 * MB)),), np.uint8)
                a[:8] = seed
                keep.append(a)
                if len(keep) > 5:
                    assert (keep.pop(0)[:8] == seed).all()
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=work, args=(k + 1,)) for k in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join(120)
    ve.load_library().ve_host_alloc = alloc
    assert not errors, errors
    gc.collect()
    pool.closed()
    assert pool._held == 0 and not pool._free and not pool.live


def test_a_renderer_that_ends_inside_the_pool(ve, pool):
    """A collection inside an allocation closes another renderer on this thread."""
    lib = ve.load_library()
    alloc = lib.ve_host_alloc
    pool.opened()

    def closing(size, out):
        pool.closed()
        return alloc(size, out)

    pool.empty((MB,), np.uint8)
    lib.ve_host_alloc = closing
    done = []
    t = threading.Thread(target=lambda: done.append(pool.empty((MB,), np.uint8)), daemon=True)
    t.start()
    t.join(20)
    assert done and pinned(pool, done[0]) and pool._renderers == 1
    done.clear()
    pool.closed()
    assert pool._renderers == 0 and not pool.live and pool._held == 0

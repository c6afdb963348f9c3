"""The page-locked blocks behind large results, with a counting stand-in for the allocator: what stays page-locked is bounded whatever the caller does with its results."""
import gc
import random
import threading

import numpy as np
import pytest

from cudapp_b200 import api

MB = 1 << 20


class Fake:
    """hands out addresses of real memory, so that arrays on them can be written"""

    def __init__(self):
        self.live, self.most, self.allocs, self.memory = {}, 0, 0, {}

    def alloc(self, size):
        a = np.empty(size, np.uint8)
        self.memory[a.ctypes.data] = a
        self.live[a.ctypes.data] = size
        self.most = max(self.most, sum(self.live.values())); self.allocs += 1
        return a.ctypes.data

    def release(self, address):
        del self.live[address], self.memory[address]


@pytest.fixture
def fake(monkeypatch):
    f = Fake()
    monkeypatch.setattr(api, "_pool", api._Pool(f.alloc, f.release))
    return f


def locked(a):
    while isinstance(a, np.ndarray):
        a = a.base
    return isinstance(a, api._Block)


def test_dropped_results_share_blocks(fake):
    for i in range(200):
        r = api._result((100, 1000), np.float32)                    # the last one is alive while the next is made
        assert locked(r) and r.shape == (100, 1000) and r.dtype == np.float32
        r[:] = i
    assert fake.allocs == 2


def test_kept_results_become_ordinary_arrays(fake):
    kept = [api._result(MB // 4, np.float32) for _ in range(40)]
    assert [locked(a) for a in kept] == [True] * api.POOL_BLOCKS + [False] * (40 - api.POOL_BLOCKS) and fake.allocs == api.POOL_BLOCKS
    for i, a in enumerate(kept):
        a[:] = i
    assert all((a == i).all() for i, a in enumerate(kept))
    del kept[1], a
    gc.collect()
    assert locked(api._result(MB // 4, np.float32)) and fake.allocs == api.POOL_BLOCKS


def test_large_sizes_stay_within_the_bound(fake):
    kept = [api._result(n * MB, np.uint8) for n in (30, 1, 33, 5) for _ in range(4)]     # 30 of them lock 32, 33 would lock 64
    assert fake.most == api.POOL_BYTES and [locked(a) for a in kept] == [True] * 4 + [False] * 12
    assert not locked(api._result(2 * api.POOL_BYTES, np.uint8))


def test_idle_blocks_make_room(fake):
    a = api._result(64 * MB, np.uint8); b = api._result(64 * MB, np.uint8)
    del a, b
    for _ in range(api.POOL_IDLE - 1):                               # alternating sizes do not push one another out
        assert not locked(api._result(32 * MB, np.uint8))
    assert locked(api._result(64 * MB, np.uint8)) and locked(api._result(64 * MB, np.uint8))
    for _ in range(api.POOL_IDLE):
        api._result(32 * MB, np.uint8)
    assert locked(api._result(32 * MB, np.uint8)) and fake.most <= api.POOL_BYTES and len(fake.live) == 2


def test_failed_allocation_is_an_ordinary_array(monkeypatch):
    monkeypatch.setattr(api, "_pool", api._Pool(lambda size: None, None))
    for _ in range(10):
        assert not locked(api._result(MB, np.uint8))
    assert api._pool.held == 0


def test_threads(fake):
    wrong = []

    def work(seed):
        rng, kept = random.Random(seed), []
        for i in range(300):
            a = api._result(rng.choice((MB // 8, MB // 4, MB)), np.uint8)
            a[:16] = seed
            kept.append(a)
            if len(kept) > 3:
                if not (kept.pop(rng.randrange(4))[:16] == seed).all():
                    wrong.append(seed)
        wrong.extend(seed for a in kept if not (a[:16] == seed).all())
    threads = [threading.Thread(target=work, args=(s,)) for s in range(8)]
    for t in threads: t.start()
    for t in threads: t.join()
    gc.collect()
    assert not wrong and fake.most <= api.POOL_BYTES
    assert api._pool.held == sum(fake.live.values()) and sum(map(len, api._pool.free.values())) == len(fake.live)

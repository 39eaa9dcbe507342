"""The host memory that large results share (lightgraph._ResultBlocks): no two
live arrays on one block, blocks used again only after the last view of it is gone,
and the bounds on what is kept."""
import threading

import numpy as np
import pytest

from lightgraph_gb300.lightgraph import Context, _ResultBlocks


def address(a):
    return a.__array_interface__["data"][0]


@pytest.mark.parametrize("shape", [(128, 128), (64, 90, 4), (65536,), (65535,), (0, 4), (3,)])
def test_arrays(shape):
    pool = _ResultBlocks()
    a, b = pool.empty(shape), pool.empty(shape)
    for x in (a, b):
        assert x.shape == shape and x.dtype == np.float32 and x.flags.c_contiguous and x.flags.writeable
    a[...] = 1.0
    b[...] = 2.0
    assert (a == 1.0).all() and (b == 2.0).all()


def test_used_again_only_when_dropped():
    pool = _ResultBlocks()
    a = pool.empty((256, 256))
    at, row = address(a), a[7]
    del a
    b = pool.empty((256, 256))
    assert address(b) != at  # a row of the first is still alive
    row[...] = 3.0
    del row
    assert address(pool.empty((128, 512))) == at  # same size, other shape
    assert address(pool.empty((256, 257))) != at


def test_bounds():
    pool = _ResultBlocks()
    held = [pool.empty((400 + k, 200)) for k in range(20)]
    assert len({address(a) for a in held}) == 20
    assert len(pool.blocks) == pool.KEEP
    del held
    pool.LIMIT = 4 * 500 * 200
    pool.empty((240, 300))
    assert sum(b.nbytes for b in pool.blocks) <= pool.LIMIT
    a = pool.empty((500, 201))  # larger than the limit by itself
    a[...] = 1.0
    assert not pool.blocks


def test_threads():
    pool, bad = _ResultBlocks(), []

    def work(k):
        for i in range(300):
            a = pool.empty((256, 256 + 16 * (i % 3)))
            a[...] = k
            b = pool.empty((256, 256))
            b[...] = -k
            if not ((a == k).all() and (b == -k).all()):
                bad.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(1, 7)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad and len(pool.blocks) <= pool.KEEP


def test_closed_context_keeps_none():
    class Lib:
        lg_destroy = staticmethod(lambda handle: None)

    ctx = Context.__new__(Context)
    ctx.lib, ctx.h, ctx._results = Lib, 1, _ResultBlocks()
    kept, dropped = ctx._results.empty((256, 256)), ctx._results.empty((300, 300))
    kept[...] = 4.0
    del dropped
    ctx.close()
    assert not ctx._results.blocks
    assert (kept == 4.0).all()
    ctx.close()

"""The one-token descriptor and the joint state reset against their general counterparts."""
import numpy as np
import pytest
import torch

from ninfer_fusion_b200.runtime.batch import SeqChunk, StepBuffers
from ninfer_fusion_b200.runtime.kv_cache import RecurrentStatePool


@pytest.mark.parametrize("mrope", [False, True])
@pytest.mark.parametrize("B,deltas", [(1, 1), (1, 0), (5, 5), (5, 3), (8, 8)])
def test_build_decode_is_build_of_one_token_chunks(B, deltas, mrope):
    rng = np.random.default_rng(B)
    rows, slots = rng.permutation(B + 3)[:B].tolist(), rng.permutation(B + 2)[:B].tolist()
    start, tokens = rng.integers(0, 5000, B).tolist(), rng.integers(0, 1000, B).tolist()
    delta = rng.integers(-7, 40, deltas).tolist()
    bufs = [StepBuffers(8, 8, "cpu", mrope=mrope, attn_block_tokens=21) for _ in range(2)]
    want = bufs[0].build([SeqChunk(r, s, p, [t], True) for r, s, p, t in zip(rows, slots, start, tokens)], rope_delta=delta)
    got = bufs[1].build_decode(rows, slots, start, tokens, delta)
    assert torch.equal(bufs[0].dev, bufs[1].dev)
    for name, value in vars(want).items():
        mine = getattr(got, name)
        assert torch.equal(mine, value) and mine.shape == value.shape if torch.is_tensor(value) else mine == value, name
    with pytest.raises(ValueError):
        bufs[1].build_decode([0] * 9, [0] * 9, [0] * 9, [0] * 9, [])


@pytest.mark.parametrize("tokens", [[3, 1, 2], [3.0, 1.0, 2.0], [np.int64(3), np.float32(1), True], (3, 1, 2), np.array([3, 1, 2]),
                                    np.array([3.0, 1.0, 2.0], dtype=np.float32)])
def test_tokens_of_any_kind(tokens):
    """Whatever numpy assigns to 32-bit integers is taken as token ids; what it refuses is refused."""
    bufs = StepBuffers(8, 8, "cpu")
    batch = bufs.build([SeqChunk(0, 0, 0, tokens, True)])
    want = np.zeros(3, dtype=np.int32)
    want[:] = tokens
    assert batch.ids.tolist() == want.tolist()
    with pytest.raises(OverflowError):
        bufs.build([SeqChunk(0, 0, 0, [2 ** 31], True)])


def test_every_upload_is_waited_for_before_the_buffer_is_written(monkeypatch):
    """An upload by itself (a speculative round that is captured) counts like the one of `build`: the buffer is not written
    before the event behind it."""
    log = []

    class Event:
        def record(self, stream=None):
            log.append("sent")

        def synchronize(self):
            log.append("wait")
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: None)
    bufs = StepBuffers(8, 8, "cpu")
    bufs._sent = Event()
    bufs.upload()
    bufs.build([SeqChunk(0, 0, 5, [3, 4], True)])
    bufs.upload()
    bufs.build_decode([0], [0], [7], [1], [0])
    assert log == ["sent", "wait", "sent", "sent", "wait", "sent"]


@pytest.mark.parametrize("shapes", [[[((3, 4), torch.bfloat16), ((2, 5), torch.float32)], [((7,), torch.float32)]], []])
@pytest.mark.parametrize("taken,n", [([], 6), ([1, 3], 2), ([0, 2], 4), ([], 0)])
def test_alloc_many_is_alloc_n_times(taken, n, shapes):
    """(`shapes` empty: a decoder without recurrent layers)"""
    pools = [RecurrentStatePool(shapes, 6, "cpu") for _ in range(2)]
    for pool in pools:
        held = [pool.alloc() for _ in range(6)]
        for s in held:
            if s not in taken:
                pool.release(s)
        for t in pool.tensors():
            t.fill_(3.0)
    one = [pools[0].alloc() for _ in range(n)]
    assert pools[1].alloc_many(n) == one
    assert all(torch.equal(a, b) for a, b in zip(pools[0].tensors(), pools[1].tensors()))
    with pytest.raises(MemoryError):
        pools[1].alloc_many(7)
    assert pools[1].alloc_many(6 - len(taken) - n) == [pools[0].alloc() for _ in range(6 - len(taken) - n)]


@pytest.mark.parametrize("native", [True, False])
def test_pages_in_one_go(native):
    """Pages for many positions, and rows given back, as page by page: the same numbers, the same free list, the same state when
    the pool runs out."""
    from ninfer_fusion_b200.models.config import TINY_DENSE
    from ninfer_fusion_b200.runtime.kv_cache import PagedKvCache, PagePool
    caches = [PagedKvCache(TINY_DENSE, 12, 16, 3, 9, "cpu") for _ in range(2)]
    for c in caches:
        c.pool = PagePool(12, use_native=native)
    bulk, single = caches

    def one_by_one(cache, row, tokens):
        for n in range(1, tokens + 1):
            cache.ensure(row, n)

    def same():
        assert torch.equal(bulk.table_host, single.table_host) and bulk.row_pages == single.row_pages
        assert bulk._dirty_rows == single._dirty_rows and bulk.pool.free_pages == single.pool.free_pages
        bulk.publish(), single.publish()
        assert torch.equal(bulk.table, bulk.table_host) and torch.equal(single.table, single.table_host)
    for row, n in ((0, 50), (1, 16), (2, 33), (0, 90)):
        bulk.ensure(row, n)
        one_by_one(single, row, n)
        same()
    for c in caches:
        c.free_row(1)
        c.free_row(0)
    same()
    bulk.ensure(1, 9 * 16)
    one_by_one(single, 1, 9 * 16)
    same()
    for grow in (lambda: bulk.ensure(0, 40), lambda: one_by_one(single, 0, 40)):   # three pages wanted, none or few left
        with pytest.raises(MemoryError):
            grow()
    same()
    with pytest.raises(RuntimeError):
        bulk.pool.release_many([bulk.row_pages[1][0], 11 if bulk.pool.refcount_of(11) == 0 else bulk.row_pages[1][0]])

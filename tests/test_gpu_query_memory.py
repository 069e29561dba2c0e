"""Queries wherever a caller's memory has them: separate allocations gigabytes
apart, one pinned and one not, records of one array.  The responses are those
of the same queries in one array."""
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

R = 2048


@pytest.fixture(scope="module")
def env():
    import inspire_b200 as ib
    s = ib.Server(R * ib.RING_N // 64, 120, ib.fill_db(R * ib.RING_N, 5), db_rows=R, max_batch=6, crs_seed=bytes(64))
    qs = ib.synth_queries_host(R, 13, 0, 6)
    yield s, qs, s.answer_batch(list(qs))
    s.close()


def _words(n):
    """n u64 words of untouched address space."""
    return np.frombuffer(mmap.mmap(-1, 8 * n, mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS), np.uint64)


def _placed(words, qs, step):
    out = [words[k * step:k * step + q.size] for k, q in enumerate(qs)]
    for o, q in zip(out, qs):
        o[:] = q
    return out


@pytest.mark.parametrize("count", [2, 6])   # copied as a small batch, and in parts
def test_queries_gigabytes_apart(env, count):
    s, qs, want = env
    step = 3 << 27                            # 3.2 GB: beyond the documented pitch of a 2-D copy
    words = _words(step * (count - 1) + qs.shape[1])
    assert (s.answer_batch(_placed(words, qs[:count], step)) == want[:count]).all()


@pytest.mark.parametrize("pinned", [0, 1])
def test_one_query_pinned_and_one_not(env, pinned):
    import torch
    s, qs, want = env
    n = qs.shape[1]                           # whole pages
    placed = _placed(_words(3 * n), qs[:2], 2 * n)
    rt = torch.cuda.cudart()
    assert int(rt.cudaHostRegister(placed[pinned].ctypes.data, 8 * n, 0)) == 0
    try:
        assert (s.answer_batch(placed) == want[:2]).all()
    finally:
        assert int(rt.cudaHostUnregister(placed[pinned].ctypes.data)) == 0


@pytest.mark.parametrize("pin", [False, True])
@pytest.mark.parametrize("pad", [0, 40])
def test_records_of_one_array(env, pin, pad):
    import torch
    s, qs, want = env
    n = qs.shape[1] + pad
    words = torch.empty(6 * n, dtype=torch.int64, pin_memory=pin).numpy().view(np.uint64)
    assert (s.answer_batch(_placed(words, qs, n)) == want).all()

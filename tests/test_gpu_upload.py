"""Preprocessing of large databases from pageable memory (several threads
copying through pinned slots, from 128 MB) against pinned memory (one direct
copy): 134 MB in one encode pass, just at the limit, 268 MB in two passes over
several chunks, a database of one group that is not encoded, and a shard."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pinned_copy(db):
    import torch
    p = torch.empty(db.size, dtype=torch.int16, pin_memory=True)
    p.numpy().view(np.uint16)[:] = db
    return p.numpy().view(np.uint16)


def _db(rows, groups):
    import inspire_b200 as ib
    db = ib.fill_db(rows * groups * ib.RING_N, groups)
    return db, _pinned_copy(db)


@pytest.mark.parametrize("rows,groups", [(2048, 16), (2048, 32), (32768, 1)])
def test_pageable_equals_pinned(rows, groups):
    import inspire_b200 as ib
    q = ib.synth_queries_host(rows, 17, 0, 1)[0]
    got = []
    for db in _db(rows, groups):
        with ib.Server(rows * groups * ib.RING_N // 64, 120, db, db_rows=rows, max_batch=1, crs_seed=bytes(64)) as s:
            got.append((s.export_db(0, rows), s.answer(q)))
    (enc0, ans0), (enc1, ans1) = got
    assert (enc0 == enc1).all()
    assert (ans0 == ans1).all()


def test_pageable_shard_equals_pinned():
    import inspire_b200 as ib
    import torch
    rows, groups, lo, hi = 2048, 32, 5, 9
    qs = list(ib.synth_queries_host(rows, 19, 0, 2))
    out = []
    for db in _db(rows, groups):
        sh = ib.Shard(rows * groups * ib.RING_N // 64, 120, db, lo, hi, bytes(64), db_rows=rows, max_batch=2)
        o = torch.empty((2, hi - lo, 2 * ib.RING_N), dtype=torch.int32, device="cuda")
        sh.pack(qs, o.data_ptr())
        out.append(o.cpu())
        sh.close()
    assert torch.equal(out[0], out[1])

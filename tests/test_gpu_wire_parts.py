"""Packed queries copied and unpacked in parts (batches above 1 MB of wire
bytes) against the same queries flat: one slice and two, a chunked schedule, a
database of few and one of many rows, and the last batch copied whole (5
queries of 2048 rows) beside the first in parts (6)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,groups,counts,hchunks", [
    (2048, 8, (5, 6, 11, 33, 64), 0),
    (2048, 32, (6, 11), 3),
    (32768, 1, (2, 3, 9), 0),
])
def test_packed_in_parts_equals_flat(rows, groups, counts, hchunks):
    import inspire_b200 as ib
    from wire import pack_query
    cols = groups * ib.RING_N
    n = max(counts)
    qs = ib.synth_queries_host(rows, 91, 0, n)
    packed = np.stack([pack_query(q, rows) for q in qs])
    srv = ib.Server(rows * cols // 64, 120, ib.fill_db(rows * cols, 9), db_rows=rows, max_batch=n, crs_seed=bytes(64))
    try:
        for c in counts:
            want = srv.answer_batch(list(qs[:c]))
            if hchunks:
                srv.set_schedule(c, matvec_tc=1, horner_cluster=1, hchunks=hchunks)
            assert (srv.answer_wire(packed[:c], c, ib.RESP_FLAT) == want).all(), c
            assert (srv.answer_wire(packed[::-1][:c], c, ib.RESP_FLAT) == srv.answer_batch(list(qs[::-1][:c]))).all(), c
    finally:
        srv.close()

"""What the schedules of small databases promise beyond equal answers (those
split the SMs between the tensor pass and the mat-vec by default)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

R, G = 2048, 8


@pytest.fixture(scope="module")
def srv():
    import inspire_b200 as ib
    cols = G * ib.RING_N
    s = ib.Server(R * cols // 64, 120, ib.fill_db(R * cols, 3), db_rows=R, max_batch=3, crs_seed=bytes(64))
    yield s
    s.close()


@pytest.fixture(scope="module")
def queries():
    import inspire_b200 as ib
    return list(ib.synth_queries_host(R, 31, 0, 3))


def test_stage_times_separate_the_two_passes(srv, queries):
    """Timed, the tensor pass has its own stage: at least its 0.54 GB at the
    memory's nominal 8 TB/s."""
    assert srv.schedule(1)["tp_sms"] > 0
    want = srv.answer(queries[0])
    srv.enable_stage_timing(True)
    got = srv.answer(queries[0])
    st = srv.stage_times()
    srv.enable_stage_timing(False)
    assert (got == want).all()
    assert st["collapse"] > 0.067, st
    assert all(v > 0 for v in st.values()), st

"""What the schedules of small databases promise beyond equal answers (those
split the SMs between the tensor pass and the mat-vec by default)."""
import pytest

pytestmark = pytest.mark.gpu

R, G = 2048, 32


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
    """Timed, the tensor pass has its own stage: at least its 2.1 GB at the
    memory's nominal 8 TB/s."""
    assert srv.schedule(1)["tp_sms"] > 0
    want = srv.answer(queries[0])
    srv.enable_stage_timing(True)
    got = srv.answer(queries[0])
    st = srv.stage_times()
    srv.enable_stage_timing(False)
    assert (got == want).all()
    assert st["collapse"] > 0.26, st
    assert all(v > 0 for v in st.values()), st


def test_a_schedule_read_back_takes_chunks_and_the_cuda_core_matvec(srv, queries):
    """The default split of the SMs gives way to what it excludes; a split that
    was asked for stands."""
    first = srv.schedule(2)
    want = srv.answer_batch(queries[:2])

    def launches(**kw):
        srv.set_schedule(2, **{**first, **kw})
        n0 = srv.launch_count()
        assert (srv.answer_batch(queries[:2]) == want).all(), kw
        return srv.launch_count() - n0

    split = first["tp_sms"]
    assert split > 0 and first["hchunks"] == 0
    whole = launches()
    assert srv.schedule(2) == first
    assert launches(hchunks=2) > whole       # two chunks: two mat-vecs, two finalizes
    assert (srv.schedule(2)["tp_sms"], srv.schedule(2)["hchunks"]) == (0, 2)
    launches(matvec_tc=0)
    assert (srv.schedule(2)["tp_sms"], srv.schedule(2)["matvec_tc"]) == (0, 0)
    assert launches(hchunks=2, tp_sms=40) == whole and srv.schedule(2)["tp_sms"] == 40
    assert launches(hchunks=2, horner_cluster=0) == whole and srv.schedule(2)["tp_sms"] == split
    with pytest.raises(Exception):
        launches(matvec_tc=0, tp_sms=40)
    srv.set_schedule(2, **first)


@pytest.mark.parametrize("count", [1, 15, 16, 17])
def test_eight_cta_chains_alone_on_their_sms_and_not(count):
    """Chains of 8 CTAs that all fit with an SM per CTA (15 on a whole B200), and
    more, give the responses of the other Horner kernels."""
    import inspire_b200 as ib
    cols = 4 * ib.RING_N
    qs = list(ib.synth_queries_host(R, 37, 0, count))
    with ib.Server(R * cols // 64, 120, ib.fill_db(R * cols, 3), db_rows=R, max_batch=count, crs_seed=bytes(64)) as s:
        got = []
        for hc in (2, 1, 0):
            s.set_schedule(count, horner_cluster=hc)
            got.append(s.answer_batch(qs))
    assert (got[0] == got[1]).all() and (got[0] == got[2]).all()

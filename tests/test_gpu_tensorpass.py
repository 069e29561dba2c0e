"""The tensor pass on the GPU against the oracle (integer work: tolerance 0)
at the edges of its work split: one group (a tile per item) and several (two),
odd group counts (shards), one query up to a full pass of two slices and the
16-column edges between, scan segments of a few tiles; and the resident order of the
tensors seen from outside, through the export and the checkpoint's D section.
Queries are uniform residues, as ciphertexts are."""
import functools

import numpy as np
import pytest

from oracle_lib import N, NSTEPS, Oracle, crs_seed_from

pytestmark = pytest.mark.gpu

R = 2048
SEED = crs_seed_from(21)


@functools.lru_cache(maxsize=None)
def case(groups):
    """(entries, db, oracle's encoded DB and tensors) of `groups` groups on 2048 rows."""
    o = Oracle()
    cols = groups * N
    db = o.fill_db(R * cols, 40 + groups)
    return R * cols // 64, db, o.preprocess(SEED, db, R, cols, 256)


@functools.lru_cache(maxsize=None)
def queries():
    import inspire_b200 as ib
    return ib.synth_queries_host(R, 77, 0, 64)


@functools.lru_cache(maxsize=None)
def answer(groups, k):
    _, _, (dbe, pre) = case(groups)
    return Oracle().answer(dbe, R, groups * N, 256, pre, queries()[k])


def server(groups, **kw):
    import inspire_b200 as ib
    n, db, _ = case(groups)
    return ib.Server(n, 120, db, db_rows=R, crs_seed=SEED, **kw)


@pytest.mark.parametrize("groups", [1, 2, 4])
@pytest.mark.parametrize("count", [1, 4, 5, 31, 33, 64])
def test_answers_equal_the_oracle(groups, count):
    with server(groups, max_batch=count) as srv:
        got = srv.answer_batch(list(queries()[:count]))
    for k in sorted({0, min(32, count // 2), count - 1}):
        assert (got[k] == answer(groups, k)).all(), k


def test_odd_group_shards_equal_the_oracle():
    import inspire_b200 as ib
    import torch
    n, db, _ = case(4)
    count, parts, a = 6, [], []
    for lo, hi in [(0, 3), (3, 4)]:
        sh = ib.Shard(n, 120, db, lo, hi, SEED, db_rows=R, max_batch=count)
        out = torch.empty((count, hi - lo, 2 * N), dtype=torch.int32, device="cuda")
        sh.pack(list(queries()[:count]), out.data_ptr())
        parts.append(out)
        a.append(sh.export_a())
        params = sh.params
        sh.close()
    packed = torch.cat(parts, 1).contiguous()
    owner = ib.HornerOwner(params, np.concatenate(a), max_batch=count)
    got = owner.answer(packed.data_ptr(), list(queries()[:count]), stream=torch.cuda.current_stream().cuda_stream)
    owner.close()
    for k in (0, count - 1):
        assert (got[k] == answer(4, k)).all(), k


@pytest.mark.parametrize("segments", [2, 64])
def test_scan_segments_equal_the_oracle(segments):
    import inspire_b200 as ib
    with server(4, max_batch=2) as srv:
        with ib.ServeLoop([srv], max_batch=8, scan_segments=segments, autotune=False) as loop:
            tickets = [loop.submit(0, queries()[k]) for k in range(5)]
            out = np.zeros((5, 4 * N), np.uint64)
            for t, o in zip(tickets, out):
                loop.wait(t, o)
    for k in range(5):
        assert (out[k] == answer(4, k)).all(), k


def test_export_equals_the_oracle():
    _, _, (_, (pa, pdp, pdm, pdf)) = case(2)
    with server(2, max_batch=1) as srv:
        for g in (0, 1):
            for got, want in zip(srv.export_precomp(g), (pa, pdp, pdm, pdf)):
                assert (got == want[g * got.size:(g + 1) * got.size]).all(), g


def test_checkpoint_keeps_its_d_section_order(tmp_path):
    """The file's D section: [limb][slot][g * 4 + byte][(dir * 1023 + step) * 2
    + digit], padded with zeros to 4096 positions; and a handle restored from
    it answers as the oracle."""
    import inspire_b200 as ib
    G = 2
    _, _, (_, (_, pdp, pdm, _)) = case(G)
    path = tmp_path / "d.ckpt"
    with server(G, max_batch=1) as srv:
        srv.save(path)
    raw = np.fromfile(path, np.uint8)
    off = 256 + R * G * N * 2 + G * 2 * N * 4
    sec = raw[off:off + 2 * N * 4 * G * 4096].reshape(2, N, G, 4, 4096)
    assert not sec[..., 4 * NSTEPS:].any()
    got = sec[..., :4 * NSTEPS].reshape(2, N, G, 4, 2, NSTEPS, 2)       # l, i, g, byte, dir, step, digit
    for dr, src in enumerate((pdp, pdm)):
        want = src.reshape(G, 2, NSTEPS, 2, N).transpose(1, 4, 0, 2, 3)  # l, i, g, step, digit
        for b in range(4):
            assert (got[:, :, :, b, dr] == (want >> (8 * b)).astype(np.uint8)).all(), (dr, b)
    back = ib.Server.load(path, max_batch=1)
    assert (back.answer(queries()[0]) == answer(G, 0)).all()
    back.close()

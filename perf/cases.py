"""The work that users of this server have it do, as timed cases.

Every case goes through the package's public entry points:

* ``answer``  -- Server.answer_batch: flat u64 queries in pinned host memory in,
  flat responses in pinned host memory out (the blocking call of the C ABI);
* ``wire``    -- Server.answer_wire: packed queries in, compressed responses out;
* ``staged``  -- Server.run + Server.fetch on queries staged in device memory;
* ``serve``   -- ServeLoop: a burst of requests submitted and collected;
* ``shard``   -- Shard.pack: one GPU's part of a database split by group ranges;
* ``matvec``  -- matvec: the exact database pass on the caller's device memory;
* ``create``  -- Server(...): a database generation preprocessed, then its first
  answer.

Geometries are those of the tests and of bench.py: ``rows`` database rows,
``groups`` packing groups of 2048 columns, entries of ``entry_bytes`` bytes.
Queries are uniform residues per limb, as ciphertexts are; databases are the
package's splitmix64 fill.
"""
import os
import sys

import numpy as np
import torch

_REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_REPO, "inspire-gpu_b200"))

import inspire_b200 as ib  # noqa: E402

N = ib.RING_N
QS = (ib.Q0, ib.Q1)
BLK = ib.D_EFF * 2 * N  # u64 words of one key-switching key's b part


def listed():
    return [
        # One lookup in the smallest database the tests use (256 entries of 120 B,
        # 8 MB): launches and the host path are all of it.
        {"name": "answer_8mb_b1", "kind": "answer", "rows": 2048, "groups": 1, "entry_bytes": 120, "batch": 1},
        # One lookup, 1 GB database (2^25 entries of 30 B): the sequential plain answer.
        {"name": "answer_1gb_b1", "kind": "answer", "rows": 32768, "groups": 8, "entry_bytes": 30, "batch": 1},
        # A full batch from one caller on the 1 GB database.
        {"name": "answer_1gb_b32", "kind": "answer", "rows": 32768, "groups": 8, "entry_bytes": 30, "batch": 32},
        # One lookup, 16 GB database (2^29 entries of 30 B): bench.py's plain answer.
        {"name": "answer_16gb_b1", "kind": "answer", "rows": 32768, "groups": 128, "entry_bytes": 30, "batch": 1},
        # bench.py's end-to-end step: 32 queries over the 16 GB database.
        {"name": "answer_16gb_b32", "kind": "answer", "rows": 32768, "groups": 128, "entry_bytes": 30, "batch": 32},
        # A ragged batch in the wire formats on the 4 GB database of 960 B entries.
        {"name": "wire_4gb_b11", "kind": "wire", "rows": 32768, "groups": 32, "entry_bytes": 960, "batch": 11},
        # A batch above one database pass, queries already on the GPU, many groups on few rows.
        {"name": "staged_g128_b64", "kind": "staged", "rows": 2048, "groups": 128, "entry_bytes": 120, "batch": 64},
        # A burst of requests at the serving loop over a 1 GB database (lane batches).
        {"name": "serve_1gb_burst40", "kind": "serve", "rows": 32768, "groups": 8, "entry_bytes": 30, "batch": 40},
        # The larger share of the 4 GB database split unevenly over two GPUs: an odd number of groups.
        {"name": "shard_21of32_b8", "kind": "shard", "rows": 32768, "groups": 32, "entry_bytes": 960, "batch": 8,
         "lo": 11, "hi": 32},
        # The database pass alone on a caller's 8 GB matrix.
        {"name": "matvec_8gb_b16", "kind": "matvec", "rows": 32768, "cols": 131072, "batch": 16},
        # The same on a small odd-shaped matrix.
        {"name": "matvec_5120x8576_b5", "kind": "matvec", "rows": 5120, "cols": 8576, "batch": 5},
        # A 1 GB database refreshed: preprocessing from host memory, then the first lookup.
        {"name": "create_1gb", "kind": "create", "rows": 32768, "groups": 8, "entry_bytes": 30, "batch": 1},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["answer", "answer", "answer", "wire", "staged", "serve", "shard", "matvec", "matvec", "create"])
    if kind == "matvec":
        rows = 1024 * _log_int(rng, 1, 32)
        cols = 128 * _log_int(rng, 1, (1 << 31) // (128 * rows))
        return {"kind": kind, "rows": rows, "cols": cols, "batch": _log_int(rng, 1, 48)}
    rows = rng.choice([2048, 4096, 8192, 32768, 32768, 32768])
    most = {2048: 7, 4096: 7, 8192: 7, 32768: 5}[rows]  # databases up to 4 GB
    groups = 1 << rng.randint(1 if kind == "shard" else 0, 4 if kind == "create" else most)
    case = {"kind": kind, "rows": rows, "groups": groups, "entry_bytes": rng.choice([30, 120, 960]),
            "batch": 1 if kind == "create" else _log_int(rng, 1, 48)}
    if kind == "shard":
        case["lo"] = rng.randint(0, groups - 1)
        case["hi"] = rng.randint(case["lo"] + 1, groups)
    return case


def _cpe(entry_bytes):
    return (8 * entry_bytes + 14) // 15  # 15-bit columns of one entry


def _n_entries(case):
    return case["rows"] * case["groups"] * N // _cpe(case["entry_bytes"])


def _pinned(shape, dtype=torch.int64):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _u64(a):
    return a.view(np.uint64)


def _queries(rows, seed, count):
    """count flat queries in one pinned host array."""
    qn = 2 * rows + 6 * BLK
    dev = torch.empty((count, qn), dtype=torch.int64, device="cuda")
    ib.synth_queries_device(rows, seed, 0, count, dev.data_ptr(), torch.cuda.current_stream().cuda_stream)
    host = _pinned((count, qn))
    host[:] = dev.cpu().numpy()
    return _u64(host)


def _pack(rows, flat):
    """The packed wire form of flat queries: per coefficient the CRT value of
    its two residues (53 bits), MSB first."""
    inv = pow(ib.Q1, -1, ib.Q0)
    out = []
    for f in flat:
        b0, b1 = f[:rows], f[rows:2 * rows]
        polys = f[2 * rows:].reshape(-1, 2, N)
        v0 = np.concatenate([b0, polys[:, 0].reshape(-1)]).astype(np.int64)
        v1 = np.concatenate([b1, polys[:, 1].reshape(-1)]).astype(np.int64)
        v = v1 + ib.Q1 * ((v0 - v1) % ib.Q0 * inv % ib.Q0)
        bits = np.unpackbits(v.astype(">u8").view(np.uint8).reshape(-1, 8), axis=1)[:, 11:]
        out.append(np.packbits(bits.reshape(-1)))
    host = _pinned((len(out), out[0].size), torch.uint8)
    host[:] = np.stack(out)
    return host


def prepare(case, seed):
    kind, rows, batch = case["kind"], case["rows"], case["batch"]
    if kind == "matvec":
        cols = case["cols"]
        db = torch.empty(rows * cols, dtype=torch.int16, device="cuda")
        ib.fill_db_device(db.data_ptr(), rows * cols, seed, torch.cuda.current_stream().cuda_stream)
        g = torch.Generator(device="cuda").manual_seed(seed)
        q = torch.stack([torch.randint(0, m, (batch, rows), device="cuda", generator=g) for m in QS], 1).contiguous()
        return {"kind": kind, "case": case, "db": db, "q": q,
                "out": torch.empty((batch, 2, cols), dtype=torch.int32, device="cuda")}
    db = ib.fill_db(rows * case["groups"] * N, seed)
    crs = np.random.default_rng(seed).bytes(64)
    queries = _queries(rows, seed, batch)
    state = {"kind": kind, "queries": list(queries)}
    make = dict(n_entries=_n_entries(case), entry_bytes=case["entry_bytes"], db=db, db_rows=rows, crs_seed=crs)
    if kind == "create":
        return {**state, "make": make}
    if kind == "shard":
        sh = ib.Shard(group_lo=case["lo"], group_hi=case["hi"], max_batch=batch, **make)
        return {**state, "shard": sh,
                "out": torch.empty((batch, sh.groups, 2, N), dtype=torch.int32, device="cuda")}
    srv = ib.Server(max_batch=batch, **make)
    state["srv"] = srv
    state["out"] = _u64(_pinned((batch, ib.response_u64s(srv.params))))
    if kind == "wire":
        state["packed"] = _pack(rows, queries)
        state["out"] = _pinned((batch, srv.wire_sizes()[2]), torch.uint8)
    if kind == "staged":
        srv.stage(queries)
        srv.sync()
    if kind == "serve":
        state["loop"] = ib.ServeLoop([srv], max_batch=16, queue_slots=64, autotune=False)
    return state


def run(state):
    kind = state["kind"]
    if kind == "matvec":
        c = state["case"]
        ib.matvec(state["db"].data_ptr(), c["rows"], c["cols"], state["q"].data_ptr(), c["batch"],
                  state["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return state["out"]
    queries = state["queries"]
    if kind == "create":
        with ib.Server(max_batch=1, **state["make"]) as srv:
            return srv.answer(queries[0])
    if kind == "shard":
        state["shard"].pack(queries, state["out"].data_ptr())
        return state["out"]
    srv, out = state["srv"], state["out"]
    if kind == "answer":
        return srv.answer_batch(queries, out)
    if kind == "wire":
        return srv.answer_wire(state["packed"], len(queries), ib.RESP_COMPRESSED, out)
    if kind == "staged":
        srv.run(len(queries))
        return srv.fetch(len(queries), out)
    tickets = [state["loop"].submit(0, q) for q in queries]
    for t, o in zip(tickets, out):
        state["loop"].wait(t, o)
    return out


def work(case):
    """Bytes: the database (and its precomputed tensors, 67 MB a group) read
    once, queries and responses moved once.  Operations: two per
    multiply-accumulate of the two dot products with the database and of the
    tensor pass, per limb."""
    rows, batch = case["rows"], case["batch"]
    if case["kind"] == "matvec":
        cols = case["cols"]
        return {"bytes": 2 * rows * cols + 8 * batch * 2 * rows + 4 * batch * 2 * cols,
                "flops": 2 * 2 * rows * cols * batch}
    groups = case["hi"] - case["lo"] if case["kind"] == "shard" else case["groups"]
    cols = groups * N
    tensors = groups * 4 * 2 * N * (2 * ib.D_EFF * ib.NSTEPS + ib.D_EFF + 1)
    cts = max(1, groups // 256)
    query = 8 * (2 * rows + 6 * BLK)
    return {"bytes": 2 * rows * cols + tensors + batch * (query + 8 * cts * 4 * N),
            "flops": 2 * 2 * batch * (rows * cols + groups * N * 2 * ib.D_EFF * ib.NSTEPS)}


def exact(case, seed):
    """The database pass in 64-bit floating point (each half of a residue's
    products sums to less than 2^53, so every value is exact); the answers have
    no such form."""
    if case["kind"] != "matvec":
        return None
    s = prepare(case, seed)
    rows, cols = case["rows"], case["cols"]
    db = s["db"].view(rows, cols)
    out = torch.empty((case["batch"], 2, cols), dtype=torch.int64, device="cuda")
    step = max(128, (1 << 28) // rows)
    for c0 in range(0, cols, step):
        d = (db[:, c0:c0 + step].to(torch.int32) & 0xFFFF).to(torch.float64)
        for l, m in enumerate(QS):
            lo = (s["q"][:, l] & 0x3FFF).to(torch.float64) @ d
            hi = (s["q"][:, l] >> 14).to(torch.float64) @ d
            out[:, l, c0:c0 + step] = (lo.to(torch.int64) + (hi.to(torch.int64) % m << 14)) % m
    return out.to(torch.int32)

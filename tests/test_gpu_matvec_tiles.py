"""The tensor-core mat-vec against exact products (tolerance 0) around the
edges of its work items: one and two m' tiles per item (an odd number of
tiles takes one), accumulators double-buffered or not (9 and 10 queries), the
last batch that two tiles serve (18) and the first that they do not, one K
chunk and several.  Entries and residues include their extremes."""
import numpy as np
import pytest

from oracle_lib import QS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,kchunk", [(1024, 128, 0), (1024, 384, 1024), (4096, 256, 4096), (8192, 512, 4096)])
@pytest.mark.parametrize("count", [1, 5, 9, 10, 18, 19, 32])
def test_matvec_item_shapes(rows, cols, kchunk, count):
    import inspire_b200 as ib
    import torch
    rng = np.random.default_rng(rows + cols + count)
    db = rng.integers(0, 65535, (rows, cols), dtype=np.uint16)
    db[:7] = 65534
    q = np.stack([rng.integers(0, m, (count, rows)) for m in QS], 1).astype(np.int64)
    q[0, :, :9] = np.array(QS)[:, None] - 1
    d_db = torch.from_numpy(db.view(np.int16)).cuda()
    d_q = torch.from_numpy(q).cuda()
    out = torch.zeros((count, 2, cols), dtype=torch.int32, device="cuda")
    ib.matvec_ex(d_db.data_ptr(), rows, cols, d_q.data_ptr(), count, out.data_ptr(), kchunk_rows=kchunk,
                 stream=torch.cuda.current_stream().cuda_stream)
    # exact in float64: products of 16-bit entries and 14-bit halves over <= 8192 rows stay below 2^44
    f = db.astype(np.float64)
    for l, m in enumerate(QS):
        lo = (q[:, l] & 0x3FFF).astype(np.float64) @ f
        hi = (q[:, l] >> 14).astype(np.float64) @ f
        want = (lo.astype(np.int64) + (hi.astype(np.int64) % m << 14)) % m
        assert (out[:, l].cpu().numpy() == want).all(), l


@pytest.mark.parametrize("rows,cols", [(17408, 3072), (31744, 2432), (17408, 1024), (32768, 38528), (4096, 49024)])
@pytest.mark.parametrize("count", [1, 9])
def test_default_chunks(rows, cols, count):
    """Rows an odd multiple of 1024 above 16384 with few columns: the default
    K chunk is halved until the halves are no longer whole stages; and an odd
    number of tiles, halved once more and not."""
    import inspire_b200 as ib
    import torch
    g = torch.Generator(device="cuda").manual_seed(rows + cols + count)
    db = torch.randint(0, 65536, (rows, cols), device="cuda", generator=g, dtype=torch.int32)
    db16 = db.to(torch.int16)
    q = torch.stack([torch.randint(0, m, (count, rows), device="cuda", generator=g) for m in QS], 1).contiguous()
    out = torch.zeros((count, 2, cols), dtype=torch.int32, device="cuda")
    ib.matvec(db16.data_ptr(), rows, cols, q.data_ptr(), count, out.data_ptr(),
              torch.cuda.current_stream().cuda_stream)
    f = db.to(torch.float64)  # 16-bit entries, 14-bit halves, < 2^15 rows: sums below 2^45, exact
    for l, m in enumerate(QS):
        lo = (q[:, l] & 0x3FFF).to(torch.float64) @ f
        hi = (q[:, l] >> 14).to(torch.float64) @ f
        want = (lo.to(torch.int64) + (hi.to(torch.int64) % m << 14)) % m
        assert (out[:, l] == want).all(), l

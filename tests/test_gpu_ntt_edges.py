"""The lazily reduced NTTs and the digit extraction on the GPU against the
oracle (tolerance 0) where their bounds are tight: polynomials of extreme
residues (all 0, all q - 1, alternating, sparse), and decompositions of the
values around every carry and the centering point of the CRT lift."""
import numpy as np
import pytest

from oracle_lib import N, Q0, Q1, QS, Oracle

pytestmark = pytest.mark.gpu


def extremes(limb):
    q = QS[limb]
    x = np.arange(N)
    rng = np.random.default_rng(limb)
    return np.stack([
        np.zeros(N), np.full(N, q - 1), (x & 1) * (q - 1), (x >> 10) * (q - 1), (x == 0) * (q - 1),
        (x == N - 1) * (q - 1), ((x >> 3) & 1) * (q - 1), rng.integers(0, 2, N) * (q - 1), rng.integers(q - 9, q, N),
    ]).astype(np.uint32)


@pytest.mark.parametrize("inverse", [False, True])
def test_ntt_of_extreme_residues(inverse):
    import inspire_b200 as ib
    o = Oracle()
    polys = np.stack([extremes(0), extremes(1)], 1).reshape(-1, N)  # limbs alternate
    got = ib.ntt(polys, limb_run=1, inverse=inverse)
    for i, p in enumerate(polys):
        want = (o.ntt_inverse if inverse else o.ntt_forward)(p.astype(np.uint64), i & 1)
        assert (got[i] == want).all(), i


def test_decomposition_around_carries_and_the_centre():
    import inspire_b200 as ib
    Q = Q0 * Q1
    marks = [0, 1 << 17, 1 << 18, 1 << 35, 1 << 36, (1 << 35) + (1 << 17), (1 << 36) - (1 << 17), Q // 2, Q // 4,
             Q0, Q1, (Q // 2) // (1 << 36) * (1 << 36)]
    vals = sorted({(s * m + d) % Q for m in marks for s in (1, -1) for d in range(-40, 41)})
    vals += [(k * 0x9E3779B97F4A7C15) % Q for k in range(-len(vals) % N)]
    f = np.array([[v % Q0 for v in vals], [v % Q1 for v in vals]], np.uint32)
    polys = f.reshape(2, -1, N).transpose(1, 0, 2).copy()
    got = ib.decomp(polys).reshape(len(polys), -1)
    o = Oracle()
    for i, p in enumerate(polys):
        assert (got[i] == o.decomp(p.reshape(-1).astype(np.uint64))).all(), i

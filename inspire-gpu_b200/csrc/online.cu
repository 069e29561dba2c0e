// online.cu -- per-query kernels of the B200 InsPIRe server.
//
// One answer (gpu_answer / gpu_answer_batch, reference src/gpu_protocol.cu:
// 1121-1535) runs these launches on one stream:
//   qprep     key-switching keys to NTT form (KSK5 as byte planes), RGSW to
//             u32 residues, LWE vectors to the mat-vec's byte planes
//   matvec    r_l[j] = sum_i db[i][j] * b_l[i] mod q_l   (DB pass, HBM bound)
//   tensor pass (tensorpass_tc.cu): sum_{dir,s,j} D[s][j][i] * K5[j][perm_s(i)]
//   finalize  per group: NTT(r slice) - tensor partials - D_final (.) Kneg1
//   horner    one persistent CTA per response ciphertext runs the whole
//             ExtProd chain (INTT, decomp, NTT, MAC) in shared memory
// All arithmetic is exact mod q_l, so every output equals the reference's.
#include <algorithm>
#include <atomic>

#include "ipb_common.cuh"
#include "host_util.h"
#include "ipb_launch.h"

namespace ipb {

namespace {

__device__ __forceinline__ void ld8(const uint32_t* p, uint32_t (&v)[8]) {
    uint4 a = *reinterpret_cast<const uint4*>(p);
    uint4 b = *reinterpret_cast<const uint4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void st8(uint32_t* p, const uint32_t (&v)[8]) {
    *reinterpret_cast<uint4*>(p) = make_uint4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<uint4*>(p + 4) = make_uint4(v[4], v[5], v[6], v[7]);
}

// ------------------------------------------------------------------ qprep
// Query preparation, grid (nq, n_key + n_rgsw + n_plane), any of the three parts:
//   8 blocks       one key poly NTT (key, digit, limb) each.  The client sends
//                  KSK b-parts in coefficient form and RGSW in NTT form
//                  (capi.h:47-54); the reference NTTs the keys on the server
//                  (src/gpu_protocol.cu:1059-1094).  KSK5 leaves as the tensor
//                  pass's N operand: byte planes kplanes[q][limb][byte][4096],
//                  digit j's slots in the order of T.slot_of at positions
//                  j * N ..; KSK-1 as keys[q][limb][digit][N].
//   16 blocks      an eighth of a row of the RGSW u64 -> u32 reduction each.
//   rows / 1024    CRT byte planes of 1024 LWE coefficients each:
//                  planes[7q + k][rows] = byte k of B[i] = CRT(b_0[i] mod q0,
//                  b_1[i] mod q1) < q0 q1 (Garner: b_1 + q1 ((b_0 - b_1) q1^-1
//                  mod q0)).
// Inputs are reduced mod q (identical to the reference on canonical inputs).
// Bound by latency at few queries: every thread's loads are independent, so a
// block waits for memory once (the RGSW part took 14 us as 4 blocks of 32
// dependent rounds).
constexpr int kKeyBlocks = 8, kRgswBlocks = 16;
constexpr int kPlanes = 7;
__global__ void __launch_bounds__(256) qprep_kernel(const uint64_t* __restrict__ qraw, size_t qstride,
                                                    size_t rows, const DevTables* __restrict__ T,
                                                    uint8_t* __restrict__ kplanes, uint32_t* __restrict__ keys,
                                                    uint32_t* __restrict__ rgsw32, uint8_t* __restrict__ planes,
                                                    int n_key, int n_rgsw) {
    __shared__ __align__(16) uint32_t sbuf[kNttBuf], slots[kN];
    let_next_start();
    after_previous();
    const int b = blockIdx.x, y = blockIdx.y;
    const uint32_t t = threadIdx.x;
    const uint64_t* qr = qraw + (size_t)b * qstride;
    const size_t blk = (size_t)kDeff * 2 * kN;
    if (y < n_key) {
        const int key = y >> 2, j = (y >> 1) & 1, l = y & 1;
        const LimbTables& L = T->limb[l];
        const uint64_t* src = qr + 2 * rows + key * blk + (size_t)(j * 2 + l) * kN;
        uint32_t r[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) r[e] = mod_u64(src[t + 256 * e], L.cr, L.q);
        ntt_fwd(r, sbuf, L.fwd, L.q, t, 0);
        if (key == 1) {
            st8(keys + ((size_t)(b * 2 + l) * kDeff + j) * kN + 8 * t, r);
            return;
        }
        st8(slots + 8 * t, r);
        __syncthreads();
        const uint4 so = *reinterpret_cast<const uint4*>(T->slot_of + 8 * t);
        const uint32_t sw[4] = {so.x, so.y, so.z, so.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) r[e] = slots[(sw[e >> 1] >> (16 * (e & 1))) & 0xFFFFu];
        uint8_t* dst = kplanes + ((size_t)(b * 2 + l) * 4) * (kDeff * kN) + (size_t)j * kN + 8 * t;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            uint32_t w[2] = {0, 0};
#pragma unroll
            for (int e = 0; e < 8; ++e) w[e >> 2] |= ((r[e] >> (8 * p)) & 0xFFu) << (8 * (e & 3));
            *reinterpret_cast<uint2*>(dst + (size_t)p * (kDeff * kN)) = make_uint2(w[0], w[1]);
        }
    } else if (y < n_key + n_rgsw) {
        // 16 polynomials of N words, [row][digit][limb]
        const size_t i0 = (size_t)(y - n_key) * kN + t;
        const LimbTables& L = T->limb[(y - n_key) & 1];
        const uint64_t* src = qr + 2 * rows + 2 * blk + i0;
        uint32_t* dst = rgsw32 + (size_t)b * 4 * blk + i0;
#pragma unroll
        for (int e = 0; e < 8; ++e) dst[256 * e] = mod_u64(src[256 * e], L.cr, L.q);
    } else {
        const size_t i4 = ((size_t)(y - n_key - n_rgsw) * 256 + t) * 4;
        uint64_t B[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const uint32_t v0 = mod_u64(qr[i4 + c], T->limb[0].cr, kQ0);
            const uint32_t v1 = mod_u64(qr[rows + i4 + c], T->limb[1].cr, kQ1);
            const uint32_t v1r = v1 >= kQ0 ? v1 - kQ0 : v1;
            const uint32_t diff = v0 >= v1r ? v0 - v1r : v0 + kQ0 - v1r;
            const uint32_t h = csub(shoup_mul(diff, T->crt_c[0], T->crt_cp[0], kQ0), kQ0);
            B[c] = (uint64_t)v1 + (uint64_t)kQ1 * h;
        }
#pragma unroll
        for (int k = 0; k < kPlanes; ++k) {
            uint32_t packed = 0;
#pragma unroll
            for (int c = 0; c < 4; ++c) packed |= (uint32_t)((B[c] >> (8 * k)) & 0xFFu) << (8 * c);
            *reinterpret_cast<uint32_t*>(planes + ((size_t)kPlanes * b + k) * rows + i4) = packed;
        }
    }
}

// ------------------------------------------------------------------ matvec
// Row-split dual-limb mat-vec.  CTA (x, y): columns [x*256*CPT, +256*CPT),
// rows [y*rpc, +rpc).  Each thread streams CPT u16 columns with one 16- or
// 8-byte load per row and keeps 2*BT*CPT u64 accumulators; the query words
// of the chunk are reduced mod q once into shared memory.  Products are
// < 2^43, so rpc <= 2^20 rows need no intermediate reduction.
template <int BT, int CPT>
__global__ void __launch_bounds__(256) matvec_kernel(const uint16_t* __restrict__ db, size_t rows, size_t cols,
                                                     int rpc, const uint64_t* __restrict__ qraw, size_t qstride,
                                                     const DevTables* __restrict__ T, uint32_t* __restrict__ part,
                                                     size_t part_qstride, int nq) {
    extern __shared__ __align__(16) uint32_t sb[];  // [BT][2][rpc]
    const int chunk = blockIdx.y;
    const size_t r0 = (size_t)chunk * rpc;
    for (int b = 0; b < BT; ++b) {
        const int src = b < nq ? b : 0;
        for (int l = 0; l < 2; ++l) {
            const uint64_t* qb = qraw + (size_t)src * qstride + (size_t)l * rows + r0;
            for (int i = threadIdx.x; i < rpc; i += 256)
                sb[(b * 2 + l) * rpc + i] = mod_u64(qb[i], T->limb[l].cr, T->limb[l].q);
        }
    }
    __syncthreads();
    const size_t col0 = ((size_t)blockIdx.x * 256 + threadIdx.x) * CPT;
    uint64_t acc[BT][2][CPT];
#pragma unroll
    for (int b = 0; b < BT; ++b)
#pragma unroll
        for (int c = 0; c < CPT; ++c) { acc[b][0][c] = 0; acc[b][1][c] = 0; }
    const uint16_t* p = db + r0 * cols + col0;
#pragma unroll 4
    for (int i = 0; i < rpc; ++i) {
        uint32_t w[CPT / 2];
        if (CPT == 8) {
            uint4 v = __ldcs(reinterpret_cast<const uint4*>(p + (size_t)i * cols));
            w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
        } else {
            uint2 v = __ldcs(reinterpret_cast<const uint2*>(p + (size_t)i * cols));
            w[0] = v.x; w[1] = v.y;
        }
#pragma unroll
        for (int b = 0; b < BT; ++b) {
            const uint32_t b0 = sb[(b * 2 + 0) * rpc + i];
            const uint32_t b1 = sb[(b * 2 + 1) * rpc + i];
#pragma unroll
            for (int c = 0; c < CPT; ++c) {
                const uint32_t d = (c & 1) ? (w[c >> 1] >> 16) : (w[c >> 1] & 0xFFFFu);
                acc[b][0][c] += (uint64_t)d * b0;
                acc[b][1][c] += (uint64_t)d * b1;
            }
        }
    }
#pragma unroll
    for (int b = 0; b < BT; ++b) {
        if (b >= nq) break;
#pragma unroll
        for (int l = 0; l < 2; ++l) {
            uint32_t o[CPT];
#pragma unroll
            for (int c = 0; c < CPT; ++c) o[c] = mod_u64(acc[b][l][c], T->limb[l].cr, T->limb[l].q);
            uint32_t* dst = part + (size_t)b * part_qstride + ((size_t)chunk * 2 + l) * cols + col0;
            if (CPT == 8) {
                *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
                *reinterpret_cast<uint4*>(dst + 4) = make_uint4(o[4 % CPT], o[5 % CPT], o[6 % CPT], o[7 % CPT]);
            } else {
                *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
            }
        }
    }
}

// ------------------------------------------------------------------ finalize
// Per (group, limb, query): b = NTT(sum of the mat-vec partials of the
// group's N columns) - tensor pass - sum_j D_final[j] (.) Kneg1[j]
// (reference src/gpu_protocol.cu:1233-1274, src/gpu_online.cu:547-559).
// The tensor pass result is tp_out[q][g][l][N] (tensorpass_tc.cu), laid out as
// packed_b is.
__global__ void __launch_bounds__(256, 4) finalize_kernel(
    const uint32_t* __restrict__ mvpart, size_t mv_qstride, int mv_chunks, size_t cols,
    const uint32_t* __restrict__ tp_out, int g0,
    const uint32_t* __restrict__ df, const uint32_t* __restrict__ keys, size_t key_qstride,
    const DevTables* __restrict__ T, uint32_t* __restrict__ packed_b, size_t pb_qstride) {
    __shared__ __align__(16) uint32_t sbuf[kNttBuf];
    let_next_start();
    const int g = g0 + (int)blockIdx.x, l = blockIdx.y, b = blockIdx.z;
    const uint32_t t = threadIdx.x;
    const LimbTables& L = T->limb[l];
    uint32_t d0[8], d1[8];
    ld8(df + ((size_t)g * 2 + l) * kDeff * kN + 8 * t, d0);
    ld8(df + (((size_t)g * 2 + l) * kDeff + 1) * kN + 8 * t, d1);
    after_previous();
    // Everything the block reads is asked for before the transform: one memory
    // latency per block, not three.
    uint32_t o[8], k0[8], k1[8];
    ld8(tp_out + (size_t)b * pb_qstride + ((size_t)g * 2 + l) * kN + 8 * t, o);
    const uint32_t* kn = keys + (size_t)b * key_qstride + (size_t)l * kDeff * kN;
    ld8(kn + 8 * t, k0);
    ld8(kn + kN + 8 * t, k1);
    const uint32_t* mp = mvpart + (size_t)b * mv_qstride + (size_t)l * cols + (size_t)g * kN + t;
    uint32_t r[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) r[e] = mp[256 * e];
    if (mv_chunks > 1) {
        uint64_t s[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) s[e] = r[e];
        for (int y = 1; y < mv_chunks; ++y) {
            mp += 2 * cols;
#pragma unroll
            for (int e = 0; e < 8; ++e) s[e] += mp[256 * e];
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) r[e] = mod_u64(s[e], L.cr, L.q);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e)
        o[e] = add_mod(o[e], mod_u64((uint64_t)d0[e] * k0[e] + (uint64_t)d1[e] * k1[e], L.cr, L.q), L.q);
    ntt_fwd(r, sbuf, L.fwd, L.q, t, 0);
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = sub_mod(r[e], o[e], L.q);
    st8(packed_b + (size_t)b * pb_qstride + ((size_t)g * 2 + l) * kN + 8 * t, o);
}

// ------------------------------------------------------------------ horner
// HornerEval (reference src/crypto.cpp:264-279, src/gpu_protocol.cu:1300-1334):
// acc = packed[start+L-1]; for i = L-2..0: acc = ExtProd(rgsw, acc) + packed[start+i].
// One CTA of four 256-thread NTT groups runs a whole chain; group (p, l)
// owns polynomial p (0 = a, 1 = b) in limb l.  Per step: inverse NTT, CRT
// exchange with the partner limb through shared memory, gadget digits,
// two forward NTTs, the RGSW multiply-accumulate (digits of a meet the top
// row, digits of b the bottom row) and a cross-group sum.  The chain never
// leaves the SM; the reference spends ~12 launches per step.
constexpr size_t kHornerSmem = 4 * kN * sizeof(uint2) + (4 * kNttBuf + 2 * 2 * kN + 2 * 2 * kN) * sizeof(uint32_t);

__global__ void __launch_bounds__(1024, 1) horner_kernel(const uint32_t* __restrict__ pre_a,
                                                         const uint32_t* __restrict__ packed_b, size_t pb_qstride,
                                                         const uint32_t* __restrict__ rgsw32,
                                                         const DevTables* __restrict__ T, size_t groups,
                                                         size_t d_act, uint64_t* __restrict__ resp,
                                                         size_t resp_qstride) {
    extern __shared__ __align__(16) uint8_t smem[];
    uint2* tw = reinterpret_cast<uint2*>(smem);                       // [fwd0|fwd1|inv0|inv1][N]
    uint32_t* nbuf = reinterpret_cast<uint32_t*>(smem + 4 * kN * sizeof(uint2));  // [4][kNttBuf]
    uint32_t* xcoef = nbuf + 4 * kNttBuf;                             // [p][l][N]
    uint32_t* xch = xcoef + 2 * 2 * kN;                               // [p][l][N]
    const int ct = blockIdx.x, b = blockIdx.y;
    const int gp = threadIdx.x >> 8, p = gp >> 1, l = gp & 1;
    const uint32_t t = threadIdx.x & 255;
    const int bar = 1 + gp;
    for (int i = threadIdx.x; i < kN; i += 1024) {
        tw[i] = T->limb[0].fwd[i];
        tw[kN + i] = T->limb[1].fwd[i];
        tw[2 * kN + i] = T->limb[0].inv[i];
        tw[3 * kN + i] = T->limb[1].inv[i];
    }
    __syncthreads();
    const LimbTables& L = T->limb[l];
    const uint32_t q = L.q;
    const uint2* twf = tw + l * kN;
    const uint2* twi = tw + (2 + l) * kN;
    uint32_t* mybuf = nbuf + gp * kNttBuf;
    const size_t start = (size_t)ct * d_act;
    const size_t len = (start + d_act <= groups) ? d_act : groups - start;
    const uint32_t* pbq = packed_b + (size_t)b * pb_qstride;
    auto src_of = [&](size_t i) -> const uint32_t* {
        return p ? pbq + (i * 2 + l) * kN : pre_a + (i * 2 + l) * kN;
    };
    uint32_t acc[8];
    ld8(src_of(start + len - 1) + 8 * t, acc);
    const uint32_t* rg = rgsw32 + (size_t)b * (4 * kDeff * 2 * kN);
    const uint32_t* Ra0 = rg + (size_t)(((2 * p + 0) * kDeff + 0) * 2 + l) * kN;
    const uint32_t* Ra1 = rg + (size_t)(((2 * p + 0) * kDeff + 1) * 2 + l) * kN;
    const uint32_t* Rb0 = rg + (size_t)(((2 * p + 1) * kDeff + 0) * 2 + l) * kN;
    const uint32_t* Rb1 = rg + (size_t)(((2 * p + 1) * kDeff + 1) * 2 + l) * kN;
    uint32_t* xc_me = xcoef + (p * 2 + l) * kN;
    const uint32_t* xc_ot = xcoef + (p * 2 + (1 - l)) * kN;
    uint32_t* xch_out = xch + ((1 - p) * 2 + l) * kN;
    const uint32_t* xch_in = xch + (p * 2 + l) * kN;
    for (long i = (long)len - 2; i >= 0; --i) {
        ntt_inv(acc, mybuf, twi, q, L.scale_crt, t, bar);
#pragma unroll
        for (int e = 0; e < 8; ++e) xc_me[t + 256 * e] = acc[e];
        __syncthreads();
        uint32_t d0[8], d1[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const uint32_t o = xc_ot[t + 256 * e];
            int32_t s1, s2;
            decomp_lifted(l ? o : acc[e], l ? acc[e] : o, s1, s2);
            d0[e] = q + (uint32_t)s1;
            d1[e] = q + (uint32_t)s2;
        }
        ntt_fwd(d0, mybuf, twf, q, t, bar);
        ntt_fwd(d1, mybuf, twf, q, t, bar);
        uint32_t a0[8], a1[8], b0[8], b1[8];
        ld8(Ra0 + 8 * t, a0);
        ld8(Ra1 + 8 * t, a1);
        ld8(Rb0 + 8 * t, b0);
        ld8(Rb1 + 8 * t, b1);
        uint32_t own[8], oth[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const uint32_t ca = mod_u64((uint64_t)d0[e] * a0[e] + (uint64_t)d1[e] * a1[e], L.cr, q);
            const uint32_t cb = mod_u64((uint64_t)d0[e] * b0[e] + (uint64_t)d1[e] * b1[e], L.cr, q);
            own[e] = p ? cb : ca;
            oth[e] = p ? ca : cb;
        }
        st8(xch_out + 8 * t, oth);
        __syncthreads();
        uint32_t o2[8], pk[8];
        ld8(xch_in + 8 * t, o2);
        ld8(src_of(start + (size_t)i) + 8 * t, pk);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] = add_mod(add_mod(own[e], o2[e], q), pk[e], q);
    }
    uint64_t* dst = resp + (size_t)b * resp_qstride + ((size_t)ct * 4 + p * 2 + l) * kN + 8 * t;
#pragma unroll
    for (int e = 0; e < 8; e += 2)
        *reinterpret_cast<ulonglong2*>(dst + e) = make_ulonglong2(acc[e], acc[e + 1]);
}

// floor(w 2^32 / q) for w < q, without a 64-bit division.
__device__ __forceinline__ uint32_t shoup_factor(uint32_t w, uint64_t cr, uint32_t q) {
    const uint64_t x = (uint64_t)w << 32;
    const uint64_t f = __umul64hi(x, cr);  // low by at most 1
    return (uint32_t)f + (x - f * q >= q ? 1u : 0u);
}
// Digit j + 1 as a residue in (0, 2q) from the lift terms of this limb and the
// other one (q and q_oth their primes).
__device__ __forceinline__ uint32_t digit_res(uint32_t own, uint32_t oth, uint32_t q, uint32_t q_oth, uint64_t carry,
                                              int j) {
    const uint64_t v = lift_plus(own, oth, q, q_oth, carry);
    return q + (uint32_t)(j ? digit2(v) : digit1(v));
}
// Eight values per thread in shared memory, four and four N/2 words apart: the
// lanes of a warp access consecutive 16 bytes.
__device__ __forceinline__ void ld8_sh(const uint32_t* s, uint32_t t, uint32_t (&v)[8]) {
    const uint4 a = *reinterpret_cast<const uint4*>(s + 4 * t), b = *reinterpret_cast<const uint4*>(s + kHalf + 4 * t);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void st8_sh(uint32_t* s, uint32_t t, const uint32_t (&v)[8]) {
    *reinterpret_cast<uint4*>(s + 4 * t) = make_uint4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<uint4*>(s + kHalf + 4 * t) = make_uint4(v[4], v[5], v[6], v[7]);
}

// ------------------------------------------------------------------ horner (cluster)
// The same chain on a cluster of four CTAs, CTA rank r = 2p + l owning
// polynomial p (0 = a, 1 = b) in limb l.  Each CTA has two NTT groups:
// group 0 holds the accumulator and runs the inverse NTT (scaled so that its
// output is the CRT lift's term t_l, not the coefficient); both groups then
// lift (which needs the partner limb's terms) and transform one gadget digit
// each, and multiply it by the RGSW rows of their polynomial (held in
// registers for the whole chain).  Group 0 sums the two digits' contributions
// to the own polynomial, group 1 those to the other polynomial, which it
// sends to that polynomial's CTA.  Values stay unreduced where the next
// multiplication takes any word.
// A step crosses SMs twice, 8 KB each way (partner terms, contributions): an
// exchange between two SMs costs about 320 cycles and 50 more per KB with
// st.async (bulk copies and plain remote stores measured 200-300 cycles more),
// so the contributions are summed before they leave.  Data moves straight from
// registers into the receiver's shared memory, in the order of the receiving
// threads, and completes bytes on the receiver's mbarriers; the loop has no
// cluster-wide barrier.  Received buffers alternate with the step parity; a
// remote write for step t is issued only after its receiver has finished
// reading the same buffer at step t - 2 (it depends on data the receiver sent
// after that read).  Every wait is bounded.
constexpr size_t kHornerClSmem = 2 * kN * sizeof(uint2) + (2 * kNttBuf + (1 + 2 + 2 + 2) * kN) * sizeof(uint32_t) + 64;

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_peer(const void* local, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(r)
                 : "r"((uint32_t)__cvta_generic_to_shared(local)), "r"(rank));
    return r;
}
// 16 bytes into a peer CTA's shared memory, completing 16 bytes on its mbarrier.
__device__ __forceinline__ void st_async4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d,
                                          uint32_t mbar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                     addr),
                 "r"(a), "r"(b), "r"(c), "r"(d), "r"(mbar)
                 : "memory");
}
__device__ __forceinline__ void hb_init(uint64_t* b) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((uint32_t)__cvta_generic_to_shared(b)));
}
__device__ __forceinline__ void hb_expect(uint64_t* b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(b)),
                 "r"(bytes)
                 : "memory");
}
// Bounded wait on a cluster-filled mbarrier phase; false (and *err set) on timeout.
__device__ __forceinline__ bool hb_wait(uint64_t* b, uint32_t parity, int* err, int code) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(b);
    for (uint32_t it = 0; it < (1u << 22); ++it) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    atomicCAS(err, 0, code);
    return false;
}

__global__ void __cluster_dims__(4, 1, 1) __launch_bounds__(512, 1)
    horner_cl_kernel(const uint32_t* __restrict__ pre_a, const uint32_t* __restrict__ packed_b, size_t pb_qstride,
                     const uint32_t* __restrict__ rgsw32, const DevTables* __restrict__ T, size_t groups,
                     size_t d_act, uint64_t* __restrict__ resp, size_t resp_qstride, int* err, HornerRange hr) {
    extern __shared__ __align__(16) uint8_t smem[];
    uint2* twf = reinterpret_cast<uint2*>(smem);
    uint2* twi = twf + kN;
    uint32_t* nbuf = reinterpret_cast<uint32_t*>(twi + kN);         // [group][kNttBuf]
    uint32_t* xown = nbuf + 2 * kNttBuf;                            // own lift terms, for group 1
    uint32_t* xpart = xown + kN;                                    // [parity] partner limb's lift terms
    uint32_t* cown = xpart + 2 * kN;                                // [group 0's to the other poly | group 1's to the own]
    uint32_t* cin = cown + 2 * kN;                                  // [parity] the other poly's contribution
    uint64_t* mbx = reinterpret_cast<uint64_t*>(cin + 2 * kN);      // [parity] partner terms
    uint64_t* mbc = mbx + 2;                                        // [parity] contribution
    __shared__ volatile int abort_flag;
    let_next_start();
    const uint32_t rank = cluster_rank();
    const int p = (int)(rank >> 1), l = (int)(rank & 1);
    const int ct = blockIdx.x >> 2, b = blockIdx.y;
    const int gp = threadIdx.x >> 8;
    const uint32_t t = threadIdx.x & 255;
    const int bar = 1 + gp;
    const LimbTables& L = T->limb[l];
    const uint32_t q = L.q, q_oth = T->limb[1 - l].q;
    const uint64_t carry = gp ? kCarry2 : kCarry1;
    const NttScale scale = L.scale_crt;
    const size_t start = (size_t)ct * d_act;
    const size_t len = (start + d_act <= groups) ? d_act : groups - start;
    const long i_first = hr.i_first < 0 ? (long)len - 2 : (long)hr.i_first;
    const bool steps = i_first >= (long)hr.i_last;  // one group: the response is its packed ciphertext
    for (int i = threadIdx.x; steps && i < kN; i += 512) { twf[i] = L.fwd[i]; twi[i] = L.inv[i]; }
    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int k = 0; k < 2; ++k) { hb_init(&mbx[k]); hb_init(&mbc[k]); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    after_previous();  // the tables above are constant; what follows was written by this answer's kernels
    const uint32_t rank_limb = (uint32_t)((p << 1) | (1 - l));   // same poly, other limb
    const uint32_t rank_poly = (uint32_t)(((1 - p) << 1) | l);   // other poly, same limb
    const uint32_t* pbq = packed_b + (size_t)b * pb_qstride;
    auto src_of = [&](size_t i) -> const uint32_t* {
        return p ? pbq + (i * 2 + l) * kN : pre_a + (i * 2 + l) * kN;
    };
    // RGSW rows of this poly for digit gp: to own output (p' = p) and to the other (p' = 1 - p)
    const uint32_t* rg = rgsw32 + (size_t)b * (4 * kDeff * 2 * kN);
    uint32_t r_self[8] = {}, r_oth[8] = {};
    if (steps) ld8(rg + (size_t)(((2 * p + p) * kDeff + gp) * 2 + l) * kN + 8 * t, r_self);
    if (steps) ld8(rg + (size_t)(((2 * p + (1 - p)) * kDeff + gp) * 2 + l) * kN + 8 * t, r_oth);
    // Shoup factors of the fixed RGSW values: each product below is then
    // exact with one high multiply instead of a 64-bit Barrett reduction.
    uint32_t r_self_p[8], r_oth_p[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        r_self_p[e] = shoup_factor(r_self[e], L.cr, q);
        r_oth_p[e] = shoup_factor(r_oth[e], L.cr, q);
    }
    uint32_t acc[8] = {};
    uint32_t* const st_part = hr.state + (((size_t)b * (gridDim.x >> 2) + ct) * 4 + p * 2 + l) * kN;
    if (gp == 0) ld8((hr.i_first < 0 ? src_of(start + len - 1) : st_part) + 8 * t, acc);
    cluster_sync_all();  // every CTA runs and its mbarriers are initialised before any remote access
    const uint32_t peer_x = map_peer(xpart, rank_limb);
    const uint32_t peer_c = map_peer(cin, rank_poly);
    const uint32_t peer_mbx = map_peer(mbx, rank_limb);
    const uint32_t peer_mbc = map_peer(mbc, rank_poly);
    int step = 0;
    for (long i = i_first; i >= (long)hr.i_last; --i, ++step) {
        const int par = step & 1;
        const uint32_t ph = (uint32_t)(step >> 1) & 1;
        if (threadIdx.x == 0) {
            hb_expect(&mbx[par], kN * 4);
            hb_expect(&mbc[par], kN * 4);
        }
        uint32_t pk[8];
        if (gp == 0) {
            ld8(src_of(start + (size_t)i) + 8 * t, pk);
            ntt_inv(acc, nbuf, twi, q, scale, t, bar);   // acc: t_l at index t + 256 e
            const uint32_t dst = peer_x + (uint32_t)(par * kN + 4 * t) * 4;
            st_async4(dst, acc[0], acc[1], acc[2], acc[3], peer_mbx + 8 * par);
            st_async4(dst + kHalf * 4, acc[4], acc[5], acc[6], acc[7], peer_mbx + 8 * par);
            st8_sh(xown, t, acc);
        }
        __syncthreads();  // xown complete; abort_flag is read only here, after a block barrier,
                          // so every thread takes the same branch
        if (abort_flag) break;
        uint32_t d[8], v[8];
        ld8_sh(xown, t, d);
        if (!hb_wait(&mbx[par], ph, err, 31)) abort_flag = 1;
        ld8_sh(xpart + par * kN, t, v);
#pragma unroll
        for (int e = 0; e < 8; ++e) d[e] = digit_res(d[e], v[e], q, q_oth, carry, gp);
        ntt_fwd_lazy(d, nbuf + gp * kNttBuf, twf, q, t, bar);
        // The contribution that stays with this group, and the other one through
        // shared memory ([0, 2q) each).
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const uint32_t es = shoup_mul(d[e], r_self[e], r_self_p[e], q);
            const uint32_t eo = shoup_mul(d[e], r_oth[e], r_oth_p[e], q);
            d[e] = gp ? eo : es;
            v[e] = gp ? es : eo;
        }
        st8_sh(cown + gp * kN, t, v);
        __syncthreads();
        ld8_sh(cown + (1 - gp) * kN, t, v);
#pragma unroll
        for (int e = 0; e < 8; ++e) d[e] += v[e];
        if (gp) {
            const uint32_t dst = peer_c + (uint32_t)(par * kN + 4 * t) * 4;
            st_async4(dst, d[0], d[1], d[2], d[3], peer_mbc + 8 * par);
            st_async4(dst + kHalf * 4, d[4], d[5], d[6], d[7], peer_mbc + 8 * par);
        } else {
            if (!hb_wait(&mbc[par], ph, err, 32)) abort_flag = 1;
            ld8_sh(cin + par * kN, t, v);
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] = red2(d[e] + v[e] + pk[e], q);  // of at most 9q
        }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = csub(acc[e], q);
    if (gp == 0 && hr.i_last == 0) {
        uint64_t* dst = resp + (size_t)b * resp_qstride + ((size_t)ct * 4 + p * 2 + l) * kN + 8 * t;
#pragma unroll
        for (int e = 0; e < 8; e += 2)
            *reinterpret_cast<ulonglong2*>(dst + e) = make_ulonglong2(acc[e], acc[e + 1]);
    } else if (gp == 0) {
        st8(st_part + 8 * t, acc);  // the chain resumes from here in the next launch
    }
    cluster_sync_all();  // no CTA leaves while a peer may still write into its shared memory
}

// ------------------------------------------------------------------ horner (8-CTA cluster)
// The chain on a cluster of eight CTAs of 256 threads, CTA rank
// r = 4p + 2l + j owning polynomial p, limb l and gadget digit j.  Both digit
// CTAs of (p, l) hold the same accumulator and run its inverse NTT; each
// sends its lift terms to the other limb's CTA of the same digit (the lift
// needs both limbs), decomposes and forward-transforms only its digit, and
// multiplies it by the RGSW rows of its polynomial.  The contribution to its
// own polynomial goes to the sibling digit CTA, the one to the other
// polynomial to both digit CTAs of that polynomial; every CTA then sums its
// own, its sibling's and the two other-polynomial contributions (both
// siblings add the same residues: their accumulators agree mod q).
// Remote data moves with st.async and completes on the receiver's
// transaction mbarriers (8 KB of lift terms, 24 KB of contributions per
// step); buffers alternate with the step parity, and every remote write for
// step t depends on data its receiver sent after reading the same buffer at
// step t - 2.  Half the warps per SM of the 4-CTA version, twice the SMs.
constexpr size_t kHornerCl8Smem =
    2 * kN * sizeof(uint2) + (kNttBuf + 2 * kN + 2 * 3 * kN) * sizeof(uint32_t) + 64;
constexpr size_t kHornerCl8AloneSmem = 116 * 1024;  // more than half an SM's
static_assert(kHornerCl8Smem <= kHornerCl8AloneSmem, "room for the kernel's own");

__global__ void __cluster_dims__(8, 1, 1) __launch_bounds__(256, 1)
    horner_cl8_kernel(const uint32_t* __restrict__ pre_a, const uint32_t* __restrict__ packed_b, size_t pb_qstride,
                      const uint32_t* __restrict__ rgsw32, const DevTables* __restrict__ T, size_t groups,
                      size_t d_act, uint64_t* __restrict__ resp, size_t resp_qstride, int* err, HornerRange hr) {
    extern __shared__ __align__(16) uint8_t smem[];
    uint2* twf = reinterpret_cast<uint2*>(smem);
    uint2* twi = twf + kN;
    uint32_t* nbuf = reinterpret_cast<uint32_t*>(twi + kN);  // NTT scratch
    uint32_t* xc = nbuf + kNttBuf;                           // [parity] partner limb's lift terms
    uint32_t* cin = xc + 2 * kN;                             // [parity][sibling | other j0 | other j1]
    uint64_t* mbx = reinterpret_cast<uint64_t*>(cin + 2 * 3 * kN);  // [parity] partner terms
    uint64_t* mbc = mbx + 2;                                         // [parity] contributions
    __shared__ volatile int abort_flag;
    let_next_start();
    const uint32_t rank = cluster_rank();
    const int p = (int)(rank >> 2), l = (int)((rank >> 1) & 1), j = (int)(rank & 1);
    const int ct = blockIdx.x >> 3, b = blockIdx.y;
    const uint32_t t = threadIdx.x;
    const LimbTables& L = T->limb[l];
    const uint32_t q = L.q;
    const uint32_t q_oth = T->limb[1 - l].q;
    const uint64_t carry = j ? kCarry2 : kCarry1;
    const NttScale scale = L.scale_crt;
    const size_t start = (size_t)ct * d_act;
    const size_t len = (start + d_act <= groups) ? d_act : groups - start;
    const long i_first = hr.i_first < 0 ? (long)len - 2 : (long)hr.i_first;
    const bool steps = i_first >= (long)hr.i_last;  // one group: the response is its packed ciphertext
    for (int i = threadIdx.x; steps && i < kN; i += 256) { twf[i] = L.fwd[i]; twi[i] = L.inv[i]; }
    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int k = 0; k < 2; ++k) { hb_init(&mbx[k]); hb_init(&mbc[k]); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    after_previous();  // the tables above are constant; what follows was written by this answer's kernels
    const uint32_t rank_limb = (uint32_t)((p << 2) | ((1 - l) << 1) | j);   // same poly and digit, other limb
    const uint32_t rank_sib = (uint32_t)((p << 2) | (l << 1) | (1 - j));    // same poly and limb, other digit
    const uint32_t rank_o0 = (uint32_t)(((1 - p) << 2) | (l << 1) | 0);     // other poly, same limb, digit 0
    const uint32_t rank_o1 = (uint32_t)(((1 - p) << 2) | (l << 1) | 1);     //                        digit 1
    const uint32_t* pbq = packed_b + (size_t)b * pb_qstride;
    auto src_of = [&](size_t i) -> const uint32_t* {
        return p ? pbq + (i * 2 + l) * kN : pre_a + (i * 2 + l) * kN;
    };
    const uint32_t* rg = rgsw32 + (size_t)b * (4 * kDeff * 2 * kN);
    uint32_t r_self[8] = {}, r_oth[8] = {};
    if (steps) ld8(rg + (size_t)(((2 * p + p) * kDeff + j) * 2 + l) * kN + 8 * t, r_self);
    if (steps) ld8(rg + (size_t)(((2 * p + (1 - p)) * kDeff + j) * 2 + l) * kN + 8 * t, r_oth);
    // Shoup factors of the fixed RGSW values: each product below is then
    // exact with one high multiply instead of a 64-bit Barrett reduction.
    uint32_t r_self_p[8], r_oth_p[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        r_self_p[e] = shoup_factor(r_self[e], L.cr, q);
        r_oth_p[e] = shoup_factor(r_oth[e], L.cr, q);
    }
    uint32_t acc[8];
    uint32_t* const st_part = hr.state + (((size_t)b * (gridDim.x >> 3) + ct) * 4 + p * 2 + l) * kN;
    ld8((hr.i_first < 0 ? src_of(start + len - 1) : st_part) + 8 * t, acc);
    cluster_sync_all();  // every CTA runs and its mbarriers are initialised before any remote access
    const uint32_t peer_x = map_peer(xc, rank_limb);
    const uint32_t peer_mbx = map_peer(mbx, rank_limb);
    const uint32_t sib_c = map_peer(cin, rank_sib), sib_mbc = map_peer(mbc, rank_sib);
    const uint32_t o0_c = map_peer(cin, rank_o0), o0_mbc = map_peer(mbc, rank_o0);
    const uint32_t o1_c = map_peer(cin, rank_o1), o1_mbc = map_peer(mbc, rank_o1);
    int step = 0;
    for (long i = i_first; i >= (long)hr.i_last; --i, ++step) {
        const int par = step & 1;
        const uint32_t ph = (uint32_t)(step >> 1) & 1;
        const uint32_t* xpart = xc + par * kN;
        uint32_t* cp = cin + (size_t)par * 3 * kN;
        if (threadIdx.x == 0) {
            hb_expect(&mbx[par], kN * 4);
            hb_expect(&mbc[par], 3 * kN * 4);
        }
        uint32_t pk[8];
        ld8(src_of(start + (size_t)i) + 8 * t, pk);
        ntt_inv_head(acc, nbuf, twi, q, t, 0);
        // Read between the transform's two block barriers: the first follows
        // every write of the previous step, the second precedes this step's,
        // so every thread takes the same branch.
        const int stop = abort_flag;
        ntt_inv_tail(acc, nbuf, twi, q, scale, t, 0);   // acc: t_l at index t + 256 e
        if (stop) break;
        {
            const uint32_t dst = peer_x + (uint32_t)(par * kN + 4 * t) * 4;
            st_async4(dst, acc[0], acc[1], acc[2], acc[3], peer_mbx + 8 * par);
            st_async4(dst + kHalf * 4, acc[4], acc[5], acc[6], acc[7], peer_mbx + 8 * par);
        }
        if (!hb_wait(&mbx[par], ph, err, 33)) abort_flag = 1;
        uint32_t d[8];
        ld8_sh(xpart, t, d);
#pragma unroll
        for (int e = 0; e < 8; ++e) d[e] = digit_res(acc[e], d[e], q, q_oth, carry, j);
        ntt_fwd_lazy(d, nbuf, twf, q, t, 0);
        uint32_t es[8], eo[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {  // [0, 2q)
            es[e] = shoup_mul(d[e], r_self[e], r_self_p[e], q);
            eo[e] = shoup_mul(d[e], r_oth[e], r_oth_p[e], q);
        }
        const uint32_t off = (uint32_t)((size_t)par * 3 * kN + 4 * t) * 4;
        const uint32_t off_o = off + (uint32_t)(1 + j) * kN * 4;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t o = h * kHalf * 4;
            st_async4(sib_c + off + o, es[4 * h], es[4 * h + 1], es[4 * h + 2], es[4 * h + 3], sib_mbc + 8 * par);
            st_async4(o0_c + off_o + o, eo[4 * h], eo[4 * h + 1], eo[4 * h + 2], eo[4 * h + 3], o0_mbc + 8 * par);
            st_async4(o1_c + off_o + o, eo[4 * h], eo[4 * h + 1], eo[4 * h + 2], eo[4 * h + 3], o1_mbc + 8 * par);
        }
        if (!hb_wait(&mbc[par], ph, err, 34)) abort_flag = 1;
        uint32_t v1[8], w0[8], w1[8];
        ld8_sh(cp, t, v1);
        ld8_sh(cp + kN, t, w0);
        ld8_sh(cp + 2 * kN, t, w1);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] = red2(es[e] + v1[e] + w0[e] + w1[e] + pk[e], q);  // sum < 9q
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = csub(acc[e], q);
    if (j == 0 && hr.i_last == 0) {
        uint64_t* dst = resp + (size_t)b * resp_qstride + ((size_t)ct * 4 + p * 2 + l) * kN + 8 * t;
#pragma unroll
        for (int e = 0; e < 8; e += 2)
            *reinterpret_cast<ulonglong2*>(dst + e) = make_ulonglong2(acc[e], acc[e + 1]);
    } else if (j == 0) {
        st8(st_part + 8 * t, acc);  // the chain resumes from here in the next launch
    }
    cluster_sync_all();  // no CTA leaves while a peer may still write into its shared memory
}

// ------------------------------------------------------------------ primitives
__global__ void __launch_bounds__(1024) ntt_batch_kernel(uint32_t* polys, size_t n, int limb_run, bool inverse,
                                                         const DevTables* __restrict__ T) {
    extern __shared__ __align__(16) uint32_t nb[];
    const int gp = threadIdx.x >> 8;
    const uint32_t t = threadIdx.x & 255;
    const size_t idx = (size_t)blockIdx.x * 4 + gp;
    if (idx >= n) return;  // whole group leaves; only group-local barriers follow
    const int l = (int)((idx / (size_t)limb_run) & 1);
    const LimbTables& L = T->limb[l];
    uint32_t* pp = polys + idx * kN;
    uint32_t r[8];
    if (!inverse) {
#pragma unroll
        for (int e = 0; e < 8; ++e) r[e] = pp[t + 256 * e];
        ntt_fwd(r, nb + gp * kNttBuf, L.fwd, L.q, t, 1 + gp);
        st8(pp + 8 * t, r);
    } else {
        ld8(pp + 8 * t, r);
        ntt_inv(r, nb + gp * kNttBuf, L.inv, L.q, L.scale_n, t, 1 + gp);
#pragma unroll
        for (int e = 0; e < 8; ++e) pp[t + 256 * e] = r[e];
    }
}

__global__ void decomp_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, size_t n,
                              const DevTables* __restrict__ T) {
    const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n * kN) return;
    const size_t i = k / kN, x = k % kN;
    int32_t s1, s2;
    decomp2(in[(i * 2) * kN + x], in[(i * 2 + 1) * kN + x], *T, s1, s2);
    uint32_t* o = out + i * kDeff * 2 * kN;
    o[(0 * 2 + 0) * kN + x] = signed_res(s1, kQ0);
    o[(0 * 2 + 1) * kN + x] = signed_res(s1, kQ1);
    o[(1 * 2 + 0) * kN + x] = signed_res(s2, kQ0);
    o[(1 * 2 + 1) * kN + x] = signed_res(s2, kQ1);
}

__global__ void __launch_bounds__(256) fill_db_kernel(uint16_t* __restrict__ out, size_t count, uint64_t seed) {
    for (size_t k = (size_t)blockIdx.x * 256 + threadIdx.x; k < count; k += (size_t)gridDim.x * 256) {
        uint64_t x = (seed ^ k) + 0x9e3779b97f4a7c15ULL;
        x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
        x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
        x ^= x >> 31;
        out[k] = (uint16_t)(x % 65535u);
    }
}

__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
    x += 0x9e3779b97f4a7c15ULL;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
    return x ^ (x >> 31);
}

// Synthetic queries for load generation: word k of query `id` (flat layout
// [b limb0: R][b limb1: R][6 blocks of [digit][limb][N]]) is
// splitmix64(splitmix64(seed ^ id * C) ^ k) mod q_l, l the limb of word k.
// Grid-stride over count * qstride words, coalesced writes.
__global__ void __launch_bounds__(256) synth_query_kernel(uint64_t* __restrict__ out, size_t rows, size_t qstride,
                                                          size_t count, uint64_t seed, uint64_t first_id) {
    const size_t total = count * qstride;
    for (size_t w = (size_t)blockIdx.x * 256 + threadIdx.x; w < total; w += (size_t)gridDim.x * 256) {
        const size_t j = w / qstride, k = w - j * qstride;
        const uint64_t h = splitmix64(seed ^ ((first_id + j) * 0xd1b54a32d192ed03ULL));
        const uint64_t x = splitmix64(h ^ k);
        const int l = k < rows ? 0 : k < 2 * rows ? 1 : (int)(((k - 2 * rows) / kN) & 1);
        out[w] = x % (l ? kQ1 : kQ0);
    }
}

}  // namespace

cudaError_t launch_synth_queries(uint64_t* out, size_t rows, size_t count, uint64_t seed, uint64_t first_id,
                                 cudaStream_t s) {
    if (count == 0) return cudaSuccess;
    const size_t qstride = 2 * rows + 6 * (size_t)kDeff * 2 * kN;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const size_t blocks = std::min<size_t>((count * qstride + 255) / 256, (size_t)sms * 16);
    synth_query_kernel<<<(unsigned)blocks, 256, 0, s>>>(out, rows, qstride, count, seed, first_id);
    return cudaGetLastError();
}

cudaError_t launch_fill_db(uint16_t* out, size_t count, uint64_t seed, cudaStream_t s) {
    if (count == 0) return cudaSuccess;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const size_t blocks = std::min<size_t>((count + 255) / 256, (size_t)sms * 16);
    fill_db_kernel<<<(unsigned)blocks, 256, 0, s>>>(out, count, seed);
    return cudaGetLastError();
}

// ==================================================================== wrappers
cudaError_t launch_qprep(const uint64_t* qraw, size_t qstride, size_t rows, const DevTables* T, uint8_t* kplanes,
                         uint32_t* keys, uint32_t* rgsw32, uint8_t* planes, int nq, int parts, cudaStream_t s) {
    if (nq <= 0) return cudaSuccess;
    if (parts < 1 || parts > (kPrepKeys | kPrepRgsw | kPrepPlanes)) return cudaErrorInvalidValue;
    if ((parts & kPrepPlanes) && rows % 1024) return cudaErrorInvalidValue;
    const int n_key = (parts & kPrepKeys) ? kKeyBlocks : 0, n_rgsw = (parts & kPrepRgsw) ? kRgswBlocks : 0;
    const int n_plane = (parts & kPrepPlanes) ? (int)(rows / 1024) : 0;
    return launch_overlapped(qprep_kernel, dim3(nq, n_key + n_rgsw + n_plane), 256, 0, s, qraw, qstride, rows, T, kplanes,
                             keys, rgsw32, planes, n_key, n_rgsw);
}

cudaError_t launch_matvec(const uint16_t* db, size_t rows, size_t cols, int chunks, const uint64_t* qraw,
                          size_t qstride, const DevTables* T, uint32_t* part, size_t part_qstride, int nq,
                          cudaStream_t s) {
    if (nq <= 0) return cudaSuccess;
    if (nq > 4 || chunks <= 0 || rows % (size_t)chunks) return cudaErrorInvalidValue;
    const int rpc = (int)(rows / chunks);
    if (rpc > (1 << 20)) return cudaErrorInvalidValue;
    const int bt = nq == 1 ? 1 : (nq == 2 ? 2 : 4);
    const size_t smem = (size_t)bt * 2 * rpc * sizeof(uint32_t);
    cudaError_t e;
    if (bt == 1) {
        auto k = matvec_kernel<1, 8>;
        if ((e = allow_max_smem(k))) return e;
        k<<<dim3((unsigned)(cols / 2048), chunks), 256, smem, s>>>(db, rows, cols, rpc, qraw, qstride, T, part,
                                                                   part_qstride, nq);
    } else if (bt == 2) {
        auto k = matvec_kernel<2, 4>;
        if ((e = allow_max_smem(k))) return e;
        k<<<dim3((unsigned)(cols / 1024), chunks), 256, smem, s>>>(db, rows, cols, rpc, qraw, qstride, T, part,
                                                                   part_qstride, nq);
    } else {
        auto k = matvec_kernel<4, 4>;
        if ((e = allow_max_smem(k))) return e;
        k<<<dim3((unsigned)(cols / 1024), chunks), 256, smem, s>>>(db, rows, cols, rpc, qraw, qstride, T, part,
                                                                   part_qstride, nq);
    }
    return cudaGetLastError();
}

cudaError_t launch_finalize(const uint32_t* mvpart, size_t mv_qstride, int mv_chunks, size_t cols,
                            const uint32_t* tp_out, const uint32_t* df, const uint32_t* keys, size_t key_qstride,
                            const DevTables* T, uint32_t* packed_b, size_t pb_qstride, size_t groups, int nq,
                            cudaStream_t s) {
    return launch_finalize_range(mvpart, mv_qstride, mv_chunks, cols, tp_out, df, keys, key_qstride, T, packed_b,
                                 pb_qstride, groups, 0, groups, nq, s);
}

cudaError_t launch_finalize_range(const uint32_t* mvpart, size_t mv_qstride, int mv_chunks, size_t cols,
                                  const uint32_t* tp_out, const uint32_t* df, const uint32_t* keys,
                                  size_t key_qstride, const DevTables* T, uint32_t* packed_b, size_t pb_qstride,
                                  size_t groups, size_t g0, size_t gn, int nq, cudaStream_t s) {
    if (nq <= 0) return cudaSuccess;
    if (gn == 0 || g0 + gn > groups) return cudaErrorInvalidValue;
    return launch_overlapped(finalize_kernel, dim3((unsigned)gn, 2, nq), 256, 0, s, mvpart, mv_qstride, mv_chunks, cols,
                             tp_out, (int)g0, df, keys, key_qstride, T, packed_b, pb_qstride);
}

cudaError_t launch_horner(const uint32_t* pre_a, const uint32_t* packed_b, size_t pb_qstride,
                          const uint32_t* rgsw32, const DevTables* T, size_t groups, size_t d_act,
                          size_t num_cts, uint64_t* resp, size_t resp_qstride, int nq, cudaStream_t s) {
    if (nq <= 0) return cudaSuccess;
    cudaError_t e = allow_max_smem(horner_kernel);
    if (e) return e;
    horner_kernel<<<dim3((unsigned)num_cts, nq), 1024, kHornerSmem, s>>>(pre_a, packed_b, pb_qstride, rgsw32, T,
                                                                          groups, d_act, resp, resp_qstride);
    return cudaGetLastError();
}

static bool horner_range_ok(const HornerRange& hr, size_t d_act) {
    if (hr.i_first < 0 && hr.i_last == 0) return true;  // the whole chain
    return hr.state && hr.i_last >= 0 && hr.i_first < (long)d_act - 1 && (hr.i_first < 0 || hr.i_first >= hr.i_last);
}

cudaError_t launch_horner_cluster(const uint32_t* pre_a, const uint32_t* packed_b, size_t pb_qstride,
                                  const uint32_t* rgsw32, const DevTables* T, size_t groups, size_t d_act,
                                  size_t num_cts, uint64_t* resp, size_t resp_qstride, int nq, int* err,
                                  cudaStream_t s, HornerRange hr) {
    if (nq <= 0) return cudaSuccess;
    if (!horner_range_ok(hr, d_act)) return cudaErrorInvalidValue;
    cudaError_t e = allow_max_smem(horner_cl_kernel);
    if (e) return e;
    return launch_overlapped(horner_cl_kernel, dim3((unsigned)(4 * num_cts), nq), 512, kHornerClSmem, s, pre_a, packed_b,
                             pb_qstride, rgsw32, T, groups, d_act, resp, resp_qstride, err, hr);
}

size_t horner_cl8_chains() {
    static std::atomic<int> known[64];
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    if ((n = known[dev].load()) > 0) return (size_t)n;
    cudaLaunchConfig_t cfg{};  // the cluster's size is the kernel's own
    cfg.gridDim = dim3(8);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = kHornerCl8AloneSmem;
    if (allow_max_smem(horner_cl8_kernel) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, horner_cl8_kernel, &cfg) != cudaSuccess || n < 1) {
        cudaGetLastError();
        return 0;
    }
    known[dev].store(n);
    return (size_t)n;
}

cudaError_t launch_horner_cluster8(const uint32_t* pre_a, const uint32_t* packed_b, size_t pb_qstride,
                                   const uint32_t* rgsw32, const DevTables* T, size_t groups, size_t d_act,
                                   size_t num_cts, uint64_t* resp, size_t resp_qstride, int nq, int* err,
                                   cudaStream_t s, HornerRange hr) {
    if (nq <= 0) return cudaSuccess;
    if (!horner_range_ok(hr, d_act)) return cudaErrorInvalidValue;
    cudaError_t e = allow_max_smem(horner_cl8_kernel);
    if (e) return e;
    // A whole chain starts while the kernel before it still holds SMs.  Two of its
    // CTAs fit one SM, and clusters that are placed so share it for the whole chain
    // (10 queries, 128 groups on 2048 rows: 2037 us, started late 1811).  Chains that
    // can all have SMs of their own ask for so much shared memory that they get
    // them (1810).
    const bool alone = hr.i_first < 0 && hr.i_last == 0 && (size_t)nq * num_cts <= horner_cl8_chains();
    return launch_overlapped(horner_cl8_kernel, dim3((unsigned)(8 * num_cts), nq), 256,
                             alone ? kHornerCl8AloneSmem : kHornerCl8Smem, s, pre_a, packed_b, pb_qstride, rgsw32, T,
                             groups, d_act, resp, resp_qstride, err, hr);
}

cudaError_t launch_ntt_batch(uint32_t* polys, size_t n, int limb_run, bool inverse, const DevTables* T,
                             cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const size_t smem = 4 * kNttBuf * sizeof(uint32_t);
    cudaError_t e = allow_max_smem(ntt_batch_kernel);
    if (e) return e;
    ntt_batch_kernel<<<(unsigned)((n + 3) / 4), 1024, smem, s>>>(polys, n, limb_run, inverse, T);
    return cudaGetLastError();
}

cudaError_t launch_decomp(const uint32_t* in, uint32_t* out, size_t n, const DevTables* T, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    decomp_kernel<<<(unsigned)((n * kN + 255) / 256), 256, 0, s>>>(in, out, n, T);
    return cudaGetLastError();
}

}  // namespace ipb

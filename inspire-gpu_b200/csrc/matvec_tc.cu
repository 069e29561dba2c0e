// matvec_tc.cu -- exact database x query mat-vec on the tcgen05 tensor cores.
//
//   r_l[q][j] = sum_i db[i][j] * b_{q,l}[i]  mod q_l      (reference src/gpu_online.cu:23-175)
//
// The row-major u16 DB is read, unchanged, as a u8 matrix A'[m'][i] with
// m' = 2j + byte (lo byte at even m', hi byte at odd m'): consecutive m' are
// contiguous, i.e. an MN-major operand.  A query's two limbs are combined
// by CRT into one word B[i] < q0*q1 < 2^53 (B = b_{q,l}[i] mod q_l for both
// limbs), split into 7 bytes: B[n][i] with n = 7q + k holds byte k of query
// q's B[i] (K-major rows built by qplanes_kernel).  One
// tcgen05.mma.kind::i8 chain accumulates D[m'][n] = sum_i A'[m'][i] B[n][i]
// in s32 TMEM.  With K <= 32768 rows per chunk every D entry is
// <= 255*255*32768 < 2^31: exact.  The epilogue forms, per limb, the sum over
// both byte rows of sum_k (256^(k + byte) mod q_l) D[m'][n_k] (< 2^62) and
// reduces it: the exact sum_i db[i][j] b_{q,l}[i] mod q_l.  All arithmetic
// stays exact, so the result equals the reference's.  Seven planes per query instead of four
// per limb: 12.5 % fewer MMAs and query-plane bytes.
//
// CTA roles (384 threads): warp 0 issues TMA loads (DB tile 256 x 64 rows as
// two 128-byte boxes, query planes N x 64), warp 1 allocates TMEM and one
// thread issues the MMAs, warps 4..11 drain TMEM (tcgen05.ld), four each half
// of the tile, and write partial sums.  Stages are recycled through mbarriers; every wait is
// bounded and reports a timeout through *err instead of hanging.
//
// Work items (m'-tile, K-chunk) are handed out dynamically: the producer
// thread takes the next item from an atomic counter (zero between launches: a
// launch's last CTA puts it back) and publishes it to the MMA thread and the epilogue through a
// ring of kRing shared slots; -1 ends the sequence.  SMs that other kernels
// hold when this one starts (the previous batch's Horner, another lane)
// simply take fewer items instead of delaying the whole pass.
#include <cuda.h>

#include "ipb_common.cuh"
#include "host_util.h"
#include "ipb_launch.h"
#include "matvec_rules.h"
#include "tc_ptx.cuh"

namespace ipb {

namespace {
using namespace tc;

constexpr int kRing = 8;          // published work items in flight
struct TcParams {
    uint32_t* part;        // [q][chunk][limb][ld], first column of the range at part
    size_t part_qstride;
    size_t cols;           // columns in the range
    size_t ld;             // columns per (chunk, limb) row of part
    int nq;                // queries in this pass (<= 32)
    int npad;              // N = 16 ceil(7 nq / 16) (<= 224)
    uint32_t c[2][kPlanes + 1];  // 256^k mod q_l
    int n_mtiles;
    int mt_per_range;      // > 0: the m' tiles cover ranges of this many tiles, range r starting
    int range_stride_m;    // r * range_stride_m m' rows after the first (several column ranges in one
                           // launch); 0: one contiguous range
    int n_kchunks;
    int kchunk_rows;
    int stages;
    int acc_stages;
    uint32_t tmem_cols;
    int* err;
    unsigned* tiles;       // [0] work-item counter, [1] CTAs done: both zero between launches
    const DevTables* T;
    int has_qmap;          // output row of pass query q: qmap[q] (else q)
    uint8_t qmap[32];
    int abort_after;       // > 0: the MMA issuer stops after this many m' tiles and reports code 99 (a test of
                           // the abort path, IPB_TEST_ABORT_AFTER_ITEMS); 0: off
};

// First m' row (2 x column, relative to the launch's first column) of m'
// tile mt: tiles of one contiguous range, or of several equal ranges
// range_stride_m apart.
__device__ __forceinline__ int mtile_m0(const TcParams& P, int mt) {
    return P.mt_per_range ? (mt / P.mt_per_range) * P.range_stride_m + (mt % P.mt_per_range) * kMT : mt * kMT;
}

constexpr int kMvThreads = 384;
constexpr int kEpiThreads = 256;

// MT: m' tiles per work item, 1 or 2 (two adjacent ones, 512 bytes of a row,
// that share a stage's query planes; mv_tiles has the rule).
// Bound by HBM up to about 8 queries and by power beyond: the same launch takes
// 3.05 ms alone and 3.9 ms back to back at 32 queries over 16 GB.  Two tiles
// halve the planes' way from L2 through shared memory: back to back over 16 GB
// 2.78 -> 2.59 ms at 8 queries, 3.17 -> 2.93 at 16; over 4 GB, where fewer,
// longer items also leave less of a tail, 0.69 -> 0.64 at 1 and 0.79 -> 0.75 at
// 16.
template <int MT>
__global__ void __launch_bounds__(kMvThreads, 1) mv_tc_kernel(const __grid_constant__ CUtensorMap map_a,
                                                       const __grid_constant__ CUtensorMap map_b, TcParams P) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int S = P.stages;
    constexpr uint32_t a_bytes = kKT * 128;          // one 128-byte m' box x kKT rows
    const uint32_t b_bytes = (uint32_t)P.npad * kKT;
    const uint32_t stage_bytes = 2 * MT * a_bytes + b_bytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)S * stage_bytes);
    uint64_t* full = bars;
    uint64_t* empty = bars + S;
    uint64_t* tfull = bars + 2 * S;
    uint64_t* tempty = bars + 2 * S + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S + 4);
    __shared__ volatile int abort_flag;
    __shared__ volatile int item_ring[kRing];
    __shared__ uint64_t ifull[kRing], iempty[kRing];
    __shared__ uint64_t mma_done;  // the MMA issuer's final commit: all its MMAs have completed

    let_next_start();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < S; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(&tfull[a], 1); mbar_init(&tempty[a], kEpiThreads); }
        for (int r = 0; r < kRing; ++r) { mbar_init(&ifull[r], 1); mbar_init(&iempty[r], 1 + kEpiThreads); }
        mbar_init(&mma_done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(P.tmem_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    after_previous();
    const uint32_t tmem_base = *tmem_slot;
    const int n_mitems = P.n_mtiles / MT, n_items = n_mitems * P.n_kchunks;
    const int ktiles = P.kchunk_rows / kKT;

    if (warp == 0) {
        // ---------------- TMA producer
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 0;
            unsigned issued = 0;  // stage loads issued
            for (int it = 0;; ++it) {
                const int r = it % kRing;
                int item = -1;
                if (!abort_flag && mbar_wait_ab(&iempty[r], ((uint32_t)(it / kRing) & 1) ^ 1, P.err, 6, &abort_flag)) {
                    const unsigned t = atomicAdd(P.tiles, 1u);
                    if (t < (unsigned)n_items) item = (int)t;
                } else {
                    abort_flag = 1;
                }
                item_ring[r] = item;
                mbar_arrive(&ifull[r]);
                if (item < 0) break;
                const int mt = item % n_mitems * MT, kc = item / n_mitems;
                const int m0 = mtile_m0(P, mt);
                for (int kt = 0; kt < ktiles; ++kt) {
                    if (!mbar_wait_ab(&empty[s], ph ^ 1, P.err, 1, &abort_flag)) { abort_flag = 1; break; }
                    uint8_t* st = smem + (size_t)s * stage_bytes;
                    mbar_expect_tx(&full[s], stage_bytes);
                    const int k0 = kc * P.kchunk_rows + kt * kKT;
#pragma unroll
                    for (int h = 0; h < 2 * MT; ++h)
                        tma_load_2d(st + h * a_bytes, &map_a, &full[s], m0 + 128 * h, k0);
                    tma_load_2d(st + 2 * MT * a_bytes, &map_b, &full[s], k0, 0);
                    ++issued;
                    if (++s == S) { s = 0; ph ^= 1; }
                }
            }
            // Drain: every issued load has landed in shared memory before the
            // CTA exits, also when the MMA issuer stopped early (a timeout) and
            // never consumed them.  Load n went to stage n % S with phase
            // (n / S) & 1; no later load reuses a stage, so each wait is exact.
            for (unsigned i = 0; i < (unsigned)S && i < issued; ++i) {
                const unsigned n = issued - 1 - i;
                mbar_wait(&full[n % S], (n / S) & 1u, P.err, 2);
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer
        if (lane == 0) {
            const uint32_t idesc = idesc_i8(P.npad), desc0 = smem_desc_lo(smem, 0);
            int s = 0, as = 0;
            uint32_t ph = 0, aph = 0;
            bool it_mma = false;  // any MMA issued
            for (int it = 0;; ++it) {
                const int r = it % kRing;
                if (!mbar_wait_ab(&ifull[r], (uint32_t)(it / kRing) & 1, P.err, 7, &abort_flag)) {
                    abort_flag = 1;
                    break;
                }
                const int item = item_ring[r];
                mbar_arrive(&iempty[r]);
                if (item < 0 || abort_flag) break;
                if (P.abort_after > 0 && it * MT >= P.abort_after) {  // test hook: the designed early stop
                    atomicCAS(P.err, 0, 99);
                    abort_flag = 1;
                    break;
                }
                if (!mbar_wait_ab(&tempty[as], aph ^ 1, P.err, 3, &abort_flag)) { abort_flag = 1; break; }
                tc_fence_after();
                const uint32_t d0 = tmem_base + (uint32_t)(as * 2 * MT * P.npad);
                for (int kt = 0; kt < ktiles; ++kt) {
                    if (!mbar_wait_ab(&full[s], ph, P.err, 4, &abort_flag)) { abort_flag = 1; break; }
                    tc_fence_after();
                    // A: MN-major, rows of 128 bytes, 8-row swizzle atoms (SBO 1024 B);
                    // K advances 32 rows = 4096 bytes per MMA.
                    // B: K-major, 64-byte rows (SWIZZLE_64B), 8-row groups 512 B apart; K advances 32 bytes.
                    if (MT == 1) {
                        // Whole descriptors, which takes the thread longer: at 32 queries
                        // and a burst of launches 1.55 ms over 8 GB against 1.55-1.89 with
                        // the MMAs issued at once.
                        const uint8_t* st = smem + (size_t)s * stage_bytes;
#pragma unroll
                        for (int kk = 0; kk < kKT / 32; ++kk) {
                            const uint64_t a0 = smem_desc(st + kk * 4096, 0, 1024);
                            const uint64_t a1 = smem_desc(st + a_bytes + kk * 4096, 0, 1024);
                            const uint64_t b = smem_desc_sw64(st + 2 * a_bytes + kk * 32, 512);
                            const uint32_t acc = (kt > 0 || kk > 0) ? 1u : 0u;
                            mma_i8(d0, a0, b, idesc, acc);
                            mma_i8(d0 + (uint32_t)P.npad, a1, b, idesc, acc);
                        }
                    } else {
                        // A descriptor is one 32-bit add (the address field of its low word).
                        const uint32_t ad = desc0 + (uint32_t)s * (stage_bytes >> 4);
                        const uint32_t bd = ad + (2 * MT * a_bytes >> 4) + (1u << 16);
#pragma unroll
                        for (int kk = 0; kk < kKT / 32; ++kk)
#pragma unroll
                            for (int h = 0; h < 2 * MT; ++h)
                                mma_i8_lo(d0 + (uint32_t)(h * P.npad), ad + h * (a_bytes >> 4) + kk * 256, bd + kk * 2,
                                          smem_desc_hi_sw128(1024), smem_desc_hi_sw64(512), idesc,
                                          (kt > 0 || kk > 0) ? 1u : 0u);
                    }
                    it_mma = true;
                    mma_commit(&empty[s]);
                    if (++s == S) { s = 0; ph ^= 1; }
                }
                mma_commit(&tfull[as]);
                if (++as == P.acc_stages) { as = 0; aph ^= 1; }
            }
            // Every MMA this thread issued has completed (also after an early
            // stop) before TMEM is deallocated and shared memory released.
            if (it_mma) {
                mma_commit(&mma_done);
                mbar_wait(&mma_done, 0, P.err, 9);
            }
        }
    } else if (warp >= 4) {
        // ---------------- epilogue: TMEM -> u64 dot products -> mod q
        // An accumulator set of more than 256 columns (more than 18 queries, or
        // 9 with two tiles) is not double-buffered: the MMAs wait while it is drained, so the
        // epilogue's length counts.  Two warps per TMEM lane quarter, one half
        // of each m' tile each; the weights of the lane's byte row (lo bytes in
        // even lanes, hi in odd) are in registers, and the pair of lanes of a
        // column meets once per query in 64 bits: the even lane reduces and
        // writes limb 0, the odd one limb 1.
        const int wq = warp & 3, mb = (warp - 4) >> 2, hi = lane & 1;
        const uint32_t lane_base = (uint32_t)(wq * 32) << 16;
        int as = 0;
        uint32_t aph = 0;
        const uint64_t cr = P.T->limb[hi].cr;
        const uint32_t ql = hi ? kQ1 : kQ0;
        uint32_t w0[kPlanes], w1[kPlanes];
#pragma unroll
        for (int k = 0; k < kPlanes; ++k) {
            w0[k] = P.c[0][k + hi];
            w1[k] = P.c[1][k + hi];
        }
        for (int it = 0;; ++it) {
            const int r = it % kRing;
            if (!mbar_wait_ab(&ifull[r], (uint32_t)(it / kRing) & 1, P.err, 8, &abort_flag)) { abort_flag = 1; break; }
            const int item = item_ring[r];
            mbar_arrive(&iempty[r]);
            if (item < 0) break;
            if (!mbar_wait_ab(&tfull[as], aph, P.err, 5, &abort_flag)) { abort_flag = 1; break; }
            tc_fence_after();
            const int mt = item % n_mitems * MT, kc = item / n_mitems;
            const int m0 = mtile_m0(P, mt);
#pragma unroll
            for (int hb = mb; hb < 2 * MT; hb += 2) {  // 128-row halves of the item
                const size_t col = ((size_t)m0 + hb * 128 + wq * 32 + lane) >> 1;
                uint32_t* const out = P.part + ((size_t)kc * 2 + hi) * P.ld + col;
                const uint32_t acc = tmem_base + lane_base + (uint32_t)(as * 2 * MT * P.npad + hb * P.npad);
                for (int q0 = 0; q0 < P.nq; q0 += 8) {
                    // queries q0..q0+7: columns 7 q0 .. 7 q0 + 55, seven 8-column
                    // loads (those at or past N are not loaded: they hold no query)
                    uint32_t t[kPlanes][8];
#pragma unroll
                    for (int c = 0; c < kPlanes; ++c) {
                        const int n = kPlanes * q0 + 8 * c;
                        if (n < P.npad) {
                            tmem_ld8_issue(acc + (uint32_t)n, t[c]);
                        } else {
#pragma unroll
                            for (int e = 0; e < 8; ++e) t[c][e] = 0;
                        }
                    }
                    uint32_t v[kPlanes * 8];
#pragma unroll
                    for (int c = 0; c < kPlanes; ++c) {
                        tmem_wait8(t[c]);  // one wait for all seven loads; the others are no-ops
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[8 * c + e] = t[c][e];
                    }
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        if (q0 + e >= P.nq) break;
                        uint64_t a0 = 0, a1 = 0;
#pragma unroll
                        for (int k = 0; k < kPlanes; ++k) {
                            a0 += (uint64_t)w0[k] * v[kPlanes * e + k];
                            a1 += (uint64_t)w1[k] * v[kPlanes * e + k];
                        }
                        const uint64_t sum = (hi ? a1 : a0) + __shfl_xor_sync(0xffffffffu, hi ? a0 : a1, 1);
                        const int qo = P.has_qmap ? P.qmap[q0 + e] : q0 + e;
                        out[(size_t)qo * P.part_qstride] = mod_u64(sum, cr, ql);
                    }
                }
            }
            tc_fence_before();
            mbar_arrive(&tempty[as]);
            if (++as == P.acc_stages) { as = 0; aph ^= 1; }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0) release_counter(P.tiles);
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(P.tmem_cols));
    }
}

// out[q][l][c] = sum over K-chunks of part[q][chunk][l][c]  mod q_l.
__global__ void __launch_bounds__(256) mv_chunk_reduce_kernel(const uint32_t* __restrict__ part, size_t part_qstride,
                                                              int chunks, size_t cols, const DevTables* __restrict__ T,
                                                              uint32_t* __restrict__ out, size_t out_qstride) {
    const int q = blockIdx.y;
    const size_t idx = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (idx >= 2 * cols) return;
    const int l = (int)(idx / cols);
    const size_t c = idx % cols;
    uint64_t s = 0;
#pragma unroll 8
    for (int ch = 0; ch < chunks; ++ch) s += part[(size_t)q * part_qstride + ((size_t)ch * 2 + l) * cols + c];
    out[(size_t)q * out_qstride + (size_t)l * cols + c] = mod_u64(s, T->limb[l].cr, T->limb[l].q);
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) == cudaSuccess &&
            qr == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

}  // namespace

size_t mv_tc_planes_bytes(size_t rows, int max_queries) { return (size_t)kPlanes * max_queries * rows + 16 * rows; }
size_t mv_tc_planes_offset(size_t first_query, size_t rows) { return (size_t)kPlanes * first_query * rows; }

cudaError_t launch_mv_chunk_reduce(const uint32_t* part, size_t part_qstride, int chunks, size_t cols,
                                   const DevTables* T, uint32_t* out, size_t out_qstride, int nq, cudaStream_t s) {
    if (nq <= 0) return cudaSuccess;
    mv_chunk_reduce_kernel<<<dim3((unsigned)((2 * cols + 255) / 256), nq), 256, 0, s>>>(part, part_qstride, chunks,
                                                                                         cols, T, out, out_qstride);
    return cudaGetLastError();
}

cudaError_t launch_matvec_tc(const uint16_t* db, size_t rows, size_t cols, const uint8_t* planes, int nq,
                             const DevTables* T, uint32_t* part, size_t part_qstride, int* err, unsigned* tiles,
                             int num_sms, int kchunk_rows, cudaStream_t s) {
    return launch_matvec_tc_range(db, rows, cols, 0, cols, planes, nq, T, part, part_qstride, nullptr, err, tiles,
                                  num_sms, kchunk_rows, s);
}

cudaError_t launch_matvec_tc_range(const uint16_t* db, size_t rows, size_t ld, size_t c0, size_t c1,
                                   const uint8_t* planes, int nq, const DevTables* T, uint32_t* part,
                                   size_t part_qstride, const uint8_t* qmap, int* err, unsigned* tiles, int num_sms,
                                   int kchunk_rows, cudaStream_t s) {
    if (c1 <= c0) return nq <= 0 ? cudaSuccess : cudaErrorInvalidValue;
    return launch_matvec_tc_ranges(db, rows, ld, c0, c1 - c0, 1, 0, planes, nq, T, part, part_qstride, qmap, err,
                                   tiles, num_sms, kchunk_rows, s);
}

cudaError_t launch_matvec_tc_ranges(const uint16_t* db, size_t rows, size_t ld, size_t c0, size_t cols_per_range,
                                    int n_ranges, size_t range_stride, const uint8_t* planes, int nq,
                                    const DevTables* T, uint32_t* part, size_t part_qstride, const uint8_t* qmap,
                                    int* err, unsigned* tiles, int num_sms, int kchunk_rows, cudaStream_t s,
                                    bool overlap) {
    if (nq <= 0) return cudaSuccess;
    if (n_ranges < 1 || cols_per_range == 0 || cols_per_range % 128 || c0 % 128 ||
        (n_ranges > 1 && (range_stride < cols_per_range || range_stride % 128)))
        return cudaErrorInvalidValue;
    // the launch's columns span [c0, c0 + cols): the ranges and the gaps between them
    const size_t cols = (size_t)(n_ranges - 1) * range_stride + cols_per_range;
    if (c0 + cols > ld) return cudaErrorInvalidValue;
    db += c0;
    part += c0;
    if (nq > 32 || rows % kKT || cols % 128 || !tiles) return cudaErrorInvalidValue;
    EncodeTiledFn enc = encode_fn();
    if (!enc) return cudaErrorNotSupported;
    const int npad = ((kPlanes * nq + 15) / 16) * 16;
    const int kchunk = kchunk_rows;
    if (!mv_kchunk_ok(rows, kchunk)) return cudaErrorInvalidValue;
    CUtensorMap ma, mb;
    {
        cuuint64_t dims[2] = {(cuuint64_t)(2 * cols), (cuuint64_t)rows};
        cuuint64_t strides[1] = {(cuuint64_t)(2 * ld)};
        cuuint32_t box[2] = {128, (cuuint32_t)kKT};
        cuuint32_t es[2] = {1, 1};
        if (enc(&ma, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)db, dims, strides, box, es,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    {
        cuuint64_t dims[2] = {(cuuint64_t)rows, (cuuint64_t)npad};
        cuuint64_t strides[1] = {(cuuint64_t)rows};
        cuuint32_t box[2] = {(cuuint32_t)kKT, (cuuint32_t)npad};
        cuuint32_t es[2] = {1, 1};
        if (enc(&mb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)planes, dims, strides, box, es,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    TcParams P{};
    P.part = part;
    P.part_qstride = part_qstride;
    P.cols = cols;
    P.ld = ld;
    P.has_qmap = qmap != nullptr;
    if (qmap)
        for (int q = 0; q < nq; ++q) P.qmap[q] = qmap[q];
    P.nq = nq;
    P.npad = npad;
    P.abort_after = test_abort_after_items();
    {
        const uint32_t qs[2] = {kQ0, kQ1};
        for (int l = 0; l < 2; ++l) {
            uint64_t c = 1;
            for (int k = 0; k <= kPlanes; ++k, c = c * 256 % qs[l]) P.c[l][k] = (uint32_t)c;
        }
    }
    P.mt_per_range = n_ranges > 1 ? (int)((2 * cols_per_range) / kMT) : 0;
    P.range_stride_m = n_ranges > 1 ? (int)(2 * range_stride) : 0;
    P.n_mtiles = n_ranges > 1 ? n_ranges * P.mt_per_range : (int)((2 * cols) / kMT);
    P.kchunk_rows = kchunk;
    P.n_kchunks = (int)(rows / kchunk);
    const int mt = mv_tiles(nq, rows, ld, kchunk, P.n_mtiles % 2 == 0 && P.mt_per_range % 2 == 0);
    P.acc_stages = (4 * mt * npad <= 512) ? 2 : 1;
    uint32_t need = (uint32_t)(P.acc_stages * 2 * mt * npad);
    uint32_t tc = 32;
    while (tc < need) tc <<= 1;
    P.tmem_cols = tc;
    P.err = err;
    P.tiles = tiles;
    P.T = T;
    const size_t stage_bytes = 2 * mt * (size_t)kKT * 128 + (size_t)npad * kKT;
    const size_t budget = 200 * 1024;
    P.stages = (int)std::min<size_t>(8, budget / stage_bytes);
    if (P.stages < 2) return cudaErrorInvalidValue;
    const size_t smem = 1024 + (size_t)P.stages * stage_bytes + (2 * P.stages + 4) * 8 + 16;
    const auto kernel = mt == 2 ? mv_tc_kernel<2> : mv_tc_kernel<1>;
    cudaError_t e = allow_max_smem(kernel);
    if (e) return e;
    const int items = P.n_mtiles / mt * P.n_kchunks;
    const int grid = std::min(items, std::max(1, num_sms));
    return launch_overlapped_if(overlap, kernel, grid, kMvThreads, smem, s, ma, mb, P);
}

}  // namespace ipb

// Target of the device code this library carries, read back from the loaded
// module (cudaFuncGetAttributes on the tensor-core mat-vec kernel):
// binaryVersion is 100 for sm_100a cubins.  No counterpart in the reference.
extern "C" int ipir_b200_kernel_binary_version(int* out) {
    if (!out) return 1;
    cudaFuncAttributes a{};
    cudaError_t e = cudaFuncGetAttributes(&a, ipb::mv_tc_kernel<1>);
    if (e != cudaSuccess) {
        ipb::set_last_error(cudaGetErrorString(e));
        return 4;
    }
    *out = a.binaryVersion;
    return 0;
}



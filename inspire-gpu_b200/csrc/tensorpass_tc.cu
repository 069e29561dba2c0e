// tensorpass_tc.cu -- the online tensor pass (InspiRINGOnline) as one int8
// tcgen05 GEMM per limb.
//
// For group g, limb l and NTT slot i the reference subtracts
//   T_g[l][i] = sum_{dir, s, j} D_g[dir][l][s][j][i] * K5[l][j][perm_{t(dir,s)}(i)],
// t(dir, s) = +-5^(1022-s) (src/gpu_online.cu:593-714, permutations of
// src/gpu_protocol.cu:169-215), re-reading and re-permuting the query key for
// every group.
//
// Slot i is the evaluation at psi^odd, odd = 2 BR(i) + 1 = sigma 5^k mod 2N
// (sigma = +-1; 5 generates the residues = 1 mod 4), and perm_t(i) is the slot
// of t * odd = +-sigma 5^(k + 1022 - s).  So the terms of slot i meet the
// key's slots in one fixed order, whatever i is, once D is indexed by the key
// position instead of the step: with rho = dir xor (sigma < 0) and
// m = (k + 1022 - s) mod 1024, u = j * 2048 + rho * 1024 + m and
//   D'_g[l][i][u] = D_g[dir][l][s][j][i]     (0 where s would be 1023),
//   K'[l][u]      = K5[l][j][slot of (-1)^rho 5^m],
//   T_g[l][i]     = sum_u D'_g[l][i][u] * K'[l][u].
// K' depends on neither the slot nor the group: per limb the pass over all
// groups, slots and queries is one GEMM, M = (group, slot), N = queries,
// K = 4096, whose N operand is 16 KB per query and limb.  (With D in step
// order every slot needed its own permuted key, gathered from L2 by the
// kernel: 67 MB per query, which bounded the pass at few groups.)
//
// Both operands are < 2^27: split each into four bytes, D's planes in M (row
// 4 i + a) and K's planes in N (column 4 q + b); tcgen05.mma.kind::i8
// accumulates sum_u over bytes exactly in s32 (255^2 * 4096 < 2^31), and the
// epilogue forms sum_{a,b} (256^(a+b) mod q_l) * P[4 i + a][4 q + b] < 2^59
// and reduces mod q_l.  Exact, so equal to the reference.
//
// Layouts.  D' is stored as the kernel reads it: tile t = (2 g + l) * 64 +
// i / 32 holds the 128 rows of 32 slots, as 32 K blocks of 128 rows x 128
// bytes (16 KB), rows already in the SWIZZLE_128B pattern.  A block is one
// contiguous bulk copy, and the pass streams the tensors in address order.
// K' planes: kplanes[q][l][b][4096] u8, written by the query prep.  Output:
// tp_out[q][g][l][N] u32, reduced.
#include <cuda.h>

#include <algorithm>

#include "ipb_common.cuh"
#include "host_util.h"
#include "ipb_launch.h"
#include "tc_ptx.cuh"

namespace ipb {

namespace {
using namespace tc;

constexpr int kK = 4096;                // u range
constexpr int kKBlock = 128;            // bytes of K per stage
constexpr int kKTiles = kK / kKBlock;
constexpr uint32_t kTile = 128 * 128;   // bytes of one 128-row K block
constexpr int kTilesPerPoly = kN / 32;  // 128-row tiles of one (group, limb)
constexpr int kRing = 8;                // published work items in flight
constexpr int kEpiWarps = 8;
constexpr int kTpThreads = 64 + 32 * kEpiWarps;

// Byte (row 4 i + a, position u) of group-limb gl = 2 g + l.
__device__ __forceinline__ size_t dt_addr(size_t gl, uint32_t i, uint32_t a, uint32_t u) {
    const uint32_t r = (i & 31) * 4 + a;
    return ((gl * kTilesPerPoly + (i >> 5)) * kKTiles + (u >> 7)) * kTile + r * 128 +
           ((((u >> 4) ^ r) & 7) << 4) + (u & 15);
}
// Step of slot exponent k at key exponent m (1023: no such step).
__device__ __forceinline__ uint32_t dt_step(uint32_t k, uint32_t m) { return (k + kHalf - 2 - m) & (kHalf - 1); }

// ------------------------------------------------------------------ D re-layout
// Source: one wave of groups in the reference layout [l][s][j][N] (u32) for
// each direction.  CTA: 8 slots x all steps of one (direction, digit), read a
// 32-byte sector per step, written as whole 128-byte rows of the K blocks.
constexpr int kTrStride = kHalf + 4;  // tile row stride: the 8 slots of a step land in distinct banks
__global__ void __launch_bounds__(256) dt_transpose_kernel(const uint32_t* __restrict__ dp,
                                                           const uint32_t* __restrict__ dm, size_t g0,
                                                           const DevTables* __restrict__ T, uint8_t* __restrict__ Dt) {
    __shared__ uint32_t tile[8 * kTrStride];
    const uint32_t i0 = blockIdx.x * 8;
    const int dir = blockIdx.y >> 1, j = blockIdx.y & 1;
    const int gw = blockIdx.z >> 1, l = blockIdx.z & 1;
    const uint32_t t = threadIdx.x;
    const uint32_t* src = (dir ? dm : dp) + (size_t)gw * (2 * (size_t)kSteps * kDeff * kN) +
                          ((size_t)l * kSteps * kDeff + j) * kN + i0 + (t & 7);
    for (uint32_t s = t >> 3; s < (uint32_t)kHalf; s += 32)
        tile[(t & 7) * kTrStride + s] = s < (uint32_t)kSteps ? src[(size_t)s * kDeff * kN] : 0u;
    __syncthreads();
    const size_t gl = (g0 + gw) * 2 + l;
#pragma unroll
    for (uint32_t x = 0; x < 8; ++x) {
        const uint32_t i = i0 + x, ex = T->exp_of[i];
        const uint32_t k = ex & (kHalf - 1), rho = (uint32_t)dir ^ (ex >> 10);
        uint32_t v[4];
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) v[e] = tile[x * kTrStride + dt_step(k, 4 * t + e)];
#pragma unroll
        for (uint32_t a = 0; a < 4; ++a) {
            uint32_t w = 0;
#pragma unroll
            for (int e = 0; e < 4; ++e) w |= ((v[e] >> (8 * a)) & 0xFFu) << (8 * e);
            *reinterpret_cast<uint32_t*>(Dt + dt_addr(gl, i, a, j * kN + rho * kHalf + 4 * t)) = w;
        }
    }
}

// Inverse of the re-layout for one group (precomp export): [l][s][j][N] u32.
__global__ void __launch_bounds__(256) dt_export_kernel(const uint8_t* __restrict__ Dt, size_t g,
                                                        const DevTables* __restrict__ T, uint32_t* __restrict__ dp,
                                                        uint32_t* __restrict__ dm) {
    const size_t idx = (size_t)blockIdx.x * 256 + threadIdx.x;  // over l, i, u
    const uint32_t u = (uint32_t)(idx % kK), i = (uint32_t)(idx / kK % kN), l = (uint32_t)(idx / kK / kN);
    const uint32_t ex = T->exp_of[i], j = u >> 11, rho = (u >> 10) & 1;
    const uint32_t s = dt_step(ex & (kHalf - 1), u & (kHalf - 1));
    if (s >= (uint32_t)kSteps) return;
    uint32_t v = 0;
#pragma unroll
    for (uint32_t a = 0; a < 4; ++a) v |= (uint32_t)Dt[dt_addr(g * 2 + l, i, a, u)] << (8 * a);
    ((rho ^ (ex >> 10)) ? dm : dp)[(((size_t)l * kSteps + s) * kDeff + j) * kN + i] = v;
}

// Rows [row0, row0 + gridDim.x) of the checkpoint files' order of the same
// bytes: row ((l * N + i) * G + g) * 4 + a, positions (dir * 1023 + s) * 2 + j
// (4092 used, the last four zero).  One CTA copies one row to or from the
// resident layout.
template <bool kToFile>
__global__ void __launch_bounds__(256) dt_file_rows_kernel(uint8_t* __restrict__ Dt, size_t G, size_t row0,
                                                           uint8_t* __restrict__ file,
                                                           const DevTables* __restrict__ T) {
    __shared__ __align__(16) uint8_t row[kK];
    const size_t fr = row0 + blockIdx.x;
    const uint32_t a = (uint32_t)(fr & 3);
    const size_t g = (fr >> 2) % G, li = (fr >> 2) / G;
    const uint32_t i = (uint32_t)(li % kN), l = (uint32_t)(li / kN);
    const uint32_t t = threadIdx.x, ex = T->exp_of[i], k = ex & (kHalf - 1), neg = ex >> 10;
    uint8_t* frow = file + (size_t)blockIdx.x * kK + 16 * t;
    uint8_t* drow = Dt + dt_addr(g * 2 + l, i, a, 16 * t);
    *reinterpret_cast<uint4*>(row + 16 * t) = *reinterpret_cast<const uint4*>(kToFile ? drow : frow);
    __syncthreads();
    uint32_t out[4] = {0, 0, 0, 0};
#pragma unroll
    for (uint32_t e = 0; e < 16; ++e) {
        const uint32_t p = 16 * t + e;
        uint32_t src;
        bool used;
        if (kToFile) {
            const uint32_t w = p >> 1, j = p & 1, dir = w >= (uint32_t)kSteps, s = w - dir * kSteps;
            used = w < 2u * kSteps;
            src = j * kN + (dir ^ neg) * kHalf + dt_step(k, s);  // m and s are each other's step
        } else {
            const uint32_t s = dt_step(k, p & (kHalf - 1)), dir = ((p >> 10) & 1) ^ neg;
            used = s < (uint32_t)kSteps;
            src = (dir * kSteps + s) * 2 + (p >> 11);
        }
        if (used) out[e >> 2] |= (uint32_t)row[src] << (8 * (e & 3));
    }
    *reinterpret_cast<uint4*>(kToFile ? frow : drow) = make_uint4(out[0], out[1], out[2], out[3]);
}

// One lane's row (slot, a) over 4 queries' 16 accumulator columns (byte plane
// b of query k at column 4k + b): part_k = sum_b (256^(a+b) mod q) P[4k + b]
// (< 2^60, unreduced), then summed over the 4 lanes a of a slot as a
// reduce-scatter, so that lane a returns query a's total.  Round 1 (xor 1)
// keeps queries a & 1 and (a & 1) + 2, round 2 (xor 2) keeps query a.
__device__ __forceinline__ uint64_t tp_reduce4(const uint32_t (&v)[16], const uint32_t (&c)[4], int a) {
    uint64_t part[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
        part[k] = (uint64_t)c[0] * v[4 * k] + (uint64_t)c[1] * v[4 * k + 1] + (uint64_t)c[2] * v[4 * k + 2] +
                  (uint64_t)c[3] * v[4 * k + 3];
    const int b0 = a & 1, b1 = (a >> 1) & 1;
    const uint64_t keep0 = b0 ? part[1] : part[0], keep1 = b0 ? part[3] : part[2];
    const uint64_t send0 = b0 ? part[0] : part[1], send1 = b0 ? part[2] : part[3];
    const uint64_t s0 = keep0 + __shfl_xor_sync(0xffffffffu, send0, 1);
    const uint64_t s1 = keep1 + __shfl_xor_sync(0xffffffffu, send1, 1);
    return (b1 ? s1 : s0) + __shfl_xor_sync(0xffffffffu, b1 ? s0 : s1, 2);
}

// ------------------------------------------------------------------ GEMM
struct TpParams {
    const uint8_t* dt;     // D' tiles
    uint32_t* out;         // tp_out, row of query 0 of the pass (row qmap[0] .. with a map)
    size_t out_qstride;
    int nq;                // queries in this pass
    int nb;                // N = roundup16(4 nq)
    int tile0;             // first 128-row tile of this launch
    int n_items;           // work items of MTI tiles
    int stages;
    int acc_stages;
    uint32_t tmem_cols;
    int* err;
    unsigned* tiles;       // [0] work-item counter, [1] CTAs done: both zero between launches
    int has_qmap;          // output row of pass query p: qmap[p] (else p)
    uint8_t qmap[32];
    uint32_t c[2][7];      // 256^k mod q_l
    uint64_t cr[2];
    uint32_t q[2];
    int abort_after;       // > 0: the MMA issuer stops after this many items and reports code 99 (a test of
                           // the abort path, IPB_TEST_ABORT_AFTER_ITEMS); 0: off
};

// Persistent, one CTA per SM, work items (MTI consecutive tiles) taken from an
// atomic counter by the producer and published to the MMA thread
// and the epilogue through a ring of shared slots (-1 ends it), so SMs held
// by other kernels at launch take fewer items.  Warps: 0 producer (one
// thread: MTI bulk copies of 16 KB and one key-plane tile per stage), 1 TMEM
// allocation and MMA issue (one thread), 2..9 epilogue (two warps per TMEM
// lane quarter).
// Bound by HBM: the tensors are read once, 67 MB a group; 8.59 GB at 128
// groups take 1.16 ms with 1 query (7.4 TB/s) and 1.23 ms with 32, 0.54 GB at
// 8 groups 86 and 92 us.  (With the key planes gathered per slot: 1.20, 1.60,
// 0.13 and 0.66 ms; 1 group, and any odd number, filled 4 rows of 128: 0.72 ms
// against 20 us.)
template <int MTI>
__global__ void __launch_bounds__(kTpThreads, 1) tp_tc_kernel(const __grid_constant__ CUtensorMap map_b, TpParams P) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int S = P.stages;
    constexpr uint32_t a_region = (uint32_t)MTI * kTile;
    const uint32_t stage_bytes = a_region + (uint32_t)P.nb * kKBlock;
    const uint32_t tx_bytes = a_region + (uint32_t)P.nq * 4 * kKBlock;
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
        for (int a = 0; a < 2; ++a) { mbar_init(&tfull[a], 1); mbar_init(&tempty[a], 32 * kEpiWarps); }
        for (int r = 0; r < kRing; ++r) { mbar_init(&ifull[r], 1); mbar_init(&iempty[r], 1 + 32 * kEpiWarps); }
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
    const int acc_cols = MTI * P.nb;

    if (warp == 0) {
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 0;
            unsigned issued = 0;  // stage loads issued
            for (int it = 0;; ++it) {
                const int r = it % kRing;
                int item = -1;
                if (!abort_flag && mbar_wait_ab(&iempty[r], ((uint32_t)(it / kRing) & 1) ^ 1, P.err, 16, &abort_flag)) {
                    const unsigned t = atomicAdd(P.tiles, 1u);
                    if (t < (unsigned)P.n_items) item = (int)t;
                } else {
                    abort_flag = 1;
                }
                item_ring[r] = item;
                mbar_arrive(&ifull[r]);
                if (item < 0) break;
                const int t0 = P.tile0 + item * MTI;
                const int l = (t0 / kTilesPerPoly) & 1;  // an item's tiles are of one limb
                const uint8_t* src = P.dt + (size_t)t0 * kKTiles * kTile;
                for (int kt = 0; kt < kKTiles; ++kt) {
                    if (!mbar_wait_ab(&empty[s], ph ^ 1, P.err, 11, &abort_flag)) { abort_flag = 1; break; }
                    uint8_t* st = smem + (size_t)s * stage_bytes;
                    mbar_expect_tx(&full[s], tx_bytes);
#pragma unroll
                    for (int mt = 0; mt < MTI; ++mt)
                        bulk_load(st + mt * kTile, src + ((size_t)mt * kKTiles + kt) * kTile, kTile, &full[s]);
                    tma_load_4d(st + a_region, &map_b, &full[s], kt * kKBlock, 0, l, 0);
                    ++issued;
                    if (++s == S) { s = 0; ph ^= 1; }
                }
            }
            // Drain: every issued load has landed before the CTA exits, also
            // when the MMA issuer stopped early and never consumed them.  Load n
            // went to stage n % S with phase (n / S) & 1; no later load reuses
            // a stage, so each wait is exact.
            for (unsigned i = 0; i < (unsigned)S && i < issued; ++i) {
                const unsigned n = issued - 1 - i;
                mbar_wait(&full[n % S], (n / S) & 1u, P.err, 12);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // One thread issues every MMA: descriptors are one 32-bit add each
            // (address field of the low word), the loops unrolled.
            const uint32_t idesc = idesc_i8_kk(P.nb);
            constexpr uint32_t kDescHi = smem_desc_hi_sw128(1024);
            const uint32_t desc0 = smem_desc_lo(smem, 16);
            int s = 0, as = 0;
            uint32_t ph = 0, aph = 0;
            bool any_mma = false;
            for (int it = 0;; ++it) {
                const int r = it % kRing;
                if (!mbar_wait_ab(&ifull[r], (uint32_t)(it / kRing) & 1, P.err, 17, &abort_flag)) { abort_flag = 1; break; }
                const int item = item_ring[r];
                mbar_arrive(&iempty[r]);
                if (item < 0 || abort_flag) break;
                if (P.abort_after > 0 && it >= P.abort_after) {  // test hook: the designed early stop
                    atomicCAS(P.err, 0, 99);
                    abort_flag = 1;
                    break;
                }
                if (!mbar_wait_ab(&tempty[as], aph ^ 1, P.err, 13, &abort_flag)) { abort_flag = 1; break; }
                tc_fence_after();
                const uint32_t d0 = tmem_base + (uint32_t)(as * acc_cols);
                for (int kt = 0; kt < kKTiles; ++kt) {
                    if (!mbar_wait_ab(&full[s], ph, P.err, 14, &abort_flag)) { abort_flag = 1; break; }
                    tc_fence_after();
                    const uint32_t ad = desc0 + (uint32_t)s * (stage_bytes >> 4), bd = ad + (a_region >> 4);
#pragma unroll
                    for (int kk = 0; kk < kKBlock / 32; ++kk)
#pragma unroll
                        for (int mt = 0; mt < MTI; ++mt)
                            mma_i8_lo(d0 + (uint32_t)(mt * P.nb), ad + mt * (kTile >> 4) + kk * 2, bd + kk * 2, kDescHi,
                                      kDescHi, idesc, (kt > 0 || kk > 0) ? 1u : 0u);
                    mma_commit(&empty[s]);
                    any_mma = true;
                    if (++s == S) { s = 0; ph ^= 1; }
                }
                mma_commit(&tfull[as]);
                if (++as == P.acc_stages) { as = 0; aph ^= 1; }
            }
            // Every MMA this thread issued has completed (also after an early
            // stop) before TMEM is deallocated and shared memory released.
            if (any_mma) {
                mma_commit(&mma_done);
                mbar_wait(&mma_done, 0, P.err, 22);
            }
        }
    } else {
        // ---------------- epilogue: TMEM -> reduced tensor-pass values.  The
        // two warps of a lane quarter take alternate 16-column chunks.
        const int wq = warp & 3, share = (warp - 2) >> 2;
        const uint32_t lane_base = (uint32_t)(wq * 32) << 16;
        const int a = lane & 3;
        const int nqc = (P.nq + 3) / 4, chunks = MTI * nqc;
        int as = 0;
        uint32_t aph = 0;
        for (int it = 0;; ++it) {
            const int r = it % kRing;
            if (!mbar_wait_ab(&ifull[r], (uint32_t)(it / kRing) & 1, P.err, 18, &abort_flag)) { abort_flag = 1; break; }
            const int item = item_ring[r];
            mbar_arrive(&iempty[r]);
            if (item < 0) break;
            if (!mbar_wait_ab(&tfull[as], aph, P.err, 15, &abort_flag)) { abort_flag = 1; break; }
            tc_fence_after();
            const int t0 = P.tile0 + item * MTI;
            const int l = (t0 / kTilesPerPoly) & 1;
            const uint64_t cr = P.cr[l];
            const uint32_t q = P.q[l];
            uint32_t c[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) c[b] = P.c[l][a + b];
            for (int ch = share; ch < chunks; ch += kEpiWarps / 4) {
                const int mt = ch / nqc, q0 = (ch - mt * nqc) * 4;
                const uint32_t ta = tmem_base + lane_base + (uint32_t)(as * acc_cols + mt * P.nb + 4 * q0);
                uint32_t v[16];
                tmem_ld16(ta, v);
                const uint64_t tot = tp_reduce4(v, c, a);
                if (q0 + a < P.nq) {
                    const int qo = P.has_qmap ? P.qmap[q0 + a] : q0 + a;
                    P.out[(size_t)qo * P.out_qstride + (size_t)(t0 + mt) * 32 + wq * 8 + (lane >> 2)] =
                        mod_u64(tot, cr, q);
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

// kplanes[q][l][b][4096] of nq queries; box: one K block of every (q, b) row
// of one limb, rows 4 q + b of the B tile.
bool make_map_b(CUtensorMap* m, const void* base, int nq) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) return false;
    cuuint64_t dims[4] = {(cuuint64_t)kK, 4, 2, (cuuint64_t)nq};
    cuuint64_t strides[3] = {(cuuint64_t)kK, (cuuint64_t)4 * kK, (cuuint64_t)8 * kK};
    cuuint32_t box[4] = {(cuuint32_t)kKBlock, 4, 1, (cuuint32_t)nq};
    cuuint32_t es[4] = {1, 1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<void*>(base), dims, strides, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

uint32_t powmod_host(uint64_t b, uint64_t e, uint64_t q) {
    uint64_t r = 1;
    b %= q;
    while (e) {
        if (e & 1) r = r * b % q;
        b = b * b % q;
        e >>= 1;
    }
    return (uint32_t)r;
}

}  // namespace

size_t tp_dt_bytes(size_t groups) { return (size_t)2 * kN * 4 * groups * kK; }
int tp_tiles(size_t groups) { return (int)(2 * groups) * kTilesPerPoly; }

cudaError_t launch_dt_transpose(const uint32_t* dp, const uint32_t* dm, size_t g0, size_t nw, const DevTables* T,
                                uint8_t* Dt, cudaStream_t s) {
    if (nw == 0) return cudaSuccess;
    dt_transpose_kernel<<<dim3(kN / 8, 4, (unsigned)(nw * 2)), 256, 0, s>>>(dp, dm, g0, T, Dt);
    return cudaGetLastError();
}

cudaError_t launch_dt_export(const uint8_t* Dt, size_t g, const DevTables* T, uint32_t* dp, uint32_t* dm,
                             cudaStream_t s) {
    dt_export_kernel<<<(unsigned)((size_t)2 * kN * kK / 256), 256, 0, s>>>(Dt, g, T, dp, dm);
    return cudaGetLastError();
}

cudaError_t launch_dt_file_rows(uint8_t* Dt, size_t G, size_t row0, size_t nrows, uint8_t* file, bool to_file,
                                const DevTables* T, cudaStream_t s) {
    if (nrows == 0) return cudaSuccess;
    if (to_file)
        dt_file_rows_kernel<true><<<(unsigned)nrows, 256, 0, s>>>(Dt, G, row0, file, T);
    else
        dt_file_rows_kernel<false><<<(unsigned)nrows, 256, 0, s>>>(Dt, G, row0, file, T);
    return cudaGetLastError();
}

cudaError_t launch_tensor_pass(const uint8_t* Dt, int tile0, int n_tiles, const uint8_t* kplanes, int nq,
                               const uint8_t* qmap, uint32_t* tp_out, size_t out_qstride, int* err, unsigned* tiles,
                               int num_sms, cudaStream_t s) {
    if (nq <= 0) return cudaSuccess;
    if (nq > kTpMaxPass || (qmap && nq > 32) || !tiles || tile0 < 0 || n_tiles <= 0) return cudaErrorInvalidValue;
    TpParams P{};
    P.dt = Dt;
    P.out = tp_out;
    P.out_qstride = out_qstride;
    P.nq = nq;
    P.nb = (4 * nq + 15) / 16 * 16;
    P.tile0 = tile0;
    P.has_qmap = qmap != nullptr;
    if (qmap)
        for (int p = 0; p < nq; ++p) P.qmap[p] = qmap[p];
    const int sms = std::max(1, num_sms);
    // Two tiles per item (their MMAs share a stage's key planes) once that
    // leaves an item per SM.  G = 1 (128 tiles), 32 queries: 20 us with one tile,
    // 25 with two; G = 128, 32 queries: 1255 and 1227 us (four tiles, whose
    // accumulators cannot be double-buffered: 1300); between, within 3 %.
    // More than 32 queries: one tile, so that its 256 columns stay
    // double-buffered (G = 128, 64 queries: 1648 us, two tiles 1683, two passes
    // of 32 queries 2450).
    const int mti = nq <= 32 && n_tiles % 2 == 0 && tile0 % 2 == 0 && n_tiles >= 2 * sms ? 2 : 1;
    const auto kernel = mti == 2 ? tp_tc_kernel<2> : tp_tc_kernel<1>;
    P.n_items = n_tiles / mti;
    P.acc_stages = 2;  // at most 2 x 2 x 128 or 2 x 256 columns
    uint32_t need = (uint32_t)(P.acc_stages * mti * P.nb), tc = 32;
    while (tc < need) tc <<= 1;
    P.tmem_cols = tc;
    P.err = err;
    P.tiles = tiles;
    P.abort_after = test_abort_after_items();
    const uint32_t qs[2] = {kQ0, kQ1};
    for (int l = 0; l < 2; ++l) {
        for (int k = 0; k < 7; ++k) P.c[l][k] = powmod_host(256, k, qs[l]);
        P.cr[l] = ~0ULL / qs[l];
        P.q[l] = qs[l];
    }
    const size_t stage_bytes = (size_t)mti * kTile + (size_t)P.nb * kKBlock;
    // As many stages as the device's shared memory takes (1 KB alignment
    // slack, 512 B of barriers).
    size_t max_dyn = 0;
    cudaError_t e = allow_max_smem(kernel, &max_dyn);
    if (e) return e;
    P.stages = (int)std::min<size_t>(12, (max_dyn - 1024 - 512) / stage_bytes);
    if (P.stages < 2) return cudaErrorInvalidValue;
    CUtensorMap mb;
    if (!make_map_b(&mb, kplanes, nq)) return cudaErrorInvalidValue;
    const size_t smem = 1024 + (size_t)P.stages * stage_bytes + (2 * P.stages + 4) * 8 + 16;
    // The items take `waves` rounds; the SMs that would have none in the last
    // round are left to the mat-vec (1 group, 128 items, beside on 98 SMs: 64 CTAs
    // end as soon, 42 -> 38 us for the answer's kernels).
    const int waves = (P.n_items + sms - 1) / sms;
    return launch_overlapped(kernel, (P.n_items + waves - 1) / waves, kTpThreads, smem, s, mb, P);
}

}  // namespace ipb

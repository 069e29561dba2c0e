// ipb_common.cuh -- constants, exact modular arithmetic and the 2048-point
// negacyclic NTT shared by every kernel of the B200 InsPIRe server.
//
// Ring Z_q[X]/(X^2048+1), q = q0*q1 with the two 27-bit NTT primes of the
// reference (src/params.h:15-18).  Residues are u32 in [0, q).
//
// NTT convention (must match the reference's CPU/GPU NTT bit for bit,
// src/ntt.cpp:107-149): Cooley-Tukey DIT forward with twiddles
// fwd[i] = psi^BR(i), Gentleman-Sande inverse with inv[i] = fwd[i]^-1 and a
// final N^-1 scale.  Output slot i holds the evaluation at psi^(2 BR(i)+1).
// Every stage here computes the same mathematical transform lazily and
// reduces to [0, q) at the end, so results are identical.  A 27-bit q leaves
// room for 45 q in a word and Shoup multiplication takes any word, so a
// forward stage only adds (its values grow by 2 q) and no forward transform
// reduces before its end; an inverse stage doubles its sums, and two of a
// thread's eight values are reduced after each three stages.  (With a
// conditional subtraction in every butterfly a Horner step took 6.0 us on
// 4 CTAs and 4.5 us on 8.)
//
// The transform runs on one "NTT group" of 256 threads holding 8 elements
// each in registers; three shared-memory exchanges (four words of padding per
// 32: bank-conflict free, and every address of a thread is one register plus a
// constant) move between the four register layouts
//   L1: x = t + 256 e        stages s = 10, 9, 8
//   L2: x = (t&31) + 32 e + 256 (t>>5)   s = 7, 6, 5
//   L3: x = (t&3) + 4 e + 32 (t>>2)      s = 4, 3, 2
//   L4: x = 8 t + e          stages s = 1, 0
// A forward NTT takes L1 in and leaves L4; the inverse takes L4 to L1.
// Only L1 <-> L2 moves data between warps: in L2, L3 and L4 warp w holds
// x in [256w, 256w + 256), its own part of the buffer, so those exchanges need
// warp barriers only.  Each transform starts with a group barrier before its
// first store, which orders it after the previous transform's reads.
// Several groups can share a CTA, each synchronising on its own named
// barrier (bar.sync id, 256).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace ipb {

constexpr int kN = 2048;
constexpr int kLogN = 11;
constexpr int kHalf = kN / 2;
constexpr int kSteps = kHalf - 1;      // collapse steps per direction
constexpr int kDgsw = 3;               // gadget digits (src/params.h:26-29)
constexpr int kDeff = 2;               // digits kept (digit 0 dropped)
constexpr int kBaseLog = 18;
constexpr uint32_t kQ0 = 94519297u;
constexpr uint32_t kQ1 = 95293441u;
constexpr uint32_t kP = 65535u;        // plaintext modulus (Mersenne)
constexpr uint64_t kQFull = (uint64_t)kQ0 * kQ1;

// Per-limb tables, one set per device.  Entries are (w, floor(w 2^32/q)),
// stored at tw_index.
// An inverse transform scales by a constant c of its last stage: NttScale is
// (c, c inv[1]) with Shoup factors.
struct NttScale {
    uint2 c, w;
};
struct LimbTables {
    alignas(16) uint2 fwd[kN];
    alignas(16) uint2 inv[kN];
    NttScale scale_n;            // N^-1
    NttScale scale_crt;          // N^-1 times the limb's CRT factor crt_c
    uint32_t q;
    uint32_t inv_n, inv_n_p;     // N^-1 and its Shoup factor
    uint64_t cr;                 // floor(2^64 / q), exact u64 Barrett
};
struct DevTables {
    LimbTables limb[2];
    uint32_t crt_c[2], crt_cp[2];  // q1^-1 mod q0, q0^-1 mod q1 and Shoup factors
    // The slots' odd exponents 2 BR(slot) + 1 = (-1)^rho 5^m mod 2N:
    // slot_of[rho * N/2 + m] and its inverse.
    alignas(16) uint16_t slot_of[kN];
    uint16_t exp_of[kN];
};

// ------------------------------------------------------------ arithmetic
__device__ __forceinline__ uint32_t shoup_mul(uint32_t x, uint32_t w, uint32_t wp, uint32_t q) {
    // x < 2^32, w < q: returns x*w mod q in [0, 2q).
    uint32_t t = __umulhi(x, wp);
    return x * w - t * q;
}
__device__ __forceinline__ uint32_t csub(uint32_t x, uint32_t m) {
    // x < 2m  ->  x mod m (unsigned wrap makes x-m huge when x < m).
    return min(x, x - m);
}
__device__ __forceinline__ uint32_t add_mod(uint32_t a, uint32_t b, uint32_t q) { return csub(a + b, q); }
__device__ __forceinline__ uint32_t sub_mod(uint32_t a, uint32_t b, uint32_t q) { return csub(a + q - b, q); }
__device__ __forceinline__ uint32_t mod_u64(uint64_t x, uint64_t cr, uint32_t q) {
    // Exact for every u64: the quotient estimate is low by at most 1.
    uint64_t t = __umul64hi(x, cr);
    uint64_t r = x - t * (uint64_t)q;
    return (uint32_t)(r >= q ? r - q : r);
}
__device__ __forceinline__ uint32_t brev11(uint32_t x) { return __brev(x) >> (32 - kLogN); }

// Slot permutation of the automorphism tau_t in NTT form: result slot x is
// source slot perm(t, x) (src/gpu_preprocess.cu:158-194).  `odd` = 2 BR(x)+1.
__device__ __forceinline__ uint32_t perm_from_odd(uint32_t t, uint32_t odd) {
    uint32_t e = (t * odd) & (2 * kN - 1);
    return brev11((e - 1) >> 1);
}

// ------------------------------------------------------------ launch overlap
// Kernels of the answer pipeline launch with programmatic stream
// serialization: the next one may start, and run its prologue, while this one
// is still running.  after_previous() waits until the previous kernel of the
// stream has completed and its writes are visible; every read or write of
// memory that another kernel touches comes after it.  let_next_start() is
// called first thing, so the next kernel's blocks take whatever this one leaves
// free.  Both are no-ops in an ordinary launch.
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ------------------------------------------------------------ barriers
__device__ __forceinline__ void gsync(int bar) {
    if (bar == 0) __syncthreads();
    else asm volatile("bar.sync %0, 256;" ::"r"(bar) : "memory");
}
constexpr int kNttBuf = kN + kN / 8;  // words of one group's exchange buffer
// Where the tables hold twiddle i: the four entries that one thread reads for
// stage 0 (i = 1024 + 4t ..) and stage 2 (256 + 4h ..) lie as two pairs half
// the stage's range apart, so the lanes of a warp read consecutive 16 bytes.
__host__ __device__ constexpr int tw_index(int i) {
    const int n = i >= 1024 ? 1024 : i >= 256 && i < 512 ? 256 : 0;
    return n == 0 ? i : n + ((i >> 1) & 1) * (n / 2) + (i - n) / 4 * 2 + (i & 1);
}

// x mod q up to one q, for any word: [0, 2q).  floor(2^32 / q) is 45 for both
// primes; the estimate of the quotient (< 46) is low by less than 1.5.
__device__ __forceinline__ uint32_t red2(uint32_t x, uint32_t q) { return x - __umulhi(x, 45u) * q; }
static_assert((1ull << 32) / kQ0 == 45 && (1ull << 32) / kQ1 == 45, "red2");

// Layout helpers: a thread's first exchange-buffer word and the distance of
// its elements (x + 4 (x >> 5) at the layout's x) per layout id (1..4).
template <int L> __device__ __forceinline__ uint32_t lay_base(uint32_t t);
template <> __device__ __forceinline__ uint32_t lay_base<1>(uint32_t t) { return t + 4 * (t >> 5); }
template <> __device__ __forceinline__ uint32_t lay_base<2>(uint32_t t) { return (t & 31) + 288 * (t >> 5); }
template <> __device__ __forceinline__ uint32_t lay_base<3>(uint32_t t) { return (t & 3) + 36 * (t >> 2); }
template <> __device__ __forceinline__ uint32_t lay_base<4>(uint32_t t) { return 8 * t + 4 * (t >> 2); }
template <int L> struct LayStep;
template <> struct LayStep<1> { static constexpr int v = 288; };
template <> struct LayStep<2> { static constexpr int v = 36; };
template <> struct LayStep<3> { static constexpr int v = 4; };
template <> struct LayStep<4> { static constexpr int v = 1; };

template <int L>
__device__ __forceinline__ void lay_store(const uint32_t (&r)[8], uint32_t* s, uint32_t t) {
    uint32_t* p = s + lay_base<L>(t);
    if (L == 4) {
        *reinterpret_cast<uint4*>(p) = make_uint4(r[0], r[1], r[2], r[3]);
        *reinterpret_cast<uint4*>(p + 4) = make_uint4(r[4], r[5], r[6], r[7]);
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) p[e * LayStep<L>::v] = r[e];
    }
}
template <int L>
__device__ __forceinline__ void lay_load(uint32_t (&r)[8], const uint32_t* s, uint32_t t) {
    const uint32_t* p = s + lay_base<L>(t);
    if (L == 4) {
        uint4 a = *reinterpret_cast<const uint4*>(p);
        uint4 b = *reinterpret_cast<const uint4*>(p + 4);
        r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w;
        r[4] = b.x; r[5] = b.y; r[6] = b.z; r[7] = b.w;
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) r[e] = p[e * LayStep<L>::v];
    }
}

// ------------------------------------------------------------ twiddles
// The twiddles of one register pass over layout L: w[0] for k = 2, w[1..2]
// for k = 1, w[3..6] for k = 0 (stage s = B0 + k, k = bit of the register
// index; L4 has k = 1, 0 only).  Entry of stage s at x: number 2^(10-s) + (x >> (s+1)).
struct Tw {
    uint2 w[7];
};
__device__ __forceinline__ void ld_tw2(uint2 (&w)[7], int i, const uint2* p) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    w[i] = make_uint2(v.x, v.y);
    w[i + 1] = make_uint2(v.z, v.w);
}
template <int L>
__device__ __forceinline__ Tw load_tw(const uint2* __restrict__ tw, uint32_t t) {
    Tw r;
    if (L == 4) {
        ld_tw2(r.w, 1, tw + 512 + 2 * t);
        ld_tw2(r.w, 3, tw + 1024 + 2 * t);
        ld_tw2(r.w, 5, tw + 1536 + 2 * t);
    } else if (L == 3) {
        r.w[0] = tw[64 + (t >> 2)];
        ld_tw2(r.w, 1, tw + 128 + 2 * (t >> 2));
        ld_tw2(r.w, 3, tw + 256 + 2 * (t >> 2));
        ld_tw2(r.w, 5, tw + 384 + 2 * (t >> 2));
    } else {
        const uint32_t h = L == 1 ? 0u : t >> 5;
        constexpr int b = L == 1 ? 1 : 8;
        r.w[0] = tw[b + h];
        ld_tw2(r.w, 1, tw + 2 * b + 2 * h);
        ld_tw2(r.w, 3, tw + 4 * b + 4 * h);
        ld_tw2(r.w, 5, tw + 4 * b + 4 * h + 2);
    }
    return r;
}

// Register pass of a forward transform: stages k = K - 1 .. 0.  Values grow
// by 2q per stage.
template <int K>
__device__ __forceinline__ void pass_fwd(uint32_t (&r)[8], const Tw& T, uint32_t q) {
    const uint32_t q2 = 2 * q;
#pragma unroll
    for (int k = K - 1; k >= 0; --k)
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            if (e & (1 << k)) continue;
            const uint2 w = T.w[(1 << (2 - k)) - 1 + (e >> (k + 1))];
            const uint32_t v = shoup_mul(r[e | (1 << k)], w.x, w.y, q), u = r[e];
            r[e] = u + v;
            r[e | (1 << k)] = u + q2 - v;
        }
}
// Register pass of an inverse transform: stages k = 0 .. K - 1 on values
// <= B q.  bound[] (compile-time, in q) follows each value; what ends above
// 4q is reduced, so the pass leaves values <= 4q.
template <int K, int B>
__device__ __forceinline__ void pass_inv(uint32_t (&r)[8], const Tw& T, uint32_t q) {
    int bound[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) bound[e] = B;
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            if (e & (1 << k)) continue;
            const int e2 = e | (1 << k);
            const uint2 w = T.w[(1 << (2 - k)) - 1 + (e >> (k + 1))];
            const uint32_t u = r[e], v = r[e2];
            r[e] = u + v;
            r[e2] = shoup_mul(u + (uint32_t)bound[e2] * q - v, w.x, w.y, q);
            bound[e] += bound[e2];
            bound[e2] = 2;
        }
#pragma unroll
    for (int e = 0; e < 8; ++e)
        if (bound[e] > 4) r[e] = red2(r[e], q);
}
// The last pass of an inverse transform (stages 8, 9, 10) on values <= 4q:
// the scale goes into the last stage's two multiplications.  Leaves [0, q).
__device__ __forceinline__ void pass_inv_last(uint32_t (&r)[8], const Tw& T, const NttScale& c, uint32_t q) {
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            if (e & (1 << k)) continue;
            const int e2 = e | (1 << k);
            const uint2 w = T.w[(1 << (2 - k)) - 1 + (e >> (k + 1))];
            const uint32_t u = r[e], v = r[e2];
            // bounds: k = 0: 4, 4; k = 1: 8, 8 (e even), 2, 2 (e odd)
            r[e] = u + v;
            r[e2] = shoup_mul(u + (k == 0 ? 4u : (e & 1) ? 2u : 8u) * q - v, w.x, w.y, q);
        }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const uint32_t u = r[e], v = r[e + 4];  // <= 16q (e = 0), 4q, 2q
        r[e] = csub(shoup_mul(u + v, c.c.x, c.c.y, q), q);
        r[e + 4] = csub(shoup_mul(u + 16u * q - v, c.w.x, c.w.y, q), q);
    }
}

// Forward NTT without the final reduction: r in L1 (values <= 4q) -> r in L4,
// values < 26q.  buf: kNttBuf u32 private to this group.  All 256 threads must
// call.
__device__ __forceinline__ void ntt_fwd_lazy(uint32_t (&r)[8], uint32_t* buf, const uint2* __restrict__ tw, uint32_t q,
                                             uint32_t t, int bar) {
    pass_fwd<3>(r, load_tw<1>(tw, t), q);
    const Tw w2 = load_tw<2>(tw, t);
    gsync(bar);
    lay_store<1>(r, buf, t); gsync(bar); lay_load<2>(r, buf, t);
    pass_fwd<3>(r, w2, q);
    const Tw w3 = load_tw<3>(tw, t);
    __syncwarp(); lay_store<2>(r, buf, t); __syncwarp(); lay_load<3>(r, buf, t);
    pass_fwd<3>(r, w3, q);
    const Tw w4 = load_tw<4>(tw, t);
    __syncwarp(); lay_store<3>(r, buf, t); __syncwarp(); lay_load<4>(r, buf, t);
    pass_fwd<2>(r, w4, q);
}
// Forward NTT: r in L1 (values <= 4q) -> r in L4, canonical [0, q).
__device__ __forceinline__ void ntt_fwd(uint32_t (&r)[8], uint32_t* buf, const uint2* __restrict__ tw,
                                        uint32_t q, uint32_t t, int bar) {
    ntt_fwd_lazy(r, buf, tw, q, t, bar);
#pragma unroll
    for (int e = 0; e < 8; ++e) r[e] = csub(red2(r[e], q), q);
}

// Inverse NTT times a constant: r in L4 (values <= 2q) -> r in L1, canonical.
// In two halves around the exchange between warps, for callers that read
// shared state between the two group barriers.
__device__ __forceinline__ void ntt_inv_head(uint32_t (&r)[8], uint32_t* buf, const uint2* __restrict__ tw, uint32_t q,
                                             uint32_t t, int bar) {
    pass_inv<2, 2>(r, load_tw<4>(tw, t), q);
    const Tw w3 = load_tw<3>(tw, t);
    gsync(bar);
    lay_store<4>(r, buf, t); __syncwarp(); lay_load<3>(r, buf, t);
    pass_inv<3, 4>(r, w3, q);
    const Tw w2 = load_tw<2>(tw, t);
    __syncwarp(); lay_store<3>(r, buf, t); __syncwarp(); lay_load<2>(r, buf, t);
    pass_inv<3, 4>(r, w2, q);
    __syncwarp(); lay_store<2>(r, buf, t);
}
__device__ __forceinline__ void ntt_inv_tail(uint32_t (&r)[8], uint32_t* buf, const uint2* __restrict__ tw, uint32_t q,
                                             const NttScale& c, uint32_t t, int bar) {
    const Tw w1 = load_tw<1>(tw, t);
    gsync(bar);
    lay_load<1>(r, buf, t);
    pass_inv_last(r, w1, c, q);
}
__device__ __forceinline__ void ntt_inv(uint32_t (&r)[8], uint32_t* buf, const uint2* __restrict__ tw, uint32_t q,
                                        const NttScale& c, uint32_t t, int bar) {
    ntt_inv_head(r, buf, tw, q, t, bar);
    ntt_inv_tail(r, buf, tw, q, c, t, bar);
}

// ------------------------------------------------------------ gadget decomposition
// One coefficient: CRT lift of (c0 mod q0, c1 mod q1) to [0, Q), center to
// r in (-Q/2, Q/2], three signed base-2^18 digits, digit 0 dropped
// (src/ring.cpp:205-246).  t_l = c_l crt_c[l] mod q_l (canonical), so the lift
// is t0 q1 + t1 q0 mod Q; digit 1 is bits 18..35 of r + 2^17 as a signed
// number and digit 2 the bits from 36 on of r + 2^17 + 2^35 (the carries of
// the balanced digits below).  lift_plus returns r + c from the
// terms ta, tb of the two limbs (primes qa, qb) in either order.
__device__ __forceinline__ uint64_t lift_plus(uint32_t ta, uint32_t tb, uint32_t qa, uint32_t qb, uint64_t c) {
    uint64_t v = (uint64_t)ta * qb + ((uint64_t)tb * qa + c);  // < 2Q + c
    uint64_t n = v > kQFull / 2 + c ? kQFull : 0;
    if (v > kQFull + kQFull / 2 + c) n = 2 * kQFull;
    return v - n;
}
constexpr uint64_t kCarry1 = 1ull << (kBaseLog - 1), kCarry2 = kCarry1 + (1ull << (2 * kBaseLog - 1));
__device__ __forceinline__ int32_t digit1(uint64_t r_carry1) { return (int32_t)(r_carry1 >> 4) >> 14; }
__device__ __forceinline__ int32_t digit2(uint64_t r_carry2) { return (int32_t)(r_carry2 >> 32) >> 4; }
static_assert(kBaseLog == 18, "digit1, digit2");

__device__ __forceinline__ void decomp_lifted(uint32_t t0, uint32_t t1, int32_t& d1, int32_t& d2) {
    const uint64_t r = lift_plus(t0, t1, kQ0, kQ1, kCarry1);
    d1 = digit1(r);
    d2 = digit2(r + (kCarry2 - kCarry1));
}
__device__ __forceinline__ void decomp2(uint32_t c0, uint32_t c1, const DevTables& T, int32_t& d1, int32_t& d2) {
    decomp_lifted(csub(shoup_mul(c0, T.crt_c[0], T.crt_cp[0], kQ0), kQ0),
                  csub(shoup_mul(c1, T.crt_c[1], T.crt_cp[1], kQ1), kQ1), d1, d2);
}
__device__ __forceinline__ uint32_t signed_res(int32_t d, uint32_t q) { return d >= 0 ? (uint32_t)d : q + (uint32_t)d; }

}  // namespace ipb

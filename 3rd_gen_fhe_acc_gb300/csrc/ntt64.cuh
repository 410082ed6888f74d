// ntt64.cuh -- negacyclic NTT / inverse NTT of a 2048-point polynomial with
// 64-bit words (Q < 2^62), computed in shared memory by a group of threads.
//
// Same transforms as the reference's NTT / iNTT (FHE_ACC_runtime/src/
// nbt.cpp:423-454 and 456-491), so canonical outputs are bit-identical.
//
// A 64-bit Shoup multiplication (w' = floor(w 2^64 / Q)) costs about five
// times a 32-bit one, so shared-memory traffic matters less here than in the
// 32-bit path: the polynomial stays in shared memory and each thread runs
// radix-8 / radix-16 passes (three or four butterfly stages per load/store of
// 8 or 16 words: 3 passes per forward transform, 4 per inverse), with one
// group barrier per pass.
// Forward butterflies leave the upper input unreduced
// (bound grows by 2Q a stage: inputs < Q end below 23Q < 2^59 for Q < 2^54);
// the inverse ends canonical.
//
// The transforms are bound by the 32-bit multiply pipe, so the modular
// multiplication decides their time. Two forms, chosen by the modulus
// (template parameter PM):
//   PM = true: Q = 2^b - c with 48 <= b <= 54 and c <= 2^(b-36), which every Q
//     picked as the largest prime below a power of two satisfies (pm64_shift).
//     A constant w is kept as (w, w 2^30 mod Q); x = x1 2^30 + x0 gives
//     x w = x0 w + x1 (w 2^30) below 2^(b+32), and the bits above 2^b fold
//     back times c: five 32 x 32 -> 64 multiplies (20 issue slots of the
//     multiply pipe's 16 lanes) where Shoup's form takes 33. A register-only
//     butterfly loop: 34 cycles per warp against 42 with Shoup's. The blind
//     rotation, products and expansion of such a Q are in block form
//     (block64.cuh); of the transforms here they use the whole-polynomial ones.
//   PM = false: Shoup's multiplication, any Q < 2^58.
#pragma once
#include <cstdint>

namespace fheacc {
namespace dev {

// Shared-memory layouts of a 2048-word polynomial, chosen by the template
// parameter P of the transforms: P = false, word e at e; P = true, one padding
// word after every 16, word e at px(e). A 64-bit shared access takes a half
// warp at a time: padded, its 16 words fall on 16 different bank pairs in
// every pass (consecutive words; 8 consecutive words of two tuples 136 words
// apart; the first words of 16 octets), and a tuple's offsets stay
// compile-time constants.
constexpr int kPoly64 = 2048 + 128;
__host__ __device__ __forceinline__ constexpr int px(int e) { return e + (e >> 4); }
template <bool P>
__host__ __device__ __forceinline__ constexpr int pi(int e) { return P ? px(e) : e; }
template <bool P>
__host__ __device__ constexpr int poly_words64() { return P ? kPoly64 : 2048; }

struct Ntt64Consts {
    uint64_t Q, twoQ;
    uint64_t iN, iNs;       // N^-1 as a constant pair (w, companion)
    uint64_t iw1N, iw1Ns;   // irou[1] * N^-1
    uint64_t mu64;          // floor(2^64 / Q)
    uint32_t pm_c;          // 2^b - Q where the PM form applies (else 0)
    uint32_t pm_s;          // 64 - b
};

// 64 - b if Q = 2^b - c with 48 <= b <= 54 and c <= 2^(b-36), else 0. The
// bounds make every product of mul64<true> less than (1 + 2^-4) 2^b < 2Q, and
// b <= 54 keeps a residue in two 27-bit limbs (mac27 in block64.cuh).
inline int pm64_shift(uint64_t Q)
{
    for (int b = 48; b <= 54; b++) {
        const uint64_t p = (uint64_t)1 << b;
        if (Q < p && Q > p / 2) return p - Q <= (uint64_t)1 << (b - 36) ? 64 - b : 0;
    }
    return 0;
}

// a b, and a b + s as one instruction: from (uint64_t)a * b + s the compiler often
// makes a multiply and a 64-bit add, both on the multiply pipe (a step of the blind
// rotation: 70 k instructions of that pipe, 50 k with the chains written out).
__device__ __forceinline__ uint64_t mul_wide64(uint32_t a, uint32_t b)
{
    uint64_t d;
    asm("mul.wide.u32 %0, %1, %2;" : "=l"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint64_t mad_wide64(uint32_t a, uint32_t b, uint64_t s)
{
    uint64_t d;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(s));
    return d;
}

// 2^-s (U + 2^32 V) mod Q of products with constants times 2^s (PM): the part
// above 2^b is the word above 2^64.
__device__ __forceinline__ uint64_t fold64(uint64_t U, uint64_t V, const Ntt64Consts &c)
{
    V += U >> 32;
    const uint64_t low = (V << 32) | (uint32_t)U;
    return mad_wide64((uint32_t)(V >> 32), c.pm_c, low >> c.pm_s);
}

// x w mod Q for a constant pair w, in [0, 2Q).
// PM: w = (w << s, (w 2^30 mod Q) << s), s = 64 - b; x < 2^61. With U and V the
// sums of the low and high word products, 2^s x w = U + 2^32 V; the word above
// 2^64 is the part of x w above 2^b. Bounds: x0 < 2^30 and x1 < 2^31 keep both
// sums below 2^62 + 2^63 + 2^32.
// Shoup: w = (w, floor(w 2^64 / Q)), any x.
template <bool PM>
__device__ __forceinline__ uint64_t mul64(uint64_t x, ulonglong2 w, const Ntt64Consts &c)
{
    if (PM) {
        const uint32_t x0 = (uint32_t)x & 0x3fffffffu, x1 = (uint32_t)(x >> 30);
        const uint64_t U = mad_wide64(x1, (uint32_t)w.y, mul_wide64(x0, (uint32_t)w.x));
        const uint64_t V = mad_wide64(x1, (uint32_t)(w.y >> 32), mul_wide64(x0, (uint32_t)(w.x >> 32)));
        return fold64(U, V, c);
    }
    const uint64_t t = __umul64hi(x, w.y);
    return x * w.x - t * c.Q;
}

// Any 64-bit x to [0, 2Q). PM: x = x1 2^b + x0 folds to x0 + c x1 < 2^b + 2^34.
template <bool PM>
__device__ __forceinline__ uint64_t reduce64(uint64_t x, const Ntt64Consts &c)
{
    if (PM) {
        const uint32_t b = 64 - c.pm_s;
        return mad_wide64((uint32_t)(x >> b), c.pm_c, x & (~0ull >> c.pm_s));
    }
    return x - __umul64hi(x, c.mu64) * c.Q;
}

template <bool PM>
__device__ __forceinline__ uint64_t canonical64(uint64_t x, const Ntt64Consts &c)
{
    const uint64_t v = reduce64<PM>(x, c);
    return v >= c.Q ? v - c.Q : v;
}

template <bool PM>
__device__ __forceinline__ void ct64(uint64_t &x, uint64_t &y, ulonglong2 w, const Ntt64Consts &c)
{
    const uint64_t t = mul64<PM>(y, w, c);
    y = x + c.twoQ - t;
    x = x + t;
}

// Gentleman-Sande butterfly of inputs below 2^K Q. Shoup: K = 1, the sum is
// brought back below 2Q. PM: the sum is left at 2^(K+1) Q.
template <bool PM, int K>
__device__ __forceinline__ void gs64(uint64_t &x, uint64_t &y, ulonglong2 w, const Ntt64Consts &c)
{
    uint64_t u = x + y;
    if (!PM) u = u >= c.twoQ ? u - c.twoQ : u;
    const uint64_t v = mul64<PM>(x - y + (PM ? c.Q << K : c.twoQ), w, c);
    x = u;
    y = v;
}

__device__ __forceinline__ void group_sync(int bar_id, int threads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "r"(threads) : "memory");
}

// One radix-2^R forward pass: stages t, t/2, ..., t/2^(R-1) (m = N / 2t) on
// the tuples e0 + k t/2^(R-1) (k < 2^R) of every 2t-block.
template <bool PM, int G, int R, bool P>
__device__ __forceinline__ void fwd_passR(uint64_t *a, const ulonglong2 *__restrict__ tw, const Ntt64Consts &c,
                                          int tid, int t, int m)
{
    constexpr int K = 1 << R;
    const int h = t >> (R - 1);
    for (int oc = tid; oc < 2048 / K; oc += G) {
        const int grp = oc / h, j = oc - grp * h;
        // e0 + k h in the layout: base + pi(k h), as j < h and h divides 16 or 16 divides h
        uint64_t *const b = a + pi<P>(grp * 2 * t + j);
        uint64_t x[K];
#pragma unroll
        for (int k = 0; k < K; k++) x[k] = b[pi<P>(k * h)];
#pragma unroll
        for (int st = 0; st < R; st++) {
            const int d = K >> (st + 1);
#pragma unroll
            for (int k = 0; k < K; k++) {
                if (k & d) continue;
                ct64<PM>(x[k], x[k + d], __ldg(tw + (m << st) + (grp << st) + (k >> (R - st))), c);
            }
        }
#pragma unroll
        for (int k = 0; k < K; k++) b[pi<P>(k * h)] = x[k];
    }
}

// Forward NTT of a[poly_words64<P>()] (layout pi<P>) in shared memory by `G` threads (tid < G) that share
// the named barrier `bar`. tw[k] = (psi^bitrev(k), companion). Input < Q,
// output < 23Q, bit-reversed order as the reference's. Two radix-16 passes
// (stages t = 1024..128, 64..8) and one radix-8 pass (t = 4, 2, 1).
template <bool PM, int G, bool P>
__device__ __forceinline__ void ntt64_fwd_2048(uint64_t *a, const ulonglong2 *__restrict__ tw, const Ntt64Consts &c,
                                               int tid, int bar)
{
    fwd_passR<PM, G, 4, P>(a, tw, c, tid, 1024, 1);   // t = 1024 .. 128
    group_sync(bar, G);
    fwd_passR<PM, G, 4, P>(a, tw, c, tid, 64, 16);    // t = 64 .. 8
    group_sync(bar, G);
    fwd_passR<PM, G, 3, P>(a, tw, c, tid, 4, 256);    // t = 4, 2, 1
    group_sync(bar, G);
}

// Forward NTT as ntt64_fwd_2048 of the polynomial whose word e is load(j, k),
// e = j + 128 k, into a (layout pi<P>): the first pass (stages t = 1024 .. 128)
// needs no pass of its own to write the words before it. Output < 23Q.
template <bool PM, int G, bool P, class Load>
__device__ __forceinline__ void ntt64_fwd_2048_load(uint64_t *a, Load load, const ulonglong2 *__restrict__ tw,
                                                    const Ntt64Consts &c, int tid, int bar)
{
    for (int j = tid; j < 128; j += G) {
        uint64_t x[16];
#pragma unroll
        for (int k = 0; k < 16; k++) x[k] = load(j, k);
#pragma unroll
        for (int st = 0; st < 4; st++) {
            const int d = 16 >> (st + 1);
#pragma unroll
            for (int k = 0; k < 16; k++) {
                if (k & d) continue;
                ct64<PM>(x[k], x[k + d], __ldg(tw + (1 << st) + (k >> (4 - st))), c);
            }
        }
        uint64_t *const b = a + pi<P>(j);
#pragma unroll
        for (int k = 0; k < 16; k++) b[pi<P>(k * 128)] = x[k];
    }
    group_sync(bar, G);
    fwd_passR<PM, G, 4, P>(a, tw, c, tid, 64, 16);    // t = 64 .. 8
    group_sync(bar, G);
    fwd_passR<PM, G, 3, P>(a, tw, c, tid, 4, 256);    // t = 4, 2, 1
    group_sync(bar, G);
}

// The gadget digit (src >> sh) & mask of a canonical time-domain polynomial src
// (layout pi<P>), for ntt64_fwd_2048_load.
template <bool P>
struct LoadDigit64 {
    const uint64_t *src;
    uint32_t sh, mask;
    __device__ __forceinline__ uint64_t operator()(int j, int k) const
    {
        return (uint32_t)(src[pi<P>(j) + pi<P>(k * 128)] >> sh) & mask;
    }
};

// One radix-8 inverse pass: stages t, 2t, 4t (m = N / 2t) on the octets
// e0 + k t (k < 8) of every 8t-block. Inputs below 2^K Q (PM; else 2Q); PM
// outputs below 2^(K+3) Q, or below 2Q with FOLD (the products, x[4..7], are).
template <bool PM, int G, bool P, int K, bool FOLD>
__device__ __forceinline__ void inv_pass8(uint64_t *a, const ulonglong2 *__restrict__ itw, const Ntt64Consts &c,
                                          int tid, int t, int m)
{
    for (int oc = tid; oc < 256; oc += G) {
        int grp = oc / t;
        const int j = oc - grp * t;
        // t = 8, padded: a half warp takes blocks two apart (136 words, the other
        // eight bank pairs) rather than neighbours (68 words)
        if (P && t == 8) grp = (grp & ~3) | ((grp & 1) << 1) | ((grp >> 1) & 1);
        uint64_t *const b = a + pi<P>(grp * 8 * t + j);
        uint64_t x[8];
#pragma unroll
        for (int k = 0; k < 8; k++) x[k] = b[pi<P>(k * t)];
#pragma unroll
        for (int k = 0; k < 4; k++) gs64<PM, K>(x[2 * k], x[2 * k + 1], __ldg(itw + m + 4 * grp + k), c);
        const ulonglong2 w2a = __ldg(itw + (m >> 1) + 2 * grp), w2b = __ldg(itw + (m >> 1) + 2 * grp + 1);
        gs64<PM, K + 1>(x[0], x[2], w2a, c);
        gs64<PM, K + 1>(x[1], x[3], w2a, c);
        gs64<PM, K + 1>(x[4], x[6], w2b, c);
        gs64<PM, K + 1>(x[5], x[7], w2b, c);
        const ulonglong2 w4 = __ldg(itw + (m >> 2) + grp);
        gs64<PM, K + 2>(x[0], x[4], w4, c);
        gs64<PM, K + 2>(x[1], x[5], w4, c);
        gs64<PM, K + 2>(x[2], x[6], w4, c);
        gs64<PM, K + 2>(x[3], x[7], w4, c);
        if (PM && FOLD) {
#pragma unroll
            for (int k = 0; k < 4; k++) x[k] = reduce64<PM>(x[k], c);
        }
#pragma unroll
        for (int k = 0; k < 8; k++) b[pi<P>(k * t)] = x[k];
    }
}

// Inverse NTT of a[poly_words64<P>()] (layout pi<P>; values < 2Q, bit-reversed order) in shared memory
// -> canonical coefficients times N^-1. itw[k] = (psi^-bitrev(k), companion).
// Three radix-8 passes (stages t = 1..4, 8..32, 64..256) and one radix-4 pass
// (t = 512 and the last stage, t = 1024, with N^-1 folded into both outputs).
template <bool PM, int G, bool P>
__device__ __forceinline__ void ntt64_inv_2048(uint64_t *a, const ulonglong2 *__restrict__ itw, const Ntt64Consts &c,
                                               int tid, int bar)
{
    inv_pass8<PM, G, P, 1, false>(a, itw, c, tid, 1, 1024);   // 2Q -> 16Q
    group_sync(bar, G);
    inv_pass8<PM, G, P, 4, true>(a, itw, c, tid, 8, 128);     // 16Q -> 2Q
    group_sync(bar, G);
    inv_pass8<PM, G, P, 1, false>(a, itw, c, tid, 64, 16);    // 2Q -> 16Q
    group_sync(bar, G);
    for (int b = tid; b < 512; b += G) {
        uint64_t x0 = a[pi<P>(b)], x1 = a[pi<P>(b + 512)], x2 = a[pi<P>(b + 1024)], x3 = a[pi<P>(b + 1536)];
        gs64<PM, 4>(x0, x1, __ldg(itw + 2), c);   // t = 512, m = 2, block 0
        gs64<PM, 4>(x2, x3, __ldg(itw + 3), c);   // block 1
        // t = 1024, m = 1, with N^-1 folded into both outputs
        const uint64_t bias = PM ? c.Q << 5 : c.twoQ;
        const ulonglong2 wu = make_ulonglong2(c.iN, c.iNs), wv = make_ulonglong2(c.iw1N, c.iw1Ns);
        uint64_t u = mul64<PM>(x0 + x2, wu, c);
        uint64_t v = mul64<PM>(x0 - x2 + bias, wv, c);
        a[pi<P>(b)] = u >= c.Q ? u - c.Q : u;
        a[pi<P>(b + 1024)] = v >= c.Q ? v - c.Q : v;
        u = mul64<PM>(x1 + x3, wu, c);
        v = mul64<PM>(x1 - x3 + bias, wv, c);
        a[pi<P>(b + 512)] = u >= c.Q ? u - c.Q : u;
        a[pi<P>(b + 1536)] = v >= c.Q ? v - c.Q : v;
    }
    group_sync(bar, G);
}

}  // namespace dev
}  // namespace fheacc

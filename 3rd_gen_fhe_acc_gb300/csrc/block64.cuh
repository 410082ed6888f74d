// block64.cuh -- the 64-bit path's block form of an RLWE x RGSW step: transforms cut into
// their residues mod the factors X^M - zeta of X^2048 + 1 (see blind_rotate64.cu), for
// moduli Q = 2^b - c. Shared by the blind rotation, the RLWE x RGSW products
// (products64.cu) and expand_RLWE (expand.cu).
#pragma once
#include "br64.cuh"
#include <cooperative_groups.h>

namespace fheacc {
namespace dev {

namespace cg = cooperative_groups;

// Threads of a CTA: the 10 digits' 512-word blocks are 640 octets (digitG = 6), all
// at once in the latency form (kTB), half of them for each of the throughput form's two
// workers in a CTA (kTP).
constexpr int kTB = 640, kTP = 320;
// A worker alone on its SM (digitG = 7 and 8, whose work areas fill more than half of the
// shared memory) has kTB threads: 1000 products at digitG = 8 451 us with kTP, 344 so;
// 912 gates of n = 32 19.8 ms, 16.2 so.
__host__ __device__ constexpr int worker_threads64(int W) { return W == 1 ? kTB : kTP; }

// x w of the MAC, x = x1 2^27 + x0 < 2^59 and limbs w < 2^27: the sums of x0 w0, of
// (x0 + x1) (w0 + w1) and of x1 w1, three multiplies (Karatsuba; four without: 2048 gates
// 1 % slower). At most 16 products: the middle sum < 16 2^31.6 2^28 < 2^64.
__device__ __forceinline__ void mac27(uint64_t (&s)[3], uint32_t x0, uint32_t x1, uint2 w)
{
    s[0] += mul_wide64(x0, w.x);
    s[1] += mul_wide64(x0 + x1, w.x + w.y);
    s[2] += mul_wide64(x1, w.y);
}

// The value sums[0] + 2^27 (sums[1] - sums[0] - sums[2]) + 2^54 sums[2] mod Q, below 2Q:
// c54 (2^54 mod Q, below 2^19) folds the part Y above 2^54 (Y < 2^64) twice.
__device__ __forceinline__ uint64_t mac27_reduce(const uint64_t (&s)[3], uint32_t c54, const Ntt64Consts &c)
{
    constexpr uint64_t m27 = (1u << 27) - 1;
    const uint64_t T = s[1] - s[0] - s[2] + (s[0] >> 27);
    const uint64_t low = (s[0] & m27) | ((T & m27) << 27);
    const uint64_t Y = s[2] + (T >> 27);
    const uint64_t zl = mul_wide64((uint32_t)Y, c54);
    const uint64_t zm = mad_wide64((uint32_t)(Y >> 32), c54, zl >> 32);   // Z = zm 2^32 + low word of zl
    const uint64_t z0 = ((zm << 32) | (uint32_t)zl) & (((uint64_t)1 << 54) - 1);
    return reduce64<true>(mad_wide64((uint32_t)(zm >> 22), c54, low + z0), c);
}

template <int B, int C>
struct BlockLayout {
    static constexpr int M = 2048 / B, NB = B / C, ME = M + M / 16;   // words of a block, blocks of a CTA
    static constexpr int GBUF = C > 1 ? 2 : 1;
    static constexpr size_t g_off = 0;                                  // [GBUF][2][2048]
    static constexpr size_t acc_off = (size_t)GBUF * 2 * 2048 * 8;      // [2][NB * ME], layout px
    static size_t __host__ __device__ work_off(int) { return acc_off + (size_t)2 * NB * ME * 8; }
    // digit NTTs [2 (DG - 1)][ME]; the inverse NTT's [2][NB * ME] before them
    static size_t __host__ __device__ work_words(int DG)
    {
        const int d = 2 * (DG - 1), i = 2 * NB;
        return (size_t)(d > i ? d : i) * ME;
    }
    // the latency form's key buffer: the rows of one block
    static size_t __host__ __device__ key_off(int DG) { return work_off(DG) + work_words(DG) * 8; }
    static size_t __host__ __device__ key_bytes(int DG) { return (size_t)DG * 4 * M * 8; }
};

// Threads that share a 512- or 256-word transform: GS = 32 or 64 consecutive ones,
// group gi of the CTA. A transform's passes then need no CTA barrier between them.
template <int GS>
__device__ __forceinline__ void group_sync64(int gi)
{
    if (GS == 32) __syncwarp();
    else group_sync(1 + gi, GS);
}

// One radix-2^R forward pass of a digit's block d (M words, layout px) by a group:
// stages t, t/2, ..; blk: the block, gt: the thread in the group.
template <int M, int R, int GS>
__device__ __forceinline__ void blk_fwd_pass(uint64_t *d, int blk, int t, int gt, const ulonglong2 *__restrict__ tw,
                                             const Ntt64Consts &c)
{
    constexpr int K = 1 << R, per = M / K;
    const int h = t >> (R - 1), m = 1024 / t;
    for (int q = gt; q < per; q += GS) {
        const int gl = q / h, j = q - gl * h;
        const int grp = blk * (M / (2 * t)) + gl;
        uint64_t *const b = d + px(gl * 2 * t + j);
        uint64_t x[K];
#pragma unroll
        for (int k = 0; k < K; k++) x[k] = b[px(k * h)];
#pragma unroll
        for (int st = 0; st < R; st++) {
            const int dl = K >> (st + 1);
#pragma unroll
            for (int k = 0; k < K; k++) {
                if (k & dl) continue;
                ct64<true>(x[k], x[k + dl], __ldg(tw + ((m + grp) << st) + (k >> (R - st))), c);
            }
        }
#pragma unroll
        for (int k = 0; k < K; k++) b[px(k * h)] = x[k];
    }
}

// A word of a digit's residue: y(0) plus z[i - 1] (zeta^i times 2^pm_s) times y(i), y < 2^30.
template <int B, class Y>
__device__ __forceinline__ uint64_t digit_residue(const uint64_t (&z)[B - 1], const Ntt64Consts &c, Y y)
{
    uint64_t U = 0, V = 0;
#pragma unroll
    for (int i = 1; i < B; i++) {
        const uint32_t v = y(i);
        U = mad_wide64(v, (uint32_t)z[i - 1], U);
        V = mad_wide64(v, (uint32_t)(z[i - 1] >> 32), V);
    }
    return fold64(U, V, c) + y(0);
}

// The first pass (M = 512: t = 256 .. 64; 256: t = 128, 64) of a polynomial's residue mod
// X^M - zeta, computed as it loads: word(j, k) is word j + 64 k of the residue.
template <int B, int GS, class Word>
__device__ __forceinline__ void blk_fwd_first(uint64_t *d, Word word, int blk, int gt,
                                              const ulonglong2 *__restrict__ tw, const Ntt64Consts &c)
{
    constexpr int M = 2048 / B, R = M == 512 ? 3 : 2, K = 1 << R;
    for (int j = gt; j < 64; j += GS) {
        uint64_t v[K];
#pragma unroll
        for (int k = 0; k < K; k++) v[k] = word(j, k);
#pragma unroll
        for (int st = 0; st < R; st++) {
            const int dl = K >> (st + 1);
#pragma unroll
            for (int k = 0; k < K; k++) {
                if (k & dl) continue;
                ct64<true>(v[k], v[k + dl], __ldg(tw + ((B + blk) << st) + (k >> (R - st))), c);
            }
        }
        uint64_t *const o = d + px(j);
#pragma unroll
        for (int k = 0; k < K; k++) o[px(64 * k)] = v[k];
    }
}

// One radix-8 inverse pass of a block (M words, layout px) by a group, src to
// out(word, x); stages t, 2t, 4t. Inputs below 2^K0 Q, outputs below 2^(K0+3) Q, or
// below 2Q with FOLD.
template <int M, int K0, bool FOLD, int GS, class Out>
__device__ __forceinline__ void blk_inv_pass8(const uint64_t *src, int blk, int t, int gt,
                                              const ulonglong2 *__restrict__ itw, const Ntt64Consts &c, Out out)
{
    constexpr int per = M / 8;
    const int m = 1024 / t;
    for (int q = gt; q < per; q += GS) {
        int gl = q / t;
        const int j = q - gl * t;
        if (t == 8) gl = (gl & ~3) | ((gl & 1) << 1) | ((gl >> 1) & 1);   // as inv_pass8
        const int grp = blk * (M / (8 * t)) + gl, e0 = gl * 8 * t + j;
        const uint64_t *b = src + px(e0);
        uint64_t x[8];
#pragma unroll
        for (int k = 0; k < 8; k++) x[k] = b[px(k * t)];
#pragma unroll
        for (int k = 0; k < 4; k++) gs64<true, K0>(x[2 * k], x[2 * k + 1], __ldg(itw + m + 4 * grp + k), c);
        const ulonglong2 w2a = __ldg(itw + (m >> 1) + 2 * grp), w2b = __ldg(itw + (m >> 1) + 2 * grp + 1);
        gs64<true, K0 + 1>(x[0], x[2], w2a, c);
        gs64<true, K0 + 1>(x[1], x[3], w2a, c);
        gs64<true, K0 + 1>(x[4], x[6], w2b, c);
        gs64<true, K0 + 1>(x[5], x[7], w2b, c);
        const ulonglong2 w4 = __ldg(itw + (m >> 2) + grp);
#pragma unroll
        for (int k = 0; k < 4; k++) gs64<true, K0 + 2>(x[k], x[k + 4], w4, c);
        if (FOLD) {
#pragma unroll
            for (int k = 0; k < 4; k++) x[k] = reduce64<true>(x[k], c);
        }
        out(e0, x);
    }
}

// The last inverse stages (t = M .. 1024, N^-1 folded in) of the tuple x_i = word
// j + i M, canonical; inputs below 2^K Q (K <= 4).
template <int B>
__device__ __forceinline__ void blk_inv_last(uint64_t (&x)[B], const ulonglong2 *__restrict__ itw, const Ntt64Consts &c)
{
    if (B == 8) {
#pragma unroll
        for (int i = 0; i < B / 2; i++) gs64<true, 3>(x[2 * i], x[2 * i + 1], __ldg(itw + 4 + i), c);
#pragma unroll
        for (int i = 0; i < B / 4; i++) {
            const ulonglong2 w = __ldg(itw + 2 + i);
            gs64<true, 4>(x[4 * i], x[4 * i + 2], w, c);
            gs64<true, 4>(x[4 * i + 1], x[4 * i + 3], w, c);
        }
    } else {
#pragma unroll
        for (int i = 0; i < B / 2; i++) gs64<true, 4>(x[2 * i], x[2 * i + 1], __ldg(itw + 2 + i), c);
    }
    const ulonglong2 wu = make_ulonglong2(c.iN, c.iNs), wv = make_ulonglong2(c.iw1N, c.iw1Ns);
#pragma unroll
    for (int i = 0; i < B / 2; i++) {
        const uint64_t a = x[i], b = x[i + B / 2];
        const uint64_t u = mul64<true>(a + b, wu, c), v = mul64<true>(a - b + (c.Q << 5), wv, c);
        x[i] = u >= c.Q ? u - c.Q : u;
        x[i + B / 2] = v >= c.Q ? v - c.Q : v;
    }
}

// What a CTA of a cluster of C brings to a step.
template <int B, int C>
struct BlockCta {
    uint64_t *g, *acc, *work;      // shared memory (BlockLayout); g: the buffer of this step
    uint64_t *peer[C];             // the cluster's g buffers of this step
    const uint64_t (*zeta)[B - 1]; // powers of the blocks' zeta, times 2^pm_s
    int rank;
};

// The accumulator's inverse NTT by T threads (tid < T) that share the named barrier `bar`
// (0: the whole CTA): canonical coefficients of its NP polys in s.g.
template <int B, int C, int T, int NP = 2>
__device__ __forceinline__ void block_to_time(const BlockCta<B, C> &s, const ulonglong2 *__restrict__ itw,
                                              const Ntt64Consts &c, int tid, int bar)
{
    using L = BlockLayout<B, C>;
    constexpr int M = L::M, NB = L::NB, ME = L::ME, NW = NB * M;
    uint64_t *const work = s.work, *const acc = s.acc;
    constexpr int GS = M == 512 && T == kTB ? 64 : 32, NG = T / GS;
    const int gi = tid / GS, gt = tid - gi * GS;
    // ---- 1. inverse stages inside the blocks, a group per block
    for (int u = gi; u < NP * NB; u += NG) {
        const int p = u / NB, lb = u - p * NB, blk = s.rank * NB + lb, base = p * 2048 + blk * M;
        uint64_t *const w = work + u * ME;
        blk_inv_pass8<M, 1, false, GS>(acc + p * px(NW) + lb * ME, blk, 1, gt, itw, c, [&](int e0, uint64_t (&x)[8]) {
#pragma unroll
            for (int k = 0; k < 8; k++) w[px(e0) + k] = x[k];   // 2Q -> 16Q
        });
        group_sync64<GS>(gi);
        blk_inv_pass8<M, 4, true, GS>(w, blk, 8, gt, itw, c, [&](int e0, uint64_t (&x)[8]) {   // -> 2Q
#pragma unroll
            for (int k = 0; k < 8; k++) w[px(e0) + px(8 * k)] = x[k];
        });
        group_sync64<GS>(gi);
        if (B == 8) {   // t = 64, 128: 2Q -> 8Q
            for (int j = gt; j < 64; j += GS) {
                uint64_t x[4];
#pragma unroll
                for (int k = 0; k < 4; k++) x[k] = w[px(j) + px(64 * k)];
                gs64<true, 1>(x[0], x[1], __ldg(itw + 16 + 2 * blk), c);
                gs64<true, 1>(x[2], x[3], __ldg(itw + 16 + 2 * blk + 1), c);
                const ulonglong2 w2 = __ldg(itw + 8 + blk);
                gs64<true, 2>(x[0], x[2], w2, c);
                gs64<true, 2>(x[1], x[3], w2, c);
#pragma unroll
                for (int r = 0; r < C; r++)
#pragma unroll
                    for (int k = 0; k < 4; k++) s.peer[r][base + j + 64 * k] = x[k];
            }
        } else {        // t = 64, 128, 256: 2Q -> 16Q
            blk_inv_pass8<M, 1, false, GS>(w, blk, 64, gt, itw, c, [&](int e0, uint64_t (&x)[8]) {
#pragma unroll
                for (int r = 0; r < C; r++)
#pragma unroll
                    for (int k = 0; k < 8; k++) s.peer[r][base + e0 + 64 * k] = x[k];
            });
        }
    }
    if (C > 1) cg::this_cluster().sync();
    else group_sync(bar, T);
    // ---- 2. last inverse stages of all words
    for (int u = tid; u < NP * M; u += T) {
        uint64_t *const b = s.g + (u / M) * 2048 + u % M;
        uint64_t x[B];
#pragma unroll
        for (int i = 0; i < B; i++) x[i] = b[i * M];
        blk_inv_last<B>(x, itw, c);
#pragma unroll
        for (int i = 0; i < B; i++) b[i * M] = x[i];
    }
    group_sync(bar, T);
}

// One step of the CTA's blocks by T threads (tid < T) that share the named barrier `bar`
// (0: the whole CTA). A: digitG, bg_bits and c54. keys(lb): waits for and returns
// the key rows of block lb, [DG][2][2] rows of M words `row` words apart (KG: in global
// memory, read past L1, which then keeps the twiddles of the block);
// done(lb) runs after the block's products.
template <int B, int C, int T, bool KG, class Args, class Keys, class Done>
__device__ __forceinline__ void block_step(const BlockCta<B, C> &s, const Args &A,
                                           const ulonglong2 *__restrict__ tw, const ulonglong2 *__restrict__ itw,
                                           const Ntt64Consts &c, size_t row, int tid, int bar, Keys keys,
                                           Done done)
{
    using L = BlockLayout<B, C>;
    constexpr int M = L::M, NB = L::NB, ME = L::ME, NW = NB * M;
    const int DG = A.DG, nd = 2 * (DG - 1);
    const uint32_t mask = (1u << A.bg_bits) - 1;
    uint64_t *const work = s.work, *const acc = s.acc;
    constexpr int GS = M == 512 && T == kTB ? 64 : 32, NG = T / GS;
    const int gi = tid / GS, gt = tid - gi * GS;
    block_to_time<B, C, T>(s, itw, c, tid, bar);   // 1. and 2.
    for (int lb = 0; lb < NB; lb++) {
        const int blk = s.rank * NB + lb;
        // ---- 3. the digits' NTTs in the block, a group per digit
        for (int dd = gi; dd < nd; dd += NG) {
            const int p = dd / (DG - 1), h = dd - p * (DG - 1);
            uint64_t z[B - 1];
#pragma unroll
            for (int i = 0; i < B - 1; i++) z[i] = s.zeta[lb][i];
            uint64_t *const d = work + dd * ME;
            const uint64_t *const x = s.g + p * 2048;
            const uint32_t sh = A.bg_bits * (uint32_t)h;
            blk_fwd_first<B, GS>(d, [&](int j, int k) {
                const uint64_t *b = x + j + 64 * k;
                return digit_residue<B>(z, c, [&](int i) { return (uint32_t)(b[i * M] >> sh) & mask; });
            }, blk, gt, tw, c);
            group_sync64<GS>(gi);
            blk_fwd_pass<M, 3, GS>(d, blk, 32, gt, tw, c);   // t = 32 .. 8
            group_sync64<GS>(gi);
            blk_fwd_pass<M, 3, GS>(d, blk, 4, gt, tw, c);    // t = 4, 2, 1
        }
        const uint2 *const kb = keys(lb);
        group_sync(bar, T);
        // ---- multiply-accumulate
        for (int k = tid; k < M; k += T) {
            uint64_t sa[3] = {0, 0, 0}, sb[3] = {0, 0, 0};
            const uint2 *kk = kb + k;
            uint64_t *const a0 = acc + lb * ME + px(k);
#pragma unroll 6
            for (int h = 0; h < DG; h++, kk += 4 * row) {
#pragma unroll
                for (int p = 0; p < 2; p++) {
                    const uint64_t v = h < DG - 1 ? work[(p * (DG - 1) + h) * ME + px(k)] : a0[p * px(NW)];
                    const uint32_t x0 = (uint32_t)v & ((1u << 27) - 1), x1 = (uint32_t)(v >> 27);
                    mac27(sa, x0, x1, KG ? __ldcg(kk + (p * 2 + 0) * row) : kk[(p * 2 + 0) * row]);
                    mac27(sb, x0, x1, KG ? __ldcg(kk + (p * 2 + 1) * row) : kk[(p * 2 + 1) * row]);
                }
            }
            a0[0] = mac27_reduce(sa, A.c54, c);
            a0[px(NW)] = mac27_reduce(sb, A.c54, c);
        }
        group_sync(bar, T);
        done(lb);
    }
}

// Powers 1 .. B - 1 of the zeta of blocks first .. first + NB - 1.
template <int B, int NB>
__device__ __forceinline__ void block_zeta(uint64_t (*zeta)[B - 1], int first, const ulonglong2 *tw, const Ntt64Consts &c)
{
    const int tid = threadIdx.x;
    if (tid < NB) {
        const int d = first + tid;
        const uint64_t w = tw[B / 2 + d / 2].x >> c.pm_s, z = (d & 1) ? c.Q - w : w;
        uint64_t v = z;
        for (int i = 0; i < B - 1; i++) {
            zeta[tid][i] = v << c.pm_s;
            v = (uint64_t)((unsigned __int128)v * z % c.Q);
        }
    }
}

}  // namespace dev
}  // namespace fheacc

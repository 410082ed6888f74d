// blind_rotate64.cu -- blind rotation of the 64-bit-word path (N = 2048) for
// moduli Q = 2^b - c (pm64_shift in ntt64.cuh); other moduli take br64_kernel
// (bootstrap64.cu).
//
// Reference behaviour: the accumulate loop of eval_bootstrap
// (FHE_ACC_runtime/src/RLWE.cpp:733-767) -- LWE_evaluate (LWE.cpp:203-222),
// acc_initialization (RLWE.cpp:706-724), an RLWE_mult_RGSW (RLWE.cpp:642-704)
// per non-zero refresh residue -- then the NTT_a_transpose and inverse NTT that
// open LWE_keyswitch (LWE.cpp:235-238).
//
// Block form of a step. X^N + 1 splits into B factors X^M - zeta_d, M = N / B:
// the words [d M, (d + 1) M) of a bit-reversed NTT depend on the polynomial only
// through its residue mod X^M - zeta_d, x_0 + zeta_d x_M + zeta_d^2 x_2M + ...
// So one CTA can own some of the B blocks of the accumulator, the digit NTTs and
// the key rows, and needs the other CTAs only between the two halves of the
// inverse NTT. A cluster of C CTAs works on one ciphertext, each on B / C blocks:
//   1. the first stages of the inverse NTT of its blocks of the accumulator
//      (blocks are closed under them), written to every CTA's shared memory;
//      one cluster barrier per step;
//   2. the last log2 B inverse stages of all words (every CTA needs them all),
//      in registers: canonical coefficients x_j, x_{j+M}, ...;
//   3. per block, the digits' residues mod X^M - zeta_d from those registers (a
//      digit times a constant: two 32 x 32 -> 64 multiplies), three passes of
//      butterflies, and the multiply-accumulate of all digits with the block's
//      key rows, whose sums stay in registers: each key word is two limbs of 27
//      bits (8 bytes, half of a constant pair's), each product four multiplies into
//      three 64-bit sums, reduced once per output.
// The last digit's NTT is the accumulator itself (DevParams::last_digit_from_acc).
//
// Two kernels. br64_cluster_kernel (up to one ciphertext per SM) is for latency: per
// step 8.5 us on 8 CTAs, 10.5 on 4, 17.6 on 2, 31.4 on one, where a 256-thread worker
// took 75 us (40 with its register spills gone). br64_items_kernel is for batches: 27.8
// us per step and SM (2048 gates: 451 ms; 582 before the moduli's fold form). Both are
// bound by the multiply pipe: 48 k of its instructions a step, of which 29 k are
// 32 x 32 -> 64 multiplies; a loop of butterflies on registers alone keeps the pipe 74 %
// busy, the items form 62 %.
#include "br64.cuh"
#include <algorithm>
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace fheacc {
namespace dev {

// Threads of a CTA: the 10 digits' 512-word blocks are 640 octets (digitG = 6), all
// at once in the latency form, half of them in the throughput form (two CTAs per SM).
constexpr int kTB = 640, kTP = 320;

// Polls of an mbarrier before a key wait gives up and flags the launch.
constexpr unsigned kKeyWaitLimit = 1u << 22;

struct BlockArgs {
    const uint2 *btkey;   // [(i*digitR + j)*Br + r][digitG][2][2][2048] limb words (limb_word64)
    uint64_t *accs;       // [count][2][2048], NTT domain, values < 2Q
    const uint8_t *res;   // [count][n * digitR] residues
    size_t count;
    int S, DG;            // steps, digits
    uint32_t bg_bits, Br, flags;
    uint32_t c54;         // 2^54 mod Q
    unsigned *status;
    unsigned wait_limit;
};

// x w of the MAC: sums[0] + 2^27 sums[1] + 2^54 sums[2] (x < 2^59, limbs < 2^27,
// at most 16 products: sums[1] < 16 (2^59 + 2^54) < 2^64).
__device__ __forceinline__ void mac27(uint64_t (&s)[3], uint32_t x0, uint32_t x1, uint2 w)
{
    s[0] += mul_wide64(x0, w.x);
    s[1] += mul_wide64(x0, w.y);
    s[1] += mul_wide64(x1, w.x);
    s[2] += mul_wide64(x1, w.y);
}

// The value of the sums mod Q, below 2Q: c54 (2^54 mod Q, below 2^19) folds the part
// Y above 2^54 (Y < 2^64) twice.
__device__ __forceinline__ uint64_t mac27_reduce(const uint64_t (&s)[3], uint32_t c54, const Ntt64Consts &c)
{
    constexpr uint64_t m27 = (1u << 27) - 1;
    const uint64_t T = s[1] + (s[0] >> 27);
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

// The first pass (M = 512: t = 256 .. 64; 256: t = 128, 64) with the digit's residue
// mod X^M - zeta computed as it loads: word j is the digit of x[j] plus
// z[i - 1] times the digit of x[j + i M].
template <int B, int GS>
__device__ __forceinline__ void blk_fwd_first(uint64_t *d, const uint64_t *x, const uint64_t (&z)[B - 1], uint32_t sh,
                                              uint32_t mask, int blk, int gt, const ulonglong2 *__restrict__ tw,
                                              const Ntt64Consts &c)
{
    constexpr int M = 2048 / B, R = M == 512 ? 3 : 2, K = 1 << R;
    for (int j = gt; j < 64; j += GS) {
        uint64_t v[K];
#pragma unroll
        for (int k = 0; k < K; k++) {
            const uint64_t *b = x + j + 64 * k;
            uint64_t U = 0, V = 0;
#pragma unroll
            for (int i = 1; i < B; i++) {
                const uint32_t y = (uint32_t)(b[i * M] >> sh) & mask;
                U = mad_wide64(y, (uint32_t)z[i - 1], U);
                V = mad_wide64(y, (uint32_t)(z[i - 1] >> 32), V);
            }
            v[k] = fold64(U, V, c) + ((uint32_t)(b[0] >> sh) & mask);
        }
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

__device__ __forceinline__ int next_issued(const uint8_t *res, int s, int S, int mode)
{
    for (s++; s < S; s++)
        if (step_issued(res, s, mode)) return s;
    return S;
}

// What a CTA of a cluster of C brings to a step.
template <int B, int C>
struct BlockCta {
    uint64_t *g, *acc, *work;      // shared memory (BlockLayout); g: the buffer of this step
    uint64_t *peer[C];             // the cluster's g buffers of this step
    const uint64_t (*zeta)[B - 1]; // powers of the blocks' zeta, times 2^pm_s
    int rank;
};

// One step of the CTA's blocks by T threads (tid < T) that share the named barrier
// `bar` (0: the whole CTA). keys(lb): waits for and returns
// the key rows of block lb, [DG][2][2] rows of M words `row` words apart (KG: in global
// memory, read past L1, which then keeps the twiddles of the block);
// done(lb) runs after the block's products.
template <int B, int C, int T, bool KG, class Keys, class Done>
__device__ __forceinline__ void block_step(const BlockCta<B, C> &s, const BlockArgs &A,
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
    // ---- 1. inverse stages inside the blocks, a group per block
    for (int u = gi; u < 2 * NB; u += NG) {
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
    for (int u = tid; u < 2 * M; u += T) {
        uint64_t *const b = s.g + (u / M) * 2048 + u % M;
        uint64_t x[B];
#pragma unroll
        for (int i = 0; i < B; i++) x[i] = b[i * M];
        blk_inv_last<B>(x, itw, c);
#pragma unroll
        for (int i = 0; i < B; i++) b[i * M] = x[i];
    }
    group_sync(bar, T);
    for (int lb = 0; lb < NB; lb++) {
        const int blk = s.rank * NB + lb;
        // ---- 3. the digits' NTTs in the block, a group per digit
        for (int dd = gi; dd < nd; dd += NG) {
            const int p = dd / (DG - 1), h = dd - p * (DG - 1);
            uint64_t z[B - 1];
#pragma unroll
            for (int i = 0; i < B - 1; i++) z[i] = s.zeta[lb][i];
            uint64_t *const d = work + dd * ME;
            blk_fwd_first<B, GS>(d, s.g + p * 2048, z, A.bg_bits * (uint32_t)h, mask, blk, gt, tw, c);
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

// Latency form: one ciphertext per cluster of C CTAs at a time, its accumulator in
// shared memory for all its steps, a block's keys by bulk copies issued as soon as
// the products of the block before are done.
template <int B, int C>
__global__ void __launch_bounds__(kTB, 1) br64_cluster_kernel(const __grid_constant__ BlockArgs A,
                                                             const ulonglong2 *__restrict__ tw,
                                                             const ulonglong2 *__restrict__ itw,
                                                             const __grid_constant__ Ntt64Consts c)
{
    using L = BlockLayout<B, C>;
    constexpr int M = L::M, NB = L::NB, NW = NB * M, T = kTB;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    uint64_t *const g = reinterpret_cast<uint64_t *>(smem_raw + L::g_off);
    uint64_t *const acc = reinterpret_cast<uint64_t *>(smem_raw + L::acc_off);
    uint64_t *const work = reinterpret_cast<uint64_t *>(smem_raw + L::work_off(A.DG));
    uint2 *const kbuf = reinterpret_cast<uint2 *>(smem_raw + L::key_off(A.DG));
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint64_t zeta[NB][B - 1];
    const int tid = threadIdx.x, DG = A.DG;
    const int rank = C > 1 ? (int)(blockIdx.x % C) : 0, first = rank * NW;
    const int mode = issue_mode(A.flags);
    const size_t rgsw = (size_t)DG * 4 * 2048;
    uint64_t *peer[C];
    peer[0] = g;
    if (C > 1) {
        cg::cluster_group cl = cg::this_cluster();
#pragma unroll
        for (int r = 0; r < C; r++) peer[r] = cl.map_shared_rank(g, r);
    }
    block_zeta<B, NB>(zeta, rank * NB, tw, c);
    if (tid == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
    }
    if (C > 1) cg::this_cluster().sync();
    else __syncthreads();
    unsigned parity = 0;
    bool failed = false, pending = false;   // pending: a key copy not yet waited for

    for (size_t gid = blockIdx.x / C; gid < A.count; gid += gridDim.x / C) {
        const uint8_t *res = A.res + gid * (size_t)A.S;
        uint64_t *ga = A.accs + gid * 4096;
        for (int u = tid; u < 2 * NW; u += T) {
            const int p = u / NW, e = u - p * NW;
            acc[p * px(NW) + px(e)] = __ldcg(ga + p * 2048 + first + e);
        }
        __syncthreads();
        // rows of block lb of step s into kbuf (warp 0)
        auto fetch = [&](int s, int lb) {
            if (tid >= 32 || failed) return;
            if (tid == 0) mbar_expect_tx(&bar, (unsigned)L::key_bytes(DG));
            __syncwarp();
            const uint2 *src = A.btkey + ((size_t)s * A.Br + res[s]) * rgsw + first + lb * M;
            if (tid < DG * 4) bulk_copy_g2s(kbuf + tid * M, src + (size_t)tid * 2048, M * 8, &bar);
        };
        int s = next_issued(res, -1, A.S, mode);
        if (s < A.S) {
            fetch(s, 0);
            pending = !failed;
        }
        for (int buf = 0; s < A.S; buf ^= C > 1) {
            const int next = next_issued(res, s, A.S, mode);
            BlockCta<B, C> cta{g + buf * 4096, acc, work, {}, zeta, rank};
#pragma unroll
            for (int r = 0; r < C; r++) cta.peer[r] = peer[r] + buf * 4096;
            block_step<B, C, T, false>(
                cta, A, tw, itw, c, M, tid, 0,
                [&](int) {
                    if (pending && !failed) {
                        if (mbar_wait_bounded(&bar, parity, (int)A.wait_limit)) {
                            parity ^= 1u;
                        } else {
                            // flag the launch and let the cluster run to its end without
                            // keys: its barriers need every CTA
                            failed = true;
                            if (tid == 0) atomicOr(A.status, kStatusWaitLimit);
                        }
                    }
                    return (const uint2 *)kbuf;
                },
                [&](int lb) {
                    if (lb + 1 < NB) fetch(s, lb + 1);
                    else if (next < A.S) fetch(next, 0);
                    else pending = pending && failed;   // nothing in flight, but for a copy that was given up
                });
            s = next;
        }
        for (int u = tid; u < 2 * NW; u += T) {
            const int p = u / NW, e = u - p * NW;
            ga[p * 2048 + first + e] = acc[p * px(NW) + px(e)];
        }
        __syncthreads();
    }
    // a copy that was given up must land before the CTA's shared memory goes
    if (failed && tid == 0) mbar_wait_bounded(&bar, parity, (int)kKeyWaitLimit);
    if (C > 1) cg::this_cluster().sync();
}

// Polls of a worker waiting for another worker's item of the same ciphertext
// (about 60 ns each) before it gives up and flags the launch.
constexpr unsigned kItemWaitLimit = 1u << 26;

// Steps of an item: long enough that taking it, and the accumulator's way through L2
// and back, cost little, short enough that the keys in use (9 MB a step) stay in L2 and
// the batch ends evenly. 2048 gates, us per step and SM: 29.2 with 1 step, 28.3 with 2,
// 27.8 with 4 and with 6, 28.2 with 8.
constexpr int kItemSteps = 4;

// Throughput form: W workers of kTP threads per CTA (two, so that one's barriers and
// loads overlap the other's arithmetic; in one CTA, because their 20 warps then spread
// evenly over the SM's four schedulers: as two CTAs of 10 warps, two schedulers get 6
// and two get 4, 30.0 against 29.4 us per step and SM). Each worker takes items,
// kItemSteps consecutive steps of one ciphertext, from one cursor that walks them
// step-major, so all workers stream the same few steps' keys (9 MB a step) through L2
// and the batch ends evenly whatever its size. Accumulators live in global memory
// between items (L2, evict-last). An item is run once the item of the same ciphertext
// before it has finished (done[]); that one was taken earlier, by a worker that is
// running, so the wait ends whether or not the whole grid is resident.
template <int B, int W>
__global__ void __launch_bounds__(W * kTP, 1) br64_items_kernel(const __grid_constant__ BlockArgs A,
                                                           unsigned long long *cursor, int *done,
                                                           const ulonglong2 *__restrict__ tw,
                                                           const ulonglong2 *__restrict__ itw,
                                                           const __grid_constant__ Ntt64Consts c)
{
    using L = BlockLayout<B, 1>;
    constexpr int T = kTP;
    extern __shared__ __align__(128) unsigned char smem_all[];
    const int wk = threadIdx.x / T, tid = threadIdx.x - wk * T, bar = 1 + wk;
    unsigned char *const smem_raw = smem_all + wk * L::key_off(A.DG);
    uint64_t *const g = reinterpret_cast<uint64_t *>(smem_raw + L::g_off);
    uint64_t *const acc = reinterpret_cast<uint64_t *>(smem_raw + L::acc_off);
    uint64_t *const work = reinterpret_cast<uint64_t *>(smem_raw + L::work_off(A.DG));
    __shared__ uint64_t zeta[B][B - 1];
    __shared__ int plans[W][2];   // item of the ciphertext (-1: none left), ciphertext
    int *const plan = plans[wk];
    const int mode = issue_mode(A.flags);
    const size_t rgsw = (size_t)A.DG * 4 * 2048;
    block_zeta<B, B>(zeta, 0, tw, c);
    __syncthreads();
    const unsigned long long items = (unsigned long long)((A.S + kItemSteps - 1) / kItemSteps) * A.count;
    for (;;) {
        if (tid == 0) {
            const unsigned long long v = atomicAdd(cursor, 1ull);
            const int it = v < items ? (int)(v / A.count) : -1;
            const size_t k = it < 0 ? 0 : (size_t)(v - (unsigned long long)it * A.count);
            plan[0] = it;
            plan[1] = (int)k;
            if (it >= 0) {
                const volatile int *d = done + k;
                unsigned polls = 0;
                while (*d != it - 1) {
                    if (++polls > A.wait_limit) {
                        atomicOr(A.status, kStatusWaitLimit);
                        plan[0] = -1;
                        break;
                    }
                    __nanosleep(32);
                }
                __threadfence();
            }
        }
        group_sync(bar, T);
        const int it = plan[0], k = plan[1];
        if (it < 0) break;
        const uint8_t *const res = A.res + (size_t)k * A.S;
        uint64_t *const ga = A.accs + (size_t)k * 4096;
        {
            const uint64_t pol = l2_keep_policy();
            for (int e = tid; e < 4096; e += T)
                acc[(e >> 11) * px(2048) + px(e & 2047)] = ld_keep64(ga + e, pol);
        }
        group_sync(bar, T);
        const BlockCta<B, 1> cta{g, acc, work, {g}, zeta, 0};
        const int end = min(A.S, (it + 1) * kItemSteps);
        for (int st = it * kItemSteps; st < end; st++) {
            if (!step_issued(res, st, mode)) continue;
            const uint2 *const key = A.btkey + ((size_t)st * A.Br + res[st]) * rgsw;
            block_step<B, 1, T, true>(
                cta, A, tw, itw, c, 2048, tid, bar, [&](int lb) { return key + lb * L::M; }, [](int) {});
        }
        {
            const uint64_t pol = l2_keep_policy();
            for (int e = tid; e < 4096; e += T) st_keep64(ga + e, acc[(e >> 11) * px(2048) + px(e & 2047)], pol);
        }
        __threadfence();
        group_sync(bar, T);
        if (tid == 0) atomicExch(done + k, it);
    }
}

// Residues and initial accumulators, one CTA per ciphertext.
__global__ void __launch_bounds__(kT64) br64_begin_kernel(const __grid_constant__ Br64Args A, uint8_t *res, int *done,
                                                         const ulonglong2 *__restrict__ tw,
                                                         const __grid_constant__ Ntt64Consts c)
{
    __shared__ uint64_t buf[kPoly64];
    __shared__ uint32_t bv[3];
    const size_t gid = blockIdx.x;
    if (threadIdx.x == 0) done[gid] = -1;
    br64_residues(A, gid, res + gid * (size_t)(A.n * (int)A.digitR), &bv[0], &bv[1], &bv[2], threadIdx.x, kT64);
    __syncthreads();
    br64_acc_init<true, true>(A, c, tw, gid, bv[0], bv[1], bv[2], buf, threadIdx.x, 1);
}

__global__ void __launch_bounds__(kT64) br64_end_kernel(const __grid_constant__ Br64Args A,
                                                       const ulonglong2 *__restrict__ itw,
                                                       const __grid_constant__ Ntt64Consts c)
{
    __shared__ uint64_t buf[2][kPoly64];
    br64_output<true, true>(A, c, itw, blockIdx.x, buf[0], buf[1], threadIdx.x, 1);
}

// Key words (reduced mod Q) as limbs of 27 bits.
__global__ void limb_words64_kernel(const uint64_t *__restrict__ in, uint2 *__restrict__ out, size_t n, uint64_t Q)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const uint64_t w = in[i] % Q;
        out[i] = make_uint2((uint32_t)w & ((1u << 27) - 1), (uint32_t)(w >> 27));
    }
}

}  // namespace dev

int launch_limb_words64(Context &c, const uint64_t *d_in, uint2 *d_out, size_t n, cudaStream_t st)
{
    if (!n) return FHEACC_OK;
    dev::limb_words64_kernel<<<(unsigned)std::min<size_t>((n + 255) / 256, 4096), 256, 0, st>>>(d_in, d_out, n, c.p.Q);
    c.launches++;
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? FHEACC_OK : c.cuda_fail(e, "limb words launch");
}

static int sm_count64(Context &c)
{
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, c.device);
    return v > 0 ? v : 1;
}

template <int B, int C>
static int launch_cluster(Context &c, const dev::BlockArgs &A, int max_ctas, cudaStream_t st, bool *fits)
{
    auto kern = dev::br64_cluster_kernel<B, C>;
    const size_t smem = dev::BlockLayout<B, C>::key_off(A.DG) + dev::BlockLayout<B, C>::key_bytes(A.DG);
    *fits = false;
    if (smem > 227 * 1024 || (max_ctas > 0 && max_ctas < C)) return FHEACC_OK;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return c.cuda_fail(e, "blind rotation smem attribute");
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(dev::kTB);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = C > 1 ? 1 : 0;
    size_t clusters = (size_t)sm_count64(c);
    if (C > 1) {
        int n = 0;
        cfg.gridDim = dim3(C);
        if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
            cudaGetLastError();
            return FHEACC_OK;
        }
        clusters = (size_t)n;
        if (A.count > clusters) return FHEACC_OK;   // more than one round: fewer CTAs per ciphertext
    }
    if (max_ctas > 0) clusters = std::min<size_t>(clusters, (size_t)(max_ctas / C));
    *fits = true;
    cfg.gridDim = dim3((unsigned)(std::min<size_t>(A.count, clusters) * C));
    e = cudaLaunchKernelEx(&cfg, kern, A, (const ulonglong2 *)c.d_tw64, (const ulonglong2 *)c.d_itw64, c.nc64);
    c.launches++;
    if (e == cudaSuccess) e = cudaGetLastError();
    return e == cudaSuccess ? FHEACC_OK : c.cuda_fail(e, "blind rotation launch");
}

template <int B, int W>
static int launch_items(Context &c, dev::BlockArgs A, unsigned long long *cursor, int *done, int max_ctas,
                        cudaStream_t st)
{
    auto kern = dev::br64_items_kernel<B, W>;
    const size_t smem = W * dev::BlockLayout<B, 1>::key_off(A.DG);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return c.cuda_fail(e, "blind rotation smem attribute");
    // an SM per ciphertext while there are enough: the surplus workers wait their turn
    size_t blocks = std::min<size_t>((size_t)sm_count64(c), A.count * std::max(c.tune.br_pipes, 1));
    if (max_ctas > 0) blocks = std::min<size_t>(blocks, (size_t)max_ctas);
    e = cudaMemsetAsync(cursor, 0, sizeof(*cursor), st);
    if (e != cudaSuccess) return c.cuda_fail(e, "blind rotation cursor reset");
    A.wait_limit = c.tune.debug_wait_limit >= 0 ? (unsigned)c.tune.debug_wait_limit : dev::kItemWaitLimit;
    kern<<<(unsigned)blocks, W * dev::kTP, smem, st>>>(A, cursor, done, c.d_tw64, c.d_itw64, c.nc64);
    c.launches++;
    e = cudaGetLastError();
    return e == cudaSuccess ? FHEACC_OK : c.cuda_fail(e, "blind rotation launch");
}

int launch_blind_rotate64_blocks(Context &c, const dev::Br64Args &R, int max_ctas, cudaStream_t st)
{
    dev::BlockArgs A{};
    A.btkey = c.d_btkey64_limbs; A.accs = R.accs; A.count = R.count;
    A.S = c.p.n * (int)c.p.digitR; A.DG = (int)c.p.digitG;
    A.bg_bits = c.p.BG_bits; A.Br = c.p.Br; A.flags = R.flags;
    A.c54 = c.nc64.pm_c << (c.nc64.pm_s - 10);   // 2^54 = 2^(54-b) 2^b
    A.status = c.d_status;
    A.wait_limit = c.tune.debug_wait_limit >= 0 ? (unsigned)c.tune.debug_wait_limit : dev::kKeyWaitLimit;
    // after the accumulators: claim words, done words, residues
    unsigned long long *cursor = reinterpret_cast<unsigned long long *>(R.accs + R.count * 4096);
    int *done = reinterpret_cast<int *>(cursor + kClaimWords / 2);
    uint8_t *res = reinterpret_cast<uint8_t *>(done + R.count);
    A.res = res;
    dev::br64_begin_kernel<<<(unsigned)R.count, dev::kT64, 0, st>>>(R, res, done, c.d_tw64, c.nc64);
    c.launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return c.cuda_fail(e, "blind rotation begin launch");
    // up to one ciphertext per SM the latency form, on as many CTAs per ciphertext as
    // run at once; beyond that the items form (an explicit worker count asks for it)
    bool fits = false;
    int rc = FHEACC_OK;
    if (c.tune.br_pipes == 0 && R.count <= (size_t)sm_count64(c)) {
        if (c.p.BG_bits <= 29) rc = launch_cluster<8, 8>(c, A, max_ctas, st, &fits);
        if (!rc && !fits) rc = launch_cluster<4, 4>(c, A, max_ctas, st, &fits);
        if (!rc && !fits) rc = launch_cluster<4, 2>(c, A, max_ctas, st, &fits);
        if (!rc && !fits) rc = launch_cluster<4, 1>(c, A, max_ctas, st, &fits);
    }
    if (!rc && !fits)   // digitG = 7 and 8: one worker's work area more than fills half an SM
        rc = 2 * dev::BlockLayout<4, 1>::key_off(A.DG) <= 227 * 1024 ? launch_items<4, 2>(c, A, cursor, done, max_ctas, st)
                                                                     : launch_items<4, 1>(c, A, cursor, done, max_ctas, st);
    if (rc) return rc;
    dev::br64_end_kernel<<<(unsigned)R.count, dev::kT64, 0, st>>>(R, c.d_itw64, c.nc64);
    c.launches++;
    e = cudaGetLastError();
    return e == cudaSuccess ? FHEACC_OK : c.cuda_fail(e, "blind rotation end launch");
}

}  // namespace fheacc

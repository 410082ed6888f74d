// expand.cu -- the X -> X^k automorphism, the RLWE key switch and
// expand_RLWE, for both word widths.
//
// Reference behaviour: RLWE_substitute (FHE_ACC_runtime/src/RLWE.cpp:444-462)
// with poly_substitute (RLWE.cpp:23-37), RLWE_keyswitch (RLWE.cpp:464-510),
// RLWE_rotate_freq (RLWE.cpp:411-430) and application::expand_RLWE
// (app.cpp:26-76); on the FPGA the RLWESUBS instruction (subs_module.sv +
// the NTT/MAC chain) and fpga_expand_RLWE (myfpga.cpp:1662-1790).
//
// An RLWE is an "item": of one CTA (32-bit words, and 64-bit moduli without a fold form),
// or of a cluster of CTAs or a worker (block form). The substitution is applied while the
// time-domain coefficients are read: out[e] = in[i'] when i' < N, else
// -in[i' - N], with i' = e * power^-1 mod 2N and power = N / 2^f + 1 (odd) --
// the inverse of poly_substitute's scatter out[i * power mod N] = +-in[i]. The
// key switch then decomposes sigma(a) in base 2^Bks_R_bits, transforms each
// digit and multiply-accumulates with the key rows. Of sigma(b) only the NTT is needed,
// whose words the automorphism permutes (subs_ntt_src; the moduli without a fold form
// transform it). Modes:
//   SUBS      out = RLWE_substitute(c, f)
//   KS        out = RLWE_keyswitch(c, ksk)                (f = 0 is the identity)
//   SUBS_KS   out = RLWE_keyswitch(RLWE_substitute(c, f), ksk)
//   EXPAND    r[j] <- r[j] + s, r[j + 2^f] <- (r[j] - s) * NTT(-X^(N - 2^f)),
//             s = SUBS_KS(r[j], f, subs_key[f]), for every j < 2^f (one level)
#include "block64.cuh"
#include "ctx.hpp"
#include "step32.cuh"
#include <algorithm>

namespace fheacc {
namespace dev {

enum ExpMode { kSubs = 0, kKs = 1, kSubsKs = 2, kExpand = 3 };

struct ExpArgs {
    const uint64_t *in;      // items [count][2N] (EXPAND: the r arrays)
    uint64_t *out;           // [count][2N] (EXPAND: the r arrays, in place)
    size_t count;
    size_t batches;          // EXPAND: independent r arrays, bstride words apart (else 1)
    size_t bstride;
    int mode, f, logN, L;    // L = digitKS_R
    uint32_t bits;           // Bks_R_bits
    uint32_t ipow;           // (N / 2^f + 1)^-1 mod 2N
    const uint32_t *ksk32;   // [L][2][N] u32 (narrow)
    const ulonglong2 *ksk64; // [L][2][N] Shoup pairs (wide, other moduli)
    const uint2 *ksk_limbs;  // the same as limb words (wide, block form)
    uint32_t c54, power;     // 2^54 mod Q (block form); N / 2^f + 1 (KS: 1)
    const uint64_t *rot;     // [N] NTT(-X^(N - 2^f)) (EXPAND, narrow)
    const ulonglong2 *rot64; // rot as constant pairs (mul64 in ntt64.cuh; wide)
    uint64_t Q, mu64;
};

__device__ __forceinline__ uint32_t subs_src(uint32_t e, uint32_t ipow, uint32_t N, bool &neg)
{
    const uint32_t ip = (e * ipow) & (2 * N - 1);   // 2 N a power of two: the low word is enough
    neg = ip >= N;
    return neg ? ip - N : ip;
}

// Where word e of the NTT of the substituted polynomial comes from: word j of an NTT is
// the value at psi^(2 rev(j) + 1), and p(X^power) there is p at psi^(power (2 rev(j) + 1)).
__device__ __forceinline__ uint32_t subs_ntt_src(uint32_t e, uint32_t power, int logN)
{
    const uint32_t x = ((2 * (__brev(e) >> (32 - logN)) + 1) * power) & ((2u << logN) - 1);
    return __brev(x >> 1) >> (32 - logN);
}

// ---------------------------------------------------------------- narrow
// 8 warps: warp 0 the inverse NTT of a, then warps 0..L-1 the digits of sigma(a),
// then all threads the MAC and the epilogue. Only NTT(sigma(b)) is needed, whose words
// the automorphism permutes (subs_ntt_src), so b takes no transform, nor does SUBS.
__global__ void __launch_bounds__(256) expand32_kernel(const __grid_constant__ ExpArgs A,
                                                      const __grid_constant__ Ntt32Consts c,
                                                      const uint2 *__restrict__ fwd_tw,
                                                      const uint2 *__restrict__ inv_tw, uint32_t mu32)
{
    __shared__ __align__(16) uint32_t t[2][kPadN];
    __shared__ __align__(16) uint32_t d[4][kPadN];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t Q = c.Q;
    const int L = A.L;
    const size_t per = A.mode == kExpand ? ((size_t)1 << A.f) : A.count;
    const size_t items = per * A.batches;
    for (size_t it = blockIdx.x; it < items; it += gridDim.x) {
        const size_t bo = it / per * A.bstride, jt = it % per;   // batch offset, item within the batch
        const uint64_t *in = A.in + bo + jt * 2048;
        // a to the time domain (warp 0); b, and a of SUBS, as NTTs (subs_ntt_src)
        if (warp == 0 && A.mode != kSubs) {
            uint32_t x[32];
#pragma unroll
            for (int r = 0; r < 32; r++) x[r] = (uint32_t)in[32 * lane + r];
            ntt_inv_1024(x, c, inv_tw, d[warp], lane);
#pragma unroll
            for (int r = 0; r < 32; r++) t[0][pad32(lane + 32 * r)] = x[r];
        } else if (warp >= 1) {
            for (int e = threadIdx.x - 32; e < 1024; e += blockDim.x - 32) {
                const uint32_t v = (uint32_t)in[1024 + e];
                t[1][pad32(e)] = min(v, v - Q);
                if (A.mode == kSubs) {
                    const uint32_t u = (uint32_t)in[e];
                    t[0][pad32(e)] = min(u, u - Q);
                }
            }
        }
        __syncthreads();
        if (A.mode != kSubs && warp < L) {   // the digits of sigma(a)
            const uint32_t sh = A.bits * (uint32_t)warp, mask = (1u << A.bits) - 1;
            uint32_t x[32];
#pragma unroll
            for (int r = 0; r < 32; r++) {
                bool neg;
                uint32_t v = t[0][pad32(subs_src(lane + 32 * r, A.ipow, 1024, neg))];   // ipow = 1 for KS
                if (neg && v) v = Q - v;
                x[r] = (v >> sh) & mask;
            }
            ntt_fwd_1024(x, c, fwd_tw, d[warp], lane);
#pragma unroll
            for (int r = 0; r < 32; r++) d[warp][33 * lane + r] = reduce32(x[r], mu32, Q);
        }
        __syncthreads();
        uint64_t *out = A.out + bo + jt * 2048;
        for (int k = threadIdx.x; k < 1024; k += blockDim.x) {
            uint64_t oa, ob;
            if (A.mode == kSubs) {
                const uint32_t j = subs_ntt_src((uint32_t)k, A.power, 10);
                oa = t[0][pad32(j)];
                ob = t[1][pad32(j)];
            } else {
                uint64_t sa = 0, sb = 0;
                for (int h = 0; h < L; h++) {
                    const uint64_t dv = d[h][pad32(k)];
                    sa += dv * A.ksk32[(h * 2 + 0) * 1024 + k];
                    sb += dv * A.ksk32[(h * 2 + 1) * 1024 + k];
                }
                const uint32_t ra = barrett64_lazy(sa, A.mu64, Q), rb = barrett64_lazy(sb, A.mu64, Q);
                const uint32_t ca = min(ra, ra - Q), cb = min(rb, rb - Q);
                oa = ca ? Q - ca : 0;
                const uint32_t nb = t[1][pad32(subs_ntt_src((uint32_t)k, A.power, 10))];
                ob = nb >= cb ? nb - cb : nb + Q - cb;
            }
            if (A.mode == kExpand) {
                const uint64_t ta = in[k], tb = in[1024 + k];
                const uint64_t rot = A.rot[k];
                uint64_t *hi = A.out + bo + (jt + per) * 2048;
                out[k] = (ta + oa) % Q;
                out[1024 + k] = (tb + ob) % Q;
                hi[k] = ((ta + Q - oa) % Q) * rot % Q;
                hi[1024 + k] = ((tb + Q - ob) % Q) * rot % Q;
            } else {
                out[k] = oa;
                out[1024 + k] = ob;
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------- wide
// Word e = j + 128 k of the substituted polynomial (subs_src) for
// ntt64_fwd_2048_load, or its digit (v >> sh) & mask (mask = 0: the word).
struct LoadSubs64 {
    const uint64_t *t;
    uint64_t Q;
    uint32_t ipow, sh, mask;
    __device__ __forceinline__ uint64_t operator()(int j, int k) const
    {
        bool neg;
        const uint32_t s = subs_src((uint32_t)(j + 128 * k), ipow, 2048, neg);
        uint64_t v = t[px(s)];
        if (neg && v) v = Q - v;
        return mask ? (uint64_t)((uint32_t)(v >> sh) & mask) : v;
    }
};

// 256 threads in two 128-thread groups; group g transforms poly g.
__global__ void __launch_bounds__(256, 2) expand64_kernel(const __grid_constant__ ExpArgs A,
                                                      const ulonglong2 *__restrict__ tw,
                                                      const ulonglong2 *__restrict__ itw,
                                                      const __grid_constant__ Ntt64Consts c)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t(*t)[kPoly64] = reinterpret_cast<uint64_t(*)[kPoly64]>(smem_raw);   // [2], layout px
    uint64_t(*buf)[kPoly64] = t + 2;                                            // [2]
    const int tid = threadIdx.x, grp = tid >> 7, gtid = tid & 127;
    const uint64_t Q = c.Q;
    const int L = A.L;
    const size_t per = A.mode == kExpand ? ((size_t)1 << A.f) : A.count;
    const size_t items = per * A.batches;
    for (size_t it = blockIdx.x; it < items; it += gridDim.x) {
        const size_t bo = it / per * A.bstride, jt = it % per;   // batch offset, item within the batch
        const uint64_t *in = A.in + bo + jt * 4096;
        for (int e = gtid; e < 2048; e += 128) t[grp][px(e)] = in[grp * 2048 + e];
        group_sync(1 + grp, 128);
        ntt64_inv_2048<false, 128, true>(t[grp], itw, c, gtid, 1 + grp);
        __syncthreads();
        // transforms: L digits of sigma(a) and sigma(b) (SUBS: sigma(a), sigma(b)),
        // two at a time; MAC after each pair
        const int nt = A.mode == kSubs ? 2 : L + 1;
        uint64_t sa[8], sb[8], fb[8];
#pragma unroll
        for (int i = 0; i < 8; i++) sa[i] = sb[i] = fb[i] = 0;
        for (int base = 0; base < nt; base += 2) {
            const int tr = base + grp;   // transform index of this group
            if (tr < nt) {
                const int poly = A.mode == kSubs ? tr : (tr == L ? 1 : 0);
                // A.ipow = 1 is the identity (kKs)
                if (A.mode != kSubs && tr < L) {
                    ntt64_fwd_2048_load<false, 128, true>(
                        buf[grp], LoadSubs64{t[poly], Q, A.ipow, A.bits * (uint32_t)tr, (1u << A.bits) - 1}, tw, c, gtid,
                        1 + grp);
                } else {
                    ntt64_fwd_2048_load<false, 128, true>(buf[grp], LoadSubs64{t[poly], Q, A.ipow, 0, 0}, tw, c,
                                                               gtid, 1 + grp);
                }
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int k = tid + 256 * i;
#pragma unroll
                for (int g2 = 0; g2 < 2; g2++) {
                    const int tr = base + g2;
                    if (tr >= nt) continue;
                    const uint64_t dv = buf[g2][px(k)];
                    if (A.mode == kSubs || tr == L) {
                        const uint64_t v = reduce64<false>(dv, c);
                        if (A.mode == kSubs && tr == 0) sa[i] = v;
                        else fb[i] = v;
                    } else {
                        const ulonglong2 ka = __ldg(A.ksk64 + (size_t)(tr * 2 + 0) * 2048 + k);
                        const ulonglong2 kb = __ldg(A.ksk64 + (size_t)(tr * 2 + 1) * 2048 + k);
                        sa[i] += mul64<false>(dv, ka, c);
                        sb[i] += mul64<false>(dv, kb, c);
                    }
                }
            }
            __syncthreads();
        }
        uint64_t *out = A.out + bo + jt * 4096;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int k = tid + 256 * i;
            uint64_t oa, ob;
            if (A.mode == kSubs) {
                oa = sa[i] >= Q ? sa[i] - Q : sa[i];
                ob = fb[i] >= Q ? fb[i] - Q : fb[i];
            } else {
                uint64_t ra = reduce64<false>(sa[i], c), rb = reduce64<false>(sb[i], c);
                ra = ra >= Q ? ra - Q : ra;
                rb = rb >= Q ? rb - Q : rb;
                const uint64_t nb = fb[i] >= Q ? fb[i] - Q : fb[i];
                oa = ra ? Q - ra : 0;
                ob = nb >= rb ? nb - rb : nb + Q - rb;
            }
            if (A.mode == kExpand) {
                const uint64_t ta = in[k], tb = in[2048 + k];
                const ulonglong2 rot = __ldg(A.rot64 + k);
                uint64_t *hi = A.out + bo + (jt + per) * 4096;
                const uint64_t s1 = ta + oa, s2 = tb + ob;
                out[k] = s1 >= Q ? s1 - Q : s1;
                out[2048 + k] = s2 >= Q ? s2 - Q : s2;
                const uint64_t d1 = ta >= oa ? ta - oa : ta + Q - oa, d2 = tb >= ob ? tb - ob : tb + Q - ob;
                const uint64_t h1 = mul64<false>(d1, rot, c), h2 = mul64<false>(d2, rot, c);
                hi[k] = h1 >= Q ? h1 - Q : h1;
                hi[2048 + k] = h2 >= Q ? h2 - Q : h2;
            } else {
                out[k] = oa;
                out[2048 + k] = ob;
            }
        }
        __syncthreads();
    }
}

// An expand_RLWE level of few RLWEs (64-bit words), split over the transform
// pairs for latency: CTA (item, pair p) takes the item's inverse NTTs, transforms
// 2p and 2p + 1 of the L + 1 (the key-switch digits of sigma(a), transform L
// sigma(b)) and their share of the key multiply-accumulate, written to
// part[item][p] as [sa | sb | fb][2048], each word < 4Q. expand64_combine_kernel
// adds the shares and applies the level's epilogue. One RLWE's transforms then
// take two rounds instead of 1 + ceil((L + 1) / 2).
__global__ void __launch_bounds__(256) expand64_split_kernel(const __grid_constant__ ExpArgs A,
                                                            uint64_t *__restrict__ part, int P,
                                                            const ulonglong2 *__restrict__ tw,
                                                            const ulonglong2 *__restrict__ itw,
                                                            const __grid_constant__ Ntt64Consts c)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t(*t)[kPoly64] = reinterpret_cast<uint64_t(*)[kPoly64]>(smem_raw);   // [2], layout px
    uint64_t(*buf)[kPoly64] = t + 2;                                            // [2]
    const int tid = threadIdx.x, grp = tid >> 7, gtid = tid & 127;
    const uint64_t Q = c.Q;
    const int L = A.L, nt = L + 1;
    const size_t per = (size_t)1 << A.f;
    const size_t it = blockIdx.x / (unsigned)P;
    const int p = (int)(blockIdx.x - it * (unsigned)P);
    const size_t bo = it / per * A.bstride, jt = it % per;
    const uint64_t *in = A.in + bo + jt * 4096;
    for (int e = gtid; e < 2048; e += 128) t[grp][px(e)] = in[grp * 2048 + e];
    group_sync(1 + grp, 128);
    ntt64_inv_2048<false, 128, true>(t[grp], itw, c, gtid, 1 + grp);
    __syncthreads();
    const int tr = 2 * p + grp;
    if (tr < nt) {
        if (tr < L)
            ntt64_fwd_2048_load<false, 128, true>(
                buf[grp], LoadSubs64{t[0], Q, A.ipow, A.bits * (uint32_t)tr, (1u << A.bits) - 1}, tw, c, gtid, 1 + grp);
        else
            ntt64_fwd_2048_load<false, 128, true>(buf[grp], LoadSubs64{t[1], Q, A.ipow, 0, 0}, tw, c, gtid,
                                                       1 + grp);
    }
    __syncthreads();
    uint64_t *o = part + (it * (unsigned)P + (unsigned)p) * 3 * 2048;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int k = tid + 256 * i;
        uint64_t sa = 0, sb = 0, fb = 0;
#pragma unroll
        for (int g2 = 0; g2 < 2; g2++) {
            const int tq = 2 * p + g2;
            if (tq >= nt) continue;
            const uint64_t dv = buf[g2][px(k)];
            if (tq == L) {
                fb = reduce64<false>(dv, c);
            } else {
                const ulonglong2 ka = __ldg(A.ksk64 + (size_t)(tq * 2 + 0) * 2048 + k);
                const ulonglong2 kb = __ldg(A.ksk64 + (size_t)(tq * 2 + 1) * 2048 + k);
                sa += mul64<false>(dv, ka, c);
                sb += mul64<false>(dv, kb, c);
            }
        }
        o[k] = sa;
        o[2048 + k] = sb;
        o[4096 + k] = fb;
    }
}

// The shares of expand64_split_kernel added (P of them, < 4PQ < 2^64, checked
// by the launcher) and the expand level's epilogue, one thread per item word:
// s = (-sa, sigma(b) - sb), r[j] <- r[j] + s, r[j + 2^f] <- (r[j] - s) * rot.
__global__ void expand64_combine_kernel(const __grid_constant__ ExpArgs A, const uint64_t *__restrict__ part, int P,
                                        size_t items, const __grid_constant__ Ntt64Consts c)
{
    const uint64_t Q = c.Q;
    const size_t per = (size_t)1 << A.f;
    for (size_t w = (size_t)blockIdx.x * blockDim.x + threadIdx.x; w < items * 2048;
         w += (size_t)gridDim.x * blockDim.x) {
        const size_t it = w / 2048;
        const int k = (int)(w - it * 2048);
        const size_t bo = it / per * A.bstride, jt = it % per;
        const uint64_t *pp = part + it * (unsigned)P * 3 * 2048 + k;
        uint64_t sa = 0, sb = 0, fb = 0;
        for (int p = 0; p < P; p++) {
            sa += pp[(size_t)(p * 3 + 0) * 2048];
            sb += pp[(size_t)(p * 3 + 1) * 2048];
            fb += pp[(size_t)(p * 3 + 2) * 2048];
        }
        uint64_t ra = reduce64<false>(sa, c), rb = reduce64<false>(sb, c);
        ra = ra >= Q ? ra - Q : ra;
        rb = rb >= Q ? rb - Q : rb;
        const uint64_t nb = fb >= Q ? fb - Q : fb;
        const uint64_t oa = ra ? Q - ra : 0;
        const uint64_t ob = nb >= rb ? nb - rb : nb + Q - rb;
        const uint64_t *in = A.in + bo + jt * 4096;
        uint64_t *out = A.out + bo + jt * 4096;
        uint64_t *hi = A.out + bo + (jt + per) * 4096;
        const uint64_t ta = in[k], tb = in[2048 + k];
        const ulonglong2 rot = __ldg(A.rot64 + k);
        const uint64_t s1 = ta + oa, s2 = tb + ob;
        out[k] = s1 >= Q ? s1 - Q : s1;
        out[2048 + k] = s2 >= Q ? s2 - Q : s2;
        const uint64_t d1 = ta >= oa ? ta - oa : ta + Q - oa, d2 = tb >= ob ? tb - ob : tb + Q - ob;
        const uint64_t h1 = mul64<false>(d1, rot, c), h2 = mul64<false>(d2, rot, c);
        hi[k] = h1 >= Q ? h1 - Q : h1;
        hi[2048 + k] = h2 >= Q ? h2 - Q : h2;
    }
}

// ---- Block form (moduli Q = 2^b - c; block64.cuh), every mode. The automorphism permutes
// the words of an NTT (subs_ntt_src), so sigma(b), of which only the NTT is needed, takes no
// transform (nor does SUBS), and a step is one inverse NTT and the L digits' instead of
// two and L + 1. A cluster of C CTAs per RLWE up to one RLWE per SM (a level of few RLWEs
// is a chain of transforms: 16 us, 36 split over transform pairs with a second launch for
// their sum), else three workers of 192 threads per CTA, a warp per digit. The large
// levels are bound by the multiply pipe.

// Shared memory: as BlockLayout with one poly to transform; g: [GBUF][2][2048] (a's
// coefficients; b as it came in), acc: sigma(a) afterwards (C = 1).
template <int B, int C>
struct ExpandLayout {
    using L = BlockLayout<B, C>;
    static constexpr size_t work_off = L::acc_off + (size_t)(C == 1 ? px(2048) : L::NB * L::ME) * 8;
    static size_t __host__ __device__ bytes(int nd) { return work_off + (size_t)(nd > L::NB ? nd : L::NB) * L::ME * 8; }
};

// RLWE `it` on the CTA's blocks by T threads.
template <int B, int C, int T>
__device__ __forceinline__ void expand_item(const BlockCta<B, C> &s, const ExpArgs &A, size_t it,
                                            const ulonglong2 *__restrict__ tw, const ulonglong2 *__restrict__ itw,
                                            const Ntt64Consts &c, int tid, int bar)
{
    using L = BlockLayout<B, C>;
    constexpr int M = L::M, NB = L::NB, ME = L::ME, NW = NB * M;
    constexpr int GS = M == 512 && T == kTB ? 64 : 32, NG = T / GS;
    const int gi = tid / GS, gt = tid - gi * GS, first = s.rank * NW;
    const size_t per = A.mode == kExpand ? ((size_t)1 << A.f) : A.count;
    const size_t bo = it / per * A.bstride, jt = it % per;   // batch offset, item within the batch
    const uint64_t *in = A.in + bo + jt * 4096;
    uint64_t *out = A.out + bo + jt * 4096;
    const uint64_t Q = c.Q;
    uint64_t *const gb = s.g + 2048;   // b
    for (int e = tid; e < 2048; e += T) gb[e] = canonical64<true>(in[2048 + e], c);
    if (A.mode == kSubs) {
        for (int e = tid; e < 2048; e += T) s.g[e] = canonical64<true>(in[e], c);
        if (C > 1) cg::this_cluster().sync();   // out may be in
        else group_sync(bar, T);
        for (int u = tid; u < 2 * NW; u += T) {
            const int p = u / NW, e = first + u - p * NW;
            out[p * 2048 + e] = s.g[p * 2048 + subs_ntt_src((uint32_t)e, A.power, 11)];
        }
        group_sync(bar, T);
        return;
    }
    for (int e = tid; e < NW; e += T) s.acc[px(e)] = in[first + e];
    group_sync(bar, T);
    block_to_time<B, C, T, 1>(s, itw, c, tid, bar);
    // sigma(a) once for all digits, into the accumulator's words (C = 1, free by now) or
    // the other g buffer (one RLWE per cluster: free)
    uint64_t *const sg = C == 1 ? s.acc : s.g + 4096;
    for (int e = tid; e < 2048; e += T) {
        bool neg;
        const uint64_t v = s.g[subs_src((uint32_t)e, A.ipow, 2048, neg)];
        sg[e] = neg && v ? Q - v : v;
    }
    group_sync(bar, T);
    const int nd = A.L;
    const uint32_t mask = (1u << A.bits) - 1;
    for (int lb = 0; lb < NB; lb++) {
        const int blk = s.rank * NB + lb;
        for (int dd = gi; dd < nd; dd += NG) {
            uint64_t *const d = s.work + dd * ME;
            const uint32_t sh = A.bits * (uint32_t)dd;
            uint64_t z[B - 1];
#pragma unroll
            for (int i = 0; i < B - 1; i++) z[i] = s.zeta[lb][i];
            blk_fwd_first<B, GS>(d, [&](int j, int k) {
                const uint64_t *b = sg + j + 64 * k;
                return digit_residue<B>(z, c, [&](int i) { return (uint32_t)(b[i * M] >> sh) & mask; });
            }, blk, gt, tw, c);
            group_sync64<GS>(gi);
            blk_fwd_pass<M, 3, GS>(d, blk, 32, gt, tw, c);
            group_sync64<GS>(gi);
            blk_fwd_pass<M, 3, GS>(d, blk, 4, gt, tw, c);
        }
        group_sync(bar, T);
        for (int k = tid; k < M; k += T) {
            const int e = blk * M + k;
            uint64_t sa[3] = {0, 0, 0}, sb[3] = {0, 0, 0};
            const uint2 *kk = A.ksk_limbs + e;
#pragma unroll 3
            for (int h = 0; h < nd; h++, kk += 4096) {
                const uint64_t v = s.work[h * ME + px(k)];
                const uint32_t x0 = (uint32_t)v & ((1u << 27) - 1), x1 = (uint32_t)(v >> 27);
                mac27(sa, x0, x1, __ldcg(kk));
                mac27(sb, x0, x1, __ldcg(kk + 2048));
            }
            uint64_t ra = mac27_reduce(sa, A.c54, c), rb = mac27_reduce(sb, A.c54, c);
            ra = ra >= Q ? ra - Q : ra;
            rb = rb >= Q ? rb - Q : rb;
            const uint64_t nb = gb[subs_ntt_src((uint32_t)e, A.power, 11)];
            const uint64_t oa = ra ? Q - ra : 0;
            const uint64_t ob = nb >= rb ? nb - rb : nb + Q - rb;
            if (A.mode == kExpand) {
                const uint64_t ta = in[e], tb = gb[e];
                const ulonglong2 rot = __ldg(A.rot64 + e);
                uint64_t *hi = A.out + bo + (jt + per) * 4096;
                const uint64_t s1 = ta + oa, s2 = tb + ob;
                out[e] = s1 >= Q ? s1 - Q : s1;
                out[2048 + e] = s2 >= Q ? s2 - Q : s2;
                const uint64_t d1 = ta >= oa ? ta - oa : ta + Q - oa, d2 = tb >= ob ? tb - ob : tb + Q - ob;
                const uint64_t h1 = mul64<true>(d1, rot, c), h2 = mul64<true>(d2, rot, c);
                hi[e] = h1 >= Q ? h1 - Q : h1;
                hi[2048 + e] = h2 >= Q ? h2 - Q : h2;
            } else {
                out[e] = oa;
                out[2048 + e] = ob;
            }
        }
        group_sync(bar, T);
    }
}

template <int B, int C>
__global__ void __launch_bounds__(kTB, 1) expand64_cluster_kernel(const __grid_constant__ ExpArgs A, size_t items,
                                                                 const ulonglong2 *__restrict__ tw,
                                                                 const ulonglong2 *__restrict__ itw,
                                                                 const __grid_constant__ Ntt64Consts c)
{
    using L = BlockLayout<B, C>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint64_t zeta[L::NB][B - 1];
    uint64_t *const g = reinterpret_cast<uint64_t *>(smem_raw + L::g_off);
    const int rank = C > 1 ? (int)(blockIdx.x % C) : 0;
    BlockCta<B, C> cta{g, reinterpret_cast<uint64_t *>(smem_raw + L::acc_off),
                       reinterpret_cast<uint64_t *>(smem_raw + ExpandLayout<B, C>::work_off), {}, zeta, rank};
    cta.peer[0] = g;
    if (C > 1) {
        cg::cluster_group cl = cg::this_cluster();
#pragma unroll
        for (int r = 0; r < C; r++) cta.peer[r] = cl.map_shared_rank(g, r);
    }
    block_zeta<B, L::NB>(zeta, rank * L::NB, tw, c);
    if (C > 1) cg::this_cluster().sync();
    else __syncthreads();
    // one RLWE per cluster (the launcher's rule)
    if (blockIdx.x / C < items)
        expand_item<B, C, kTB>(cta, A, blockIdx.x / C, tw, itw, c, threadIdx.x, 0);
    if (C > 1) cg::this_cluster().sync();
}

constexpr int kTE = 192;   // threads of an expand worker

template <int B, int W>
__global__ void __launch_bounds__(W * kTE, 1) expand64_workers_kernel(const __grid_constant__ ExpArgs A, size_t items,
                                                                     int worker_bytes,
                                                                     const ulonglong2 *__restrict__ tw,
                                                                     const ulonglong2 *__restrict__ itw,
                                                                     const __grid_constant__ Ntt64Consts c)
{
    using L = BlockLayout<B, 1>;
    extern __shared__ __align__(128) unsigned char smem_all[];
    __shared__ uint64_t zeta[B][B - 1];
    const int wk = threadIdx.x / kTE, tid = threadIdx.x - wk * kTE;
    unsigned char *const smem_raw = smem_all + wk * worker_bytes;
    uint64_t *const g = reinterpret_cast<uint64_t *>(smem_raw + L::g_off);
    block_zeta<B, B>(zeta, 0, tw, c);
    __syncthreads();
    const BlockCta<B, 1> cta{g, reinterpret_cast<uint64_t *>(smem_raw + L::acc_off),
                             reinterpret_cast<uint64_t *>(smem_raw + ExpandLayout<B, 1>::work_off), {g}, zeta, 0};
    for (size_t it = (size_t)wk * gridDim.x + blockIdx.x; it < items; it += (size_t)gridDim.x * W)
        expand_item<B, 1, kTE>(cta, A, it, tw, itw, c, tid, 1 + wk);
}

__global__ void to_u32_kernel(const uint64_t *__restrict__ in, uint32_t *__restrict__ out, size_t n, uint64_t Q)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = (uint32_t)(in[i] % Q);
}

}  // namespace dev

static int sms(Context &c)
{
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, c.device);
    return v > 0 ? v : 1;
}

static uint32_t inv_power(int N, int f)
{
    const uint64_t m = 2ULL * (uint64_t)N, p = (uint64_t)(N >> f) + 1;
    for (uint64_t x = 1; x < m; x += 2)
        if ((x * p) % m == 1) return (uint32_t)x;
    return 1;
}

template <int B, int C>
static int launch_expand_cluster(Context &c, const dev::ExpArgs &A, size_t items, cudaStream_t st, bool *fits)
{
    auto kern = dev::expand64_cluster_kernel<B, C>;
    const size_t smem = dev::ExpandLayout<B, C>::bytes(A.L);
    *fits = false;
    if (smem > kMaxDynamicSmem || items * C > (size_t)sms(c)) return FHEACC_OK;
    cudaError_t e = allow_dynamic_smem(kern);
    if (e != cudaSuccess) return c.cuda_fail(e, "expand smem attribute");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(items * C));
    cfg.blockDim = dim3(dev::kTB);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = C > 1 ? 1 : 0;
    if (C > 1) {
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
            cudaGetLastError();
            return FHEACC_OK;
        }
        if (items > (size_t)n) return FHEACC_OK;   // more than one round: fewer CTAs per RLWE
    }
    *fits = true;
    e = cudaLaunchKernelEx(&cfg, kern, A, items, (const ulonglong2 *)c.d_tw64, (const ulonglong2 *)c.d_itw64, c.nc64);
    c.launches++;
    if (e == cudaSuccess) e = cudaGetLastError();
    return e == cudaSuccess ? FHEACC_OK : c.cuda_fail(e, "expand launch");
}

template <int W>
static int launch_expand_workers(Context &c, const dev::ExpArgs &A, size_t items, cudaStream_t st)
{
    auto kern = dev::expand64_workers_kernel<4, W>;
    const int bytes = (int)dev::ExpandLayout<4, 1>::bytes(A.L);
    cudaError_t e = allow_dynamic_smem(kern);
    if (e != cudaSuccess) return c.cuda_fail(e, "expand smem attribute");
    kern<<<(unsigned)std::min<size_t>(items, (size_t)sms(c)), W * dev::kTE, W * bytes, st>>>(
        A, items, bytes, c.d_tw64, c.d_itw64, c.nc64);
    c.launches++;
    e = cudaGetLastError();
    return e == cudaSuccess ? FHEACC_OK : c.cuda_fail(e, "expand launch");
}

// The block form of a launch of `items` RLWEs.
static int launch_expand_blocks(Context &c, const dev::ExpArgs &A, size_t items, cudaStream_t st)
{
    bool fits = false;
    int rc = FHEACC_OK;
    if (A.bits <= 29) rc = launch_expand_cluster<8, 8>(c, A, items, st, &fits);
    if (!rc && !fits) rc = launch_expand_cluster<4, 4>(c, A, items, st, &fits);
    if (!rc && !fits) rc = launch_expand_cluster<4, 2>(c, A, items, st, &fits);
    if (!rc && !fits) rc = launch_expand_cluster<4, 1>(c, A, items, st, &fits);
    if (rc || fits) return rc;
    return 3 * dev::ExpandLayout<4, 1>::bytes(A.L) <= kMaxDynamicSmem ? launch_expand_workers<3>(c, A, items, st)
                                                                     : launch_expand_workers<2>(c, A, items, st);
}

// ksk: narrow, u32 [L][2][N] device words; wide, limb words (block form,
// products64_apply) or Shoup pairs.
int launch_expand(Context &c, int mode, const uint64_t *d_in, uint64_t *d_out, size_t count, int f,
                  const void *ksk, cudaStream_t st, size_t batches, size_t bstride)
{
    const int logN = c.wide ? 11 : 10;
    if (f < 0 || f >= logN) return c.fail(FHEACC_EINVAL, "substitution factor out of range");
    dev::ExpArgs A{};
    A.in = d_in; A.out = d_out; A.count = count; A.mode = mode; A.f = f; A.logN = logN;
    A.batches = mode == dev::kExpand ? batches : 1;
    A.bstride = bstride;
    A.L = (int)c.p.digitKS_R; A.bits = c.p.Bks_R_bits; A.ipow = inv_power(c.p.N, mode == dev::kKs ? 0 : f);
    A.Q = c.p.Q; A.mu64 = c.dp.mu64;
    if (mode == dev::kKs) A.ipow = 1;
    A.power = mode == dev::kKs ? 1u : (uint32_t)(c.p.N >> f) + 1u;
    if (mode == dev::kExpand) {
        if (c.wide) A.rot64 = c.d_rot64 + (size_t)f * c.p.N;
        else A.rot = c.d_rot + (size_t)f * c.p.N;
    }
    const size_t items = (mode == dev::kExpand ? ((size_t)1 << f) : count) * A.batches;
    if (!items) return FHEACC_OK;
    size_t blocks = std::min<size_t>(items, (size_t)sms(c) * 4);
    cudaError_t e;
    if (c.wide) {
        if (A.L > 8) return c.fail(FHEACC_EINVAL, "digitKS_R too large");
        if (products64_apply(c)) {
            A.ksk_limbs = (const uint2 *)ksk;
            A.c54 = limb_c54(c);
            return launch_expand_blocks(c, A, items, st);
        }
        A.ksk64 = (const ulonglong2 *)ksk;
        const size_t smem = 4 * dev::kPoly64 * sizeof(uint64_t);
        // an expand level of at most two CTAs per SM of (item, transform pair)
        // splits each item over its transform pairs, for latency
        const int P = (A.L + 2) / 2;
        if (mode == dev::kExpand && items * P <= (size_t)sms(c) * 2 && (uint64_t)4 * P < UINT64_MAX / c.p.Q) {
            const size_t words = items * P * 3 * 2048;
            int rc = ensure_scratch(c, c.expand, words * sizeof(uint64_t));
            if (rc) return rc;
            uint64_t *part = (uint64_t *)c.expand.ptr;
            auto split = dev::expand64_split_kernel;
            cudaFuncSetAttribute(split, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            split<<<(unsigned)(items * P), 256, smem, st>>>(A, part, P, c.d_tw64, c.d_itw64, c.nc64);
            c.launches++;
            e = cudaGetLastError();
            if (e != cudaSuccess) return c.cuda_fail(e, "expand split launch");
            const unsigned cb = (unsigned)std::min<size_t>((items * 2048 + 255) / 256, (size_t)sms(c) * 4);
            auto combine = dev::expand64_combine_kernel;
            combine<<<cb, 256, 0, st>>>(A, part, P, items, c.nc64);
            c.launches++;
            e = cudaGetLastError();
            return e == cudaSuccess ? FHEACC_OK : c.cuda_fail(e, "expand combine launch");
        }
        auto kern = dev::expand64_kernel;
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        kern<<<(unsigned)blocks, 256, smem, st>>>(A, c.d_tw64, c.d_itw64, c.nc64);
        c.launches++;
    } else {
        if (A.L > 4) return c.fail(FHEACC_EINVAL, "digitKS_R too large for the 32-bit path");
        A.ksk32 = (const uint32_t *)ksk;
        dev::expand32_kernel<<<(unsigned)blocks, 256, 0, st>>>(A, c.nc, c.d_fwd_tw, c.d_inv_tw,
                                                              (uint32_t)((1ULL << 32) / c.p.Q));
        c.launches++;
    }
    e = cudaGetLastError();
    return e == cudaSuccess ? FHEACC_OK : c.cuda_fail(e, "expand launch");
}

int launch_to_u32(Context &c, const uint64_t *d_in, uint32_t *d_out, size_t n, cudaStream_t st)
{
    if (!n) return FHEACC_OK;
    unsigned blocks = (unsigned)std::min<size_t>((n + 255) / 256, (size_t)sms(c) * 32);
    dev::to_u32_kernel<<<blocks, 256, 0, st>>>(d_in, d_out, n, c.p.Q);
    c.launches++;
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? FHEACC_OK : c.cuda_fail(e, "convert launch");
}

}  // namespace fheacc

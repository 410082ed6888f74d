// block32.cuh -- latency form of the 32-bit blind rotation: one ciphertext per
// cluster of C CTAs (included by blind_rotate32.cu, whose prologue, epilogue and
// arithmetic it shares: outputs are identical word for word).
//
// With a gate or two per SM the pipelines have nothing to overlap: a lone
// ciphertext's steps are a serial chain, and a transform on one warp takes longer
// than all of a step's multiplications spread over the SM. X^1024 + 1 splits into
// four factors X^256 - zeta: the 256-word blocks of the bit-reversed NTTs depend on
// the polynomial only through its residue mod X^256 - zeta, so every transform is cut
// into four 256-word transforms of one warp each (8 words a lane), and a CTA of the
// cluster owns 4 / C blocks of the accumulator, the digit NTTs and the key rows:
//   1. 2 * 4 / C warps: the inverse stages t = 1 .. 128 of a block of the accumulator
//      (closed in the block), written to every CTA's shared memory; one cluster
//      barrier per step;
//   2. 512 threads: the stages t = 256, 512 of one tuple (x_j, x_{j+256}, ..) in
//      registers, the canonical coefficients' digits and the first two forward stages
//      of each digit, of which the CTA keeps its blocks' words;
//   3. a warp per digit and block: forward stages t = 128 .. 1;
//   4. multiply-accumulate of the CTA's words, keys from shared memory (copied
//      a step ahead with cp.async: on one CTA by the warps that have no part in 1, on more
//      by those that have none in 3).
// One GB300, per step: 2.0 us on 4 CTAs, 2.5 on 2, 3.4 on one; a CTA of 8 warps with one
// transform each took 3.8 (one gate) to 4.3 (152). On 4 CTAs a step is 4160 cycles: 830
// for 1 (two warps, a chain of eight stages), 685 for the cluster barrier, 865 for 2
// (every CTA does the last inverse stages of all words), 955 for 3 and 440 for 4.
// Three CTA barriers and one cluster barrier per step; the transforms' own exchanges
// stay inside a warp. Residues, accumulator, twiddles and keys live in shared memory
// for the whole bootstrap.
#pragma once

namespace fheacc {
namespace dev {

constexpr int kB32 = 256, kB32E = 256 + 32;   // words of a block, with 4 words of padding after every 32

// Padded position of word e of a block: the passes' accesses (32 consecutive words;
// words grp * 32 + j + 4 k for j < 4; four consecutive words) fall on distinct banks.
__device__ __forceinline__ constexpr int p4(int e) { return e + ((e >> 5) << 2); }

template <int DG, int C>
struct Block32Layout {
    static constexpr int NB = 4 / C, ND = 2 * (DG - 1);
    static constexpr int T = C == 1 ? 768 : 512;   // threads: 24 digit blocks (digitG = 4), or the 512 tuples
    static constexpr size_t g_off = 0;                                             // [C > 1 ? 2 : 1][2][1024]
    static constexpr size_t acc_off = (C > 1 ? 2 : 1) * 2 * kN32 * 4;              // [2 buffers][2][NB][kB32E]
    static constexpr size_t d_off = acc_off + (size_t)2 * 2 * NB * kB32E * 4;      // [ND][NB][kB32E], or [2][NB][kB32E]
    static constexpr size_t key_off = d_off + (size_t)ND * NB * kB32E * 4;         // [2][DG * 4][NB * 256]
    static constexpr size_t key_words = (size_t)DG * 4 * NB * kB32;
    static constexpr size_t tw_off = key_off + 2 * key_words * 4;                  // [fwd, inv][1024] (w, w')
    static constexpr size_t res_off = tw_off + 2 * kN32 * sizeof(uint2);
    static size_t bytes(size_t steps) { return res_off + (steps + 15) / 16 * 16; }
};

__device__ __forceinline__ void cp_async16_32(void *smem, const void *gmem)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}

// E = 1, 2 or 4 consecutive words in one shared-memory access.
template <int E>
__device__ __forceinline__ void load_words(uint32_t (&v)[E], const uint32_t *p)
{
    if constexpr (E == 4) {
        const uint4 x = *reinterpret_cast<const uint4 *>(p);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    } else if constexpr (E == 2) {
        const uint2 x = *reinterpret_cast<const uint2 *>(p);
        v[0] = x.x; v[1] = x.y;
    } else {
        v[0] = *p;
    }
}
template <int E>
__device__ __forceinline__ void store_words(uint32_t *p, const uint32_t (&v)[E])
{
    if constexpr (E == 4) *reinterpret_cast<uint4 *>(p) = make_uint4(v[0], v[1], v[2], v[3]);
    else if constexpr (E == 2) *reinterpret_cast<uint2 *>(p) = make_uint2(v[0], v[1]);
    else *p = v[0];
}

// Forward stages t = 128 .. 1 of block b (of four) at d by one warp.
__device__ __forceinline__ void block32_fwd(uint32_t *d, int b, int lane, const Ntt32Consts &c, const uint2 *ftw)
{
    const uint32_t Q = c.Q, twoQ = c.twoQ;
    {
        uint32_t x[8];
#pragma unroll
        for (int k = 0; k < 8; k++) x[k] = d[lane + 36 * k];
#pragma unroll
        for (int st = 0; st < 3; st++)
#pragma unroll
            for (int k = 0; k < 8; k++)
                if (!(k & (4 >> st))) {
                    const int i = (4 << st) + (b << st) + (k >> (3 - st));
                    ct_bfly(x[k], x[k + (4 >> st)], c.fw[i], c.fws[i], Q, twoQ);
                }
#pragma unroll
        for (int k = 0; k < 8; k++) d[lane + 36 * k] = x[k];
    }
    __syncwarp();
    {
        const int grp = lane >> 2, G = 8 * b + grp;
        uint32_t *const p = d + grp * 36 + (lane & 3);
        uint32_t x[8];
#pragma unroll
        for (int k = 0; k < 8; k++) x[k] = p[4 * k];
        const uint2 w0 = ftw[32 + G];
        const uint4 w1 = *reinterpret_cast<const uint4 *>(ftw + 64 + 2 * G);
        const uint4 w2 = *reinterpret_cast<const uint4 *>(ftw + 128 + 4 * G);
        const uint4 w3 = *reinterpret_cast<const uint4 *>(ftw + 130 + 4 * G);
#pragma unroll
        for (int k = 0; k < 4; k++) ct_bfly(x[k], x[k + 4], w0.x, w0.y, Q, twoQ);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            ct_bfly(x[k], x[k + 2], w1.x, w1.y, Q, twoQ);
            ct_bfly(x[k + 4], x[k + 6], w1.z, w1.w, Q, twoQ);
        }
        ct_bfly(x[0], x[1], w2.x, w2.y, Q, twoQ);
        ct_bfly(x[2], x[3], w2.z, w2.w, Q, twoQ);
        ct_bfly(x[4], x[5], w3.x, w3.y, Q, twoQ);
        ct_bfly(x[6], x[7], w3.z, w3.w, Q, twoQ);
#pragma unroll
        for (int k = 0; k < 8; k++) p[4 * k] = x[k];
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int q = lane + 32 * i, P = 64 * b + q;
        uint4 *const p = reinterpret_cast<uint4 *>(d + p4(4 * q));
        uint4 v = *p;
        const uint2 w0 = ftw[256 + P];
        const uint4 w1 = *reinterpret_cast<const uint4 *>(ftw + 512 + 2 * P);
        ct_bfly(v.x, v.z, w0.x, w0.y, Q, twoQ);
        ct_bfly(v.y, v.w, w0.x, w0.y, Q, twoQ);
        ct_bfly(v.x, v.y, w1.x, w1.y, Q, twoQ);
        ct_bfly(v.z, v.w, w1.z, w1.w, Q, twoQ);
        *p = v;
    }
}

// Inverse stages t = 1 .. 128 of block b at src (values < 2Q) by one warp; w: scratch
// of kB32E words; out(k, x): word lane + 32 k of the block, < 2Q.
template <class Out>
__device__ __forceinline__ void block32_inv(const uint32_t *src, uint32_t *w, int b, int lane, const Ntt32Consts &c,
                                            const uint2 *itw, Out out)
{
    const uint32_t Q = c.Q, twoQ = c.twoQ;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int q = lane + 32 * i, P = 64 * b + q;
        uint4 v = *reinterpret_cast<const uint4 *>(src + p4(4 * q));
        const uint4 w1 = *reinterpret_cast<const uint4 *>(itw + 512 + 2 * P);
        const uint2 w0 = itw[256 + P];
        gs_bfly(v.x, v.y, w1.x, w1.y, Q, twoQ);
        gs_bfly(v.z, v.w, w1.z, w1.w, Q, twoQ);
        gs_bfly(v.x, v.z, w0.x, w0.y, Q, twoQ);
        gs_bfly(v.y, v.w, w0.x, w0.y, Q, twoQ);
        *reinterpret_cast<uint4 *>(w + p4(4 * q)) = v;
    }
    __syncwarp();
    {
        const int grp = lane >> 2, G = 8 * b + grp;
        uint32_t *const p = w + grp * 36 + (lane & 3);
        uint32_t x[8];
#pragma unroll
        for (int k = 0; k < 8; k++) x[k] = p[4 * k];
        const uint4 w2 = *reinterpret_cast<const uint4 *>(itw + 128 + 4 * G);
        const uint4 w3 = *reinterpret_cast<const uint4 *>(itw + 130 + 4 * G);
        const uint4 w1 = *reinterpret_cast<const uint4 *>(itw + 64 + 2 * G);
        const uint2 w0 = itw[32 + G];
        gs_bfly(x[0], x[1], w2.x, w2.y, Q, twoQ);
        gs_bfly(x[2], x[3], w2.z, w2.w, Q, twoQ);
        gs_bfly(x[4], x[5], w3.x, w3.y, Q, twoQ);
        gs_bfly(x[6], x[7], w3.z, w3.w, Q, twoQ);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            gs_bfly(x[k], x[k + 2], w1.x, w1.y, Q, twoQ);
            gs_bfly(x[k + 4], x[k + 6], w1.z, w1.w, Q, twoQ);
        }
#pragma unroll
        for (int k = 0; k < 4; k++) gs_bfly(x[k], x[k + 4], w0.x, w0.y, Q, twoQ);
#pragma unroll
        for (int k = 0; k < 8; k++) p[4 * k] = x[k];
    }
    __syncwarp();
    uint32_t x[8];
#pragma unroll
    for (int k = 0; k < 8; k++) x[k] = w[lane + 36 * k];
#pragma unroll
    for (int st = 0; st < 3; st++)
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (!(k & (1 << st))) {
                const int i = (16 >> st) + (b << (2 - st)) + (k >> (st + 1));
                gs_bfly(x[k], x[k + (1 << st)], c.iw[i], c.iws[i], Q, twoQ);
            }
#pragma unroll
    for (int k = 0; k < 8; k++) out(k, x[k]);
}

// What a step works on: shared memory of the CTA (or worker), the cluster's g buffers
// of this step, the accumulator read and the one written.
template <int C>
struct Block32Cta {
    uint32_t *g, *acc, *acc_out, *dbuf;
    uint32_t *peer[C];
    const uint2 *ftw, *itw;
    int rank;
};

// One step of the CTA's blocks by T threads (tid < T) that share named barrier `bar` (0:
// the CTA). key: the RGSW's rows of the CTA's blocks, in B-tile order, in shared memory,
// or (KG: C = 1, global memory) in global memory but for its first KP, which are at
// head. mid(0), mid(1), mid(2): run before the barrier of 1, at the start of 3 and
// before the products.
template <int DG, int C, int T, bool KG, int KP, class Mid>
__device__ __forceinline__ void block32_step(const Block32Cta<C> &s, const PipeArgs &A, const Ntt32Consts &c,
                                             const uint32_t *key, const uint32_t *head, int tid, int bar, Mid mid)
{
    constexpr int NB = 4 / C, ND = 2 * (DG - 1), NW = T / 32;
    const int warp = tid >> 5, lane = tid & 31;
    const uint32_t Q = c.Q, twoQ = c.twoQ, fourQ = 2 * twoQ, mask = (1u << A.bg_bits) - 1;
    // ---- 1. inverse stages in the blocks
    for (int w = warp; w < 2 * NB; w += NW) {
        const int p = w / NB, lb = w - p * NB, b = s.rank * NB + lb;
        const int o = p * kN32 + b * kB32 + lane;
        block32_inv(s.acc + w * kB32E, s.dbuf + w * kB32E, b, lane, c, s.itw, [&](int k, uint32_t v) {
#pragma unroll
            for (int r = 0; r < C; r++) s.peer[r][o + 32 * k] = v;
        });
    }
    mid(0);
    if (C > 1) cg::this_cluster().sync();
    else pipe_barrier(bar, T);
    // ---- 2. last inverse stages, digits, first two forward stages
    for (int u = tid; u < 512; u += T) {
        const int p = u >> 8, j = u & 255;
        const uint32_t *const x = s.g + p * kN32 + j;
        uint32_t x0 = x[0], x1 = x[256], x2 = x[512], x3 = x[768];
        gs_bfly(x0, x1, c.iw[2], c.iws[2], Q, twoQ);
        gs_bfly(x2, x3, c.iw[3], c.iws[3], Q, twoQ);
        auto last = [&](uint32_t &a, uint32_t &b) {   // as ntt_inv_1024_noscale
            uint32_t u = a + b;
            u = min(u, u - twoQ);
            const uint32_t v = shoup32(a - b + twoQ, c.iw[1], c.iws[1], Q);
            a = min(u, u - Q);
            b = min(v, v - Q);
        };
        last(x0, x2);
        last(x1, x3);
        uint32_t *o = s.dbuf + p * (DG - 1) * NB * kB32E + p4(j);
#pragma unroll
        for (int h = 0; h < DG - 1; h++, o += NB * kB32E) {
            const uint32_t sh = A.bg_bits * h;
            const uint32_t y0 = (x0 >> sh) & mask, y1 = (x1 >> sh) & mask, y2 = (x2 >> sh) & mask,
                           y3 = (x3 >> sh) & mask;
            // y0 +- w1 y2 +- (w2 y1 + w2 w1 y3), and with w3, -w3 w1 for the
            // lower half: each < 6Q + BG
            const uint32_t a = shoup32(y2, c.fw[1], c.fws[1], Q);
            if (C == 1 || s.rank < C / 2) {
                const uint32_t z = y0 + a;
                const uint32_t v = shoup32(y1, c.fw[2], c.fws[2], Q) + shoup32(y3, A.w21, A.w21s, Q);
                if (C < 4) {
                    o[0] = z + v;
                    o[kB32E] = z + fourQ - v;
                } else {
                    o[0] = s.rank == 0 ? z + v : z + fourQ - v;
                }
            }
            if (C == 1 || s.rank >= C / 2) {
                const uint32_t z = y0 + twoQ - a;
                const uint32_t v = shoup32(y1, c.fw[3], c.fws[3], Q) + shoup32(y3, A.w31n, A.w31ns, Q);
                uint32_t *const q = C == 1 ? o + 2 * kB32E : o;
                if (C < 4) {
                    q[0] = z + v;
                    q[kB32E] = z + fourQ - v;
                } else {
                    q[0] = s.rank == 2 ? z + v : z + fourQ - v;
                }
            }
        }
    }
    pipe_barrier(bar, T);
    // ---- 3. forward stages in the blocks
    mid(1);
    for (int w = warp; w < ND * NB; w += NW)
        block32_fwd(s.dbuf + w * kB32E, s.rank * NB + w % NB, lane, c, s.ftw);
    mid(2);
    pipe_barrier(bar, T);
    // ---- 4. multiply-accumulate in the keys' B-tile order (conflict-free in the
    // blocks too): C = 1, 256 threads with 4 words of both output polys each (a
    // digit word is read once); else 512 threads with E words of one poly
    constexpr int PP = C == 1 ? 2 : 1;   // output polys per thread
    if (tid < 512 / PP) {
        constexpr int E = NB;
        const int P = tid >> 8, v = tid & 255, ch = v * E / 4, e0 = v * E % 4;
        const int q = ch / (8 * NB), l = ch % (8 * NB), e = 36 * (l & 7) + 4 * q + e0, lb = l >> 3;
        const uint32_t *const a0 = s.acc + lb * kB32E + e;
        const uint32_t *const d0 = s.dbuf + lb * kB32E + e, *ka = key + P * (NB * kB32) + v * E;
        uint64_t sum[PP][E];
#pragma unroll
        for (int o = 0; o < PP; o++)
#pragma unroll
            for (int i = 0; i < E; i++) sum[o][i] = 0;
#pragma unroll
        for (int h = 0; h < DG; h++)
#pragma unroll
            for (int p = 0; p < 2; p++, ka += 2 * NB * kB32) {
                uint32_t dv[E], kv[E];
                load_words<E>(dv, h < DG - 1 ? d0 + (p * (DG - 1) + h) * NB * kB32E : a0 + p * NB * kB32E);
#pragma unroll
                for (int o = 0; o < PP; o++) {
                    if constexpr (KG) {
                        const int row = (h * 2 + p) * 2 + o;   // compile-time: the loops are unrolled
                        const uint4 x = row < KP ? *reinterpret_cast<const uint4 *>(head + row * kN32 + 4 * v)
                                                 : __ldcg(reinterpret_cast<const uint4 *>(ka + o * NB * kB32));
                        kv[0] = x.x; kv[1] = x.y; kv[2] = x.z; kv[3] = x.w;
                    } else {
                        load_words<E>(kv, ka + o * NB * kB32);
                    }
#pragma unroll
                    for (int i = 0; i < E; i++) sum[o][i] += (uint64_t)dv[i] * kv[i];
                }
            }
#pragma unroll
        for (int o = 0; o < PP; o++) {
            uint32_t r[E];
#pragma unroll
            for (int i = 0; i < E; i++) r[i] = mont_reduce_2q(sum[o][i], Q, A.qinv_neg);
            store_words<E>(s.acc_out + ((P + o) * NB + lb) * kB32E + e, r);
        }
    }
    pipe_barrier(bar, T);
}

template <int DG, int C>
__global__ void __launch_bounds__(Block32Layout<DG, C>::T, 1)
    br32_block_kernel(const __grid_constant__ PipeArgs A, const __grid_constant__ Ntt32Consts c,
                      const uint2 *__restrict__ fwd_tw, const uint2 *__restrict__ inv_tw,
                      const uint2 *__restrict__ plain_tw, uint32_t mu32)
{
    using L = Block32Layout<DG, C>;
    constexpr int NB = L::NB, ND = L::ND, T = L::T, NW = T / 32;
    constexpr int FW = ND * NB < NW ? ND * NB : 0;   // warps with a block in 3 (0: no other warp)
    extern __shared__ __align__(16) unsigned char blk_smem[];
    uint32_t *const g = reinterpret_cast<uint32_t *>(blk_smem + L::g_off);
    uint32_t *const acc = reinterpret_cast<uint32_t *>(blk_smem + L::acc_off);
    uint32_t *const dbuf = reinterpret_cast<uint32_t *>(blk_smem + L::d_off);
    uint32_t *const keys = reinterpret_cast<uint32_t *>(blk_smem + L::key_off);
    uint2 *const ftw = reinterpret_cast<uint2 *>(blk_smem + L::tw_off), *const itw = ftw + kN32;
    uint8_t *const res = blk_smem + L::res_off;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = C > 1 ? (int)(blockIdx.x % C) : 0;
    const int S = A.n * (int)A.digitR, mode = issue_mode(A.flags);
    uint32_t *peer[C];
    peer[0] = g;
    if (C > 1) {
        cg::cluster_group cl = cg::this_cluster();
#pragma unroll
        for (int r = 0; r < C; r++) peer[r] = cl.map_shared_rank(g, r);
    }
    for (int i = tid; i < 2 * kN32; i += T) ftw[i] = __ldg(plain_tw + i);
    if (C > 1) cg::this_cluster().sync();

    // the CTA's key words of step s into buffer b: of each row, in B-tile order, the
    // chunks q * 32 + l (words 32 l + 4 q ..) of its blocks' rows l
    auto fetch = [&](int s, int b, int t0, int nt) {
        if (s < S && t0 >= 0) {
            const uint4 *src = reinterpret_cast<const uint4 *>(A.btkey + ((size_t)s * A.Br + res[s]) * ((size_t)DG * 4 * kN32));
            uint4 *dst = reinterpret_cast<uint4 *>(keys + b * L::key_words);
            for (int x = t0; x < DG * 4 * NB * 64; x += nt) {
                const int row = x / (NB * 64), y = x - row * (NB * 64), q = y / (8 * NB), l = y - q * (8 * NB);
                cp_async16_32(dst + x, src + row * 256 + q * 32 + rank * NB * 8 + l);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    for (size_t gid = blockIdx.x / C; gid < A.count; gid += gridDim.x / C) {
        // ---- LWE_evaluate, residues and the initial accumulator (global, B-tiled; the
        // CTAs of a cluster write the same words)
        if (warp == 0) pipe_init_item(A, c, fwd_tw, keys, res, gid, lane, mu32);
        __syncthreads();
        uint32_t *const ga = A.accs + gid * 2048;
        for (int u = tid; u < 2 * NB * 64; u += T) {
            const int p = u / (NB * 64), cc = u - p * (NB * 64);
            *reinterpret_cast<uint4 *>(acc + (p * NB + (cc >> 6)) * kB32E + p4(4 * (cc & 63))) = __ldcg(
                reinterpret_cast<const uint4 *>(ga) + p * 256 + (cc & 7) * 32 + rank * NB * 8 + (cc >> 3));
        }
        int s = solo_next_step(res, -1, S, mode), next = s < S ? solo_next_step(res, s, S, mode) : S;
        fetch(s, 0, tid, T);
        __syncthreads();
        int ab = 0;   // accumulator buffer
        for (int kb = 0, gb = 0; s < S; kb ^= 1, ab ^= 1, gb ^= C > 1) {
            const Block32Cta<C> cta = [&]() {
                Block32Cta<C> v{g + gb * 2048, acc + ab * (2 * NB * kB32E), acc + (ab ^ 1) * (2 * NB * kB32E), dbuf, {},
                                ftw, itw, rank};
#pragma unroll
                for (int r = 0; r < C; r++) v.peer[r] = peer[r] + gb * 2048;
                return v;
            }();
            block32_step<DG, C, T, false, 0>(cta, A, c, keys + kb * L::key_words, nullptr, tid, 0, [&](int at) {
                // warps without a block in 1 (C = 1) or in 3 start the copy of the next
                // step's keys into the buffer that the last products have freed (copies in
                // flight would hold up the cluster barrier's release: C = 4, 2.01 -> 2.18
                // us per step)
                if (at == 0 && C == 1) fetch(next, kb ^ 1, tid - 64 * NB, T - 64 * NB);
                if (at == 1 && C > 1) fetch(next, kb ^ 1, tid - 32 * FW, T - 32 * FW);
                if (at == 2) asm volatile("cp.async.wait_group 1;" ::: "memory");
            });
            s = next;
            next = s < S ? solo_next_step(res, s, S, mode) : S;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        // ---- accumulator back to global memory, then the outputs of the pipelines' epilogue
        for (int u = tid; u < 2 * NB * 64; u += T) {
            const int p = u / (NB * 64), cc = u - p * (NB * 64);
            __stcg(reinterpret_cast<uint4 *>(ga) + p * 256 + (cc & 7) * 32 + rank * NB * 8 + (cc >> 3),
                   *reinterpret_cast<const uint4 *>(acc + ab * (2 * NB * kB32E) + (p * NB + (cc >> 6)) * kB32E +
                                                      p4(4 * (cc & 63))));
        }
        if (C > 1) cg::this_cluster().sync();
        else __syncthreads();
        if (rank == 0 && warp < 2) pipe_out_poly(A, c, inv_tw, keys + warp * kN32, gid, warp, lane);
        if (C > 1) cg::this_cluster().sync();   // the next ciphertext's accumulator words, and this CTA's exit
        else __syncthreads();
    }
}

// ---- Items form (more than a gate per SM, to a few): W workers of 768 / W threads per CTA, whose
// barriers and loads overlap, take items, consecutive steps of one ciphertext, from a
// cursor that walks them step-major; the accumulator goes through L2 between items. So
// the work spreads evenly over the SMs whatever the batch, where the pipelines give whole
// ciphertexts to CTAs (333 gates: 3 each to 111 of the 152). An item waits for the item
// before it of its ciphertext (done[]), taken earlier by a worker that is running. Three
// workers of 8 warps divide every phase evenly over the four schedulers and reach 2.5 us
// per step and SM; with two of 12 the few ciphertexts of a small batch advance faster
// (blind rotation, two / three workers: 304 gates 5.6 / 6.1 ms, 512 gates 9.1 / 8.2 ms).
// Bound by the multiply pipe (70 % busy; a loop of butterflies alone reaches 82 %).
// Digit tables instead of multiplications did not pay here: 1000 gates 16.0 -> 16.1 ms.
// A step's key rows in shared memory, by one bulk copy that the transforms hide: all of
// them with one worker (160 gates 3.75 -> 3.18 ms), the first 4 of 16 with three (1000 gates
// 15.95 -> 15.70 ms), the others from L2 as they are multiplied. With two workers 4 to 12
// rows gained nothing.
constexpr int kItem32Threads = 768;   // of a CTA
__host__ __device__ constexpr int item32_key_rows(int DG, int W) { return W == 1 ? 4 * DG : W == 2 ? 0 : 4; }
constexpr int kItem32KeyWaitLimit = 1 << 22;   // polls before a key wait gives up
__host__ __device__ constexpr int item32_steps(int W) { return W == 2 ? 8 : 16; }

// Polls of such a wait (about 60 ns each) before it gives up and flags the launch.
constexpr unsigned kItem32WaitLimit = 1u << 26;

// Dynamic shared memory: twiddles, then per worker [g | acc x 2 | dbuf | key rows].
template <int DG, int W>
__host__ __device__ constexpr size_t item32_worker_bytes()
{
    return 4 * (2 * kN32 + (size_t)2 * 2 * 4 * kB32E + (size_t)2 * (DG - 1) * 4 * kB32E +
                (size_t)item32_key_rows(DG, W) * kN32);
}
template <int DG, int W>
constexpr size_t item32_bytes()
{
    return 2 * kN32 * sizeof(uint2) + W * item32_worker_bytes<DG, W>();
}

// Residues and initial accumulators, one warp per ciphertext.
__global__ void __launch_bounds__(32) br32_begin_kernel(const __grid_constant__ PipeArgs A,
                                                        const __grid_constant__ Ntt32Consts c,
                                                        const uint2 *__restrict__ fwd_tw, uint8_t *res, int *done,
                                                        uint32_t mu32)
{
    __shared__ __align__(16) uint32_t buf[kN32];
    const size_t gid = blockIdx.x;
    if (threadIdx.x == 0) done[gid] = -1;
    pipe_init_item(A, c, fwd_tw, buf, res + gid * (size_t)(A.n * (int)A.digitR), gid, threadIdx.x, mu32);
}

__global__ void __launch_bounds__(64) br32_end_kernel(const __grid_constant__ PipeArgs A,
                                                      const __grid_constant__ Ntt32Consts c,
                                                      const uint2 *__restrict__ inv_tw)
{
    __shared__ __align__(16) uint32_t buf[2][kN32];
    pipe_out_poly(A, c, inv_tw, buf[threadIdx.x >> 5], blockIdx.x, threadIdx.x >> 5, threadIdx.x & 31);
}

template <int DG, int W>
__global__ void __launch_bounds__(kItem32Threads, 1)
    br32_items_kernel(const __grid_constant__ PipeArgs A, const __grid_constant__ Ntt32Consts c,
                      const uint2 *__restrict__ plain_tw, const uint8_t *__restrict__ all_res, int *done,
                      unsigned wait_limit, int key_wait_limit)
{
    constexpr int T = kItem32Threads / W, K = item32_steps(W);
    extern __shared__ __align__(16) unsigned char blk_smem[];
    __shared__ int plans[W][2];   // item of the ciphertext (-1: none left), ciphertext
    uint2 *const ftw = reinterpret_cast<uint2 *>(blk_smem), *const itw = ftw + kN32;
    const int wk = threadIdx.x / T, tid = threadIdx.x - wk * T, bar = 1 + wk;
    uint32_t *const g = reinterpret_cast<uint32_t *>(blk_smem + 2 * kN32 * sizeof(uint2) + wk * item32_worker_bytes<DG, W>());
    uint32_t *const acc = g + 2 * kN32, *const dbuf = acc + 2 * 2 * 4 * kB32E, *const head = dbuf + 2 * (DG - 1) * 4 * kB32E;
    constexpr int KP = item32_key_rows(DG, W);
    __shared__ __align__(8) uint64_t bars[W];
    unsigned parity = 0;
    bool failed = false;
    if (tid == 0) {
        mbar_init(&bars[wk], 1);
        mbar_fence_init();
    }
    const int S = A.n * (int)A.digitR, mode = issue_mode(A.flags);
    for (int i = threadIdx.x; i < 2 * kN32; i += kItem32Threads) ftw[i] = __ldg(plain_tw + i);
    __syncthreads();
    const unsigned long long items = (unsigned long long)((S + K - 1) / K) * A.count;
    int *const plan = plans[wk];
    for (;;) {
        if (tid == 0) {
            const unsigned long long v = atomicAdd(A.claim_next, 1ull);
            const int it = v < items ? (int)(v / A.count) : -1;
            const size_t k = it < 0 ? 0 : (size_t)(v - (unsigned long long)it * A.count);
            plan[0] = it;
            plan[1] = (int)k;
            if (it >= 0) {
                const volatile int *d = done + k;
                unsigned polls = 0;
                while (*d != it - 1) {
                    if (++polls > wait_limit) {
                        atomicOr(A.status, kStatusWaitLimit);
                        plan[0] = -1;
                        break;
                    }
                    __nanosleep(32);
                }
                __threadfence();
            }
        }
        pipe_barrier(bar, T);
        const int it = plan[0], k = plan[1];
        if (it < 0) break;
        const uint8_t *const res = all_res + (size_t)k * S;
        uint4 *const ga = reinterpret_cast<uint4 *>(A.accs + (size_t)k * 2048);
        const uint64_t pol = l2_keep_policy();
        // B-tile chunk q * 32 + l holds words 32 l + 4 q ..
        for (int u = tid; u < 512; u += T)
            *reinterpret_cast<uint4 *>(acc + (u >> 8) * 4 * kB32E + 36 * (u & 31) + 4 * ((u >> 5) & 7)) = ld_keep(ga + u, pol);
        pipe_barrier(bar, T);
        int ab = 0;
        const int end = min(S, (it + 1) * K);
        for (int st = it * K; st < end; st++) {
            if (!step_issued(res, st, mode)) continue;
            const Block32Cta<1> cta{g, acc + ab * (8 * kB32E), acc + (ab ^ 1) * (8 * kB32E), dbuf, {g}, ftw, itw, 0};
            const uint32_t *const key = A.btkey + ((size_t)st * A.Br + res[st]) * ((size_t)DG * 4 * kN32);
            if (KP && tid == 0 && !failed) {
                mbar_expect_tx(&bars[wk], KP * kN32 * 4);
                bulk_copy_g2s(head, key, KP * kN32 * 4, &bars[wk]);
            }
            block32_step<DG, 1, T, true, KP>(cta, A, c, key, head, tid, bar, [&](int at) {
                // warp 0 waits, the barrier that follows is the others' wait; thread 0, which
                // alone issues the copies, does so until it gives up itself. (All threads
                // waiting: 160 gates of n = 100 0.698 -> 0.706 ms, 1000 gates 3.21 -> 3.23)
                if (!KP || at != 2 || tid >= 32 || failed) return;
                if (mbar_wait_bounded(&bars[wk], parity, key_wait_limit)) {
                    parity ^= 1u;
                } else {   // flag the launch and go on without
                    failed = true;
                    atomicOr(A.status, kStatusWaitLimit);
                }
            });
            ab ^= 1;
        }
        for (int u = tid; u < 512; u += T)
            st_keep(ga + u, *reinterpret_cast<const uint4 *>(acc + ab * (8 * kB32E) + (u >> 8) * 4 * kB32E + 36 * (u & 31) +
                                                             4 * ((u >> 5) & 7)), pol);
        __threadfence();
        pipe_barrier(bar, T);
        if (tid == 0) atomicExch(done + k, it);
    }
    // a copy that was given up must land before the CTA's shared memory goes
    if (failed && tid == 0) mbar_wait_bounded(&bars[wk], parity, kItem32KeyWaitLimit);
}

}  // namespace dev
}  // namespace fheacc

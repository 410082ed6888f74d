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
//      bits (8 bytes, half of a Shoup pair's), each product three multiplies into
//      three 64-bit sums, reduced once per output.
// The last digit's NTT is the accumulator itself (DevParams::last_digit_from_acc).
//
// Two kernels. br64_cluster_kernel (up to about 1.6 ciphertexts per SM) is for latency: per
// step 8.7 us on 8 CTAs, 10.3 on 4, 17.1 on 2, 30.7 on one, where a 256-thread worker
// took 75 us (40 with its register spills gone). br64_items_kernel is for batches: 27.5
// us per step and SM (2048 gates: 446 ms; 582 before the moduli's fold form). Both are
// bound by the multiply pipe: a loop of butterflies on registers alone keeps it 74 %
// busy, the items form 67 %, the latency form on one CTA 62 %.
#include "block64.cuh"
#include <algorithm>

namespace fheacc {
namespace dev {

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
    unsigned wait_limit;       // polls of a key wait (items form: of an item's wait)
    // latency form over items: the cursor, the ciphertexts' done words, polls of their waits
    unsigned long long *cursor;
    int *done;
    unsigned item_wait_limit;
};

__device__ __forceinline__ int next_issued(const uint8_t *res, int s, int S, int mode)
{
    for (s++; s < S; s++)
        if (step_issued(res, s, mode)) return s;
    return S;
}

// Polls of a worker waiting for another worker's item of the same ciphertext
// (about 60 ns each) before it gives up and flags the launch.
constexpr unsigned kItemWaitLimit = 1u << 26;

// Item v of the step-major cursor as (item of the ciphertext, ciphertext) in plan, once
// the item before it of that ciphertext is done: that one was taken earlier, by CTAs that
// are running, so the wait ends whether or not the whole grid is resident. plan[0] = -1:
// no item left, or the wait was given up.
__device__ __forceinline__ void take_item(unsigned long long *cursor, const int *done, size_t count,
                                          unsigned long long items, unsigned limit, unsigned *status, int (&plan)[2])
{
    const unsigned long long v = atomicAdd(cursor, 1ull);
    plan[0] = v < items ? (int)(v / count) : -1;
    plan[1] = v < items ? (int)(v % count) : 0;
    if (plan[0] < 0) return;
    const volatile int *d = done + plan[1];
    const int before = plan[0] - 1;
    unsigned polls = 0;
    while (*d != before) {
        if (++polls > limit) {
            atomicOr(status, kStatusWaitLimit);
            plan[0] = -1;
            break;
        }
        __nanosleep(32);
    }
    __threadfence();
}

// Steps of an item of the latency form: its accumulator, the barriers and the first keys
// of an item cost about a third of a step.
constexpr int kClusterItemSteps = 16;

// Latency form: one ciphertext per cluster of C CTAs at a time, its accumulator in
// shared memory for all its steps, a block's keys by bulk copies issued as soon as
// the products of the block before are done. ITEMS, for more ciphertexts than
// clusters that run at once: the clusters take items of kClusterItemSteps steps of a
// ciphertext from a cursor, the accumulators in global memory between items (100 gates on
// 76 clusters of 2: 23 us per step of all, where one CTA each took 30.7; a runtime flag
// instead of the instances cost the others 2 %).
template <int B, int C, bool ITEMS>
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
    __shared__ int plan[2];
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
    bool failed = false;   // warp 0: a key wait was given up
    const unsigned long long items =
        (unsigned long long)((A.S + kClusterItemSteps - 1) / kClusterItemSteps) * A.count;

    for (size_t at = blockIdx.x / C;; at += gridDim.x / C) {
        size_t gid = at;
        int it = 0, s = -1, end = A.S;
        if (ITEMS) {
            if (rank == 0 && tid == 0) {
                int pl[2];
                take_item(A.cursor, A.done, A.count, items, A.item_wait_limit, A.status, pl);
                plan[0] = pl[0];
                plan[1] = pl[1];
#pragma unroll
                for (int r = 1; r < C; r++) {
                    int *const q = cg::this_cluster().map_shared_rank(plan, r);
                    q[0] = pl[0];
                    q[1] = pl[1];
                }
            }
            if (C > 1) cg::this_cluster().sync();
            else __syncthreads();
            it = plan[0];
            if (it < 0) break;
            gid = (size_t)plan[1];
            s = it * kClusterItemSteps - 1;
            end = min(A.S, (it + 1) * kClusterItemSteps);
        } else if (gid >= A.count) {
            break;
        }
        const uint8_t *res = A.res + gid * (size_t)A.S;
        uint64_t *ga = A.accs + gid * 4096;
        for (int u = tid; u < 2 * NW; u += T) {
            const int p = u / NW, e = u - p * NW;
            acc[p * px(NW) + px(e)] = __ldcg(ga + p * 2048 + first + e);
        }
        __syncthreads();
        // rows of block lb of step s into kbuf (warp 0). After a lane has given up a wait the
        // warp issues no more, as one: a copy is issued whole or not at all. The launch is
        // flagged then, and the cluster runs to its end without keys, as its barriers need
        // every CTA
        auto fetch = [&](int s, int lb) {
            if (tid >= 32) return;
            if (__any_sync(~0u, failed)) {
                if (!failed) parity ^= 1u;   // back to the last phase, which this lane saw complete
                failed = true;
                return;
            }
            if (tid == 0) mbar_expect_tx(&bar, (unsigned)L::key_bytes(DG));
            __syncwarp();
            const uint2 *src = A.btkey + ((size_t)s * A.Br + res[s]) * rgsw + first + lb * M;
            if (tid < DG * 4) bulk_copy_g2s(kbuf + tid * M, src + (size_t)tid * 2048, M * 8, &bar);
        };
        s = next_issued(res, s, end, mode);
        if (s < end) fetch(s, 0);
        for (int buf = 0; s < end; buf ^= C > 1) {
            const int next = next_issued(res, s, end, mode);
            BlockCta<B, C> cta{g + buf * 4096, acc, work, {}, zeta, rank};
#pragma unroll
            for (int r = 0; r < C; r++) cta.peer[r] = peer[r] + buf * 4096;
            block_step<B, C, T, false>(
                cta, A, tw, itw, c, M, tid, 0,
                [&](int) {
                    // warp 0 waits, the barrier that follows is the others' wait (all threads
                    // waiting: a lone gate of n = 200 3.32 -> 3.34 ms, 100 gates 8.83 -> 8.94)
                    if (tid < 32) {
                        if (!failed) {
                            if (mbar_wait_bounded(&bar, parity, (int)A.wait_limit)) {
                                parity ^= 1u;
                            } else {
                                failed = true;
                                atomicOr(A.status, kStatusWaitLimit);
                            }
                        }
                        __syncwarp();
                    }
                    return (const uint2 *)kbuf;
                },
                [&](int lb) {
                    if (lb + 1 < NB) fetch(s, lb + 1);
                    else if (next < end) fetch(next, 0);
                });
            s = next;
        }
        for (int u = tid; u < 2 * NW; u += T) {
            const int p = u / NW, e = u - p * NW;
            ga[p * 2048 + first + e] = acc[p * px(NW) + px(e)];
        }
        if (ITEMS) __threadfence();
        // the whole cluster: the next ciphertext starts with the first g buffer again
        if (C > 1) cg::this_cluster().sync();
        else __syncthreads();
        if (ITEMS && rank == 0 && tid == 0) atomicExch(A.done + gid, it);
    }
    // a copy that was given up must land before the CTA's shared memory goes
    if (failed && tid == 0) mbar_wait_bounded(&bar, parity, (int)kKeyWaitLimit);
    if (C > 1) cg::this_cluster().sync();
}

// Steps of an item: long enough that taking it, and the accumulator's way through L2
// and back, cost little, short enough that the keys in use (9 MB a step) stay in L2 and
// the batch ends evenly. 2048 gates, us per step and SM: 29.2 with 1 step, 28.3 with 2,
// 27.8 with 4 and with 6, 28.2 with 8.
constexpr int kItemSteps = 4;

// Throughput form: W workers per CTA (two of kTP threads, so that one's barriers and
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
__global__ void __launch_bounds__(W * worker_threads64(W), 1) br64_items_kernel(const __grid_constant__ BlockArgs A,
                                                           unsigned long long *cursor, int *done,
                                                           const ulonglong2 *__restrict__ tw,
                                                           const ulonglong2 *__restrict__ itw,
                                                           const __grid_constant__ Ntt64Consts c)
{
    using L = BlockLayout<B, 1>;
    constexpr int T = worker_threads64(W);
    extern __shared__ __align__(128) unsigned char smem_all[];
    const int wk = threadIdx.x / T, tid = threadIdx.x - wk * T, bar = W == 1 ? 0 : 1 + wk;
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
        if (tid == 0) take_item(cursor, done, A.count, items, A.wait_limit, A.status, plans[wk]);
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

// The same with the last-digit identity (derive_keys64_kernel) applied on the way, to
// `count` RGSWs [DG][4][2048].
__global__ void derive_limbs64_kernel(const uint64_t *__restrict__ in, uint2 *__restrict__ out, size_t count, int DG,
                                      const ulonglong2 *__restrict__ cf, const __grid_constant__ Ntt64Consts c)
{
    constexpr size_t plane = 4 * 2048;
    constexpr uint32_t m27 = (1u << 27) - 1;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < count * plane;
         i += (size_t)gridDim.x * blockDim.x) {
        const size_t at = i / plane * (size_t)DG * plane + i % plane;
        const uint64_t last = in[at + (size_t)(DG - 1) * plane] % c.Q;
        for (int h = 0; h < DG; h++) {
            uint64_t m = mul64<true>(last, cf[h], c), w;
            m = m >= c.Q ? m - c.Q : m;
            if (h + 1 < DG) {
                const uint64_t k = in[at + (size_t)h * plane] % c.Q;
                w = k >= m ? k - m : k + c.Q - m;
            } else {
                w = m;
            }
            out[at + (size_t)h * plane] = make_uint2((uint32_t)w & m27, (uint32_t)(w >> 27));
        }
    }
}

}  // namespace dev

int launch_derive_limbs64(Context &c, const uint64_t *d_in, uint2 *d_out, size_t count, cudaStream_t st)
{
    if (!count) return FHEACC_OK;
    dev::derive_limbs64_kernel<<<(unsigned)std::min<size_t>(count * 32, 4096), 256, 0, st>>>(
        d_in, d_out, count, (int)c.p.digitG, c.d_cf64, c.nc64);
    c.launches++;
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? FHEACC_OK : c.cuda_fail(e, "derived limb words launch");
}

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

// Launch configuration of the latency form and the clusters that run at once (0: the form
// does not fit).
template <int B, int C, bool ITEMS>
static int cluster_config(Context &c, const dev::BlockArgs &A, cudaStream_t st, cudaLaunchConfig_t &cfg,
                          cudaLaunchAttribute (&attr)[1])
{
    auto kern = dev::br64_cluster_kernel<B, C, ITEMS>;
    const size_t smem = dev::BlockLayout<B, C>::key_off(A.DG) + dev::BlockLayout<B, C>::key_bytes(A.DG);
    if (smem > kMaxDynamicSmem) return 0;
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(dev::kTB);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = C > 1 ? 1 : 0;
    int n = sm_count64(c);
    if (allow_dynamic_smem(kern) != cudaSuccess ||
        (C > 1 && cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess)) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

template <int B, int C, bool ITEMS>
static int launch_cluster(Context &c, const dev::BlockArgs &A, int max_ctas, cudaStream_t st)
{
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    size_t clusters = (size_t)cluster_config<B, C, ITEMS>(c, A, st, cfg, attr);
    if (max_ctas > 0) clusters = std::min<size_t>(clusters, (size_t)(max_ctas / C));
    if (!clusters) return c.fail(FHEACC_EINVAL, "blind rotation latency form does not fit");
    cudaError_t e;
    if (ITEMS) {
        e = cudaMemsetAsync(A.cursor, 0, sizeof(*A.cursor), st);
        if (e != cudaSuccess) return c.cuda_fail(e, "blind rotation cursor reset");
    }
    cfg.gridDim = dim3((unsigned)(std::min<size_t>(A.count, clusters) * C));
    e = cudaLaunchKernelEx(&cfg, dev::br64_cluster_kernel<B, C, ITEMS>, A, (const ulonglong2 *)c.d_tw64,
                           (const ulonglong2 *)c.d_itw64, c.nc64);
    c.launches++;
    if (e == cudaSuccess) e = cudaGetLastError();
    return e == cudaSuccess ? FHEACC_OK : c.cuda_fail(e, "blind rotation launch");
}

// The latency form in the CTAs per ciphertext (and over items or not) that give a step of
// all ciphertexts the least time, unless the throughput form's is less (*taken = false).
// The times, us, as a + b (digitG - 2), fitted at digitG = 2, 4 and 6: a step on 8, 4, 2
// and 1 CTAs while all ciphertexts run at once; that times ciphertexts per cluster and 4 %
// over items; the throughput form's, a worker's chain up to two ciphertexts per SM. At
// digitG = 6: over items 4 CTAs from 39 to 60 gates, 2 from 77 to 131, 1 from 153 to 241.
// Blind rotation of n = 200: 50 gates 6.57 ms on 2 CTAs, 5.63 over items on 4; 62 gates 6.55
// and 6.59; 100 gates 11.9 on one, 8.8 over items on 2; 130 gates 11.7 and 11.6; 160 gates
// 19.4 in the throughput form, 12.6 over items on one; 230 gates 20.2 and 17.9; 260 gates
// 20.5 and 20.6.
static int launch_latency(Context &c, const dev::BlockArgs &A, int max_ctas, cudaStream_t st, bool *taken)
{
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    const size_t sms = (size_t)sm_count64(c), at_once = max_ctas > 0 ? (size_t)max_ctas : sms;
    struct Form {
        int (*launch)(Context &, const dev::BlockArgs &, int, cudaStream_t);
        int C, n;
        double step;
        bool items;
    };
    const int n4 = cluster_config<4, 4, false>(c, A, st, cfg, attr), n2 = cluster_config<4, 2, false>(c, A, st, cfg, attr),
              n1 = cluster_config<4, 1, false>(c, A, st, cfg, attr);
    const double d = A.DG - 2;
    const double t4 = 7.5 + 0.7 * d, t2 = 11.2 + 1.475 * d, t1 = 15.2 + 3.88 * d;
    const Form forms[] = {
        {launch_cluster<8, 8, false>, 8, c.p.BG_bits <= 29 ? cluster_config<8, 8, false>(c, A, st, cfg, attr) : 0,
         6.8 + 0.47 * d, false},
        {launch_cluster<4, 4, false>, 4, n4, t4, false}, {launch_cluster<4, 2, false>, 2, n2, t2, false},
        {launch_cluster<4, 1, false>, 1, n1, t1, false}, {launch_cluster<4, 4, true>, 4, n4, t4, true},
        {launch_cluster<4, 2, true>, 2, n2, t2, true},   {launch_cluster<4, 1, true>, 1, n1, t1, true}};
    double least = std::max(31.0 + 5.0 * d, (14.5 + 3.25 * d) * (double)A.count / sms);
    const Form *best = nullptr;
    for (const Form &f : forms) {
        if (f.n < 1 || at_once < (size_t)f.C) continue;
        const bool fits = A.count <= (size_t)f.n;
        if (f.items ? fits || max_ctas > 0 : !fits) continue;
        const double t = f.items ? 1.04 * f.step * (double)A.count / f.n : f.step;
        if (t < least) {
            best = &f;
            least = t;
        }
    }
    *taken = best != nullptr;
    return best ? best->launch(c, A, max_ctas, st) : FHEACC_OK;
}

template <int B, int W>
static int launch_items(Context &c, dev::BlockArgs A, unsigned long long *cursor, int *done, int max_ctas,
                        cudaStream_t st)
{
    auto kern = dev::br64_items_kernel<B, W>;
    const size_t smem = W * dev::BlockLayout<B, 1>::key_off(A.DG);
    cudaError_t e = allow_dynamic_smem(kern);
    if (e != cudaSuccess) return c.cuda_fail(e, "blind rotation smem attribute");
    // an SM per ciphertext while there are enough: the surplus workers wait their turn
    size_t blocks = std::min<size_t>((size_t)sm_count64(c), A.count * std::max(c.tune.br_pipes, 1));
    if (max_ctas > 0) blocks = std::min<size_t>(blocks, (size_t)max_ctas);
    e = cudaMemsetAsync(cursor, 0, sizeof(*cursor), st);
    if (e != cudaSuccess) return c.cuda_fail(e, "blind rotation cursor reset");
    A.wait_limit = c.tune.debug_wait_limit >= 0 ? (unsigned)c.tune.debug_wait_limit : dev::kItemWaitLimit;
    kern<<<(unsigned)blocks, W * dev::worker_threads64(W), smem, st>>>(A, cursor, done, c.d_tw64, c.d_itw64, c.nc64);
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
    A.c54 = limb_c54(c);
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
    A.cursor = cursor;
    A.done = done;
    A.item_wait_limit = c.tune.debug_wait_limit >= 0 ? (unsigned)c.tune.debug_wait_limit : dev::kItemWaitLimit;
    // an explicit worker count asks for the throughput form
    bool taken = false;
    int rc = c.tune.br_pipes == 0 ? launch_latency(c, A, max_ctas, st, &taken) : FHEACC_OK;
    if (!rc && !taken)   // digitG = 7 and 8: one worker's work area more than fills half an SM
        rc = 2 * dev::BlockLayout<4, 1>::key_off(A.DG) <= kMaxDynamicSmem
                 ? launch_items<4, 2>(c, A, cursor, done, max_ctas, st)
                 : launch_items<4, 1>(c, A, cursor, done, max_ctas, st);
    if (rc) return rc;
    dev::br64_end_kernel<<<(unsigned)R.count, dev::kT64, 0, st>>>(R, c.d_itw64, c.nc64);
    c.launches++;
    e = cudaGetLastError();
    return e == cudaSuccess ? FHEACC_OK : c.cuda_fail(e, "blind rotation end launch");
}

}  // namespace fheacc

// products64.cu -- RLWE x RGSW products (RLWE_mult_RGSW, RLWE.cpp:642-704) of the
// 64-bit path in block form, with what CMUX (RLWE.cpp:788-793) and the RLWE blind rotation
// (RLWE.cpp:824-838) do before and after them folded into their loads and stores: the
// subtraction c1 - c0, the NTT-domain rotation, the addition of c0; for homo_expand the
// rows of the RGSWs it builds.
//
// A CMUX was six launches (subtract, key pairs, products split over the digits, their sum,
// add; 42 us for one pair); it is two now. Up to one product per SM a product runs on a
// cluster of 8, 4 or 2 CTAs or on one, as the blind rotation's latency form; beyond that
// on two workers per CTA. Bound by the multiply pipe, as the blind rotation.
#include "block64.cuh"
#include <algorithm>

namespace fheacc {
namespace dev {

// Word e of poly p of product i's input.
__device__ __forceinline__ uint64_t product_in(const Products64 &A, size_t i, int p, int e, const Ntt64Consts &c)
{
    const size_t at = i * A.in_stride + p * 2048 + e;
    if (!A.in0) return A.in1[at];
    const uint64_t u0 = A.in0[at];
    uint64_t u1;
    if (A.rot) {
        u1 = mul64<true>(u0, __ldg(A.rot + e), c);
        u1 = u1 >= c.Q ? u1 - c.Q : u1;
    } else {
        u1 = A.in1[at];
    }
    return u1 >= u0 ? u1 - u0 : u1 + c.Q - u0;
}

// Product i on the CTA's blocks.
template <int B, int C, int T>
__device__ __forceinline__ void product_item(const BlockCta<B, C> &s, const Products64 &A, size_t i,
                                             const ulonglong2 *__restrict__ tw, const ulonglong2 *__restrict__ itw,
                                             const Ntt64Consts &c, int tid, int bar)
{
    using L = BlockLayout<B, C>;
    constexpr int NW = L::NB * L::M;
    const int first = s.rank * NW;
    uint64_t *const out = A.out + i / A.out_per * A.out_s1 + i % A.out_per * A.out_s2;
    for (int u = tid; u < 2 * NW; u += T) {
        const int p = u / NW, e = u - p * NW;
        const uint64_t v = product_in(A, i, p, first + e, c);
        s.acc[p * px(NW) + px(e)] = v;
        if (A.copy_in) out[4096 + p * 2048 + first + e] = v;
    }
    group_sync(bar, T);
    const uint2 *const key = A.keys + i * A.key_stride + first;
    block_step<B, C, T, true>(
        s, A, tw, itw, c, 2048, tid, bar, [&](int lb) { return key + lb * L::M; }, [](int) {});
    for (int u = tid; u < 2 * NW; u += T) {
        const int p = u / NW, e = u - p * NW;
        uint64_t v = s.acc[p * px(NW) + px(e)];
        v = v >= c.Q ? v - c.Q : v;
        if (A.add0) {
            v += A.in0[i * A.in_stride + p * 2048 + first + e];
            v = v >= c.Q ? v - c.Q : v;
        }
        out[p * 2048 + first + e] = v;
    }
    group_sync(bar, T);
}

template <int B, int C>
__global__ void __launch_bounds__(kTB, 1) products64_cluster_kernel(const __grid_constant__ Products64 A,
                                                                   const ulonglong2 *__restrict__ tw,
                                                                   const ulonglong2 *__restrict__ itw,
                                                                   const __grid_constant__ Ntt64Consts c)
{
    using L = BlockLayout<B, C>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    uint64_t *const g = reinterpret_cast<uint64_t *>(smem_raw + L::g_off);
    uint64_t *const acc = reinterpret_cast<uint64_t *>(smem_raw + L::acc_off);
    uint64_t *const work = reinterpret_cast<uint64_t *>(smem_raw + L::work_off(A.DG));
    __shared__ uint64_t zeta[L::NB][B - 1];
    const int rank = C > 1 ? (int)(blockIdx.x % C) : 0;
    uint64_t *peer[C];
    peer[0] = g;
    if (C > 1) {
        cg::cluster_group cl = cg::this_cluster();
#pragma unroll
        for (int r = 0; r < C; r++) peer[r] = cl.map_shared_rank(g, r);
    }
    block_zeta<B, L::NB>(zeta, rank * L::NB, tw, c);
    if (C > 1) cg::this_cluster().sync();
    else __syncthreads();
    int buf = 0;
    for (size_t i = blockIdx.x / C; i < A.count; i += gridDim.x / C, buf ^= C > 1) {
        BlockCta<B, C> cta{g + buf * 4096, acc, work, {}, zeta, rank};
#pragma unroll
        for (int r = 0; r < C; r++) cta.peer[r] = peer[r] + buf * 4096;
        product_item<B, C, kTB>(cta, A, i, tw, itw, c, threadIdx.x, 0);
    }
    if (C > 1) cg::this_cluster().sync();
}

template <int B, int W>
__global__ void __launch_bounds__(W * worker_threads64(W), 1) products64_workers_kernel(const __grid_constant__ Products64 A,
                                                                       const ulonglong2 *__restrict__ tw,
                                                                       const ulonglong2 *__restrict__ itw,
                                                                       const __grid_constant__ Ntt64Consts c)
{
    using L = BlockLayout<B, 1>;
    extern __shared__ __align__(128) unsigned char smem_all[];
    constexpr int T = worker_threads64(W);
    const int wk = threadIdx.x / T, tid = threadIdx.x - wk * T;
    unsigned char *const smem_raw = smem_all + wk * L::key_off(A.DG);
    uint64_t *const g = reinterpret_cast<uint64_t *>(smem_raw + L::g_off);
    __shared__ uint64_t zeta[B][B - 1];
    block_zeta<B, B>(zeta, 0, tw, c);
    __syncthreads();
    const BlockCta<B, 1> cta{g, reinterpret_cast<uint64_t *>(smem_raw + L::acc_off),
                             reinterpret_cast<uint64_t *>(smem_raw + L::work_off(A.DG)), {g}, zeta, 0};
    for (size_t i = (size_t)wk * gridDim.x + blockIdx.x; i < A.count; i += (size_t)gridDim.x * W)
        product_item<B, 1, T>(cta, A, i, tw, itw, c, tid, W == 1 ? 0 : 1 + wk);
}

}  // namespace dev

static int sms_products(Context &c)
{
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, c.device);
    return v > 0 ? v : 1;
}

template <int B, int C>
static int launch_products_cluster(Context &c, const Products64 &A, cudaStream_t st, bool *fits)
{
    auto kern = dev::products64_cluster_kernel<B, C>;
    const size_t smem = dev::BlockLayout<B, C>::key_off(A.DG), sms = (size_t)sms_products(c);
    *fits = false;
    if (smem > kMaxDynamicSmem || A.count * C > sms) return FHEACC_OK;
    cudaError_t e = allow_dynamic_smem(kern);
    if (e != cudaSuccess) return c.cuda_fail(e, "products smem attribute");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(A.count * C));
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
        if (A.count > (size_t)n) return FHEACC_OK;   // more than one round: fewer CTAs per product
    }
    *fits = true;
    e = cudaLaunchKernelEx(&cfg, kern, A, (const ulonglong2 *)c.d_tw64, (const ulonglong2 *)c.d_itw64, c.nc64);
    c.launches++;
    if (e == cudaSuccess) e = cudaGetLastError();
    return e == cudaSuccess ? FHEACC_OK : c.cuda_fail(e, "products launch");
}

template <int B, int W>
static int launch_products_workers(Context &c, const Products64 &A, cudaStream_t st)
{
    auto kern = dev::products64_workers_kernel<B, W>;
    const size_t smem = W * dev::BlockLayout<B, 1>::key_off(A.DG);
    cudaError_t e = allow_dynamic_smem(kern);
    if (e != cudaSuccess) return c.cuda_fail(e, "products smem attribute");
    const size_t blocks = std::min<size_t>((size_t)sms_products(c), A.count);
    kern<<<(unsigned)blocks, W * dev::worker_threads64(W), smem, st>>>(A, c.d_tw64, c.d_itw64, c.nc64);
    c.launches++;
    e = cudaGetLastError();
    return e == cudaSuccess ? FHEACC_OK : c.cuda_fail(e, "products launch");
}

// Whether the outputs (out_per = 1) overlap the inputs at `in` other than each its own: a
// product reads its inputs before it writes, but not before the others write.
static bool outputs_overlap(const Products64 &A, const uint64_t *in)
{
    if (!in || (in == A.out && (A.count == 1 || A.in_stride == A.out_s1))) return false;
    const uint64_t *in_end = in + (A.count - 1) * A.in_stride + 4096, *out_end = A.out + (A.count - 1) * A.out_s1 + 4096;
    return in < out_end && A.out < in_end;
}

int launch_products64(Context &c, Products64 A, cudaStream_t st)
{
    if (!A.count) return FHEACC_OK;
    if (A.out_per == 1 && (outputs_overlap(A, A.in0) || outputs_overlap(A, A.in1))) {
        int rc = ensure_scratch(c, c.psi, A.count * 4096 * sizeof(uint64_t));
        if (rc) return rc;
        Products64 B = A;
        B.out = (uint64_t *)c.psi.ptr;
        B.out_s1 = 4096;
        rc = launch_products64(c, B, st);
        if (rc) return rc;
        cudaError_t e = cudaMemcpy2DAsync(A.out, A.out_s1 * sizeof(uint64_t), B.out, 4096 * sizeof(uint64_t),
                                          4096 * sizeof(uint64_t), A.count, cudaMemcpyDeviceToDevice, st);
        return e == cudaSuccess ? FHEACC_OK : c.cuda_fail(e, "products copy");
    }
    A.DG = (int)c.p.digitG;
    A.bg_bits = c.p.BG_bits;
    A.c54 = limb_c54(c);
    bool fits = false;
    int rc = FHEACC_OK;
    if (c.p.BG_bits <= 29) rc = launch_products_cluster<8, 8>(c, A, st, &fits);
    if (!rc && !fits) rc = launch_products_cluster<4, 4>(c, A, st, &fits);
    if (!rc && !fits) rc = launch_products_cluster<4, 2>(c, A, st, &fits);
    if (!rc && !fits) rc = launch_products_cluster<4, 1>(c, A, st, &fits);
    if (rc || fits) return rc;
    return 2 * dev::BlockLayout<4, 1>::key_off(A.DG) <= kMaxDynamicSmem ? launch_products_workers<4, 2>(c, A, st)
                                                                     : launch_products_workers<4, 1>(c, A, st);
}

}  // namespace fheacc

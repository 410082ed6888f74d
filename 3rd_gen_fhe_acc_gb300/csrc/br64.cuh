// br64.cuh -- pieces shared by the 64-bit blind rotations (blind_rotate64.cu and
// bootstrap64.cu): launch arguments, residues, initial accumulators, outputs.
#pragma once
#include "bulk.cuh"
#include "ctx.hpp"
#include "l2hint.cuh"
#include "ntt64.cuh"

namespace fheacc {
namespace dev {

constexpr int kT64 = 256;   // threads of a worker

struct Br64Args {
    const uint64_t *c1, *c2;
    const uint32_t *idx1, *idx2;   // optional: gate g reads c1 + idx1[g] * (n+1) (else g)
    const int32_t *gates;
    size_t count;
    const ulonglong2 *btkey;   // [(i*digitR + j)*Br + r][digitG][2][2][2048] Shoup pairs
    uint64_t *accs;            // scratch [count][2][2048], NTT domain, values < 2Q
    uint64_t *acc_out;         // optional canonical NTT accumulators [count][4096]
    uint64_t *extract;         // optional [count][kExtract64]
    int group;                 // ciphertexts per claim (<= kMaxGroup64 per worker)
    int derive_last;           // last digit's NTT from the accumulator (DevParams::last_digit_from_acc)
    int n, DG;
    uint32_t q, embed, Br, digitR, bg_bits, flags;
    uint64_t gate_constant[8];
    StepWindow win;            // keeps the CTAs within a few steps of each other (window.cuh)
    unsigned long long *claim_next;   // next unclaimed ciphertext (zeroed before the launch)
    unsigned *status;          // set to kStatusWaitLimit if a worker gave up waiting
    unsigned wait_limit;       // polls before such a wait gives up (kWorkerWaitLimit)
    size_t claim_limit;        // ciphertexts [0, claim_limit) are claimed in groups
    // remainder pool: ciphertexts [pool_first, pool_first + pool_count) that all
    // CTAs share item by item (0: none); their state after the claim words
    int pool_count;
    size_t pool_first;
    unsigned long long *pool_cursor;   // next (step, pool ciphertext) item, step-major (zeroed)
    int *pool_done;            // [pool_count] last finished step (-1: none yet)
    int *pool_last;            // [pool_count] last step with a non-zero residue (-1: none)
    uint8_t *pool_res;         // [pool_count][n * digitR] residues
};

// LWE_evaluate (LWE.cpp:203-222) of ciphertext gid and the residues of its
// refresh steps, the base-Br digits of (q - a_i) mod q (RLWE.cpp:740-760), into
// res[n * digitR]; the thread that takes i = n writes the b value and the gate's
// two test-vector bounds. Threads t0, t0 + nt, ... take part.
__device__ __forceinline__ void br64_residues(const Br64Args &A, size_t gid, uint8_t *res, uint32_t *bval,
                                              uint32_t *b1, uint32_t *b2, int t0, int nt)
{
    const int n = A.n;
    const uint32_t q = A.q, qmask = q - 1;
    const int g = A.gates[gid];
    const bool x2 = (g == 4 || g == 5);
    const uint64_t *c1 = A.c1 + (A.idx1 ? (size_t)A.idx1[gid] : gid) * (size_t)(n + 1);
    const uint64_t *c2 = A.c2 + (A.idx2 ? (size_t)A.idx2[gid] : gid) * (size_t)(n + 1);
    for (int i = t0; i <= n; i += nt) {
        const uint64_t v = x2 ? 2 * (c1[i] - c2[i]) : c1[i] + c2[i];
        if (i < n) {
            uint32_t nega = (q - (uint32_t)(v & qmask)) & qmask;
            for (uint32_t j = 0; j < A.digitR; j++) {
                res[i * (int)A.digitR + (int)j] = (uint8_t)(nega % A.Br);
                nega /= A.Br;
            }
        } else {
            const uint64_t gc = A.gate_constant[(unsigned)g < 6u ? g : 6];
            *bval = (uint32_t)(v & qmask);
            *b1 = (uint32_t)(gc & qmask);
            *b2 = (*b1 + q / 2) & qmask;
        }
    }
}

// acc_initialization (RLWE.cpp:706-724) of ciphertext gid into its accumulator:
// a = 0, b = the test vector, forward NTT. buf: a shared poly (layout pi<P>)
// that the worker's second 128-thread group transforms; bar: the worker's
// barrier (its groups on bar + 1 and bar + 2).
template <bool PM, bool P>
__device__ __forceinline__ void br64_acc_init(const Br64Args &A, const Ntt64Consts &c, const ulonglong2 *tw,
                                              size_t gid, uint32_t val, uint32_t b1, uint32_t b2, uint64_t *buf,
                                              int tid, int bar)
{
    const uint32_t q = A.q, qmask = q - 1;
    const uint64_t Q8 = c.Q / 8 + 1, negQ8 = c.Q - Q8;
    for (int e = tid; e < 2048; e += kT64) {
        uint64_t v = 0;
        if (e % A.embed == 0 && (uint32_t)e / A.embed < q / 2) {
            const uint32_t tmp = (val - (uint32_t)e / A.embed) & qmask;
            if (b1 < b2) v = (tmp >= b1 && tmp < b2) ? negQ8 : Q8;
            else v = (tmp >= b2 && tmp < b1) ? Q8 : negQ8;
        }
        buf[pi<P>(e)] = v;
    }
    group_sync(bar, kT64);
    if (tid >= 128) ntt64_fwd_2048<PM, 128, P>(buf, tw, c, tid - 128, bar + 2);
    group_sync(bar, kT64);
    uint64_t *acc = A.accs + gid * 4096;
    const uint64_t pol = l2_keep_policy();
    for (int e = tid; e < 2048; e += kT64) {
        st_keep64(acc + e, 0, pol);
        st_keep64(acc + 2048 + e, canonical64<PM>(buf[pi<P>(e)], c), pol);
    }
    group_sync(bar, kT64);
}

// Output of ciphertext gid from its accumulator: the extracted RLWE
// (NTT_a_transpose, RLWE.cpp:218-226, then the inverse NTT of both polys) or
// the canonical NTT accumulator. a0, a1: shared polys (layout pi<P>).
template <bool PM, bool P>
__device__ __noinline__ void br64_output(const Br64Args &A, const Ntt64Consts &c, const ulonglong2 *itw,
                                            size_t gid, uint64_t *a0, uint64_t *a1, int tid, int bar)
{
    const uint64_t *acc = A.accs + gid * 4096;
    if (A.extract) {
        for (int e = tid; e < 2048; e += kT64) {
            a0[pi<P>(e)] = __ldcg(acc + 2047 - e);
            a1[pi<P>(e)] = __ldcg(acc + 2048 + e);
        }
        group_sync(bar, kT64);
        ntt64_inv_2048<PM, 128, P>(tid < 128 ? a0 : a1, itw, c, tid & 127, bar + 1 + (tid >> 7));
        group_sync(bar, kT64);
        uint64_t *ext = A.extract + gid * kExtract64;
        for (int e = tid; e < 2048; e += kT64) ext[e] = a0[pi<P>(e)];
        if (tid == 0) ext[2048] = a1[pi<P>(0)];
    } else {
        for (int e = tid; e < 4096; e += kT64) {
            const uint64_t v = __ldcg(acc + e);
            A.acc_out[gid * 4096 + e] = v >= c.Q ? v - c.Q : v;
        }
    }
    group_sync(bar, kT64);
}

}  // namespace dev

// Blind rotation in block form (blind_rotate64.cu); R: inputs, outputs, flags and
// the accumulator scratch, followed by the claim words and [count][n * digitR] bytes.
int launch_blind_rotate64_blocks(Context &c, const dev::Br64Args &R, int max_ctas, cudaStream_t st);
int launch_derive_limbs64(Context &c, const uint64_t *d_in, uint2 *d_out, size_t count, cudaStream_t st);
int launch_limb_words64(Context &c, const uint64_t *d_in, uint2 *d_out, size_t n, cudaStream_t st);

// RLWE x RGSW products in block form (products64.cu; moduli Q = 2^b - c). Product i: of
// in1[i] (in0 null), in1[i] - in0[i], or in0[i] times rot minus in0[i] (rot: constant
// pairs), i-th RLWEs in_stride words apart, with RGSW i (limb words with the last-digit
// identity, launch_derive_limbs64; one RGSW for all: key_stride 0); plus in0[i] with
// add0; to out + i / out_per * out_s1 + i % out_per * out_s2 words, and with copy_in the
// input after it. All RLWEs canonical NTT, [2][2048]; out may be in0 or in1 of equal
// strides.
struct Products64 {
    const uint64_t *in0, *in1;
    size_t in_stride;
    const ulonglong2 *rot;
    const uint2 *keys;
    size_t key_stride;
    uint64_t *out;
    size_t out_per, out_s1, out_s2;
    int add0, copy_in;
    size_t count;
    int DG;
    uint32_t bg_bits, c54;
};
int launch_products64(Context &c, Products64 A, cudaStream_t st);
// Whether the block form's products and key words apply to the context.
inline bool products64_apply(const Context &c) { return c.wide && c.nc64.pm_c && c.dp.last_digit_from_acc; }
inline uint32_t limb_c54(const Context &c) { return c.nc64.pm_c << (c.nc64.pm_s - 10); }   // 2^54 = 2^(54-b) 2^b

}  // namespace fheacc

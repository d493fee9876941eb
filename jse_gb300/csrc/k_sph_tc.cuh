// Spherical-Chebyshev forward on the tensor cores (tcgen05, kind::f16, FP32 accumulation in
// TMEM).  Included by k_desc.cu after the FP32-pipe kernels.
//
// For fuse matrices of the form W[tc][tn][p][n] = alpha[tc][tn][p] delta(n, p mod N1) the
// expansion coefficients of one atom are a single product over its neighbours,
//   A[p][lm] = sum_j Y_j[lm] c_j[p],   c_j[p] = alpha[tc][tn_j][p] fc_j T_{p mod N1}(r_j)
// (basis_SphericalChebyshev.hpp:264-351 with the fuse step of nnap_util.hpp:273-280), i.e.
// D = Y^T C with M = 64 rows (lm; (L+1)^2 <= 64), N = NP rounded up to 8 columns (p) and
// K = 16 neighbours per MMA.  The descriptors are then fp[p][l] = 4 pi/(2l+1) sum_m A^2 as
// in k_sph_fwd_n.
//
// Precision.  Each FP32 operand x is split into FP16 hi = fp16(x) and lo = fp16(x - hi), and
// each product is formed as hi*hi + lo*hi + hi*lo: about 22 significant bits per operand
// where lo is a normal FP16 number (|x| >= 2^-3) and an absolute error below 2^-25 (of 32 c)
// otherwise, well inside FP32 descriptor accuracy.  The operands are bounded (|Y_lm| <= 1.5
// for l <= 12, |fc T_n| <= 1), and the host uses this kernel only when every |alpha| is at
// most kTcAlphaMax, so hi never overflows FP16.
//
// Organisation.  A CTA of 4 warps takes 4 atom slots per round, one per warp.  A warp walks
// its atom's row 32 neighbours at a time (lane = neighbour): it evaluates fc T_n, c and Y
// into registers, waits for its own previous MMAs, stores the split operands into its two
// 16-neighbour chunks of shared memory (MN-major, no swizzle: core matrices of 8
// neighbours x 16 bytes, LBO = the stride between neighbour groups, SBO = 128 bytes between
// groups of 8 rows or columns), and one lane issues the 3 MMAs of each chunk into the
// atom's 32 TMEM columns and commits them to the warp's mbarrier.  After the round's last
// MMAs all 4 warps read the 4 tiles back: an M = 64 tile keeps rows 16q..16q+15 in TMEM
// lanes 32q..32q+15, which warp q reads.  They write A and form the power spectrum from
// A in shared memory (the operand buffers, free once the MMAs are done).  Every wait on
// an mbarrier is bounded; a wait that gives up raises ERRBIT_TIMEOUT.
#pragma once

#include <cuda_fp16.h>

#include "smem_limit.cuh"
#include "tc_util.cuh"

namespace nnapgb {
namespace {

constexpr int kFwdTcWarps = 4;
// c is split times this (kTcAlphaMax times it is below FP16's largest number), so that the lo
// part of a neighbour near the cutoff, where fc is small, stays clear of FP16's smallest steps.
constexpr float kTcScale = 32.f;

template <int L, int NP>
struct SphTcShape {
    static constexpr int KM = (L + 1) * (L + 1);   // tile rows in use
    static constexpr int NPN = (NP + 7) & ~7;       // MMA N
    static constexpr int NCA = (KM + 7) / 8;        // 8-row groups of Y a neighbour writes
    static constexpr int NPH = NPN / 2 <= 4 ? 4 : NPN / 2 <= 8 ? 8 : 16;  // columns a lane reads back
    static constexpr int NCB = NPN / 8;             // 8-column groups of c a neighbour writes
    static constexpr int ABYTES = 64 * 16 * 2;      // one FP16 image of a chunk's Y^T
    static constexpr int BBYTES = 16 * NPN * 2;     // one FP16 image of a chunk's C
    static constexpr int CHUNK = 2 * ABYTES + 2 * BBYTES;
    static constexpr int WARP_BYTES = 2 * CHUNK;
    static constexpr int AL_BYTES = (kFwdTypes * kFwdTypes * NPN * 4 + 127) & ~127;
    static constexpr int A2_BYTES = kFwdTcWarps * NP * KM * 4;
    static constexpr int OPS = kFwdTcWarps * WARP_BYTES > A2_BYTES ? kFwdTcWarps * WARP_BYTES : A2_BYTES;
    // at least 46 KB, so that at most four CTAs (4 x 128 TMEM columns) share an SM
    static constexpr int SMEM = AL_BYTES + OPS > 47104 ? AL_BYTES + OPS : 47104;
    // lmax 6 or 7, where the tile's 64 rows are mostly in use, and 16 or more channels.  Each MMA
    // truncates its FP32 accumulation: descriptors of the liquid are 2.4e-7 (rms; 2.5e-6 at most)
    // of a column's largest off 64 bits, the FP32 pipe's 1.5e-7 (2.0e-6).  Smaller shapes, which
    // gain less, stay there (lmax 4 with two atoms per tile: 1.65 against 2.05 ms on the 1M-atom
    // glass)
    static constexpr bool fits = KM >= 49 && KM <= 64 && NP >= 16 && NPN <= 32;
};

__device__ __forceinline__ uint64_t tc_sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;  // descriptor version for this architecture; no swizzle
    return d;
}

// 8 FP32 values -> FP16 hi and lo images (16 bytes each, element 0 at the lowest address).
__device__ __forceinline__ void split_f16x8(const float* v, uint4& hi, uint4& lo) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const __half2 hh = __floats2half2_rn(v[2 * q], v[2 * q + 1]);
        const float2 hf = __half22float2(hh);
        const float2 lf = __ffma2_rn(hf, make_float2(-1.f, -1.f), make_float2(v[2 * q], v[2 * q + 1]));
        const __half2 ll = __floats2half2_rn(lf.x, lf.y);
        h[q] = *reinterpret_cast<const uint32_t*>(&hh);
        l[q] = *reinterpret_cast<const uint32_t*>(&ll);
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// Bound: instruction issue (1816 warp instructions per atom of 54 neighbours, 52 % of the slots;
// the operand splits and stores are a third).  Angle-free harmonics, a read-back by both halves
// of each warp, the spectrum by a thread per channel and the next atom's loads ahead of their
// use: 1024-structure batch 2.00 -> 1.32 ms, 32000-atom liquid 139 -> 97 us.

// TMEM lanes 0..15 of this warp's quarter, both halves of the warp reading: lanes 0..15 the
// columns from taddr, lanes 16..31 those from taddr + H (the next 4, 8 or 16 columns of each),
// waited for in the same statement.
template <int H>
__device__ __forceinline__ void tmem_ld_halves_wait(uint32_t taddr, float* v) {
    if constexpr (H <= 4) {
        uint32_t r[4];
        asm volatile("tcgen05.ld.sync.aligned.16x32bx2.x4.b32 {%0,%1,%2,%3}, [%4], %5;\n\t"
                     "tcgen05.wait::ld.sync.aligned;"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(taddr), "n"(H)
                     : "memory");
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = __uint_as_float(r[q]);
    } else if constexpr (H <= 8) {
        uint32_t r[8];
        asm volatile("tcgen05.ld.sync.aligned.16x32bx2.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8], %9;\n\t"
                     "tcgen05.wait::ld.sync.aligned;"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(taddr), "n"(H)
                     : "memory");
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = __uint_as_float(r[q]);
    } else {
        uint32_t r[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.16x32bx2.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16], "
            "%17;\n\t"
            "tcgen05.wait::ld.sync.aligned;"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
              "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(taddr), "n"(H)
            : "memory");
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = __uint_as_float(r[q]);
    }
}

template <int L, int NP, int N1>
__global__ void __launch_bounds__(32 * kFwdTcWarps, 4) k_sph_fwd_tc(DescArgs a) {
    using S = SphTcShape<L, NP>;
    constexpr int KM = S::KM, NPN = S::NPN;
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t mbar[kFwdTcWarps];
    __shared__ uint32_t s_tmem;
    __shared__ int s_cnt[kFwdTcWarps];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ntab = a.T * kFwdTypes * NPN;  // alpha[tc][tn][p], rows padded to NPN
    float* sAl = reinterpret_cast<float*>(smem);
    uint8_t* ops = smem + S::AL_BYTES;
    float* sA = reinterpret_cast<float*>(ops);  // [warp][NP][KM] once a round's MMAs are done
    for (int q = tid; q < ntab; q += blockDim.x) {
        const int row = q / NPN, p = q - row * NPN;
        sAl[q] = p < NP ? kTcScale * a.fwd_alpha[row * NP + p] : 0.f;
    }
    if (tid == 0) {
        for (int q = 0; q < kFwdTcWarps; ++q)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc::smem_u32(&mbar[q])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // alpha belongs to the model; TMEM is taken after the previous kernel (which may hold it) ends
    pdl_enter();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(&s_tmem)),
                     "r"(32 * kFwdTcWarps)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc::fence_async_smem();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tbase = s_tmem;
    const uint32_t mb = tc::smem_u32(&mbar[warp]);
    uint32_t phase = 0;
    bool ok = true;
    const int s0 = a.range[a.t0], nslot = a.range[a.t1] - s0;
    const int M = a.P.M;
    const float rc = a.rcut, irc = 1.f / a.rcut;
    uint8_t* wops = ops + warp * S::WARP_BYTES;
    const uint32_t wops_s = tc::smem_u32(wops);
    // kind::f16: D F32, A = B = F16, both MN-major, N = NPN, M = 64
    const uint32_t idesc = (1u << 4) | (1u << 15) | (1u << 16) | ((uint32_t)(NPN >> 3) << 17) | (4u << 24);
    const uint32_t dcol = tbase + 32u * warp;
    const int ch = lane >> 4, kk = lane & 15;
    uint8_t* cbase = wops + ch * S::CHUNK;
    const int aoff = (kk >> 3) * 1024 + (kk & 7) * 16;
    const int boff = (kk >> 3) * (NPN / 8) * 128 + (kk & 7) * 16;

    // the first neighbours of the next round's atom are loaded while this round computes
    int at = 0, tc = 0, cnt = 0;
    float4 d0 = make_float4(0.f, 0.f, 1.f, __int_as_float(1));
    const int rstep = gridDim.x * kFwdTcWarps;
    int r0 = blockIdx.x * kFwdTcWarps;
    if (r0 + warp < nslot) {
        at = a.perm[s0 + r0 + warp];
        tc = a.type[at] - 1;
        cnt = min(a.P.count[at], M);
        if (lane < cnt) d0 = a.P.dx[(size_t)at * M + lane];
    }
    for (; r0 < nslot; r0 += rstep) {
        if (lane == 0) s_cnt[warp] = cnt;
        int at_n = -1, tc_n = 0, cnt_n = 0;
        float4 dn = make_float4(0.f, 0.f, 1.f, __int_as_float(1));
        if (r0 + rstep + warp < nslot) at_n = a.perm[s0 + r0 + rstep + warp];
        const float* al = sAl + tc * kFwdTypes * NPN;
        for (int b0 = 0; b0 < cnt; b0 += 32) {
            const int k = b0 + lane;
            const float4 dl = d0;
            if (k + 32 < cnt) d0 = a.P.dx[(size_t)at * M + k + 32];  // the next step's
            float y[KM];
            float c[NPN];
            // a lane without a neighbour takes c = 0 and the harmonics of the z axis
            float4 d = make_float4(0.f, 0.f, 1.f, __int_as_float(1));
            float r = 1.f;
            bool valid = false;
            if (k < cnt) {
                d = dl;
                r = sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
                valid = r < rc;
            }
            {
                const int tn = __float_as_int(d.w) - 1;
                const float u = over_rc(r, rc, irc), fc1 = 1.f - u * u, fc2 = fc1 * fc1, fc = valid ? fc2 * fc2 : 0.f;
                float fT[N1];
                cheby_f<N1>(1.f - 2.f * u, fT);
                const float4* a4 = reinterpret_cast<const float4*>(al + tn * NPN);
#pragma unroll
                for (int q = 0; q < NPN / 4; ++q) {
                    const float4 v = a4[q];
                    const float w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int p = 4 * q + e;
                        c[p] = p < NP ? w4[e] * (fc * fT[p % N1]) : 0.f;
                    }
                }
                const float ir = 1.f / r;
                sph_cart<L, true>(d.x * ir, d.y * ir, d.z * ir, y);
            }
            // the warp's previous MMAs read these chunks
            if (b0 > 0) {
                ok = tc::mbar_wait(mb, phase) && ok;
                phase ^= 1;
            } else if (at_n >= 0) {
                tc_n = a.type[at_n] - 1;
                cnt_n = min(a.P.count[at_n], M);
            }
#pragma unroll
            for (int g = 0; g < S::NCA; ++g) {
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = 8 * g + e < KM ? y[8 * g + e] : 0.f;
                uint4 hi, lo;
                split_f16x8(v, hi, lo);
                *reinterpret_cast<uint4*>(cbase + g * 128 + aoff) = hi;
                *reinterpret_cast<uint4*>(cbase + S::ABYTES + g * 128 + aoff) = lo;
            }
#pragma unroll
            for (int g = 0; g < S::NCB; ++g) {
                uint4 hi, lo;
                split_f16x8(c + 8 * g, hi, lo);
                *reinterpret_cast<uint4*>(cbase + 2 * S::ABYTES + g * 128 + boff) = hi;
                *reinterpret_cast<uint4*>(cbase + 2 * S::ABYTES + S::BBYTES + g * 128 + boff) = lo;
            }
            tc::fence_async_smem();
            __syncwarp();
            if (lane == 0) {
                tc::fence_after();
                const int nch = min(2, (cnt - b0 + 15) >> 4);
                for (int q = 0; q < nch; ++q) {
                    const uint32_t cb = wops_s + q * S::CHUNK;
                    const uint64_t ah = tc_sdesc(cb, 1024, 128), alo = tc_sdesc(cb + S::ABYTES, 1024, 128);
                    const uint64_t bh = tc_sdesc(cb + 2 * S::ABYTES, (NPN / 8) * 128, 128);
                    const uint64_t bl = tc_sdesc(cb + 2 * S::ABYTES + S::BBYTES, (NPN / 8) * 128, 128);
                    tc::mma_bf16(dcol, ah, bh, idesc, (b0 > 0 || q > 0) ? 1u : 0u);
                    tc::mma_bf16(dcol, alo, bh, idesc, 1u);
                    tc::mma_bf16(dcol, ah, bl, idesc, 1u);
                }
                tc::mma_commit(mb);
            }
            __syncwarp();
        }
        if (at_n >= 0) {
            if (cnt == 0) {
                tc_n = a.type[at_n] - 1;
                cnt_n = min(a.P.count[at_n], M);
            }
            if (lane < cnt_n) dn = a.P.dx[(size_t)at_n * M + lane];
        }
        if (cnt > 0) {
            ok = tc::mbar_wait(mb, phase) && ok;
            phase ^= 1;
        }
        tc::fence_before();
        __syncthreads();
        tc::fence_after();
        // the 4 tiles: warp q reads rows lm = 16q + (lane & 15), lanes 0..15 the first half of the
        // columns and lanes 16..31 the second
        for (int w4 = 0; w4 < kFwdTcWarps; ++w4) {
            const int sl = r0 + w4;
            if (sl >= nslot) break;
            float v[S::NPH];
            tmem_ld_halves_wait<NPN / 2>(tbase + ((uint32_t)(32 * warp) << 16) + 32u * w4, v);
            const int lm = 16 * warp + (lane & 15), p0 = (lane >> 4) * (NPN / 2);
            if (lm < KM) {
                const bool any = s_cnt[w4] > 0;
                float* Aout = a.A + (size_t)sl * NP * KM + p0 * KM + lm;
                float* sa = sA + w4 * NP * KM + p0 * KM + lm;
#pragma unroll
                for (int p = 0; p < NPN / 2; ++p) {
                    if (p0 + p < NP) {
                        const float x = any ? v[p] * (1.f / kTcScale) : 0.f;
                        Aout[p * KM] = x;
                        sa[p * KM] = x;
                    }
                }
            }
        }
        __syncthreads();
        // power spectrum: a thread per (atom, channel)
        for (int e = tid; e < kFwdTcWarps * NP; e += blockDim.x) {
            const int w4 = e / NP, p = e - w4 * NP;
            const int sl = r0 + w4;
            if (sl >= nslot) continue;
            const float* row = sA + e * KM;
            float* out = a.fp + (size_t)(s0 + sl) * a.fp_stride + a.fp_off + p * a.sl;
#pragma unroll
            for (int l = 0; l <= L; ++l) {
                float s = 0.f;
#pragma unroll
                for (int m = 0; m <= 2 * l; ++m) s = fmaf(row[l * l + m], row[l * l + m], s);
                if (l < a.nl2) out[l] = kPi4 / (float)(2 * l + 1) * s;
            }
        }
        at = at_n;
        tc = tc_n;
        cnt = cnt_n;
        d0 = dn;
        tc::fence_before();
        __syncthreads();
        tc::fence_after();
    }
    if (!ok && lane == 0 && a.err) atomicOr(a.err, ERRBIT_TIMEOUT);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(32 * kFwdTcWarps)
                     : "memory");
}

template <int L, int NP, int N1>
cudaError_t launch_sph_fwd_tc(const DescArgs& a, cudaStream_t st) {
    using S = SphTcShape<L, NP>;
    const cudaError_t e = allow_smem(k_sph_fwd_tc<L, NP, N1>, S::SMEM);
    if (e != cudaSuccess) return e;
    const int rounds = (a.nmax + kFwdTcWarps - 1) / kFwdTcWarps;
    const int grid = rounds < 4 * a.tc_sms ? rounds : 4 * a.tc_sms;
    return launch_pdl(&k_sph_fwd_tc<L, NP, N1>, dim3(grid), dim3(32 * kFwdTcWarps), (size_t)S::SMEM, st, a);
}

}  // namespace
}  // namespace nnapgb

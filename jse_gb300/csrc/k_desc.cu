// Descriptor kernels (FP32): radial Chebyshev and spherical-Chebyshev power spectrum,
// forward (descriptors) and backward (pair gradients from dE/dfp).
//
// Mathematics restated from the reference (see the oracle for an FP64 copy):
//   x = 1 - 2r/rc, R_n = T_n(x), fc = (1 - (r/rc)^2)^4            nnap_util.hpp:226-271
//   Rnp[p] = sum_n W[t_i][t_j][p][n] R_n  (internal fuse matrix)    nnap_util.hpp:273-280
//   radial:     fp[p] = sum_j fc Rnp[p]                             basis_Chebyshev.hpp:82-133
//   spherical:  A[p][lm] = sum_j fc Rnp[p] Y_lm,
//               fp[p][l] = 4 pi/(2l+1) sum_m A[p][l,m]^2            basis_SphericalChebyshev.hpp:264-351
//   backward:   g_j = -dE_i/d(x_j - x_i) through fc, R_n, theta, phi  basis_SphericalChebyshev.hpp:353-525
// Real spherical harmonics use normalised associated Legendre functions with the
// Condon-Shortley phase, Y_{l,m>0} = sqrt2 P_lm cos(m phi), Y_{l,-m} = sqrt2 P_lm sin(m phi)
// (basis_SphericalUtil.hpp:12-101); dY/dtheta uses
//   dP_lm/dtheta = 1/2 [sqrt((l-m)(l+m+1)) P_{l,m+1} - sqrt((l+m)(l-m+1)) P_{l,m-1}],
// and the pole branch (dxy == 0) takes phi = 0 and drops the phi terms like
// calYPthetaPphi (basis_SphericalUtil.hpp:160-181).
//
// Layout: one warp per atom slot (atoms are processed in species-sorted slot order);
// forward lanes first evaluate one neighbour each into a shared-memory tile, then own
// columns lm of the P x K accumulator A; backward lanes own one neighbour each and
// stream G = dE/dA from shared memory.  The radial-fuse matrices of the basis live in
// shared memory for the whole block.  In mixed precision the spherical forward of the
// one-nonzero-per-row fuse matrices runs on the tensor cores (k_sph_tc.cuh).
#include <math_constants.h>

#include <algorithm>

#include "common.cuh"
#include "pdl.cuh"
#include "smem_limit.cuh"
#include "desc.cuh"
#include "sph_math.cuh"
#include "k_sph_tc.cuh"

namespace nnapgb {

cudaError_t upload_sh_constants() { return upload_sh_tables(); }

namespace {

constexpr int kDescMaxWarps = 8;  // warps per CTA are a launch parameter (2, 4 or 8)

__device__ __forceinline__ int atom_of(const DescArgs& a, int s0, int warp) { return a.perm[s0 + warp]; }

}  // namespace

// NEP type-wise cutoffs (find_descriptor, nep_core.hpp:1074-1082 and 1117-1125): a pair's
// radial functions use its own cutoff min(rc, (R_cov,i + R_cov,j) factor), and a pair at or
// beyond it adds nothing. Sets rc / irc to the pair's values; false when r is beyond them.
template <int RB>
__device__ __forceinline__ bool pair_cut(const DescArgs& a, int tc, int tn, float r, float& rc, float& irc) {
    if constexpr (RB == kRbNEP) {
        if (a.pair_rc) {
            const float2 q = a.pair_rc[tc * a.T + tn];
            rc = q.x;
            irc = q.y;
            return r < rc;
        }
    }
    return true;
}

// =========================================================================== radial
template <int NP, int N1, int RB>
__global__ void __launch_bounds__(32 * kDescMaxWarps) k_radial_fwd(DescArgs a) {
    pdl_enter();
    extern __shared__ float sW[];
    load_fuse<NP, N1>(a.W, sW, a.T);
    __syncthreads();
    const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int s0 = a.range[a.t0], s1 = a.range[a.t1];
    if (s0 + w >= s1) return;
    const int at = atom_of(a, s0, w);
    const int tc = a.type[at] - 1;
    const int M = a.P.M, cnt = min(a.P.count[at], M);
    const float rc = a.rcut, irc = 1.f / a.rcut;
    float acc[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) acc[p] = 0.f;
    for (int k = lane; k < cnt; k += 32) {
        const float4 d = a.P.dx[(size_t)at * M + k];
        const float r = sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
        if (r >= rc) continue;
        const int tn = __float_as_int(d.w) - 1;
        float rcp = rc, ircp = irc;
        if (!pair_cut<RB>(a, tc, tn, r, rcp, ircp)) continue;
        float T[N1], sv[NP];
        const float fc = radial_f<RB, N1>(r, rcp, ircp, T);
        fuse_apply<NP, N1>(sW + (size_t)(tc * a.T + tn) * NP * Fuse<N1>::N1P, T, sv);
#pragma unroll
        for (int p = 0; p < NP; ++p) acc[p] += fc * sv[p];
    }
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[p] += __shfl_xor_sync(0xffffffffu, acc[p], o);
    float* out = a.fp + (size_t)(s0 + w) * a.fp_stride + a.fp_off;
#pragma unroll
    for (int p = 0; p < NP; ++p)
        if (lane == (p & 31)) out[p] = acc[p];
}

template <int NP, int N1, int RB>
__global__ void __launch_bounds__(32 * kDescMaxWarps) k_radial_bwd(DescArgs a) {
    pdl_enter();
    extern __shared__ float sW[];
    load_fuse<NP, N1>(a.W, sW, a.T);
    __syncthreads();
    const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int s0 = a.range[a.t0], s1 = a.range[a.t1];
    if (s0 + w >= s1) return;
    const int at = atom_of(a, s0, w);
    const int tc = a.type[at] - 1;
    const int M = a.P.M, cnt = min(a.P.count[at], M);
    const float rc = a.rcut, irc = 1.f / a.rcut;
    const float* gf = a.gfp + (size_t)(s0 + w) * a.fp_stride + a.fp_off;
    float gfp[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) gfp[p] = gf[p];
    for (int k = lane; k < cnt; k += 32) {
        const size_t e = (size_t)at * M + k;
        const float4 d = a.P.dx[e];
        const float r = sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
        float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
        const int tn = __float_as_int(d.w) - 1;
        float rcp = rc, ircp = irc;
        if (r < rc && pair_cut<RB>(a, tc, tn, r, rcp, ircp)) {
            float T[N1], TG[N1], fcg;
            const float fc = radial_g<RB, N1>(r, rcp, ircp, T, TG, &fcg);
            float v[N1];
            fuse_apply_t<NP, N1>(sW + (size_t)(tc * a.T + tn) * NP * Fuse<N1>::N1P, gfp, v);
            float dfc = 0.f, drn = 0.f;
#pragma unroll
            for (int n = 0; n < N1; ++n) {
                dfc += v[n] * T[n];
                drn += v[n] * TG[n];
            }
            const float gr = dfc * fcg + fc * drn;
            g = make_float4(gr * d.x, gr * d.y, gr * d.z, 0.f);
        }
        if (a.accumulate) {
            float4 o = a.P.g[e];
            a.P.g[e] = make_float4(o.x + g.x, o.y + g.y, o.z + g.z, 0.f);
        } else {
            a.P.g[e] = g;
        }
    }
}

// =========================================================================== spherical
template <int L, int NP>
struct SphShape {
    static constexpr int K = (L + 1) * (L + 1);
    static constexpr int COLS = (K + 31) / 32;
    static constexpr int KS = K | 1;                 // odd row stride: conflict-free lane writes
    static constexpr int NPS = (NP + 3) & ~3;        // 16-byte rows for broadcast float4 reads
    static constexpr int FWD_WARP_FLOATS =
        (((32 * KS + 32 * NPS) > NP * K ? (32 * KS + 32 * NPS) : NP * K) + 3) & ~3;
    static constexpr int BWD_WARP_FLOATS = K * NPS + 2 * K * 32;
};

// Power spectrum of one atom from A [NP][K] in shared memory, a thread per channel: its K reads
// walk the row with the loop over l unrolled.  Rows of odd length (even L) meet no bank conflicts;
// those of odd L do, on NP K of the reads.
template <int L, int NP>
__device__ __forceinline__ void power_rows(const float* A, int nl2, int sl, float* __restrict__ out, int t, int nt) {
    constexpr int K = (L + 1) * (L + 1);
    for (int p = t; p < NP; p += nt) {
        const float* row = A + p * K;
#pragma unroll
        for (int l = 0; l <= L; ++l) {
            float s = 0.f;
#pragma unroll
            for (int m = 0; m <= 2 * l; ++m) s = fmaf(row[l * l + m], row[l * l + m], s);
            if (l < nl2) out[p * sl + l] = kPi4 / (float)(2 * l + 1) * s;
        }
    }
}

template <int L, int NP, int N1, int RB>
__global__ void __launch_bounds__(32 * kDescMaxWarps) k_sph_fwd(DescArgs a) {
    pdl_enter();
    using S = SphShape<L, NP>;
    extern __shared__ float smem[];
    const int nW = a.T * a.T * NP * Fuse<N1>::N1P;
    float* sW = smem;
    load_fuse<NP, N1>(a.W, sW, a.T);
    __syncthreads();
    const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int w = blockIdx.x * (blockDim.x >> 5) + wl;
    const int s0 = a.range[a.t0], s1 = a.range[a.t1];
    if (s0 + w >= s1) return;
    float* sY = smem + ((nW + 3) & ~3) + wl * S::FWD_WARP_FLOATS;  // [32][KS]
    float* sC = sY + 32 * S::KS;                                       // [32][NPS]
    const int at = atom_of(a, s0, w);
    const int tc = a.type[at] - 1;
    const int M = a.P.M, cnt = a.sub_dx ? a.sub_count[at] : min(a.P.count[at], M);
    const float4* rdx = (a.sub_dx ? a.sub_dx : a.P.dx) + (size_t)at * M;
    const float rc = a.rcut, irc = 1.f / a.rcut;
    // accumulators in packed pairs of channels (p = 2h, 2h + 1) for paired FP32 FMAs
    constexpr int NH = (NP + 1) / 2;
    float2 acc[NH][S::COLS];
#pragma unroll
    for (int h = 0; h < NH; ++h)
#pragma unroll
        for (int c = 0; c < S::COLS; ++c) acc[h][c] = make_float2(0.f, 0.f);
    for (int base = 0; base < cnt; base += 32) {
        const int k = base + lane;
        float c[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) c[p] = 0.f;
        float* y = sY + lane * S::KS;
        bool valid = false;
        if (k < cnt) {
            const float4 d = rdx[k];
            const float r = sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
            const int tn = __float_as_int(d.w) - 1;
            float rcp = rc, ircp = irc;
            if (r < rc && pair_cut<RB>(a, tc, tn, r, rcp, ircp)) {
                valid = true;
                float T[N1], sv[NP];
                const float fc = radial_f<RB, N1>(r, rcp, ircp, T);
                fuse_apply<NP, N1>(sW + (size_t)(tc * a.T + tn) * NP * Fuse<N1>::N1P, T, sv);
#pragma unroll
                for (int p = 0; p < NP; ++p) c[p] = fc * sv[p];
                const Angles an = angles_f(d.x, d.y, d.z, r);
                sph_harm<L, false>(an, y, nullptr, 1);
            }
        }
        if (!valid)
#pragma unroll
            for (int q = 0; q < S::K; ++q) y[q] = 0.f;
#pragma unroll
        for (int p = 0; p < S::NPS; ++p) sC[lane * S::NPS + p] = p < NP ? c[p] : 0.f;
        __syncwarp();
        const int nk = min(32, cnt - base);
#pragma unroll 4
        for (int kk = 0; kk < nk; ++kk) {
            float2 cv[NH];
            const float4* crow = reinterpret_cast<const float4*>(sC + kk * S::NPS);
#pragma unroll
            for (int q = 0; q < S::NPS / 4; ++q) {
                const float4 v = crow[q];
                if (2 * q < NH) cv[2 * q] = make_float2(v.x, v.y);
                if (2 * q + 1 < NH) cv[2 * q + 1] = make_float2(v.z, v.w);
            }
            const float* yrow = sY + kk * S::KS;
#pragma unroll
            for (int col = 0; col < S::COLS; ++col) {
                const int lm = lane + 32 * col;
                const float yv = lm < S::K ? yrow[lm] : 0.f;
                const float2 yy = make_float2(yv, yv);
#pragma unroll
                for (int h = 0; h < NH; ++h) acc[h][col] = __ffma2_rn(cv[h], yy, acc[h][col]);
            }
        }
        __syncwarp();
    }
    // A to global (backward input) and to shared memory for the power spectrum
    float* Aout = a.A + (size_t)w * NP * S::K;
    float* sA = sY;
#pragma unroll
    for (int col = 0; col < S::COLS; ++col) {
        const int lm = lane + 32 * col;
        if (lm < S::K)
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                const float v = (p & 1) ? acc[p >> 1][col].y : acc[p >> 1][col].x;
                Aout[p * S::K + lm] = v;
                sA[p * S::K + lm] = v;
            }
    }
    __syncwarp();
    power_rows<L, NP>(sA, a.nl2, a.sl, a.fp + (size_t)(s0 + w) * a.fp_stride + a.fp_off, lane, 32);
}

// Forward in the space of the radial functions, for at most kFwdTypes species and fuse
// matrices whose row p has its only nonzero in column p mod N1 (every weight type but
// rfuse): W[tc][tn][p][n] = alpha[tc][tn][p] delta(n, p mod N1).  Per neighbour species
// tn the warp accumulates
//   Ah[tn][n][lm] = sum_{j of species tn} fc_j T_n(r_j) Y_j[lm]
// (N1 instead of NP products per neighbour and lm; the neighbour's species is uniform
// across the warp in the accumulation loop, so the branch does not diverge), then
//   A[p][lm] = sum_tn alpha[tc][tn][p] Ah[tn][p mod N1][lm]
// straight from the accumulator registers.  fc Rnp is never formed.
template <int L, int NP, int N1>
struct SphFNShape {
    static constexpr int K = (L + 1) * (L + 1);
    static constexpr int COLS = (K + 31) / 32;
    static constexpr int KS = K | 1;
    static constexpr int N1P = (N1 + 3) & ~3;
    static constexpr int H = (N1 + 1) / 2;
    static constexpr int EVAL = 32 * KS + 32 * N1P + 32;   // Y, fc T, species
    static constexpr int POST = NP * K;                     // A^2
    static constexpr int WARP_FLOATS = ((EVAL > POST ? EVAL : POST) + 3) & ~3;
};

// 1M-atom glass (lmax 4) 2.51 -> 2.04 ms with the angle-free harmonics and the spectrum by a
// thread per channel (1513 warp instructions per atom of 40 neighbours; the shared-memory path is
// 77 % busy: 131072 atoms).
template <int L, int NP, int N1>
__global__ void __launch_bounds__(32 * kDescMaxWarps) k_sph_fwd_n(DescArgs a) {
    using S = SphFNShape<L, NP, N1>;
    extern __shared__ float smem[];
    const int T = a.T;
    const int ntab = T * kFwdTypes * NP;  // alpha[tc][tn][p], zero for tn >= T
    float* sAl = smem;
    for (int q = threadIdx.x; q < ntab; q += blockDim.x) sAl[q] = a.fwd_alpha[q];
    pdl_enter();  // alpha belongs to the model
    __syncthreads();
    const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int w = blockIdx.x * (blockDim.x >> 5) + wl;
    const int s0 = a.range[a.t0], s1 = a.range[a.t1];
    if (s0 + w >= s1) return;
    float* base = smem + ((ntab + 3) & ~3) + (size_t)wl * S::WARP_FLOATS;
    float* sY = base;                                       // [32][KS]
    float* sF = sY + 32 * S::KS;                            // [32][N1P] fc T_n
    int* sTn = reinterpret_cast<int*>(sF + 32 * S::N1P);    // [32]
    const int at = a.perm[s0 + w];
    const int tc = a.type[at] - 1;
    const int M = a.P.M, cnt = min(a.P.count[at], M);
    const float rc = a.rcut, irc = 1.f / a.rcut;
    float2 acc[kFwdTypes][S::H][S::COLS];
#pragma unroll
    for (int t = 0; t < kFwdTypes; ++t)
#pragma unroll
        for (int h = 0; h < S::H; ++h)
#pragma unroll
            for (int c = 0; c < S::COLS; ++c) acc[t][h][c] = make_float2(0.f, 0.f);
    for (int b0 = 0; b0 < cnt; b0 += 32) {
        const int k = b0 + lane;
        float fT[S::N1P];
#pragma unroll
        for (int n = 0; n < S::N1P; ++n) fT[n] = 0.f;
        float* y = sY + lane * S::KS;
        int tn = 0;
        bool valid = false;
        if (k < cnt) {
            const float4 d = a.P.dx[(size_t)at * M + k];
            const float r = sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
            if (r < rc) {
                valid = true;
                tn = __float_as_int(d.w) - 1;
                const float u = over_rc(r, rc, irc), fc1 = 1.f - u * u, fc2 = fc1 * fc1, fc = fc2 * fc2;
                cheby_f<N1>(1.f - 2.f * u, fT);
#pragma unroll
                for (int n = 0; n < N1; ++n) fT[n] *= fc;
                const float ir = 1.f / r;
                sph_cart<L, false>(d.x * ir, d.y * ir, d.z * ir, y);
            }
        }
        if (!valid)
#pragma unroll 7
            for (int q = 0; q < S::K; ++q) y[q] = 0.f;
        float4* frow = reinterpret_cast<float4*>(sF + lane * S::N1P);
#pragma unroll
        for (int q = 0; q < S::N1P / 4; ++q) frow[q] = make_float4(fT[4 * q], fT[4 * q + 1], fT[4 * q + 2], fT[4 * q + 3]);
        sTn[lane] = tn;
        __syncwarp();
        const int nk = min(32, cnt - b0);
        // unrolled so the loads of the next neighbours overlap the FMAs of this one
#pragma unroll 4
        for (int kk = 0; kk < nk; ++kk) {
            float2 f2[S::N1P / 2];
            const float4* fr = reinterpret_cast<const float4*>(sF + kk * S::N1P);
#pragma unroll
            for (int q = 0; q < S::N1P / 4; ++q) {
                const float4 v = fr[q];
                f2[2 * q] = make_float2(v.x, v.y);
                f2[2 * q + 1] = make_float2(v.z, v.w);
            }
            float2 yy[S::COLS];
#pragma unroll
            for (int col = 0; col < S::COLS; ++col) {
                const int lm = lane + 32 * col;
                const float yv = lm < S::K ? sY[kk * S::KS + lm] : 0.f;
                yy[col] = make_float2(yv, yv);
            }
            const int t = sTn[kk];
#pragma unroll
            for (int tt = 0; tt < kFwdTypes; ++tt) {
                if (t != tt) continue;  // uniform across the warp
#pragma unroll
                for (int h = 0; h < S::H; ++h)
#pragma unroll
                    for (int col = 0; col < S::COLS; ++col) acc[tt][h][col] = __ffma2_rn(f2[h], yy[col], acc[tt][h][col]);
            }
        }
        __syncwarp();
    }
    // A from the accumulators and alpha, to global memory and to shared memory
    float* sA = base;
    float* Aout = a.A + (size_t)w * NP * S::K;
    const float* al = sAl + (size_t)tc * kFwdTypes * NP;
#pragma unroll
    for (int col = 0; col < S::COLS; ++col) {
        const int lm = lane + 32 * col;
        if (lm < S::K) {
            const float4 nlm = d_shN[lm];  // the factor that Y left out
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                const int n = p % N1;  // a constant once the loop is unrolled
                float v = 0.f;
#pragma unroll
                for (int t = 0; t < kFwdTypes; ++t)
                    v += al[t * NP + p] * ((n & 1) ? acc[t][n >> 1][col].y : acc[t][n >> 1][col].x);
                v = fmaf(v, nlm.x, v * nlm.y);
                Aout[p * S::K + lm] = v;
                sA[p * S::K + lm] = v;
            }
        }
    }
    __syncwarp();
    power_rows<L, NP>(sA, a.nl2, a.sl, a.fp + (size_t)(s0 + w) * a.fp_stride + a.fp_off, lane, 32);
}

// Backward, one warp per atom slot, one neighbour per lane.  For each neighbour,
//   dY_lm = sum_p c_p G[p][lm]        (chain into theta and phi),
//   dc_p  = sum_lm G[p][lm] Y_lm      (chain into fc and the radial functions),
// with c_p = fc Rnp_p.  G rows are read from shared memory as broadcast float4 loads;
// Y and dY/dtheta of the lane's neighbour sit in a lane column of shared memory.  Only
// c and dc stay live through the lm loop: the radial sums are formed again afterwards
// as v_n = sum_p dc_p W[p][n], so dfc = v . T and drn = v . dT.  Registers stay at or
// below 128 per thread (four CTAs of four warps per SM).
template <int L, int NP, int N1, int RB>
__global__ void __launch_bounds__(32 * kDescMaxWarps, 2) k_sph_bwd(DescArgs a) {
    pdl_enter();
    using S = SphShape<L, NP>;
    extern __shared__ float smem[];
    const int nW = a.T * a.T * NP * Fuse<N1>::N1P;
    float* sW = smem;
    load_fuse<NP, N1>(a.W, sW, a.T);
    __syncthreads();
    const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int w = blockIdx.x * (blockDim.x >> 5) + wl;
    const int s0 = a.range[a.t0], s1 = a.range[a.t1];
    if (s0 + w >= s1) return;
    float* sG = smem + nW + wl * S::BWD_WARP_FLOATS;  // [K][NPS]
    float* sY = sG + S::K * S::NPS;                  // [K][32]
    float* sYt = sY + S::K * 32;                     // [K][32]
    const int at = atom_of(a, s0, w);
    const int tc = a.type[at] - 1;
    const int M = a.P.M, cnt = a.sub_dx ? a.sub_count[at] : min(a.P.count[at], M);
    const float4* rdx = (a.sub_dx ? a.sub_dx : a.P.dx) + (size_t)at * M;
    const float rc = a.rcut, irc = 1.f / a.rcut;
    // G[p][lm] = 2 * 4pi/(2l+1) * dE/dfp[p][l] * A[p][lm], stored transposed
    {
        const float* Ain = a.A + (size_t)w * NP * S::K;
        const float* gf = a.gfp + (size_t)(s0 + w) * a.fp_stride + a.fp_off;
        for (int lm = lane; lm < S::K; lm += 32) {
            int l = 0;
            while ((l + 1) * (l + 1) <= lm) ++l;
            const float coef = l < a.nl2 ? 2.f * kPi4 / (float)(2 * l + 1) : 0.f;
            const int lc = l < a.nl2 ? l : 0;
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                float v = coef * gf[p * a.sl + lc] * Ain[p * S::K + lm];
                if (a.Gx) v += a.Gx[(size_t)w * NP * S::K + p * S::K + lm];
                sG[lm * S::NPS + p] = v;
            }
#pragma unroll
            for (int p = NP; p < S::NPS; ++p) sG[lm * S::NPS + p] = 0.f;
        }
        __syncwarp();
    }
    for (int base = 0; base < cnt; base += 32) {
        const int k = base + lane;
        float c[NP];
        float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
        float r = 1.f, rcp = rc, ircp = irc;
        bool valid = false;
        if (k < cnt) {
            d = rdx[k];
            r = sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
            valid = r < rc;
        }
        const int tn = valid ? __float_as_int(d.w) - 1 : 0;
        if (valid) valid = pair_cut<RB>(a, tc, tn, r, rcp, ircp);
        const float* Wt = sW + (size_t)(tc * a.T + tn) * NP * Fuse<N1>::N1P;
        if (valid) {
            float T[N1], sv[NP];
            const float fc = radial_f<RB, N1>(r, rcp, ircp, T);
            fuse_apply<NP, N1>(Wt, T, sv);
#pragma unroll
            for (int p = 0; p < NP; ++p) c[p] = fc * sv[p];
            const Angles an = angles_f(d.x, d.y, d.z, r);
            sph_harm<L, true>(an, sY + lane, sYt + lane, 32);
        } else {
#pragma unroll
            for (int p = 0; p < NP; ++p) c[p] = 0.f;
#pragma unroll 7
            for (int q = 0; q < S::K; ++q) { sY[q * 32 + lane] = 0.f; sYt[q * 32 + lane] = 0.f; }
        }
        // c and dc in packed channel pairs (p = 2h, 2h + 1); padded G columns are zero
        constexpr int NH = (NP + 1) / 2;
        float2 c2[NH], dc2[NH];
#pragma unroll
        for (int h = 0; h < NH; ++h) {
            c2[h] = make_float2(c[2 * h], 2 * h + 1 < NP ? c[2 * h + 1] : 0.f);
            dc2[h] = make_float2(0.f, 0.f);
        }
        float gth = 0.f, gph = 0.f;
        // one G row: returns dY_lm and adds G[.][lm] * Y_lm into dc
        auto row = [&](int lm) -> float {
            const float4* gr = reinterpret_cast<const float4*>(sG + lm * S::NPS);
            const float yv = sY[lm * 32 + lane];
            const float2 yy = make_float2(yv, yv);
            // two independent partial sums keep the dependent FMA chain short
            float2 dYa = make_float2(0.f, 0.f), dYb = make_float2(0.f, 0.f);
#pragma unroll
            for (int q = 0; q < S::NPS / 4; ++q) {
                const float4 g = gr[q];
                if (2 * q < NH) {
                    const float2 ga = make_float2(g.x, g.y);
                    dYa = __ffma2_rn(c2[2 * q], ga, dYa);
                    dc2[2 * q] = __ffma2_rn(ga, yy, dc2[2 * q]);
                }
                if (2 * q + 1 < NH) {
                    const float2 gb = make_float2(g.z, g.w);
                    dYb = __ffma2_rn(c2[2 * q + 1], gb, dYb);
                    dc2[2 * q + 1] = __ffma2_rn(gb, yy, dc2[2 * q + 1]);
                }
            }
            return (dYa.x + dYb.x) + (dYa.y + dYb.y);
        };
#pragma unroll 1
        for (int l = 0; l <= L; ++l) {
            const int c0 = l * l + l;
            gth += row(c0) * sYt[c0 * 32 + lane];
#pragma unroll 1
            for (int m = 1; m <= l; ++m) {
                const float dYp = row(c0 + m);
                const float dYm = row(c0 - m);
                gth += dYp * sYt[(c0 + m) * 32 + lane] + dYm * sYt[(c0 - m) * 32 + lane];
                gph += (float)m * (dYm * sY[(c0 + m) * 32 + lane] - dYp * sY[(c0 - m) * 32 + lane]);
            }
        }
        if (k < cnt) {
            const size_t e = (size_t)at * M + (a.sub_dx ? a.sub_pos[(size_t)at * M + k] : k);
            float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
            if (valid) {
                float T[N1], TG[N1], v[N1], fcg;
                const float fc = radial_g<RB, N1>(r, rcp, ircp, T, TG, &fcg);
                float dc[NP];
#pragma unroll
                for (int p = 0; p < NP; ++p) dc[p] = (p & 1) ? dc2[p >> 1].y : dc2[p >> 1].x;
                fuse_apply_t<NP, N1>(Wt, dc, v);
                float dfc = 0.f, drn = 0.f;
#pragma unroll
                for (int n = 0; n < N1; ++n) {
                    dfc += v[n] * T[n];
                    drn += v[n] * TG[n];
                }
                const float gr = dfc * fcg + fc * drn;
                const Angles an = angles_f(d.x, d.y, d.z, r);
                const float ir = 1.f / r;
                const float tpx = -an.ct * an.cp * ir, tpy = -an.ct * an.sp * ir, tpz = an.st * ir;
                const float ppx = an.pole ? 0.f : an.sp / an.dxy, ppy = an.pole ? 0.f : -an.cp / an.dxy;
                g.x = gr * d.x + gth * tpx + gph * ppx;
                g.y = gr * d.y + gth * tpy + gph * ppy;
                g.z = gr * d.z + gth * tpz;
            }
            if (a.accumulate) {
                if (valid) {
                    const float4 o = a.P.g[e];
                    a.P.g[e] = make_float4(o.x + g.x, o.y + g.y, o.z + g.z, 0.f);
                }
            } else {
                a.P.g[e] = g;
            }
        }
        __syncwarp();
    }
}

// Backward in the space of the radial functions (used when every column of the fuse
// matrices has at most kNz nonzero rows, e.g. the default, none, full, exfull and fuse weight
// types).  With Gh[tn][lm][n] = sum_p W[tc][tn][p][n] G[p][lm], formed once per atom,
//   dY_lm = sum_p c_p G[p][lm] = fc sum_n T_n Gh[tn][lm][n],
//   v_n   = sum_p W[p][n] dc_p = sum_lm Gh[tn][lm][n] Y_lm,
// so the per-neighbour products run over N1 instead of NP channels, and c, dc are never
// formed.  The harmonics are the monic ones of sph_math.cuh (their factors N_lm are in the Gh
// rows), walked column by column in m with everything in registers; the gradient is taken in
// Cartesian form: with a_m = sum_l Q_lm dY_lm, b_m = sum_l Q_lm dY_l,-m and a'_m, b'_m the same
// sums over dQ_lm/dz, and c_m + i s_m = (x + iy)^m,
//   d/dz = sum_m a'_m c_m + b'_m s_m,   d/dx = sum_m m (a_m c_{m-1} + b_m s_{m-1}),
//   d/dy = sum_m m (b_m c_{m-1} - a_m s_{m-1}),
// projected onto the sphere at the end.  Rows l,m and l,-m (and two rows of m = 0) sit side by
// side as float2 in shared memory, so one paired FMA serves both.
//
// Every lane reads N1 (L+1)^2 floats of Gh for each neighbour, and shared memory returns 128
// bytes per cycle and SM: that path is 84 % busy (the FMA pipe 52 %; 32000 atoms), against the angle-based
// walk with stored Legendre columns before, which issued twice the instructions.  1024-structure
// batch (488206 atoms, lmax 6) 2.55 -> 1.98 ms, 1M-atom glass (lmax 4) 3.19 -> 1.76 ms, 32000-atom
// liquid 174 -> 139 us.  Two neighbours of one species per lane halve the reads but leave 11
// warps per SM (165 registers): 2.45 ms on the batch.
// Fuse rows that are not diagonal, and those of more than kFwdTypes species, are read in sparse
// form as each atom needs them: its species' part is a few KB, the whole table 2 T^2 N1 kNz words,
// which a CTA of four atoms copied to shared memory and kept (lmax 6, nmax 8, 20000 atoms: eight
// species 322 -> 207 us, ten 600 -> 291, fifteen 1110 -> 527).
template <int L, int NP, int N1>
struct SphNShape {
    static constexpr int K = (L + 1) * (L + 1);
    static constexpr int NZ = (L + 2) / 2;                 // row pairs of m = 0: (0,1), (2,3), ..
    static constexpr int NS = NZ + L * (L + 1) / 2;        // and of (l, +-m), m ascending
    static constexpr int RF = (2 * N1 + 3) & ~3;           // floats of a row pair
    // floats of one neighbour species, an odd number of 16-byte words: lanes of different
    // species read different banks
    static constexpr int GH = (NS * RF / 4) % 2 ? NS * RF : NS * RF + 4;
    static int warp_floats(int T, int apw, bool diag) { return apw * (T * GH + (diag ? 0 : (NP * K + 3) / 4 * 4)); }
};

// First row pair of column m >= 1 (row pair of l = m).
template <int L>
__host__ __device__ constexpr int pair_start(int m) {
    int s = (L + 2) / 2;
    for (int q = 1; q < m; ++q) s += L - q + 1;
    return s;
}

// sum_n T_n Gh[n] of a row pair, and v_n += Gh[n] Y: the two contractions of the backward.
template <int N1>
__device__ __forceinline__ float2 gh_row(const float* __restrict__ gh, const float2* T2, float2 y2, float2* v2) {
    float2 dy = make_float2(0.f, 0.f);
    const float4* gr = reinterpret_cast<const float4*>(gh);
#pragma unroll
    for (int q = 0; q < N1 / 2; ++q) {
        const float4 g = gr[q];
        const float2 ga = make_float2(g.x, g.y), gb = make_float2(g.z, g.w);
        dy = __ffma2_rn(T2[2 * q], ga, dy);
        v2[2 * q] = __ffma2_rn(ga, y2, v2[2 * q]);
        dy = __ffma2_rn(T2[2 * q + 1], gb, dy);
        v2[2 * q + 1] = __ffma2_rn(gb, y2, v2[2 * q + 1]);
    }
    if (N1 & 1) {
        const float2 ga = *reinterpret_cast<const float2*>(gh + 2 * (N1 - 1));
        dy = __ffma2_rn(T2[N1 - 1], ga, dy);
        v2[N1 - 1] = __ffma2_rn(ga, y2, v2[N1 - 1]);
    }
    return dy;
}

// Columns m .. L of the walk: q is column m, (cm, sm) = (x + iy)^m, (cp, sp) the power before.
template <int L, int N1, int m>
__device__ __forceinline__ void bwd_columns(const float* __restrict__ gh, const float2* T2, float2* v2, float x, float y,
                                            float z, const float* q, float cm, float sm, float cp, float sp, float& gx,
                                            float& gy, float& gz) {
    constexpr int RF = (2 * N1 + 3) & ~3;
    float qn[L + 2];  // column m + 1
    if constexpr (m < L) monic_column<L, m + 1>(z, qn);
    float2 ab = make_float2(0.f, 0.f), abz = make_float2(0.f, 0.f);
    const float2 cs = make_float2(cm, sm);
#pragma unroll
    for (int l = m; l <= L; ++l) {
        const float2 q2 = make_float2(q[l], q[l]);
        const float2 y2 = l == m ? cs : __fmul2_rn(q2, cs);
        const float2 dy = gh_row<N1>(gh + (pair_start<L>(m) + l - m) * RF, T2, y2, v2);
        if (l == m) {
            ab = dy;
        } else {
            const float dq = (float)(l - m) * qn[l];
            ab = __ffma2_rn(q2, dy, ab);
            abz = __ffma2_rn(make_float2(dq, dq), dy, abz);
        }
    }
    if (m < L) gz = fmaf(abz.x, cm, fmaf(abz.y, sm, gz));
    gx = fmaf((float)m, fmaf(ab.x, cp, ab.y * sp), gx);
    gy = fmaf((float)m, fmaf(ab.y, cp, -(ab.x * sp)), gy);
    if constexpr (m < L)
        bwd_columns<L, N1, m + 1>(gh, T2, v2, x, y, z, qn, fmaf(x, cm, -(y * sm)), fmaf(x, sm, y * cm), cm, sm, gx, gy,
                                  gz);
}

// LPA lanes serve one atom (32 / LPA atoms per warp).  96 registers (20 warps per SM) with 32
// lanes, 80 (24 warps) with 16: each was the faster of the two for its shapes.
constexpr int kBwdWarps = 4;  // most warps per CTA
template <int L, int NP, int N1, int LPA>
__global__ void __launch_bounds__(32 * kBwdWarps, LPA == 32 ? 5 : 6) k_sph_bwd_n(DescArgs a) {
    using S = SphNShape<L, NP, N1>;
    constexpr int APW = 32 / LPA;
    extern __shared__ __align__(16) float smem[];
    const int T = a.T;
    // per row pair: N_lm of its two rows, and N_lm 2 4pi/(2l+1) (zero where there is no row or
    // no power-spectrum column)
    float2* sN = reinterpret_cast<float2*>(smem);
    float2* sCo = sN + S::NS;
    const bool diag = a.fwd_alpha != nullptr && T <= kFwdTypes;
    float* tab = smem + ((4 * S::NS + 3) & ~3);
    const int nal = diag ? T * kFwdTypes * NP : 0;
    float* sAl = tab;  // alpha[tc][tn][p] of fuse rows with their one nonzero in column p mod N1
    for (int q = threadIdx.x; q < nal; q += blockDim.x) sAl[q] = a.fwd_alpha[q];
    for (int s = threadIdx.x; s < S::NS; s += blockDim.x) {
        int l0, l1, m = 0;
        if (s < S::NZ) {
            l0 = 2 * s;
            l1 = 2 * s + 1;
        } else {
            int t = s - S::NZ;
            for (m = 1; t >= L - m + 1; ++m) t -= L - m + 1;
            l0 = l1 = m + t;
        }
        const float4 n0 = d_shN[l0 * l0 + l0 + m], n1 = d_shN[l1 <= L ? l1 * l1 + l1 + m : 0];
        sN[s] = make_float2(n0.x, l1 <= L ? n1.x : 0.f);
        sCo[s] = make_float2(l0 < a.nl2 ? n0.z : 0.f, l1 <= L && l1 < a.nl2 ? n1.z : 0.f);
    }
    pdl_enter();  // the tables above belong to the model: only what follows needs the previous kernel
    __syncthreads();
    const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = lane / LPA, sub = lane % LPA;
    const int w0 = (blockIdx.x * (blockDim.x >> 5) + wl) * APW, w = w0 + grp;
    const int s0 = a.range[a.t0], s1 = a.range[a.t1];
    if (s0 + w0 >= s1) return;
    const bool act = s0 + w < s1;
    float* sGh = tab + (nal + 3) / 4 * 4 + (size_t)(wl * APW + grp) * (T * S::GH + (diag ? 0 : (NP * S::K + 3) / 4 * 4));
    const int at = a.perm[act ? s0 + w : s0 + w0];
    const int tc = a.type[at] - 1;
    const int M = a.P.M, cnt = act ? min(a.P.count[at], M) : 0;
    int cmax = cnt;
    if (APW > 1) cmax = __reduce_max_sync(0xffffffffu, cnt);
    const float rc = a.rcut, irc = 1.f / a.rcut;
    if (act) {
        // G[p][lm] = 2 4pi/(2l+1) dE/dfp[p][l] A[p][lm] (+ the invariant columns' part) times N_lm,
        // in row pairs; lanes over row pairs
        const float* Ain = a.A + (size_t)w * NP * S::K;
        const float* Gx = a.Gx ? a.Gx + (size_t)w * NP * S::K : nullptr;
        const float* gf = a.gfp + (size_t)(s0 + w) * a.fp_stride + a.fp_off;
        for (int s = sub; s < S::NS; s += LPA) {
            int l0, l1, k0, k1;
            if (s < S::NZ) {
                l0 = 2 * s;
                l1 = min(2 * s + 1, L);
                k0 = l0 * l0 + l0;
                k1 = l1 * l1 + l1;
            } else {
                int t = s - S::NZ, m = 1;
                for (; t >= L - m + 1; ++m) t -= L - m + 1;
                l0 = l1 = m + t;
                k0 = l0 * l0 + l0 + m;
                k1 = l0 * l0 + l0 - m;
            }
            const float2 co = sCo[s], nm = sN[s];
            l0 = l0 < a.nl2 ? l0 : 0;
            l1 = l1 < a.nl2 ? l1 : 0;
            float2 g[NP];
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                g[p] = make_float2(co.x * gf[p * a.sl + l0] * Ain[p * S::K + k0],
                                   co.y * gf[p * a.sl + l1] * Ain[p * S::K + k1]);
                if (Gx) {
                    g[p].x += nm.x * Gx[p * S::K + k0];
                    g[p].y += nm.y * Gx[p * S::K + k1];
                }
            }
            if (diag) {
                for (int tn = 0; tn < T; ++tn) {
                    const float* al = sAl + (tc * kFwdTypes + tn) * NP;
                    float4* out = reinterpret_cast<float4*>(sGh + tn * S::GH + s * S::RF);
#pragma unroll
                    for (int q = 0; q < S::RF / 4; ++q) {
                        float2 v[2];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            v[h] = make_float2(0.f, 0.f);
                            const int n = 2 * q + h;
                            if (n < N1) {
#pragma unroll
                                for (int p = n; p < NP; p += N1) v[h] = __ffma2_rn(make_float2(al[p], al[p]), g[p], v[h]);
                            }
                        }
                        out[q] = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
                    }
                }
            } else {  // G transposed to [p][lm] in scratch
                float* scr = sGh + T * S::GH;
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    if (s >= S::NZ || 2 * s + 1 <= L) scr[p * S::K + k1] = g[p].y;
                    scr[p * S::K + k0] = g[p].x;
                }
            }
        }
    }
    __syncwarp();
    if (!diag) {
        if (act) {
            const float* scr = sGh + T * S::GH;
            for (int idx = sub; idx < T * S::NS; idx += LPA) {
                const int tn = idx / S::NS, s = idx - tn * S::NS;
                int k0, k1;
                if (s < S::NZ) {
                    const int l1 = min(2 * s + 1, L);
                    k0 = 4 * s * s + 2 * s;
                    k1 = 2 * s + 1 <= L ? l1 * l1 + l1 : -1;
                } else {
                    int t = s - S::NZ, m = 1;
                    for (; t >= L - m + 1; ++m) t -= L - m + 1;
                    const int l = m + t;
                    k0 = l * l + l + m;
                    k1 = l * l + l - m;
                }
                // the sparse rows of (tc, tn), kNz = 4 words each
                const int4* np4 = reinterpret_cast<const int4*>(a.nz_p) + (size_t)(tc * T + tn) * N1;
                const float4* nw4 = reinterpret_cast<const float4*>(a.nz_w) + (size_t)(tc * T + tn) * N1;
                float* out = sGh + tn * S::GH + s * S::RF;
#pragma unroll
                for (int n = 0; n < N1; ++n) {
                    float vx = 0.f, vy = 0.f;
                    const int4 p4 = np4[n];
                    const float4 w4 = nw4[n];
                    const int pz[kNz] = {p4.x, p4.y, p4.z, p4.w};
                    const float wz[kNz] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                    for (int z = 0; z < kNz; ++z) {
                        if (pz[z] >= 0) {
                            vx += wz[z] * scr[pz[z] * S::K + k0];
                            if (k1 >= 0) vy += wz[z] * scr[pz[z] * S::K + k1];
                        }
                    }
                    *reinterpret_cast<float2*>(out + 2 * n) = make_float2(vx, vy);
                }
            }
        }
        __syncwarp();
    }
    for (int base = 0; base < cmax; base += LPA) {
        const int k = base + sub;
        float4 d = make_float4(0.f, 0.f, 1.f, 0.f);
        bool valid = false;
        float r = 1.f;
        if (k < cnt) {
            d = a.P.dx[(size_t)at * M + k];
            r = sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
            valid = r < rc;
        }
        const int tn = valid ? __float_as_int(d.w) - 1 : 0;
        const float ir = 1.f / r, x = d.x * ir, y = d.y * ir, z = d.z * ir;
        const float u = over_rc(r, rc, irc), tx = 1.f - 2.f * u;
        float Tn[N1];
        cheby_f<N1>(tx, Tn);
        float2 T2[N1], v2[N1];
#pragma unroll
        for (int n = 0; n < N1; ++n) {
            T2[n] = make_float2(Tn[n], Tn[n]);
            v2[n] = make_float2(0.f, 0.f);
        }
        const float* gh = sGh + tn * S::GH;
        float gx = 0.f, gy = 0.f, gz;
        {
            float q0[L + 2], q1[L + 2];
            monic_column<L, 0>(z, q0);
            q0[L + 1] = 0.f;
            q1[0] = 0.f;
            if constexpr (L >= 1) monic_column<L, 1>(z, q1);
            q1[L + 1] = 0.f;
            float2 az = make_float2(0.f, 0.f);
#pragma unroll
            for (int s = 0; s < S::NZ; ++s) {
                const int l = 2 * s;
                const float2 dy = gh_row<N1>(gh + s * S::RF, T2, make_float2(q0[l], q0[l + 1]), v2);
                az = __ffma2_rn(make_float2((float)l * q1[l], (float)(l + 1) * q1[l + 1]), dy, az);
            }
            gz = az.x + az.y;
            if constexpr (L >= 1) bwd_columns<L, N1, 1>(gh, T2, v2, x, y, z, q1, x, y, 1.f, 0.f, gx, gy, gz);
        }
        if (k < cnt) {
            const size_t e = (size_t)at * M + k;
            float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
            if (valid) {
                // radial part: -(1/r) d/dr of fc and of T_n (n U_{n-1} 2 / (r rc))
                const float fc1 = 1.f - u * u, fc2 = fc1 * fc1, fc = fc2 * fc2;
                float dfc = v2[0].x + v2[0].y, drn = 0.f, um1 = 1.f, um2 = 0.f;
#pragma unroll
                for (int n = 1; n < N1; ++n) {
                    const float vn = v2[n].x + v2[n].y;
                    dfc = fmaf(vn, Tn[n], dfc);
                    drn = fmaf((float)n * vn, um1, drn);
                    const float un = fmaf(2.f * tx, um1, -um2);
                    um2 = um1;
                    um1 = un;
                }
                const float gr = over_rc(over_rc(8.f * fc1 * fc2 * dfc, rc, irc) + fc * (drn * (2.f * ir)), rc, irc);
                // a neighbour on the z axis has no phi terms (basis_SphericalUtil.hpp:160-181):
                // phi = 0 there, so the y component of the angular part is dropped
                if (fmaxf(fabsf(d.x), fabsf(d.y)) < 8.f * 1.17549435e-38f) gy = 0.f;
                const float f = fc * ir, un = fmaf(x, gx, fmaf(y, gy, z * gz));
                g.x = fmaf(gr, d.x, f * fmaf(x, un, -gx));
                g.y = fmaf(gr, d.y, f * fmaf(y, un, -gy));
                g.z = fmaf(gr, d.z, f * fmaf(z, un, -gz));
            }
            if (a.accumulate) {
                if (valid) {
                    const float4 o = a.P.g[e];
                    a.P.g[e] = make_float4(o.x + g.x, o.y + g.y, o.z + g.z, 0.f);
                }
            } else {
                a.P.g[e] = g;
            }
        }
    }
}

// =========================================================================== sub-rows
// Compact copy of the entries of each row within cutoff rc (same FP32 test as the
// descriptor kernels), with their positions in the full row: the spherical kernels of a
// sub-basis whose cutoff is well inside the neighbour cutoff scan these instead of the
// full rows.  One warp per atom; entries keep their row order.
__global__ void __launch_bounds__(256) k_subrows(PairBufs P, int n, float rc, float4* __restrict__ sdx,
                                                 int* __restrict__ spos, int* __restrict__ scount) {
    pdl_enter();
    const int at = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (at >= n) return;
    const int M = P.M, cnt = min(P.count[at], M);
    int c = 0;
    for (int base = 0; base < cnt; base += 32) {
        const int k = base + lane;
        float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
        bool in = false;
        if (k < cnt) {
            d = P.dx[(size_t)at * M + k];
            in = sqrtf(d.x * d.x + d.y * d.y + d.z * d.z) < rc;
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) {
            const size_t q = (size_t)at * M + c + __popc(m & ((1u << lane) - 1u));
            sdx[q] = d;
            spos[q] = k;
        }
        c += __popc(m);
    }
    if (lane == 0) scount[at] = c;
}

cudaError_t launch_subrows(const PairBufs& P, int n, float rc, float4* sdx, int* spos, int* scount,
                           cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    return launch_pdl(&k_subrows, dim3((unsigned)(((size_t)n * 32 + 255) / 256)), dim3(256), 0, st, P, n, rc, sdx,
                      spos, scount);
}

// =========================================================================== invariants
// Columns: sum over the column's terms of coefficient x product of a channel's A entries
// (calSphL3 / calSphL4, basis_SphericalUtil.hpp:395-467).  Backward: dE/dA of each
// product, one factor at a time (calGradSphL3 / L4).  One thread owns one (atom slot,
// channel) row of A, so each sum runs in term order and the results do not depend on
// scheduling.  The rows of a block are contiguous in A; the block stages them in shared
// memory with an odd row stride: the lanes of a warp apply the same term at the same time,
// so their reads of one index fall in distinct banks.
constexpr int kInvThreads = 128;

__device__ __forceinline__ int inv_stage(const InvArgs& a, float* sA, long long& r0) {
    const long long nrows = (long long)(a.range[a.t1] - a.range[a.t0]) * a.NP;
    r0 = (long long)blockIdx.x * kInvThreads;
    if (r0 >= nrows) return 0;
    const int nr = (int)min((long long)kInvThreads, nrows - r0);
    const int KS = a.K | 1;
    const float* Ab = a.A + r0 * a.K;
    for (int e = threadIdx.x; e < nr * a.K; e += kInvThreads) {
        const int r = e / a.K;
        sA[r * KS + (e - r * a.K)] = Ab[e];
    }
    return nr;
}

__global__ void __launch_bounds__(kInvThreads) k_inv_fwd(InvArgs a) {
    pdl_enter();
    extern __shared__ float sA[];  // [kInvThreads][K | 1]
    long long r0;
    const int nr = inv_stage(a, sA, r0);
    if (!nr) return;
    __syncthreads();
    const int r = threadIdx.x;
    if (r >= nr) return;
    const long long row = r0 + r;
    const int w = (int)(row / a.NP), p = (int)(row - (long long)w * a.NP);
    const float* Ap = sA + r * (a.K | 1);
    float* out = a.fp + (size_t)(a.range[a.t0] + w) * a.fp_stride + a.fp_off + p * a.sl + a.nl2;
    for (int c = 0; c < a.ncol; ++c) {
        float s = 0.f;
        for (int q = a.start[c]; q < a.start[c + 1]; ++q) {
            const int4 t = a.idx[q];
            float v = a.coef[q] * Ap[t.x] * Ap[t.y] * Ap[t.z];
            if (t.w >= 0) v *= Ap[t.w];
            s += v;
        }
        out[c] = s;
    }
}

__global__ void __launch_bounds__(kInvThreads) k_inv_bwd(InvArgs a) {
    pdl_enter();
    extern __shared__ float sA[];  // [kInvThreads][K | 1] A rows, then as many dE/dA rows
    const int KS = a.K | 1;
    float* sG = sA + kInvThreads * KS;
    long long r0;
    const int nr = inv_stage(a, sA, r0);
    if (!nr) return;
    for (int e = threadIdx.x; e < kInvThreads * KS; e += kInvThreads) sG[e] = 0.f;
    __syncthreads();
    const int r = threadIdx.x;
    if (r < nr) {
        const long long row = r0 + r;
        const int w = (int)(row / a.NP), p = (int)(row - (long long)w * a.NP);
        const float* Ap = sA + r * KS;
        float* Gp = sG + r * KS;
        const float* gf = a.gfp + (size_t)(a.range[a.t0] + w) * a.fp_stride + a.fp_off + p * a.sl + a.nl2;
        for (int c = 0; c < a.ncol; ++c) {
            const float g = gf[c];
            for (int q = a.start[c]; q < a.start[c + 1]; ++q) {
                const int4 t = a.idx[q];
                const float cg = g * a.coef[q];
                const float x = Ap[t.x], y = Ap[t.y], z = Ap[t.z];
                if (t.w < 0) {
                    Gp[t.x] += cg * y * z;
                    Gp[t.y] += cg * x * z;
                    Gp[t.z] += cg * x * y;
                } else {
                    const float u = Ap[t.w];
                    Gp[t.x] += cg * y * z * u;
                    Gp[t.y] += cg * x * z * u;
                    Gp[t.z] += cg * x * y * u;
                    Gp[t.w] += cg * x * y * z;
                }
            }
        }
    }
    __syncthreads();
    float* Gb = a.Gx + r0 * a.K;
    for (int e = threadIdx.x; e < nr * a.K; e += kInvThreads) {
        const int rr = e / a.K;
        Gb[e] = sG[rr * KS + (e - rr * a.K)];
    }
}

// u[p][nl2 + c] = -sum_terms coef sum_f (prod of the other factors) D_b A[factor f]
__global__ void __launch_bounds__(128) k_inv_jvp(InvArgs a) {
    const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int s0 = a.range[a.t0], s1 = a.range[a.t1];
    if (s0 + w >= s1) return;
    float* out = a.u + (size_t)(s0 + w) * a.fp_stride + a.fp_off;
    for (int p = lane; p < a.NP; p += 32) {
        const float* Ap = a.A + ((size_t)w * a.NP + p) * a.K;
        const float* dAp = a.dA + ((size_t)w * a.NP + p) * a.K;
        for (int c = 0; c < a.ncol; ++c) {
            float s = 0.f;
            for (int q = a.start[c]; q < a.start[c + 1]; ++q) {
                const int4 t = a.idx[q];
                const float x = Ap[t.x], y = Ap[t.y], z = Ap[t.z];
                const float dx = dAp[t.x], dy = dAp[t.y], dz = dAp[t.z];
                float v;
                if (t.w < 0) {
                    v = dx * y * z + x * dy * z + x * y * dz;
                } else {
                    const float u = Ap[t.w], du = dAp[t.w];
                    v = (dx * y * z + x * dy * z + x * y * dz) * u + x * y * z * du;
                }
                s += a.coef[q] * v;
            }
            out[p * a.sl + a.nl2 + c] = -s;
        }
    }
}

// Per channel: M1x and M2x of the radial-fuse gradient (the invariant columns' parts).
__global__ void __launch_bounds__(128) k_inv_wgrad(InvArgs a) {
    const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int s0 = a.range[a.t0], s1 = a.range[a.t1];
    if (s0 + w >= s1) return;
    const float* gf = a.gfp + (size_t)(s0 + w) * a.fp_stride + a.fp_off;
    const float* df = a.dfp + (size_t)(s0 + w) * a.fp_stride + a.fp_off;
    for (int p = lane; p < a.NP; p += 32) {
        const size_t row = ((size_t)w * a.NP + p) * a.K;
        const float* Ap = a.A + row;
        const float* dAp = a.dA + row;
        float* M1 = a.M1x + row;
        float* M2 = a.M2x + row;
        for (int k = 0; k < a.K; ++k) { M1[k] = 0.f; M2[k] = 0.f; }
        for (int c = 0; c < a.ncol; ++c) {
            const float gv = gf[p * a.sl + a.nl2 + c], dv = df[p * a.sl + a.nl2 + c];
            for (int q = a.start[c]; q < a.start[c + 1]; ++q) {
                const int4 t = a.idx[q];
                const float cf = a.coef[q];
                const int ord = t.w < 0 ? 3 : 4;
                const int id[4] = {t.x, t.y, t.z, t.w};
                float v[4], dvv[4];
#pragma unroll
                for (int f = 0; f < 4; ++f) {
                    v[f] = f < ord ? Ap[id[f]] : 1.f;
                    dvv[f] = f < ord ? dAp[id[f]] : 0.f;
                }
#pragma unroll
                for (int f = 0; f < 4; ++f) {
                    if (f >= ord) continue;
                    // d term / d A[f] and its derivative along D_b A
                    float prod = 1.f, hd = 0.f;
#pragma unroll
                    for (int o = 0; o < 4; ++o) {
                        if (o == f || o >= ord) continue;
                        float pr = dvv[o];
#pragma unroll
                        for (int o2 = 0; o2 < 4; ++o2)
                            if (o2 != f && o2 != o && o2 < ord) pr *= v[o2];
                        hd += pr;
                        prod *= v[o];
                    }
                    M1[id[f]] += cf * (dv * prod - gv * hd);
                    M2[id[f]] -= cf * gv * prod;
                }
            }
        }
    }
}

cudaError_t launch_invariants_jvp(const InvArgs& a, cudaStream_t st) {
    if (a.nmax <= 0 || a.ncol <= 0) return cudaSuccess;
    k_inv_jvp<<<(a.nmax + 3) / 4, 128, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_invariants_wgrad(const InvArgs& a, cudaStream_t st) {
    if (a.nmax <= 0 || a.ncol <= 0) return cudaSuccess;
    k_inv_wgrad<<<(a.nmax + 3) / 4, 128, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_invariants(const InvArgs& a, bool fwd, cudaStream_t st) {
    if (a.nmax <= 0 || a.ncol <= 0) return cudaSuccess;
    const int grid = (int)(((long long)a.nmax * a.NP + kInvThreads - 1) / kInvThreads);
    const size_t sm = sizeof(float) * kInvThreads * (a.K | 1) * (fwd ? 1 : 2);
    const cudaError_t e = allow_smem(fwd ? k_inv_fwd : k_inv_bwd, sm);
    if (e != cudaSuccess) return e;
    if (fwd) return launch_pdl(&k_inv_fwd, dim3(grid), dim3(kInvThreads), sm, st, a);
    return launch_pdl(&k_inv_bwd, dim3(grid), dim3(kInvThreads), sm, st, a);
}

// =========================================================================== dispatch
namespace {

template <int NP, int N1, int RB>
cudaError_t launch_radial(const DescArgs& a, bool fwd, cudaStream_t st) {
    const int n = a.nmax;
    if (n <= 0) return cudaSuccess;
    const int wpc = a.warps;
    const int grid = (n + wpc - 1) / wpc;
    const size_t sm = sizeof(float) * a.T * a.T * NP * Fuse<N1>::N1P;
    const cudaError_t e = fwd ? allow_smem(k_radial_fwd<NP, N1, RB>, sm) : allow_smem(k_radial_bwd<NP, N1, RB>, sm);
    if (e != cudaSuccess) return e;
    if (fwd) return launch_pdl(&k_radial_fwd<NP, N1, RB>, dim3(grid), dim3(32 * wpc), sm, st, a);
    return launch_pdl(&k_radial_bwd<NP, N1, RB>, dim3(grid), dim3(32 * wpc), sm, st, a);
}

template <int L, int NP, int N1, int LPA>
cudaError_t launch_sph_bwd_lanes(const DescArgs& a, cudaStream_t st) {
    using S = SphNShape<L, NP, N1>;
    constexpr int APW = 32 / LPA;
    const bool diag = a.fwd_alpha && a.T <= kFwdTypes;
    const size_t fixed = (4 * (size_t)S::NS + 3) / 4 * 4 + (diag ? (size_t)a.T * kFwdTypes * NP + 3 : 0) / 4 * 4;
    auto bytes = [&](int w) { return sizeof(float) * (fixed + (size_t)w * S::warp_floats(a.T, APW, diag)); };
    int wpc = a.warps < kBwdWarps ? a.warps : kBwdWarps;
    if (!diag) {
        // many species: the CTA size that leaves the most warps on an SM by its shared memory
        // (228 KB, 1 KB per CTA kept back) and registers
        constexpr int reg_warps = LPA == 32 ? 21 : 25;
        int best = 0;
        for (int w = wpc; w >= 1; --w) {
            const int ctas = std::min((int)(228 * 1024 / (bytes(w) + 1024)), reg_warps / w);
            if (bytes(w) <= 227 * 1024 && w * ctas > best) {
                best = w * ctas;
                wpc = w;
            }
        }
    }
    while (wpc > 1 && bytes(wpc) > 227 * 1024) wpc >>= 1;
    const size_t sm = bytes(wpc);
    if (sm > 227 * 1024) return cudaErrorInvalidValue;
    const int grid = (a.nmax + wpc * APW - 1) / (wpc * APW);
    const cudaError_t e = allow_smem(k_sph_bwd_n<L, NP, N1, LPA>, sm);
    if (e != cudaSuccess) return e;
    return launch_pdl(&k_sph_bwd_n<L, NP, N1, LPA>, dim3(grid), dim3(32 * wpc), sm, st, a);
}

template <int L, int NP, int N1>
cudaError_t launch_sph_bwd_n(const DescArgs& a, cudaStream_t st) {
    using S = SphNShape<L, NP, N1>;
    // Sixteen lanes per atom waste fewer lanes on the last neighbours of a row (40 neighbours:
    // 48 lane slots instead of 64; 1M-atom glass, lmax 4: 1.76 against 2.58 ms) while the Gh of
    // two atoms leaves shared memory for six CTAs; with larger Gh (lmax 6, three species: 12 KB)
    // thirty-two are faster (1024-structure batch 1.96 against 2.05 ms).  Below 4096 atoms the
    // SMs are not filled and the shorter walk of thirty-two lanes wins (33 atoms: 10 against 15 us).
    if (a.nmax >= 4096 && 2 * sizeof(float) * a.T * S::GH <= 6400) return launch_sph_bwd_lanes<L, NP, N1, 16>(a, st);
    return launch_sph_bwd_lanes<L, NP, N1, 32>(a, st);
}

template <int L, int NP, int N1>
cudaError_t launch_sph_fwd_n(const DescArgs& a, cudaStream_t st) {
    using S = SphFNShape<L, NP, N1>;
    const int wpc = a.warps;
    const int grid = (a.nmax + wpc - 1) / wpc;
    const size_t sm = sizeof(float) * (((size_t)a.T * kFwdTypes * NP + 3) / 4 * 4 + (size_t)wpc * S::WARP_FLOATS);
    if (sm > 227 * 1024) return cudaErrorInvalidValue;
    const cudaError_t e = allow_smem(k_sph_fwd_n<L, NP, N1>, sm);
    if (e != cudaSuccess) return e;
    return launch_pdl(&k_sph_fwd_n<L, NP, N1>, dim3(grid), dim3(32 * wpc), sm, st, a);
}

template <int L, int NP, int N1, int RB>
cudaError_t launch_sph(const DescArgs& a, bool fwd, cudaStream_t st) {
    using S = SphShape<L, NP>;
    const int n = a.nmax;
    if (n <= 0) return cudaSuccess;
    if constexpr (RB == kRbNNAP) {   // the radial-space kernels are written for the NNAP radial functions
        if (!fwd && a.nz_p && a.nz_w && N1 <= NP) return launch_sph_bwd_n<L, NP, N1>(a, st);
        if (fwd && a.fwd_alpha && N1 <= NP && a.T <= kFwdTypes) {
            if constexpr (SphTcShape<L, NP>::fits)
                if (a.tc_sms > 0) return launch_sph_fwd_tc<L, NP, N1>(a, st);
            return launch_sph_fwd_n<L, NP, N1>(a, st);
        }
    }
    const int wpc = a.warps;
    const int grid = (n + wpc - 1) / wpc;
    const size_t wbytes = sizeof(float) * ((size_t)a.T * a.T * NP * Fuse<N1>::N1P);
    const size_t sm = wbytes + sizeof(float) * wpc * (fwd ? S::FWD_WARP_FLOATS : S::BWD_WARP_FLOATS);
    const cudaError_t e = fwd ? allow_smem(k_sph_fwd<L, NP, N1, RB>, sm) : allow_smem(k_sph_bwd<L, NP, N1, RB>, sm);
    if (e != cudaSuccess) return e;
    if (fwd) return launch_pdl(&k_sph_fwd<L, NP, N1, RB>, dim3(grid), dim3(32 * wpc), sm, st, a);
    return launch_pdl(&k_sph_bwd<L, NP, N1, RB>, dim3(grid), dim3(32 * wpc), sm, st, a);
}

}  // namespace


bool desc_supported(int kind, int basis, int lmax, int np, int n1) {
    return desc_compiled(kind, basis, lmax, np, n1) || desc_generic_fits(kind, lmax, np, n1);
}

bool desc_compiled(int kind, int basis, int lmax, int np, int n1) {
#define R_CASE(P_, N_) if (kind == 0 && np == P_ && n1 == N_) return true;
#define S_CASE(L_, P_, N_) if (kind == 1 && lmax == L_ && np == P_ && n1 == N_) return true;
    if (basis == kRbNNAP) {
        NNAP_RADIAL_SHAPES(R_CASE)
        NNAP_SPH_SHAPES(S_CASE)
    } else if (basis == kRbNEP) {
        NEP_RADIAL_SHAPES(R_CASE)
        NEP_SPH_SHAPES(S_CASE)
    }
#undef R_CASE
#undef S_CASE
    return false;
}

int desc_bwd_max_warps(int kind, int basis, int lmax, int np, int n1, bool sparse) {
    if (basis == kRbNNAP && sparse) {
#define S_CASE(L_, P_, N_) if (kind == 1 && lmax == L_ && np == P_ && n1 == N_ && N_ <= P_) return kBwdWarps;
        NNAP_SPH_SHAPES(S_CASE)
        NNAP_SPH_EVAL_SHAPES(S_CASE)
#undef S_CASE
    }
    return kDescMaxWarps;
}

cudaError_t launch_descriptor(int kind, int basis, int lmax, int np, int n1, const DescArgs& a, bool fwd,
                              cudaStream_t st) {
#define R_CASE(P_, N_) if (kind == 0 && np == P_ && n1 == N_) return launch_radial<P_, N_, RB_>(a, fwd, st);
#define S_CASE(L_, P_, N_) \
    if (kind == 1 && lmax == L_ && np == P_ && n1 == N_) return launch_sph<L_, P_, N_, RB_>(a, fwd, st);
    if (basis == kRbNNAP) {
        constexpr int RB_ = kRbNNAP;
        NNAP_RADIAL_SHAPES(R_CASE)
        NNAP_SPH_SHAPES(S_CASE)
        // the evaluation shapes: the channel-space kernels keep the fuse matrices of all T^2 pairs
        // in shared memory, so beyond kEvalTypes species the any-shape kernels are the faster
        if (a.T <= kEvalTypes || (!fwd && a.nz_p && a.nz_w)) {
            NNAP_SPH_EVAL_SHAPES(S_CASE)
        }
    } else if (basis == kRbNEP) {
        constexpr int RB_ = kRbNEP;
        NEP_RADIAL_SHAPES(R_CASE)
        NEP_SPH_SHAPES(S_CASE)
    }
#undef R_CASE
#undef S_CASE
    return launch_descriptor_generic(kind, basis, lmax, np, n1, a, fwd, st);
}

}  // namespace nnapgb

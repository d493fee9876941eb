// Tensor-core evaluation of the per-species network and its input gradient (the
// mixed-precision path), on the 5th-generation tensor cores (tcgen05, TMEM accumulators).
//
// Mathematics: normedNnForward / normedNnBackward (nnap_main.hpp:267-323) with L >= 1
// SiLU hidden layers (nn_FeedForward.hpp:8-261), widths padded to multiples of 16:
//   X   = (fp - mu)/sigma                       [128 x Dp]
//   Z_l = A_{l-1} W_l^T + b_l, A_l = silu(Z_l)   [128 x Hp_l]  GEMM (N = Hp_l, K = K_l), A_0 = X
//   E   = (w_o . A_L + b_o) sigma_E + mu_E       (FP32 on the CUDA cores, FP64 output)
//   dZ_L = sigma_E w_o * silu'(Z_L)
//   dA_{l-1} = dZ_l W_l                          [128 x K_l]   GEMM (N = K_l, K = Hp_l)
//   dZ_{l-1} = dA_{l-1} * silu'(Z_{l-1})
//   dE/dfp = dA_0 / sigma
// Padded units have zero weights and biases, so they stay zero through every layer.
// Operands are BF16 and every product is split as hi*hi + lo*hi + hi*lo with x = hi + lo
// (both BF16), accumulated in FP32 in TMEM: three kind::f16 MMAs per 16-wide K step keep
// the network error near FP32 level (about 1e-6 eV per atom) while the arithmetic stays
// on the BF16 tensor pipe.
//
// A group of 128 x SPLIT threads owns a 128-atom tile; the SPLIT threads of row t read
// TMEM lane t with tcgen05.ld 32x32b, each a share of the columns.  One thread issues the
// MMAs; completion is signalled through an mbarrier (tcgen05.commit) whose waits are
// bounded in time and raise ERRBIT_TIMEOUT instead of hanging.  silu'(Z_l) of every layer
// stays in TMEM for the backward pass; dA and dX share one column range.  One shared-memory
// operand buffer holds the activation of the current GEMM and is overwritten by the next
// layer's once that GEMM has completed.  The weight images of a species are staged in
// shared memory once per species when they fit, otherwise the B operand of each GEMM is
// copied in before it (the images are small and stay in L2).
//
// A tile is a chain: load, four GEMMs of a few hundred cycles for two hidden layers, an
// epilogue after each, store; the machine waits most of the time (a third of the issue slots
// with one tile per SM).  So a CTA of G = 2 groups works on two tiles at once, each group with
// its own operand buffer, TMEM columns, mbarrier and named barrier, both with one weight image.
// Within a tile: the sigmoid has no branch, silu' is kept instead of formed again, two values
// are split per conversion, a row's sectors are loaded whole and four at a time, and the next
// tile's rows are called into L2.  Before and now: 909 -> 403 us for 1048573 atoms
// (90-64-64-1, two species), 498 -> 232 us for 488206 (126-64-64-1, three species);
// with one group 524 and 279.
//
// The next kernel is not let in early: its blocks would start on an SM as soon as the tile
// kernel's one block there ends, and keep the SM's split between shared memory and L1, which
// with 160 to 226 KiB of operands leaves the backward kernels little L1 (488206 atoms:
// 5399 us per evaluation, 5947 with the early launch; 32000 atoms 525 against 531).
// Shared-memory operands use the no-swizzle K-major canonical layout: 8x8 core
// matrices of 128 bytes, adjacent in K at LBO = 128 bytes and in M/N at
// SBO = (K/8)*128 bytes.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "net_tc.cuh"
#include "pdl.cuh"
#include "smem_limit.cuh"
#include "tc_util.cuh"

namespace nnapgb {

bool TCLayout::same(const TCLayout& o) const {
    if (nl != o.nl || Dp != o.Dp) return false;
    for (int l = 0; l < nl; ++l)
        if (Hp[l] != o.Hp[l]) return false;
    return true;
}

namespace {

using namespace ::nnapgb::tc;

constexpr int kTcSmemMax = 220 * 1024;  // dynamic shared memory; the static part (mbarrier, energies) comes on top
constexpr int kTcSmemTwo = 226 * 1024;  // the same with two tile groups (no energies in the static part)
constexpr int kTcWidthMax = 256;       // widest padded layer (one MMA N, one operand buffer)
constexpr int kTcOperandMax = 96 * 1024;  // largest single weight operand image (hi + lo)
constexpr int kOutCols = 64;           // columns of dE/dfp staged per pass

__host__ __device__ inline int align1k(int b) { return (b + 1023) & ~1023; }
inline int r16(int v) { return (v + 15) & ~15; }

// Layout of a network with descriptor length D and hidden widths H[0..nl-1]; false with a
// reason when the kernel cannot take it.
bool make_layout(int D, const std::vector<int>& H, TCLayout& L, std::string& why) {
    const int nl = (int)H.size();
    if (nl < 1 || nl > kTcMaxLayers) {
        why = "the tensor-core network takes 1 to 8 hidden layers";
        return false;
    }
    L.nl = nl;
    L.Dp = r16(D);
    L.Wmax = L.Dp;
    int in = L.Dp, off = 0, wimg = 0;
    for (int l = 0; l < nl; ++l) {
        L.K[l] = in;
        L.Hp[l] = r16(H[l]);
        L.Wmax = std::max(L.Wmax, L.Hp[l]);
        const int img = 4 * L.Hp[l] * in;  // hi + lo BF16
        wimg = std::max(wimg, img);
        L.wf[l] = off; off = align1k(off + img);
        L.wb[l] = off; off = align1k(off + img);
        in = L.Hp[l];
    }
    if (L.Wmax > kTcWidthMax) {
        why = "the tensor-core network takes descriptors and hidden layers of at most 256 (padded) columns";
        return false;
    }
    if (wimg > kTcOperandMax) {
        why = "a tensor-core weight operand would exceed 96 KiB";
        return false;
    }
    L.fvec = off;
    L.fmu = 0;
    L.fisig = L.Dp;
    int f = 2 * L.Dp;
    for (int l = 0; l < nl; ++l) { L.fb[l] = f; f += L.Hp[l]; }
    L.fwo = f;
    f += L.Hp[nl - 1];
    L.nvec = (f + 3) & ~3;
    off = align1k(off + 4 * L.nvec);
    L.bytes = off;
    L.wimg = align1k(wimg);
    // TMEM: Z of every layer, then one range for dA / dX
    int cols = 0, dmax = 0;
    for (int l = 0; l < nl; ++l) { L.z[l] = cols; cols += L.Hp[l]; dmax = std::max(dmax, L.K[l]); }
    L.dacc = cols;
    cols += dmax;
    if (cols > 512) {
        why = "the tensor-core network's accumulators would exceed the 512 TMEM columns";
        return false;
    }
    L.ncols = 32;
    while (L.ncols < cols) L.ncols *= 2;
    L.act = align1k(std::max(4 * 128 * L.Wmax, 4 * 128 * (kOutCols + 4)));
    const int staged = L.bytes + L.act;
    const int streamed = align1k(4 * L.nvec) + L.wimg + L.act;
    if (staged <= kTcSmemMax) {
        L.staged = 1;
        L.smem = staged;
    } else if (streamed <= kTcSmemMax) {
        L.staged = 0;
        L.smem = streamed;
    } else {
        why = "the tensor-core network's operands exceed shared memory";
        return false;
    }
    return true;
}

// Element (r, k) of an R x K K-major operand in the no-swizzle core-matrix layout.
inline size_t cm_index(int r, int k, int K) { return ((size_t)(r >> 3) * (K >> 3) + (k >> 3)) * 64 + (r & 7) * 8 + (k & 7); }

uint16_t bf16_bits(float f) {
    __nv_bfloat16 b = __float2bfloat16_rn(f);
    uint16_t u;
    std::memcpy(&u, &b, 2);
    return u;
}
float bf16_val(uint16_t u) {
    uint32_t w = (uint32_t)u << 16;
    float f;
    std::memcpy(&f, &w, 4);
    return f;
}

// Write the hi and lo images of an R x K matrix M(r, k).
template <class F>
void put_operand(std::vector<uint8_t>& img, int byte_off, int R, int K, F&& M) {
    uint16_t* hi = reinterpret_cast<uint16_t*>(img.data() + byte_off);
    uint16_t* lo = hi + (size_t)R * K;
    for (int r = 0; r < R; ++r)
        for (int k = 0; k < K; ++k) {
            const float v = (float)M(r, k);
            const uint16_t h = bf16_bits(v);
            const uint16_t l = bf16_bits(v - bf16_val(h));
            hi[cm_index(r, k, K)] = h;
            lo[cm_index(r, k, K)] = l;
        }
}

// 1/(1 + e^-z) without the branch of a division, so that the 16 units of a step overlap: the
// machine's approximate reciprocal and one step of Newton's iteration, which leaves the
// rounding of the last operation.  Below -87.3, where the denominator nears 2^126 and its
// reciprocal the smallest normal number, it is zero (silu is within 2e-36 of it there, and silu
// and silu' stay zero however large -z is, as with a division).  Infinities and NaN of z reach
// the results as they do with a division.
__device__ __forceinline__ float sigmoidf_(float z) {
    const float y = 1.f + expf(-z);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
    r = fmaf(r, fmaf(-y, r, 1.f), r);
    return z < -87.3f ? 0.f : r;
}

// Species t0 .. t0+nt-1 of one launch; all share one layout.  Tiles are numbered species
// by species; a CTA stages a species' image (or its FP32 vectors, in streamed mode) when
// its next tile belongs to another species than the last one.
struct TcParams {
    const int* perm;
    const int* range;     // device: first slot of each species
    int t0, nt;
    const float* fp;
    int fp_stride, D;
    float* gfp;
    double* e_atom;
    const uint8_t* img[kMaxTypes];  // weight image per species (global)
    float bo[kMaxTypes];
    double mu_e[kMaxTypes], sigma_e[kMaxTypes];
    int* err;
};

// Copy n bytes (a multiple of 16) from global to shared memory with every thread.
__device__ __forceinline__ void copy16(uint8_t* dst, const uint8_t* src, int n, int tid, int nthr) {
    const uint4* s = reinterpret_cast<const uint4*>(src);
    uint4* d = reinterpret_cast<uint4*>(dst);
    for (int q = tid; q < n / 16; q += nthr) d[q] = s[q];
}

// Barrier of the NT threads of one tile group (barrier 0 is the CTA's).
template <int NT>
__device__ __forceinline__ void group_sync(int g) {
    asm volatile("barrier.cta.sync %0, %1;" ::"r"(g + 1), "n"(NT) : "memory");
}
template <int NT>
__device__ __forceinline__ bool group_sync_and(int g, bool v) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.and.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}\n"
        : "=r"(r)
        : "r"((uint32_t)v), "r"(g + 1), "n"(NT)
        : "memory");
    return r != 0;
}

__device__ __forceinline__ void ld16(const float* src, float* v) {  // 16-byte aligned
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float4 a = reinterpret_cast<const float4*>(src)[q];
        v[4 * q] = a.x; v[4 * q + 1] = a.y; v[4 * q + 2] = a.z; v[4 * q + 3] = a.w;
    }
}

// 32 contiguous bytes, a whole sector, with one load.
__device__ __forceinline__ void ld8(const float* src, float* v) {
    asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(src));
}

template <int SPLIT, int G>
__global__ void __launch_bounds__(128 * SPLIT * G, 1) k_net_tc(TcParams p, TCLayout L) {
    pdl_wait();  // no early launch of the next kernel, see above
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t mbar[G];
    __shared__ uint32_t tmem_base;
    __shared__ int s_tstart[kMaxTypes + 1];
    constexpr int NT = 128 * SPLIT;  // threads of a group
    constexpr int ES = 4 / SPLIT;    // energy shares of a thread
    const int grp = G == 1 ? 0 : threadIdx.x / NT;
    const int tid = threadIdx.x - grp * NT, warp = tid >> 5, lane = tid & 31;
    const int part = tid >> 7;  // column share of this thread in the epilogues
    const int row = tid & 127;
    const int nl = L.nl, Dp = L.Dp;
    // shared memory: staged [image | act per group]; streamed [FP32 vectors | one operand | act]
    uint8_t* sw = smem;
    uint8_t* swb = smem + (L.staged ? 0 : align1k(4 * L.nvec));  // per-GEMM operand (streamed)
    uint8_t* sact = smem + (L.staged ? L.bytes : align1k(4 * L.nvec) + L.wimg) + grp * L.act;
    const float* fv = reinterpret_cast<const float*>(L.staged ? sw + L.fvec : sw);
    const int half = 2 * 128 * L.Wmax;  // bytes of the hi (or lo) activation image
    uint8_t* sact_lo = sact + half;

    if (threadIdx.x == 0) {
        s_tstart[0] = 0;
        for (int t = 0; t < p.nt; ++t)
            s_tstart[t + 1] = s_tstart[t] + (p.range[p.t0 + t + 1] - p.range[p.t0 + t] + 127) / 128;
        for (int g = 0; g < G; ++g)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar[g])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                     "r"(G * L.ncols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_async_smem();
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tbase = tmem_base + grp * L.ncols;
    const uint32_t tlane = tbase + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t mb = smem_u32(&mbar[grp]);
    uint32_t phase = 0;
    bool ok = true;
    const uint32_t ah = smem_u32(sact), al = ah + half;

    // one GEMM: D (TMEM column dcol) = act [128 x K] * B [N x K]^T, B the image at byte
    // offset boff of the species image (staged) or copied from global first (streamed, G = 1)
    auto gemm = [&](int ts, int boff, int N, int K, int dcol) -> bool {
        uint32_t bh;
        if (L.staged) {
            bh = smem_u32(sw + boff);
        } else {
            copy16(swb, p.img[ts] + boff, 4 * N * K, tid, NT);
            bh = smem_u32(swb);
        }
        fence_async_smem();
        group_sync<NT>(grp);
        if (tid == 0) {
            fence_after();
            issue_gemm(tbase + dcol, ah, al, bh, bh + 2 * N * K, K, N);
            mma_commit(mb);
        }
        const bool done = group_sync_and<NT>(grp, mbar_wait(mb, phase));
        phase ^= 1;
        if (done) fence_after();
        return done;
    };

    // every CTA walks the species in order; its groups share the image and take their own
    // tiles, first one per CTA, then the second ones
    const int step = gridDim.x * G;
    for (int ts = 0; ts < p.nt; ++ts) {
        const int t0 = s_tstart[ts], t1 = s_tstart[ts + 1];
        auto first = [&](int g) {  // first tile at or after t0 of group g
            const int c = g * gridDim.x + blockIdx.x;
            return c >= t0 ? c : c + (t0 - c + step - 1) / step * step;
        };
        bool any = false;
#pragma unroll
        for (int g = 0; g < G; ++g) any |= first(g) < t1;
        int gt = first(grp);
        if (!any) continue;  // uniform over the CTA
        __syncthreads();     // no group reads the last image any more, no MMA is in flight
        if (L.staged) copy16(sw, p.img[ts], L.bytes, threadIdx.x, NT * G);
        else copy16(sw, p.img[ts] + L.fvec, 4 * L.nvec, threadIdx.x, NT * G);
        fence_async_smem();
        __syncthreads();
        const int s0 = p.range[p.t0 + ts], s1 = p.range[p.t0 + ts + 1];
        const float se = (float)p.sigma_e[ts];
        for (; gt < t1 && ok; gt += step) {
            const int tile = gt - t0;
            const int slot = s0 + tile * 128 + row;
            const bool valid = slot < s1;
            // ---- X = (fp - mu) / sigma, split into hi / lo.  Warp-cooperative: the lanes of a
            // warp take 8 rows (one core-matrix block) x 4 chunks of 8 columns, so the global
            // reads are 128-byte row segments and the shared stores fill 512 contiguous bytes
            {
                const int nch = Dp >> 3;
                const bool wide = (p.fp_stride & 7) == 0;  // rows start on a sector (else on 16 bytes)
                const int r8 = lane & 7, cq = lane >> 3;
                for (int rb = warp; rb < 16; rb += 4 * SPLIT) {
                    const int r = rb * 8 + r8, sl = s0 + tile * 128 + r;
                    const float* fr = p.fp + (size_t)(sl < s1 ? sl : s1 - 1) * p.fp_stride;
                    for (int cg = cq; cg < nch; cg += 16) {  // four chunks in flight
                        float v[4][8];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int k0 = 8 * (cg + 4 * j);
#pragma unroll
                            for (int q = 0; q < 8; ++q) v[j][q] = 0.f;
                            if (wide) {
                                if (k0 < p.D) ld8(fr + k0, v[j]);
                            } else {
#pragma unroll
                                for (int q = 0; q < 8; q += 4)
                                    if (k0 + q < p.D) {
                                        const float4 a = *reinterpret_cast<const float4*>(fr + k0 + q);
                                        v[j][q] = a.x; v[j][q + 1] = a.y; v[j][q + 2] = a.z; v[j][q + 3] = a.w;
                                    }
                            }
                            if (k0 + 8 > p.D) {  // the row's padding holds anything
#pragma unroll
                                for (int q = 0; q < 8; ++q) v[j][q] = k0 + q < p.D ? v[j][q] : 0.f;
                            }
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int c = cg + 4 * j;
                            if (c >= nch) break;
                            float4 m[2], is[2];  // zero beyond D
#pragma unroll
                            for (int q = 0; q < 2; ++q) {
                                m[q] = reinterpret_cast<const float4*>(fv + L.fmu + 8 * c)[q];
                                is[q] = reinterpret_cast<const float4*>(fv + L.fisig + 8 * c)[q];
                            }
#pragma unroll
                            for (int q = 0; q < 2; ++q) {
                                v[j][4 * q] = (v[j][4 * q] - m[q].x) * is[q].x;
                                v[j][4 * q + 1] = (v[j][4 * q + 1] - m[q].y) * is[q].y;
                                v[j][4 * q + 2] = (v[j][4 * q + 2] - m[q].z) * is[q].z;
                                v[j][4 * q + 3] = (v[j][4 * q + 3] - m[q].w) * is[q].w;
                            }
                            if (sl >= s1) {
#pragma unroll
                                for (int q = 0; q < 8; ++q) v[j][q] = 0.f;
                            }
                            store_split8(sact, sact_lo, r, 8 * c, Dp, v[j]);
                        }
                    }
                }
                // the rows of this group's next tile of the species (one block) towards L2
                const int nx = s0 + (tile + step) * 128;
                if (tid == 0 && nx < s1) {
                    const int rows = s1 - nx < 128 ? s1 - nx : 128;
                    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p.fp + (size_t)nx * p.fp_stride),
                                 "r"(rows * p.fp_stride * 4)
                                 : "memory");
                }
            }
            // ---- forward through the hidden layers.  silu'(Z_l) takes the place of Z_l in TMEM
            // for the backward pass (one exponential and one division per unit).  The energy
            // sums the 16-column blocks by their index modulo 4, so it is the same for every SPLIT
            float e[ES];
#pragma unroll
            for (int q = 0; q < ES; ++q) e[q] = 0.f;
            for (int l = 0; l < nl && ok; ++l) {
                const int H = L.Hp[l];
                ok = gemm(ts, L.wf[l], H, L.K[l], L.z[l]);
                if (!ok) break;
                const bool last = l == nl - 1;
                int u = 0;
                for (int c0 = 16 * part; c0 < H; c0 += 16 * SPLIT, u ^= 1) {
                    float z[16], b[16];
                    tmem_ld16(tlane + L.z[l] + c0, z);
                    ld16(fv + L.fb[l] + c0, b);
                    if (last) {  // energy share and dZ_L = sigma_E w_o silu'(Z_L)
                        float wo[16], s16 = 0.f;
                        ld16(fv + L.fwo + c0, wo);
                        if (ES == 1) s16 = e[0];
                        else s16 = u ? e[ES - 1] : e[0];
#pragma unroll
                        for (int q = 0; q < 16; ++q) {
                            const float zz = z[q] + b[q];
                            const float s = sigmoidf_(zz);
                            s16 += wo[q] * (zz * s);
                            z[q] = se * wo[q] * (s * (1.f + zz * (1.f - s)));
                        }
                        if (ES == 1 || !u) e[0] = s16;
                        else e[ES - 1] = s16;
                    } else {
                        float d[16];
#pragma unroll
                        for (int q = 0; q < 16; ++q) {
                            const float zz = z[q] + b[q];
                            const float s = sigmoidf_(zz);
                            d[q] = s * (1.f + zz * (1.f - s));
                            z[q] = zz * s;
                        }
                        tmem_st16(tlane + L.z[l] + c0, d);
                    }
                    store_split8(sact, sact_lo, row, c0, H, z);
                    store_split8(sact, sact_lo, row, c0 + 8, H, z + 8);
                }
                if (last) {  // the shares go to the columns of Z_L that this thread has read
#pragma unroll
                    for (int q = 0; q < ES; ++q) {
                        const int c = 16 * (part + q * SPLIT);
                        if (c < H) tmem_st1(tlane + L.z[l] + c, e[q]);
                    }
                }
                tmem_st_wait();
                fence_before();
            }
            if (!ok) break;
            // energy of a row: its shares in a fixed order (after a GEMM's barriers)
            auto energy = [&]() {
                float et = tmem_ld1(tlane + L.z[nl - 1]);
                for (int c = 16; c < 64 && c < L.Hp[nl - 1]; c += 16) et += tmem_ld1(tlane + L.z[nl - 1] + c);
                if (valid) p.e_atom[p.perm[slot]] = ((double)et + (double)p.bo[ts]) * p.sigma_e[ts] + p.mu_e[ts];
            };
            // ---- backward: dA_{l-1} = dZ_l W_l; dZ_{l-1} = dA_{l-1} silu'(Z_{l-1})
            for (int l = nl - 1; l >= 1 && ok; --l) {
                ok = gemm(ts, L.wb[l], L.K[l], L.Hp[l], L.dacc);
                if (!ok) break;
                if (l == nl - 1 && part == 0) energy();
                const int H = L.Hp[l - 1];
                for (int c0 = 16 * part; c0 < H; c0 += 16 * SPLIT) {
                    float g[16], d[16];
                    tmem_ld16x2(tlane + L.dacc + c0, g, tlane + L.z[l - 1] + c0, d);
#pragma unroll
                    for (int q = 0; q < 16; ++q) g[q] *= d[q];
                    store_split8(sact, sact_lo, row, c0, H, g);
                    store_split8(sact, sact_lo, row, c0 + 8, H, g + 8);
                }
                fence_before();
            }
            if (!ok) break;
            // ---- dX = dZ_1 W_1
            ok = gemm(ts, L.wb[0], Dp, L.Hp[0], L.dacc);
            if (!ok) break;
            if (nl == 1 && part == 0) energy();
            // ---- dE/dfp = dX / sigma, staged through the (now free) operand buffer kOutCols
            // columns at a time (rows padded by 4 floats against bank conflicts) and written
            // with coalesced stores, half a warp per row
            {
                constexpr int CS = kOutCols + 4;
                float* sg = reinterpret_cast<float*>(sact);  // [128][CS]
                for (int cb = 0; cb < Dp; cb += kOutCols) {
                    const int cw = Dp - cb < kOutCols ? Dp - cb : kOutCols;
                    auto put = [&](int c0, const float* g) {
                        float is[16];
                        ld16(fv + L.fisig + cb + c0, is);
                        float4* o = reinterpret_cast<float4*>(sg + (size_t)row * CS + c0);
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            o[q] = make_float4(g[4 * q] * is[4 * q], g[4 * q + 1] * is[4 * q + 1],
                                               g[4 * q + 2] * is[4 * q + 2], g[4 * q + 3] * is[4 * q + 3]);
                    };
                    float g[16], h[16];
                    const int c0 = 16 * part, c1 = c0 + 16 * SPLIT;  // kOutCols = 64: at most two steps
                    if (SPLIT == 2 && c1 < cw) {
                        tmem_ld16x2(tlane + L.dacc + cb + c0, g, tlane + L.dacc + cb + c1, h);
                        put(c0, g);
                        put(c1, h);
                    } else if (c0 < cw) {
                        tmem_ld16(tlane + L.dacc + cb + c0, g);
                        put(c0, g);
                    }
                    group_sync<NT>(grp);
                    const int lim = p.D - cb;  // up to three zeros follow column D, inside the row's padding
                    const int k = 4 * (lane & 15);
                    if (k < lim) {
#pragma unroll
                        for (int it = 0; it < 128 / (8 * SPLIT); ++it) {
                            const int r = 2 * warp + (lane >> 4) + it * 8 * SPLIT, sl = s0 + tile * 128 + r;
                            const float4 v = *reinterpret_cast<const float4*>(sg + (size_t)r * CS + k);
                            if (sl < s1) *reinterpret_cast<float4*>(p.gfp + (size_t)sl * p.fp_stride + cb + k) = v;
                        }
                    }
                    group_sync<NT>(grp);
                }
            }
            fence_before();
            group_sync<NT>(grp);
        }
    }
    if (!ok && tid == 0) atomicOr(p.err, ERRBIT_TIMEOUT);
    fence_before();
    __syncthreads();
    fence_after();
    if (threadIdx.x < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(G * L.ncols)
                     : "memory");
}

}  // namespace

bool net_tc_prepare(const Species& sp, NetTC& tc, std::string& why) {
    tc.ready = false;
    const int D = sp.D;
    TCLayout L;
    if (!make_layout(D, sp.hidden, L, why)) return false;
    std::vector<uint8_t> img(L.bytes, 0);
    int in = D;
    for (int l = 0; l < L.nl; ++l) {
        const int H = sp.hidden[l], Hp = L.Hp[l], K = L.K[l];
        const std::vector<double>& W = sp.Wh[l];  // [H][in]
        auto Wf = [&](int o, int i) { return o < H && i < in ? W[(size_t)o * in + i] : 0.0; };
        put_operand(img, L.wf[l], Hp, K, [&](int r, int k) { return Wf(r, k); });  // [Hp][K]
        put_operand(img, L.wb[l], K, Hp, [&](int r, int k) { return Wf(k, r); });  // [K][Hp]
        in = H;
    }
    float* fv = reinterpret_cast<float*>(img.data() + L.fvec);
    for (int k = 0; k < L.Dp; ++k) {
        fv[L.fmu + k] = k < D ? (float)sp.mu[k] : 0.f;
        fv[L.fisig + k] = k < D ? (float)(1.0 / sp.sigma[k]) : 0.f;
    }
    for (int l = 0; l < L.nl; ++l)
        for (int o = 0; o < sp.hidden[l]; ++o) fv[L.fb[l] + o] = (float)sp.bh[l][o];
    for (int o = 0; o < sp.hidden.back(); ++o) fv[L.fwo + o] = (float)sp.wo[o];
    if (cudaMalloc(&tc.blob, img.size()) != cudaSuccess) {
        cudaGetLastError();
        why = "device allocation failed";
        return false;
    }
    if (cudaMemcpy(tc.blob, img.data(), img.size(), cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaGetLastError();
        why = "copy of the network image failed";
        return false;
    }
    tc.blob_bytes = img.size();
    tc.D = D;
    tc.L = L;
    tc.bo = (float)sp.bo;
    tc.ready = true;
    return true;
}

void net_tc_release(NetTC& tc) {
    if (tc.blob) cudaFree(tc.blob);
    tc.blob = nullptr;
    tc.ready = false;
}

static int max_tiles(int n, int nt) { return (n + 127) / 128 + nt; }  // over all species of a launch

// Two tiles in flight once every SM has more than two: 40000 atoms (90-64-64-1) 36 us against
// 41 with one, 200000 94 against 116; (126-64-64-1) 32000 atoms 36.5 against 35.8, 50000 51
// against 48, 70000 57 against 60, 200000 121 against 139.  Both groups of a CTA need the
// operand buffer (226 KiB in all) and TMEM columns (512).
bool net_tc_two_tiles(const NetTC& tc, int n, int nt, int sm_count) {
    const TCLayout& L = tc.L;
    return L.staged && max_tiles(n, nt) > 2 * sm_count && 2 * L.ncols <= 512 && L.smem + L.act <= kTcSmemTwo;
}

cudaError_t launch_net_tc(const NetArgs* a, const NetTC* const* tc, int nt, int* err, int sm_count, int split,
                          cudaStream_t st) {
    if (nt < 1 || nt > kMaxTypes) return cudaErrorInvalidValue;
    for (int k = 0; k < nt; ++k) {
        if (!tc[k]->ready) return cudaErrorNotSupported;
        if (tc[k]->D != tc[0]->D || !tc[k]->L.same(tc[0]->L)) return cudaErrorInvalidValue;
    }
    const int n = a[0].nmax;
    if (n <= 0) return cudaSuccess;
    const TCLayout& L = tc[0]->L;
    if (split != 2 && split != 4) return cudaErrorInvalidValue;
    const int ntiles = max_tiles(n, nt);
    const bool two = net_tc_two_tiles(*tc[0], n, nt, sm_count);
    void (*kern)(TcParams, TCLayout) = two ? k_net_tc<2, 2> : split == 2 ? k_net_tc<2, 1> : k_net_tc<4, 1>;
    const int smem = L.smem + (two ? L.act : 0);
    const cudaError_t e = allow_smem(kern, two ? kTcSmemTwo : kTcSmemMax);
    if (e != cudaSuccess) return e;
    TcParams p;
    std::memset(&p, 0, sizeof p);
    p.perm = a[0].perm;
    p.range = a[0].range;
    p.t0 = a[0].t;
    p.nt = nt;
    p.fp = a[0].fp;
    p.fp_stride = a[0].fp_stride;
    p.D = tc[0]->D;
    p.gfp = a[0].gfp;
    p.e_atom = a[0].e_atom;
    for (int k = 0; k < nt; ++k) {
        p.img[k] = reinterpret_cast<const uint8_t*>(tc[k]->blob);
        p.bo[k] = tc[k]->bo;
        p.mu_e[k] = a[k].mu_e;
        p.sigma_e[k] = a[k].sigma_e;
    }
    p.err = err;
    const int grid = ntiles < sm_count ? ntiles : sm_count;
    return launch_pdl(kern, dim3(grid), dim3(two ? 512 : 128 * split), (size_t)smem, st, p, L);
}

}  // namespace nnapgb

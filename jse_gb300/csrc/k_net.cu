// FP32 SIMT evaluation of the per-species SiLU feed-forward network and of its input
// gradient (the plain-precision path; also the tanh network of NEP models).
//
// Restates normedNnForward / normedNnBackward (nnap_main.hpp:267-323) and
// nnForward / nnBackward (nn_FeedForward.hpp:8-21, 131-261):
//   x = (fp - mu) / sigma;  h_l = silu(W_l h_{l-1} + b_l);  o = w_out . h_L + b_out;
//   E = o * sigma_E + mu_E;  dE/dfp = (sigma_E * d o / d x) / sigma.
// Atoms of one species are evaluated eight at a time, so every weight loaded is used eight
// times; threads own output units in the forward pass and input units in the backward pass, so
// all weight loads are coalesced (W^T rows forward, W rows backward).  All species run in one
// launch (blockIdx.y).  Each sum runs over slices of kSlice inputs, the slices' sums added in
// order, which two kernels share bit for bit (a model's kernels do not depend on the atom count):
//   k_net_warp  a warp per eight atoms, up to two units per lane: many atoms;
//   k_net_cta   a CTA of 256 threads per eight atoms, the slices of a unit on different threads:
//               few atoms, where the time is the chain of weight loads (500 atoms, 126-64-64
//               networks of three species: 133 us as one launch per species with a warp per
//               eight atoms -> 23 us; 100k atoms 545 -> 402).
// A single narrow network keeps the kernel without slices (k_net_fp32).
//
// Packed FP32 parameters of a species (net_pack in nnap_api.cu):
//   mu[D] | 1/sigma[D] | for each layer: W^T[in][H] | W[H][in] | b[H] | w_out[H_L] | b_out
#include "desc.cuh"
#include "pdl.cuh"
#include "smem_limit.cuh"

namespace nnapgb {
namespace {

constexpr int kNetAtoms = 8;
constexpr int kNetWarps = 4;

__device__ __forceinline__ float silu_and_grad(float z, float* grad) {
    const float s = 1.f / (1.f + expf(-z));
    *grad = s * (1.f + z * (1.f - s));
    return z * s;
}

// tanh for NEP networks (apply_ann_one_layer, nep_core.hpp:267-305)
__device__ __forceinline__ float act_and_grad(float z, float* grad, int act) {
    if (act == kActTanh) {
        const float t = tanhf(z);
        *grad = 1.f - t * t;
        return t;
    }
    return silu_and_grad(z, grad);
}

constexpr int kSlice = 32;
constexpr int kCtaThreads = 256;

__device__ __forceinline__ int widest(const NetArgs& a) {
    int h = a.D;
    for (int l = 0; l < a.nlayer; ++l) h = max(h, a.H[l]);
    return h;
}

// acc[q] = sum over k in [k0, k1) of w[k * ldw] in[k][q], in order; the slice's weights are all
// loaded before the first is used.
__device__ __forceinline__ void slice_sum(const float* __restrict__ w, int ldw, const float* in, int k0, int k1, float* acc) {
    float wv[kSlice];
#pragma unroll
    for (int k = 0; k < kSlice; ++k) wv[k] = k0 + k < k1 ? w[(size_t)(k0 + k) * ldw] : 0.f;
#pragma unroll
    for (int q = 0; q < kNetAtoms; ++q) acc[q] = 0.f;
#pragma unroll
    for (int k = 0; k < kSlice; ++k) {
        if (k0 + k < k1) {
            const float4 x0 = *reinterpret_cast<const float4*>(in + (k0 + k) * kNetAtoms);
            const float4 x1 = *reinterpret_cast<const float4*>(in + (k0 + k) * kNetAtoms + 4);
            acc[0] = fmaf(wv[k], x0.x, acc[0]); acc[1] = fmaf(wv[k], x0.y, acc[1]);
            acc[2] = fmaf(wv[k], x0.z, acc[2]); acc[3] = fmaf(wv[k], x0.w, acc[3]);
            acc[4] = fmaf(wv[k], x1.x, acc[4]); acc[5] = fmaf(wv[k], x1.y, acc[5]);
            acc[6] = fmaf(wv[k], x1.z, acc[6]); acc[7] = fmaf(wv[k], x1.w, acc[7]);
        }
    }
}

// R units per lane (u, u + 32, ..): the same sums, one read of the inputs for all of them.
template <int R, class Out>
__device__ __forceinline__ void warp_units(const float* __restrict__ W, const float* __restrict__ bias, int K, int U, int u0,
                                           const float* in, Out&& out) {
    float tot[R][kNetAtoms];
    bool has[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        has[r] = u0 + 32 * r < U;
#pragma unroll
        for (int q = 0; q < kNetAtoms; ++q) tot[r][q] = bias && has[r] ? bias[u0 + 32 * r] : 0.f;
    }
    for (int k0 = 0; k0 < K; k0 += kSlice) {
        const int k1 = min(K, k0 + kSlice);
        float acc[R][kNetAtoms];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int q = 0; q < kNetAtoms; ++q) acc[r][q] = 0.f;
#pragma unroll 8
        for (int k = k0; k < k1; ++k) {
            const float4 x0 = *reinterpret_cast<const float4*>(in + k * kNetAtoms);
            const float4 x1 = *reinterpret_cast<const float4*>(in + k * kNetAtoms + 4);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float wv = has[r] ? W[(size_t)k * U + u0 + 32 * r] : 0.f;
                acc[r][0] = fmaf(wv, x0.x, acc[r][0]); acc[r][1] = fmaf(wv, x0.y, acc[r][1]);
                acc[r][2] = fmaf(wv, x0.z, acc[r][2]); acc[r][3] = fmaf(wv, x0.w, acc[r][3]);
                acc[r][4] = fmaf(wv, x1.x, acc[r][4]); acc[r][5] = fmaf(wv, x1.y, acc[r][5]);
                acc[r][6] = fmaf(wv, x1.z, acc[r][6]); acc[r][7] = fmaf(wv, x1.w, acc[r][7]);
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int q = 0; q < kNetAtoms; ++q) tot[r][q] += acc[r][q];
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (has[r]) out(u0 + 32 * r, tot[r]);
}

// out(u, values of the eight atoms) for every unit u < U of the layer: bias[u] + sum_k W[k][u] in[k][q].
template <class Out>
__device__ __forceinline__ void warp_layer(const float* __restrict__ W, const float* __restrict__ bias, int K, int U,
                                           const float* in, int lane, Out&& out) {
    for (int u0 = lane; u0 < U + lane; u0 += 64) {
        if (U - (u0 - lane) > 32) warp_units<2>(W, bias, K, U, u0, in, out);  // warp-uniform
        else warp_units<1>(W, bias, K, U, u0, in, out);
    }
}

// The same by a CTA: threads are (slice of a round, unit) pairs; the slices' sums go through red
// [kCtaThreads][8] and are added in order.
template <class Out>
__device__ __forceinline__ void cta_layer(const float* __restrict__ W, const float* __restrict__ bias, int K, int U,
                                          const float* in, float* red, Out&& out) {
    const int tid = threadIdx.x;
    for (int u0 = 0; u0 < U; u0 += kCtaThreads) {
        const int uw = min(U - u0, kCtaThreads), uc = (uw + 31) & ~31, R = kCtaThreads / uc;
        const int r = tid / uc, u = tid - r * uc;
        // element (unit, atom) sums of this thread: e = tid + 256 i
        constexpr int E = kNetAtoms;
        float tot[E];
#pragma unroll
        for (int i = 0; i < E; ++i) {
            const int e = tid + kCtaThreads * i;
            tot[i] = bias && e < uw * kNetAtoms ? bias[u0 + e / kNetAtoms] : 0.f;
        }
        for (int kb = 0; kb < K; kb += R * kSlice) {
            const int k0 = kb + r * kSlice, k1 = min(K, k0 + kSlice);
            if (r < R && u < uw && k0 < K) {
                float acc[kNetAtoms];
                slice_sum(W + u0 + u, U, in, k0, k1, acc);
                float4* o = reinterpret_cast<float4*>(red + (size_t)(r * uc + u) * kNetAtoms);
                o[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
                o[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
            }
            __syncthreads();
            const int ns = min(R, (K - kb + kSlice - 1) / kSlice);
#pragma unroll
            for (int i = 0; i < E; ++i) {
                const int e = tid + kCtaThreads * i;
                if (e < uw * kNetAtoms)
                    for (int s = 0; s < ns; ++s) tot[i] += red[(size_t)s * uc * kNetAtoms + e];
            }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < E; ++i) {
            const int e = tid + kCtaThreads * i;
            if (e < uw * kNetAtoms) out(u0 + e / kNetAtoms, e % kNetAtoms, tot[i]);
        }
    }
}

// Energy of atom slot0 + q from the last layer's activations, by one warp.
__device__ __forceinline__ float out_sum(const float* wo, const float* cur, int H, int q, int lane) {
    float s = 0.f;
    for (int o = lane; o < H; o += 32) s = fmaf(wo[o], cur[o * kNetAtoms + q], s);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    return s;
}

// Eight atoms of a species by a warp (CTA false) or a CTA.  buf0 / buf1: [widest][8]; sd: silu'
// of every layer, [nlayer][widest][8].
template <bool CTA>
__device__ __forceinline__ void net_eight(const NetArgs& a, int slot0, int na, float* buf0, float* buf1, float* sd, float* red) {
    const int lane = threadIdx.x & 31, t = CTA ? threadIdx.x : lane, nt = CTA ? kCtaThreads : 32;
    auto sync = [] {
        if (CTA) __syncthreads();
        else __syncwarp();
    };
    // one(u, q, z) returns the value kept in dst[u][q]
    auto layer = [&](const float* W, const float* bias, int K, int U, const float* in, float* dst, auto&& one) {
        if constexpr (CTA)
            cta_layer(W, bias, K, U, in, red, [&](int u, int q, float z) { dst[u * kNetAtoms + q] = one(u, q, z); });
        else
            warp_layer(W, bias, K, U, in, lane, [&](int u, const float* z) {
                float4* d = reinterpret_cast<float4*>(dst + u * kNetAtoms);
                d[0] = make_float4(one(u, 0, z[0]), one(u, 1, z[1]), one(u, 2, z[2]), one(u, 3, z[3]));
                d[1] = make_float4(one(u, 4, z[4]), one(u, 5, z[5]), one(u, 6, z[6]), one(u, 7, z[7]));
            });
        sync();
    };
    const int Hmax = widest(a), L = a.nlayer;
    const float* mu = a.w;
    const float* isig = mu + a.D;
    // normalised input, [i][atom]
    if (CTA) {  // a warp per atom
        const int q = threadIdx.x >> 5;
        for (int i = lane; i < a.D; i += 32)
            buf0[i * kNetAtoms + q] = q < na ? (a.fp[(size_t)(slot0 + q) * a.fp_stride + i] - mu[i]) * isig[i] : 0.f;
    } else {
        for (int i = lane; i < a.D; i += 32) {
            float v[kNetAtoms];
#pragma unroll
            for (int q = 0; q < kNetAtoms; ++q)
                v[q] = q < na ? (a.fp[(size_t)(slot0 + q) * a.fp_stride + i] - mu[i]) * isig[i] : 0.f;
            float4* d = reinterpret_cast<float4*>(buf0 + i * kNetAtoms);
            d[0] = make_float4(v[0], v[1], v[2], v[3]);
            d[1] = make_float4(v[4], v[5], v[6], v[7]);
        }
    }
    sync();
    float* cur = buf0;
    float* nxt = buf1;
    const float* p = a.w + 2 * (size_t)a.D;
    int in = a.D;
    for (int l = 0; l < L; ++l) {
        const int H = a.H[l];
        const float* bias = p + 2 * (size_t)in * H;
        layer(p, bias, in, H, cur, nxt, [&](int u, int q, float z) {
            float g;
            const float h = act_and_grad(z, &g, a.act);
            sd[((size_t)l * Hmax + u) * kNetAtoms + q] = g;
            return h;
        });
        p = bias + H;
        in = H;
        float* s = cur; cur = nxt; nxt = s;
    }
    const float* wo = p;
    const float bo = wo[in];
    float eq = 0.f;  // atom q = lane's output
    if (CTA) {       // a warp per atom
        const float s = out_sum(wo, cur, in, threadIdx.x >> 5, lane);
        if (lane == 0) red[threadIdx.x >> 5] = s;
        __syncthreads();
        if (threadIdx.x < kNetAtoms) eq = red[threadIdx.x];
    } else {
        float s[kNetAtoms];
#pragma unroll
        for (int q = 0; q < kNetAtoms; ++q) s[q] = out_sum(wo, cur, in, q, lane);
#pragma unroll
        for (int q = 0; q < kNetAtoms; ++q)
            if (lane == q) eq = s[q];
    }
    if (t < na) a.e_atom[a.perm[slot0 + t]] = ((double)eq + (double)bo) * a.sigma_e + a.mu_e;
    sync();
    // backward: dz_L = sigma_E * w_out * silu'(z_L)
    const float se = (float)a.sigma_e;
    for (int e = t; e < in * kNetAtoms; e += nt) cur[e] = se * wo[e / kNetAtoms] * sd[(size_t)(L - 1) * Hmax * kNetAtoms + e];
    sync();
    for (int l = L - 1; l >= 0; --l) {
        const int H = in, lin = l ? a.H[l - 1] : a.D;
        p -= 2 * (size_t)lin * H + H;
        const float* W = p + (size_t)lin * H;
        if (l > 0) {
            layer(W, nullptr, H, lin, cur, nxt,
                  [&](int u, int q, float g) { return g * sd[((size_t)(l - 1) * Hmax + u) * kNetAtoms + q]; });
            float* s = cur; cur = nxt; nxt = s;
        } else {  // dE/dfp
            float* gf = a.gfp + (size_t)slot0 * a.fp_stride;
            if constexpr (CTA) {
                layer(W, nullptr, H, lin, cur, nxt, [&](int u, int, float g) { return g * isig[u]; });
                const int q = threadIdx.x >> 5;
                if (q < na)
                    for (int i = lane; i < lin; i += 32) gf[(size_t)q * a.fp_stride + i] = nxt[i * kNetAtoms + q];
            } else {
                warp_layer(W, nullptr, H, lin, cur, lane, [&](int u, const float* g) {
#pragma unroll
                    for (int q = 0; q < kNetAtoms; ++q)
                        if (q < na) gf[(size_t)q * a.fp_stride + u] = g[q] * isig[u];
                });
            }
        }
        in = lin;
    }
}

struct NetMulti {
    NetArgs a[kMaxTypes];
};

__global__ void __launch_bounds__(32 * kNetWarps) k_net_warp(const __grid_constant__ NetMulti m, int warp_floats) {
    pdl_enter();
    extern __shared__ __align__(16) float smem[];
    const NetArgs& a = m.a[blockIdx.y];
    const int wl = threadIdx.x >> 5;
    const int s0 = a.range[a.t], s1 = a.range[a.t + 1];
    const int slot0 = s0 + (blockIdx.x * (blockDim.x >> 5) + wl) * kNetAtoms;
    if (slot0 >= s1) return;
    const int Hm = widest(a) * kNetAtoms;
    float* b = smem + (size_t)wl * warp_floats;
    net_eight<false>(a, slot0, min(kNetAtoms, s1 - slot0), b, b + Hm, b + 2 * Hm, nullptr);
}

__global__ void __launch_bounds__(kCtaThreads) k_net_cta(const __grid_constant__ NetMulti m) {
    pdl_enter();
    extern __shared__ __align__(16) float smem[];
    const NetArgs& a = m.a[blockIdx.y];
    const int s0 = a.range[a.t], s1 = a.range[a.t + 1];
    const int slot0 = s0 + blockIdx.x * kNetAtoms;
    if (slot0 >= s1) return;
    const int Hm = widest(a) * kNetAtoms;
    float* b = smem + kCtaThreads * kNetAtoms;
    net_eight<true>(a, slot0, min(kNetAtoms, s1 - slot0), b, b + Hm, b + 2 * Hm, smem);
}

// One species with narrow layers (at most kSlice inputs, so every sum is one slice): a warp per
// eight atoms with one unit per lane and no slices, the shortest chain (11-32-32 network, 100
// atoms: 14 us against 20 by k_net_warp; 100k atoms: 61 against 75).
__global__ void __launch_bounds__(32 * kNetWarps) k_net_fp32(NetArgs a, int warp_floats) {
    pdl_enter();
    extern __shared__ float smem[];
    const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s0 = a.range[a.t], s1 = a.range[a.t + 1];
    const int slot0 = s0 + (blockIdx.x * (blockDim.x >> 5) + wl) * kNetAtoms;
    if (slot0 >= s1) return;
    const int na = min(kNetAtoms, s1 - slot0);
    int Hmax = a.D;
    for (int l = 0; l < a.nlayer; ++l) Hmax = max(Hmax, a.H[l]);
    float* buf0 = smem + (size_t)wl * warp_floats;        // [Hmax][8]
    float* buf1 = buf0 + Hmax * kNetAtoms;                  // [Hmax][8]
    float* sd = buf1 + Hmax * kNetAtoms;                    // [nlayer][Hmax][8] silu'
    const float* mu = a.w;
    const float* isig = mu + a.D;
    // normalised input, layout [i][atom]
    for (int i = lane; i < a.D; i += 32)
#pragma unroll
        for (int q = 0; q < kNetAtoms; ++q)
            buf0[i * kNetAtoms + q] = q < na ? (a.fp[(size_t)(slot0 + q) * a.fp_stride + i] - mu[i]) * isig[i] : 0.f;
    __syncwarp();
    const float* p = isig + a.D;
    const float* layerW[kNetMaxLayers];
    int in = a.D;
    float* cur = buf0;
    float* nxt = buf1;
    for (int l = 0; l < a.nlayer; ++l) {
        const int H = a.H[l];
        const float* WT = p;
        layerW[l] = p + (size_t)in * H;
        const float* b = layerW[l] + (size_t)H * in;
        for (int o = lane; o < H; o += 32) {
            float z[kNetAtoms];
#pragma unroll
            for (int q = 0; q < kNetAtoms; ++q) z[q] = b[o];
#pragma unroll 8
            for (int i = 0; i < in; ++i) {
                const float wv = WT[(size_t)i * H + o];
                const float4 x0 = *reinterpret_cast<const float4*>(cur + i * kNetAtoms);
                const float4 x1 = *reinterpret_cast<const float4*>(cur + i * kNetAtoms + 4);
                z[0] += wv * x0.x; z[1] += wv * x0.y; z[2] += wv * x0.z; z[3] += wv * x0.w;
                z[4] += wv * x1.x; z[5] += wv * x1.y; z[6] += wv * x1.z; z[7] += wv * x1.w;
            }
#pragma unroll
            for (int q = 0; q < kNetAtoms; ++q) {
                float gz;
                nxt[o * kNetAtoms + q] = act_and_grad(z[q], &gz, a.act);
                sd[((size_t)l * Hmax + o) * kNetAtoms + q] = gz;
            }
        }
        __syncwarp();
        p = b + H;
        in = H;
        float* t = cur; cur = nxt; nxt = t;
    }
    const float* wo = p;
    const float bo = wo[in];
    // output layer and energies
    float part[kNetAtoms];
#pragma unroll
    for (int q = 0; q < kNetAtoms; ++q) part[q] = 0.f;
    for (int o = lane; o < in; o += 32)
#pragma unroll
        for (int q = 0; q < kNetAtoms; ++q) part[q] += wo[o] * cur[o * kNetAtoms + q];
#pragma unroll
    for (int q = 0; q < kNetAtoms; ++q)
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) part[q] += __shfl_xor_sync(0xffffffffu, part[q], off);
    if (lane < na) {
        float outv = part[0];
#pragma unroll
        for (int q = 1; q < kNetAtoms; ++q) if (lane == q) outv = part[q];
        a.e_atom[a.perm[slot0 + lane]] = ((double)outv + (double)bo) * a.sigma_e + a.mu_e;
    }
    __syncwarp();
    // backward: dz_L = sigma_E * w_out * silu'(z_L)
    const float se = (float)a.sigma_e;
    const int L = a.nlayer;
    for (int o = lane; o < in; o += 32)
#pragma unroll
        for (int q = 0; q < kNetAtoms; ++q)
            cur[o * kNetAtoms + q] = se * wo[o] * sd[((size_t)(L - 1) * Hmax + o) * kNetAtoms + q];
    __syncwarp();
    for (int l = L - 1; l >= 0; --l) {
        const int H = a.H[l];
        const int lin = l ? a.H[l - 1] : a.D;
        const float* W = layerW[l];
        for (int i = lane; i < lin; i += 32) {
            float g[kNetAtoms];
#pragma unroll
            for (int q = 0; q < kNetAtoms; ++q) g[q] = 0.f;
#pragma unroll 8
            for (int o = 0; o < H; ++o) {
                const float wv = W[(size_t)o * lin + i];
                const float4 d0 = *reinterpret_cast<const float4*>(cur + o * kNetAtoms);
                const float4 d1 = *reinterpret_cast<const float4*>(cur + o * kNetAtoms + 4);
                g[0] += wv * d0.x; g[1] += wv * d0.y; g[2] += wv * d0.z; g[3] += wv * d0.w;
                g[4] += wv * d1.x; g[5] += wv * d1.y; g[6] += wv * d1.z; g[7] += wv * d1.w;
            }
            if (l > 0) {
#pragma unroll
                for (int q = 0; q < kNetAtoms; ++q)
                    nxt[i * kNetAtoms + q] = g[q] * sd[((size_t)(l - 1) * Hmax + i) * kNetAtoms + q];
            } else {
#pragma unroll
                for (int q = 0; q < kNetAtoms; ++q)
                    if (q < na) a.gfp[(size_t)(slot0 + q) * a.fp_stride + i] = g[q] * isig[i];
            }
        }
        __syncwarp();
        float* t = cur; cur = nxt; nxt = t;
    }
}

int net_warp_floats(int D, int nlayer, const int* H) {
    int Hmax = D;
    for (int l = 0; l < nlayer; ++l) Hmax = Hmax > H[l] ? Hmax : H[l];
    return (2 + nlayer) * Hmax * kNetAtoms;
}
constexpr size_t kNetSmemMax = 227 * 1024;

}  // namespace

bool net_fp32_fits(int D, int nlayer, const int* H) {
    return nlayer >= 1 && nlayer <= kNetMaxLayers && sizeof(float) * (size_t)net_warp_floats(D, nlayer, H) <= kNetSmemMax;
}

cudaError_t launch_net_fp32(const NetArgs* args, int count, int sms, cudaStream_t st) {
    if (count <= 0 || count > kMaxTypes) return count ? cudaErrorInvalidValue : cudaSuccess;
    const int n = args[0].nmax;
    if (n <= 0) return cudaSuccess;
    NetMulti m;
    int wf = 0;
    bool deep = false;
    for (int k = 0; k < count; ++k) {
        const NetArgs& a = args[k];
        if (!net_fp32_fits(a.D, a.nlayer, a.H)) return cudaErrorInvalidValue;
        m.a[k] = a;
        const int w = net_warp_floats(a.D, a.nlayer, a.H);
        wf = wf > w ? wf : w;
        for (int l = 0; l <= a.nlayer; ++l) deep = deep || (l ? a.H[l - 1] : a.D) > kSlice;
    }
    const size_t cta = sizeof(float) * ((size_t)wf + kCtaThreads * kNetAtoms);
    int wpc = kNetWarps;  // fewer warps per CTA for wide networks
    while (wpc > 1 && sizeof(float) * (size_t)wf * wpc > kNetSmemMax) wpc >>= 1;
    const size_t sm = sizeof(float) * (size_t)wf * wpc;
    const int per_block = kNetAtoms * wpc;
    if (count == 1 && !deep) {
        const cudaError_t e = allow_smem(k_net_fp32, sm);
        if (e != cudaSuccess) return e;
        return launch_pdl(&k_net_fp32, dim3((n + per_block - 1) / per_block), dim3(32 * wpc), sm, st, args[0], wf);
    }
    // a CTA per eight atoms up to three of them per SM.  The CTA form takes a step with each CTA that
    // an SM gets, the warp form is flat until SMs fill: up to 2400 atoms 24 against 45 us for
    // 126-64-64 and 22 against 28 for 84-32-32, from there to this limit (3648 atoms) 43 against 45
    // and 37 against 29, beyond it (5000) 58 against 49 and 51 against 31
    if (n <= 24 * sms && deep && cta <= kNetSmemMax) {
        const cudaError_t e = allow_smem(k_net_cta, cta);
        if (e != cudaSuccess) return e;
        return launch_pdl(&k_net_cta, dim3((n + kNetAtoms - 1) / kNetAtoms, count), dim3(kCtaThreads), cta, st, m);
    }
    const cudaError_t e = allow_smem(k_net_warp, sm);
    if (e != cudaSuccess) return e;
    return launch_pdl(&k_net_warp, dim3((n + per_block - 1) / per_block, count), dim3(32 * wpc), sm, st, m, wf);
}

}  // namespace nnapgb

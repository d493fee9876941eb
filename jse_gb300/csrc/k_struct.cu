// Structure kernels: FP64 wrapping and cell binning, the full neighbour list,
// the mirror index used by the atomic-free scatter, the species sort of atoms,
// the force / per-atom virial gather and the per-structure FP64 reductions.
//
// Reference behaviour restated here:
//   wrapping        IBox.wrapPBC / toDirect / toCartesian (IBox.java:145-222,
//                   BoxPrism.java:162-175), including the snap of direct coordinates
//                   within 1e-10 of an integer (MathEX.java:1213).  All FP64 operations
//                   use explicit round-to-nearest intrinsics so that no multiply-add is
//                   contracted and every rounding matches the reference's Java doubles.
//   neighbours      NeighborListGetter.forEachNeighbor_ with check=true, half=false
//                   (NeighborListGetter.java:1018-1050): all periodic images j' with
//                   |(x_j + shift) - x_i|^2 < rcut^2 evaluated in FP64, images of i
//                   itself included, (i, zero image) excluded (NeighborListGetter.java:119-173).
//   scatter         NNAP.calEnergyForceVirial + IPairPotential accumulators
//                   (NNAP.java:571-592, IPairPotential.java:919-1006): F_i -= g_ij,
//                   F_j += g_ij, per-atom virial dx_ij (x) g_ij on j; computed here as a
//                   gather over each atom's own row and the mirrored entries, without atomics.
#include "box_math.cuh"
#include "common.cuh"
#include "pdl.cuh"
#include "smem_limit.cuh"

namespace nnapgb {

// ----------------------------------------------------------------- wrap + cell binning
// One thread per atom: wrap into the box, record the float copy used by the
// candidate screen and the atom's cell, and count atoms per cell.
__global__ void k_wrap_bin(const StructDev* __restrict__ S, const int* __restrict__ sid, const double* __restrict__ x,
                           const int* __restrict__ type, int n, int ntypes, double* __restrict__ xw,
                           float4* __restrict__ xf, float4* __restrict__ xlo, int* __restrict__ cell_of,
                           int* __restrict__ cell_count, int* __restrict__ err) {
    pdl_enter();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const StructDev& st = S[sid[i]];
    const int t = type[i];
    if (t < 1 || t > ntypes) atomicOr(err, ERRBIT_BAD_TYPE);
    double p[3] = {x[3 * i], x[3 * i + 1], x[3 * i + 2]};
    to_direct(st, p);
#pragma unroll
    for (int d = 0; d < 3; ++d)
        if (p[d] < 0.0 || p[d] >= 1.0) p[d] = ds(p[d], floor(p[d]));
    // the cell comes from these wrapped direct coordinates: every atom is binned by the same
    // rule, and the stencil's slack (R cells cover at least rc plus 1e-6 of a cell) dwarfs
    // their rounding, so no second conversion of the wrapped position is needed
    const double f[3] = {p[0], p[1], p[2]};
    to_cartesian(st, p);
    xw[3 * i] = p[0]; xw[3 * i + 1] = p[1]; xw[3 * i + 2] = p[2];
    const float hx = (float)p[0], hy = (float)p[1], hz = (float)p[2];
    // the species the pair rows carry, clamped into 1..ntypes: a bad species fails the call
    // (ERRBIT_BAD_TYPE) and indexes nothing out of range meanwhile
    xf[i] = make_float4(hx, hy, hz, __int_as_float(min(max(t, 1), ntypes)));
    // x = hi + lo exactly to 48 bits: the float-float form used by the neighbour test
    xlo[i] = make_float4((float)ds(p[0], (double)hx), (float)ds(p[1], (double)hy), (float)ds(p[2], (double)hz), 0.f);
    int c[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        int ci = (int)floor(f[d] * (double)st.nc[d]);
        c[d] = min(max(ci, 0), st.nc[d] - 1);
    }
    const int cid = st.c0 + c[0] + st.nc[0] * (c[1] + st.nc[1] * c[2]);
    cell_of[i] = cid;
    if (cell_count) atomicAdd(&cell_count[cid], 1);
}

// Exclusive scan of n ints by one CTA of 1024 threads; out has n + 1 entries.  A thread takes
// kScanItems consecutive ints per round (16-byte loads; in and out are the starts of their own
// allocations), so the serial part is n / 8192 rounds: with one int per thread, 100k cells took
// 92 us, now 28.
constexpr int kScanItems = 8;

__global__ void k_scan_excl(const int* __restrict__ in, int n, int* __restrict__ out) {
    pdl_enter();
    __shared__ int warp_tot[2][32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    int carry = 0;
    int round = 0;
    for (int base = 0; base < n; base += 1024 * kScanItems, round ^= 1) {
        const int i0 = base + tid * kScanItems;
        int v[kScanItems];
        if (i0 + kScanItems <= n) {
#pragma unroll
            for (int k = 0; k < kScanItems / 4; ++k) {
                const int4 q = reinterpret_cast<const int4*>(in + i0)[k];
                v[4 * k] = q.x; v[4 * k + 1] = q.y; v[4 * k + 2] = q.z; v[4 * k + 3] = q.w;
            }
        } else {
#pragma unroll
            for (int k = 0; k < kScanItems; ++k) v[k] = i0 + k < n ? in[i0 + k] : 0;
        }
        int own = 0;
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) own += v[k];
        int s = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += u;
        }
        if (lane == 31) warp_tot[round][w] = s;
        __syncthreads();
        // every warp scans the warps' totals for itself: one barrier per round
        int t = warp_tot[round][lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += u;
        }
        const int before = w ? __shfl_sync(0xffffffffu, t, w - 1) : 0;
        int x = carry + before + s - own;
        carry += __shfl_sync(0xffffffffu, t, 31);
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            const int y = x + v[k];
            v[k] = x;
            x = y;
        }
        if (i0 + kScanItems <= n) {
#pragma unroll
            for (int k = 0; k < kScanItems / 4; ++k)
                reinterpret_cast<int4*>(out + i0)[k] = make_int4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
        } else {
#pragma unroll
            for (int k = 0; k < kScanItems; ++k)
                if (i0 + k < n) out[i0 + k] = v[k];
        }
    }
    if (tid == 0) out[n] = carry;
}

__global__ void k_fill_cells(const int* __restrict__ cell_of, int n, const int* __restrict__ cell_start,
                             int* __restrict__ cell_fill, int* __restrict__ cell_atoms) {
    pdl_enter();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int c = cell_of[i];
    cell_atoms[cell_start[c] + atomicAdd(&cell_fill[c], 1)] = i;
}

// Order each cell's atoms by index so that every neighbour row is deterministic.
// One warp per cell (8 per CTA of 256 threads): up to 32 atoms are placed by rank from
// registers; up to kSortCellMax atoms by rank from a copy of the cell in shared memory (the
// small boxes of a batch have cells of a hundred atoms); larger cells are sorted by lane 0.
constexpr int kSortCellMax = 1024;

__global__ void k_sort_cells(const int* __restrict__ cell_start, int ncells, int* __restrict__ cell_atoms) {
    pdl_enter();
    __shared__ int s_cell[8][kSortCellMax];
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) & 7;
    if (c >= ncells) return;
    const int b = cell_start[c], e = cell_start[c + 1], m = e - b;
    if (m <= 32) {
        const int v = lane < m ? cell_atoms[b + lane] : 0x7fffffff;
        int rank = 0;
        for (int q = 0; q < m; ++q) {
            const int u = __shfl_sync(0xffffffffu, v, q);
            rank += (u < v) ? 1 : 0;
        }
        __syncwarp();
        if (lane < m) cell_atoms[b + rank] = v;
    } else if (m <= kSortCellMax) {
        for (int t = lane; t < m; t += 32) s_cell[w][t] = cell_atoms[b + t];
        __syncwarp();
        for (int t = lane; t < m; t += 32) {
            const int v = s_cell[w][t];
            int rank = 0;
            for (int q = 0; q < m; ++q) rank += s_cell[w][q] < v ? 1 : 0;
            cell_atoms[b + rank] = v;
        }
    } else if (lane == 0) {
        for (int k = b + 1; k < e; ++k) {
            const int v = cell_atoms[k];
            int q = k - 1;
            while (q >= b && cell_atoms[q] > v) { cell_atoms[q + 1] = cell_atoms[q]; --q; }
            cell_atoms[q + 1] = v;
        }
    }
}

// ----------------------------------------------------------------- neighbour rows
// One warp per chunk of up to kNbAtoms consecutive cell-order positions.  The atoms of the
// chunk that share a cell share its candidates: the stencil cells' ranges, image shifts and
// pruning, and each window of 32 candidates (one per lane, shifted position in registers), are
// formed once and screened in FP32 against every atom of the run (rc^2 plus a rounding margin).
// Candidates that pass (about one in six) queue per atom in shared memory in candidate order
// and take the exact test 32 at a time, so its lanes stay busy.  Accepted pairs are compacted
// in candidate order with a ballot, so rows are deterministic and do not depend on the chunk.
// Candidate positions are read from the cell-ordered copies xfc / xloc (k_cell_order), so
// a lane's atom index and position loads are independent and a cell's candidates are
// contiguous in memory.
// Bound: instruction issue and its dependences (131072 atoms, 8 per warp: 1106 warp instructions
// per atom, 63 % of the issue slots at 20 warps per SM; one atom per warp, which set up its cells
// and looked up the cell of each candidate for itself, took 2068 at 75 % on the batch).  Neighbour stage of the batch of 1024
// structures 1.78 -> 1.40 ms, of the 1M-atom glass 3.05 -> 2.33 ms.
constexpr int kNbMaxWarps = 8;  // warps per CTA are a launch parameter (2, 4 or 8)
constexpr int kNbAtoms = 8;     // most atoms per warp
constexpr int kNbQueue = 128;   // queued candidates per atom
constexpr int kNbSpan = 4;      // most cells between the first and last atom of a run

// floor(a / b) for b >= 1 and |a| < 2^22, from a float reciprocal of b and one correction
// step (the float quotient is within one of the true one).
__device__ __forceinline__ int floor_div(int a, int b, float inv_b) {
    int q = __float2int_rd((float)a * inv_b);
    const int r = a - q * b;
    if (r < 0) --q;
    else if (r >= b) ++q;
    return q;
}

// xfc[k] = xf[cell_atoms[k]], xloc[k] = xlo[cell_atoms[k]] for the n binned atoms.
__global__ void __launch_bounds__(256) k_cell_order(const int* __restrict__ cell_atoms, int n,
                                                    const float4* __restrict__ xf, const float4* __restrict__ xlo,
                                                    float4* __restrict__ xfc, float4* __restrict__ xloc) {
    pdl_enter();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int a = cell_atoms[k];
    xfc[k] = xf[a];
    xloc[k] = xlo[a];
}

// Renumber the atoms of an evaluation in cell order: position k of the sorted cell lists
// takes the float positions and low parts (xfc / xloc), the FP64 wrapped position, the cell
// and the species of the atom there, and orig[k] records that atom; the cell lists become
// the identity.  Rows, pair keys and per-atom work arrays then use cell-order numbers, so
// the rows of atoms close in space are close in memory (the mirror search and the gather
// read the rows of each atom's neighbours).  A structure's atoms keep their index range.
__global__ void __launch_bounds__(256) k_renumber(int* __restrict__ cell_atoms, int n, const float4* __restrict__ xf,
                                                  const float4* __restrict__ xlo, const double* __restrict__ xw,
                                                  const int* __restrict__ cell_of, const int* __restrict__ type,
                                                  float4* __restrict__ xfc, float4* __restrict__ xloc,
                                                  double* __restrict__ xw2, int* __restrict__ cell_of2,
                                                  int* __restrict__ type2, int* __restrict__ orig) {
    pdl_enter();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int a = cell_atoms[k];
    xfc[k] = xf[a];
    xloc[k] = xlo[a];
    xw2[3 * (size_t)k] = xw[3 * (size_t)a];
    xw2[3 * (size_t)k + 1] = xw[3 * (size_t)a + 1];
    xw2[3 * (size_t)k + 2] = xw[3 * (size_t)a + 2];
    cell_of2[k] = cell_of[a];
    type2[k] = type[a];
    orig[k] = a;
    cell_atoms[k] = k;
}

// The cell order, the renumbering and the species order of a small evaluation by one CTA, an
// atom per thread: the work of k_scan_excl, k_fill_cells, k_sort_cells, k_renumber (or
// k_cell_order) and the species sort, with the same results.  Each of those takes 2 to 4 us of
// latency whatever its size: the stage of 33 atoms 47 -> 40 us, of 500 atoms 52 -> 44.  (With
// several atoms per thread the one CTA's loads take longer than the launches: 2000 atoms 54
// against 51, 4000 atoms 73 against 59.)
__global__ void __launch_bounds__(kOrderAtoms) k_order_small(OrderArgs a) {
    pdl_enter();
    extern __shared__ int osm[];
    __shared__ int s_warp[32], s_tot[kMaxTypes + 1];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, n = a.n, C = a.ncells, T = a.T;
    int* cnt = osm;                               // [C + 1] counts, then starts
    int* list = osm + C + 1;                      // [n] atoms by cell, in no order inside a cell
    int* wc = list + n;                           // [ceil(n / 32)][T] species counts of 32 rows
    uint8_t* stype = reinterpret_cast<uint8_t*>(wc + ((n + 31) / 32) * T);  // [n] species of each row
    for (int c = tid; c <= C; c += kOrderAtoms) cnt[c] = 0;
    // this thread's atom
    const bool have = tid < n;
    int cell = 0, rk = 0, t = 0;
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f), lo = f;
    double x0 = 0.0, x1 = 0.0, x2 = 0.0;
    if (have) {
        cell = a.cell_of[tid];
        t = a.type[tid];
        f = a.xf[tid];
        lo = a.xlo[tid];
        if (a.renumber) {
            x0 = a.xw[3 * tid];
            x1 = a.xw[3 * tid + 1];
            x2 = a.xw[3 * tid + 2];
        }
    }
    __syncthreads();
    if (have) rk = atomicAdd(&cnt[cell], 1);
    __syncthreads();
    {  // exclusive scan of the counts, in place: consecutive cells per thread
        const int per = (C + kOrderAtoms) / kOrderAtoms, b = min(C + 1, tid * per), e = min(C + 1, b + per);
        int own = 0;
        for (int c = b; c < e; ++c) own += cnt[c];
        int s = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += u;
        }
        if (lane == 31) s_warp[w] = s;
        __syncthreads();
        int tot = s_warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, tot, o);
            if (lane >= o) tot += u;
        }
        const int before = w ? __shfl_sync(0xffffffffu, tot, w - 1) : 0;
        int x = before + s - own;
        for (int c = b; c < e; ++c) {
            const int v = cnt[c];
            cnt[c] = x;
            a.cell_start[c] = x;
            x += v;
        }
    }
    __syncthreads();
    if (have) list[cnt[cell] + rk] = tid;
    __syncthreads();
    if (have) {
        const int b = cnt[cell], e = cnt[cell + 1];
        int r = b;  // the atom's place: its rank by index in its cell
        for (int q = b; q < e; ++q) r += list[q] < tid ? 1 : 0;
        a.xfc[r] = f;
        a.xloc[r] = lo;
        if (a.renumber) {
            a.xw2[3 * r] = x0;
            a.xw2[3 * r + 1] = x1;
            a.xw2[3 * r + 2] = x2;
            a.cell_of2[r] = cell;
            a.type2[r] = t;
            a.orig[r] = tid;
            a.cell_atoms[r] = r;
        } else {
            a.cell_atoms[r] = tid;
        }
        stype[a.renumber ? r : tid] = t >= 1 && t <= T ? (uint8_t)(t - 1) : 255;
    }
    __syncthreads();
    // species order, stable: counts per 32 rows, their sums before each, then the ranks
    const int ty = have ? stype[tid] : 255;
    unsigned mine = 0;
    if (tid - lane < n)
        for (int q = 0; q < T; ++q) {
            const unsigned m = __ballot_sync(0xffffffffu, ty == q);
            if (lane == 0) wc[w * T + q] = __popc(m);
            if (ty == q) mine = m;
        }
    __syncthreads();
    if (w < T) {  // kMaxTypes <= 32 warps, and at most 32 groups of rows
        const int v = lane * 32 < n ? wc[lane * T + w] : 0;
        int s = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += u;
        }
        if (lane * 32 < n) wc[lane * T + w] = s - v;
        if (lane == 31) s_tot[w] = s;
    }
    __syncthreads();
    int base = 0;
    for (int q = 0; q < T; ++q) {
        if (tid == 0) a.type_start[q] = base;
        if (q == ty) a.perm[base + wc[w * T + q] + __popc(mine & ((1u << lane) - 1u))] = tid;
        base += s_tot[q];
    }
    if (tid == 0) a.type_start[T] = base;
}

// Shared memory of k_order_small, or 0 when the evaluation is not one for it.
size_t order_small_bytes(int n, int ncells, int T) {
    if (n < 1 || n > kOrderAtoms || ncells > kOrderCells) return 0;
    return sizeof(int) * ((size_t)ncells + 1 + n + (size_t)((n + 31) / 32) * T) + ((n + 15) & ~15);
}

cudaError_t launch_order_small(const OrderArgs& a, cudaStream_t st) {
    const size_t sm = order_small_bytes(a.n, a.ncells, a.T);  // at most 24 KB
    return launch_pdl(k_order_small, dim3(1), dim3(kOrderAtoms), sm, st, a);
}

// out[orig[k]] = in[k]: a per-atom array of a cell-ordered evaluation back in atom order.
__global__ void k_unpermute(const double* __restrict__ in, const int* __restrict__ orig, int n,
                            double* __restrict__ out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) out[orig[k]] = in[k];
}

// The requested results of a small host call into one mapped host buffer (PackArgs::out, offsets
// in doubles; -1: not wanted), per-atom energies back in atom order.
__global__ void k_pack_results(PackArgs p) {
    pdl_enter();
    const int step = gridDim.x * blockDim.x, t = blockIdx.x * blockDim.x + threadIdx.x;
    auto copy = [&](int off, const double* src, int count) {
        if (off >= 0)
            for (int k = t; k < count; k += step) p.out[off + k] = src[k];
    };
    copy(p.off[0], p.energy, p.nstruct);
    copy(p.off[3], p.virial, 9 * p.nstruct);
    if (p.off[1] >= 0)
        for (int k = t; k < p.n; k += step) p.out[p.off[1] + (p.orig ? p.orig[k] : k)] = p.e_atom[k];
    copy(p.off[2], p.forces, 3 * p.n);
    copy(p.off[4], p.virials, 9 * p.n);
}

// Shared memory of one warp; SLOTS stencil cells are held at a time (all of them where the
// structure has at most SLOTS).
template <int SLOTS, int NA>
struct NbWarp {
    // per cell slot: the image shift's high parts and the packed image (one 16-byte load in
    // the candidate loop), the shift's low parts (the float-float test), and the cell-order
    // start minus the candidate start
    float4 sh4[SLOTS];
    float4 fi[NA], li[NA];  // the run's atoms
    float4 box[2];                      // and their bounding box
    float flo[SLOTS][3];
    int base[32];
    int slot_at[32];  // cell slot starting at each position of a window
    int qn[NA], cnt[NA], last[NA];  // queued, accepted, last accepted group
    int dx[NA];                                 // cells along a from the run's first
    int qk[NA][kNbQueue];       // candidates passing the FP32 screen: position in cell order,
    uint8_t qs[NA][kNbQueue];   // cell slot
};

// The exact test of the first qn queued candidates of atom q of the run (row i); accepted ones
// are appended to the row.
template <int SLOTS, int NA>
__device__ __forceinline__ void nb_drain(NbWarp<SLOTS, NA>& sm, const StructDev& st, int q, int i, int o0, int noff,
                                         int wa, int wu, const double* __restrict__ xw, const float4* __restrict__ xfc,
                                         const float4* __restrict__ xloc, const int* __restrict__ cell_atoms,
                                         const PairBufs& P, int lane) {
    const float rc2h = (float)st.rc2, rc2l = (float)(st.rc2 - (double)(float)st.rc2);
    const float tol = 1e-10f * rc2h;  // float-float d^2 is accurate to ~1e-12 relative
    const bool keep_groups = P.GS > noff;
    const int M = P.M, qn = sm.qn[q];
    const float4 fi = sm.fi[q], li = sm.li[q];
    int cnt = sm.cnt[q], last = sm.last[q];
    int* gs = P.gstart + (size_t)i * P.GS;
    const int dx = SLOTS > 32 ? sm.dx[q] : 0;
    const float inv_wu = __frcp_rn((float)wu);
    for (int b = 0; b < qn; b += 32) {
        bool acc = false;
        int j = 0, slot = 0, g = 0;
        uint32_t img = 0;
        float fw = 0.f, ox = 0.f, oy = 0.f, oz = 0.f, lx = 0.f, ly = 0.f, lz = 0.f;
        if (b + lane < qn) {
            slot = sm.qs[q][b + lane];
            const int kp = sm.qk[q][b + lane];
            j = cell_atoms[kp];
            const float4 s4 = sm.sh4[slot];
            const float sh[3] = {s4.x, s4.y, s4.z};
            img = __float_as_uint(s4.w);
            const float4 fj = xfc[kp], lj = xloc[kp];
            fw = fj.w;
            // (x_j + shift) - x_i in float-float, then d^2 in float-float
            float dh[3], dl[3];
            const float ajh[3] = {fj.x, fj.y, fj.z}, ajl[3] = {lj.x, lj.y, lj.z};
            const float aih[3] = {fi.x, fi.y, fi.z}, ail[3] = {li.x, li.y, li.z};
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                float s1, e1, s2, e2;
                two_sum(ajh[d], sh[d], s1, e1);
                two_sum(s1, -aih[d], s2, e2);
                const float lo = ((ajl[d] + sm.flo[slot][d]) - ail[d]) + (e1 + e2);
                two_sum(s2, lo, dh[d], dl[d]);
            }
            float d2h = 0.f, d2l = 0.f;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                ff_acc_prod(d2h, d2l, dh[d], dh[d]);
                d2l += 2.f * dh[d] * dl[d];
            }
            const float diff = (d2h - rc2h) + (d2l - rc2l);
            if (fabsf(diff) > tol) {
                acc = diff < 0.f;
            } else {  // within 1e-10 of the cutoff: the exact FP64 test
                int na, nb, nc;
                unpack_img(img, na, nb, nc);
                double sd[3] = {0.0, 0.0, 0.0};
                if (na | nb | nc) image_shift(st, na, nb, nc, sd);
                const double dxv = ds(da(xw[3 * (size_t)j], sd[0]), xw[3 * (size_t)i]);
                const double dyv = ds(da(xw[3 * (size_t)j + 1], sd[1]), xw[3 * (size_t)i + 1]);
                const double dzv = ds(da(xw[3 * (size_t)j + 2], sd[2]), xw[3 * (size_t)i + 2]);
                acc = da(da(dm(dxv, dxv), dm(dyv, dyv)), dm(dzv, dzv)) < st.rc2;
            }
            if (j == i && img == pack_img(0, 0, 0)) acc = false;  // the atom itself
            two_sum(dh[0], dl[0], ox, lx);
            two_sum(dh[1], dl[1], oy, ly);
            two_sum(dh[2], dl[2], oz, lz);
            g = o0 + slot;
            if (SLOTS > 32) {  // the cell's offset from this atom's own cell
                const int rest = floor_div(g, wu, inv_wu), oa = g - rest * wu - dx;
                if (oa < 0 || oa >= wa) acc = false;
                g = oa + wa * rest;
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, acc);
        const unsigned lower = m & ((1u << lane) - 1u);
        const int gp = __shfl_sync(0xffffffffu, g, lower ? 31 - __clz(lower) : 0);
        if (acc) {
            const int pos = cnt + __popc(lower);
            if (pos < M) {
                const size_t e = (size_t)i * M + pos;
                P.key[e] = pair_key(j, img);
                P.dx[e] = make_float4(ox, oy, oz, fw);
                if (P.dxlo) P.dxlo[e] = make_float4(lx, ly, lz, 0.f);
                P.grp[e] = (uint16_t)g;
            }
            // the groups after the last accepted entry's, up to this one's, start here
            if (keep_groups)
                for (int o = (lower ? gp : last) + 1; o <= g; ++o) gs[o] = pos;
        }
        if (m) last = __shfl_sync(0xffffffffu, g, 31 - __clz(m));
        cnt += __popc(m);
    }
    __syncwarp();
    if (lane == 0) {
        sm.cnt[q] = cnt;
        sm.last[q] = last;
        sm.qn[q] = 0;
    }
    __syncwarp();
}

// NA cell-order positions per warp.
template <int SLOTS, int NA>
__global__ void __launch_bounds__(32 * kNbMaxWarps, NA == 1 ? 4 : 3)
k_neighbors(const StructDev* __restrict__ S, const int* __restrict__ sid, const double* __restrict__ xw,
            const float4* __restrict__ xfc, const float4* __restrict__ xloc, const int* __restrict__ cell_of,
            const int* __restrict__ cell_start, const int* __restrict__ cell_atoms, int n, PairBufs P,
            int* __restrict__ err, int* __restrict__ max_count) {
    pdl_enter();
    extern __shared__ __align__(16) uint8_t nb_smem[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    NbWarp<SLOTS, NA>& sm = reinterpret_cast<NbWarp<SLOTS, NA>*>(nb_smem)[w];
    const int k0 = (blockIdx.x * (blockDim.x >> 5) + w) * NA;
    const int k1 = min(n, k0 + NA);
    int most = 0;
    for (int kr = k0; kr < k1;) {
        // the run [kr, kr + A): chunk positions in one cell; where cells are half the cutoff wide
        // and hold a few atoms each (SLOTS > 32), in cells of one row along a, whose stencils
        // overlap: candidates come in the same order for each of them
        const int mine = kr + (lane & (NA - 1));
        const int ia = cell_atoms[min(mine, k1 - 1)];
        const int cell = cell_of[ia];
        const int cell0 = __shfl_sync(0xffffffffu, cell, 0);
        const int s0 = sid[__shfl_sync(0xffffffffu, ia, 0)];
        const StructDev& st = S[s0];
        bool in = cell == cell0;
        if (SLOTS > 32)
            in = cell - cell0 <= kNbSpan && sid[ia] == s0 && (cell - st.c0) / st.nc[0] == (cell0 - st.c0) / st.nc[0];
        const unsigned same = __ballot_sync(0xffffffffu, lane < NA && mine < k1 && in);
        const int A = __ffs(~same) - 1;  // atoms of a cell, and cells of a row, are contiguous
        const int span = SLOTS > 32 ? __shfl_sync(0xffffffffu, cell, A - 1) - cell0 : 0;
        const int kc = kr + min((int)(lane & (NA - 1)), A - 1);
        const float4 f = xfc[kc], lo4 = xloc[kc];
        __syncwarp();
        if (lane < NA) {
            sm.fi[lane] = f;
            sm.li[lane] = lo4;
            sm.qn[lane] = 0;
            sm.cnt[lane] = 0;
            sm.last[lane] = -1;
            if (SLOTS > 32) sm.dx[lane] = cell - cell0;
        }
        // bounding box of the run's atoms (Cartesian, or direct coordinates in a skewed box)
        float bl[3], bh[3];
        if (st.kind == 0) {
            bl[0] = f.x; bl[1] = f.y; bl[2] = f.z;
        } else {
#pragma unroll
            for (int d = 0; d < 3; ++d) bl[d] = st.iv[d][0] * f.x + st.iv[d][1] * f.y + st.iv[d][2] * f.z;
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            bh[d] = bl[d];
#pragma unroll
            for (int o = NA / 2; o > 0; o >>= 1) {
                bl[d] = fminf(bl[d], __shfl_xor_sync(0xffffffffu, bl[d], o));
                bh[d] = fmaxf(bh[d], __shfl_xor_sync(0xffffffffu, bh[d], o));
            }
        }
        __syncwarp();
        if (lane == 0) {
            sm.box[0] = make_float4(bl[0], bl[1], bl[2], 0.f);
            sm.box[1] = make_float4(bh[0], bh[1], bh[2], 0.f);
        }
        __syncwarp();
        const int cl = cell0 - st.c0;
        const int ci0 = cl % st.nc[0], ci1 = (cl / st.nc[0]) % st.nc[1], ci2 = cl / (st.nc[0] * st.nc[1]);
        const int wa = 2 * st.R[0] + 1, wb = 2 * st.R[1] + 1;
        const int noff = wa * wb * (2 * st.R[2] + 1);
        const int wu = wa + span, nun = wu * wb * (2 * st.R[2] + 1);  // the run's stencil
        const float rc2_hi = st.rc2_hi;
        for (int o0 = 0; o0 < nun; o0 += SLOTS) {
            for (int w0 = 0; w0 < SLOTS && o0 + w0 < nun; w0 += 32) {
                const int o = o0 + w0 + lane;
                int ccount = 0, cs = 0;
                if (o < nun) {
                    const float inv_wu = __frcp_rn((float)wu), inv_wb = __frcp_rn((float)wb);
                    const float inv_nc0 = __frcp_rn((float)st.nc[0]), inv_nc1 = __frcp_rn((float)st.nc[1]),
                                inv_nc2 = __frcp_rn((float)st.nc[2]);
                    const int oab = floor_div(o, wu, inv_wu), ocr = floor_div(oab, wb, inv_wb);
                    const int oa = o - oab * wu - st.R[0], ob = oab - ocr * wb - st.R[1], oc = ocr - st.R[2];
                    const int q0 = ci0 + oa, q1 = ci1 + ob, q2 = ci2 + oc;
                    const int na = floor_div(q0, st.nc[0], inv_nc0);
                    const int nb = floor_div(q1, st.nc[1], inv_nc1);
                    const int nc = floor_div(q2, st.nc[2], inv_nc2);
                    const int c0 = q0 - na * st.nc[0], c1 = q1 - nb * st.nc[1], c2 = q2 - nc * st.nc[2];
                    const int cid = st.c0 + c0 + st.nc[0] * (c1 + st.nc[1] * c2);
                    cs = cell_start[cid];
                    ccount = cell_start[cid + 1] - cs;
                    const int q[3] = {q0, q1, q2};
                    const float4 b0 = sm.box[0], b1 = sm.box[1];
                    const float bl[3] = {b0.x, b0.y, b0.z}, bh[3] = {b1.x, b1.y, b1.z};
                    if (st.kind == 0) {
                        // orthogonal box: a lower bound of the distance from the run's bounding box
                        // to the target cell (unwrapped cell q spans [q, q+1) cell widths); cells
                        // beyond the screen bound (rc^2 plus its rounding margin) hold no neighbour
                        const float wd[3] = {st.fa[0] / (float)st.nc[0], st.fb[1] / (float)st.nc[1],
                                             st.fc[2] / (float)st.nc[2]};
                        float g2 = 0.f;
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            const float g =
                                fmaxf(0.f, fmaxf((float)q[d] * wd[d] - bh[d], bl[d] - (float)(q[d] + 1) * wd[d]));
                            g2 += g * g;
                        }
                        if (g2 > rc2_hi) ccount = 0;
                    } else if (st.smin2 > 0.f) {
                        // skewed box: the gap in direct coordinates times the box's smallest
                        // singular value bounds the Cartesian distance from below
                        float g2 = 0.f;
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            const float inv_n = 1.f / (float)st.nc[d];
                            const float g =
                                fmaxf(0.f, fmaxf((float)q[d] * inv_n - bh[d], bl[d] - (float)(q[d] + 1) * inv_n));
                            g2 += g * g;
                        }
                        if (st.smin2 * g2 > rc2_hi) ccount = 0;
                    }
                    // the image shift as float-float on the FP32 pipe (the exact test forms the FP64
                    // shift itself); the zero image has an exactly zero shift
                    float hi[3], lo[3];
                    image_shift_ff(st, na, nb, nc, hi, lo);
                    sm.sh4[w0 + lane] = make_float4(hi[0], hi[1], hi[2], __uint_as_float(pack_img(na, nb, nc)));
#pragma unroll
                    for (int d = 0; d < 3; ++d) sm.flo[w0 + lane][d] = lo[d];
                }
                int incl = ccount;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    int u = __shfl_up_sync(0xffffffffu, incl, d);
                    if (lane >= d) incl += u;
                }
                const int total = __shfl_sync(0xffffffffu, incl, 31);
                const int before = incl - ccount;  // candidates of the earlier cell slots
                sm.base[lane] = cs - before;
                __syncwarp();
                // The cell slot of candidate cidx: the last nonempty slot starting at or before it.
                // Per window of 32 candidates the starting positions form a bit mask (one OR
                // reduction); a lane takes the highest start at or below its position, or the slot
                // that ran into the window from the one before.
                int carry = 0, cb = 0;
                const bool last = w0 + 32 >= SLOTS || o0 + w0 + 32 >= nun;
                do {
                    bool full = false;
                    // the run's positions, read again after a drain: registers are not held over it
                    float ax[NA], ay[NA], az[NA];
                    int qn[NA];
#pragma unroll
                    for (int q = 0; q < NA; ++q) {
                        const float4 v = sm.fi[q];
                        ax[q] = v.x; ay[q] = v.y; az[q] = v.z;
                        qn[q] = sm.qn[q];
                    }
                    for (; cb < total && !full; cb += 32) {
                        const int cidx = cb + lane;
                        const bool starts = ccount > 0 && before >= cb && before < cb + 32;
                        const unsigned smask = __reduce_or_sync(0xffffffffu, starts ? 1u << (before - cb) : 0u);
                        if (starts) sm.slot_at[before - cb] = lane;
                        __syncwarp();
                        const unsigned below = smask & (0xffffffffu >> (31 - lane));
                        const int slot = below ? sm.slot_at[31 - __clz(below)] : carry;
                        carry = __shfl_sync(0xffffffffu, slot, 31);
                        // the screen reads only the candidate's cell-order position; its atom index is
                        // loaded by the exact test, which also drops the atom itself (zero image)
                        int kp = 0;
                        float px = 3e38f, py = 0.f, pz = 0.f;  // no candidate: outside every cutoff
                        if (cidx < total) {
                            kp = sm.base[slot] + cidx;
                            const float4 fj = xfc[kp];
                            const float4 sh = sm.sh4[w0 + slot];
                            px = fj.x + sh.x;
                            py = fj.y + sh.y;
                            pz = fj.z + sh.z;
                        }
#pragma unroll
                        for (int q = 0; q < NA; ++q) {
                            if (q < A) {
                                const float fx = px - ax[q], fy = py - ay[q], fz = pz - az[q];
                                const bool pass = fx * fx + fy * fy + fz * fz < rc2_hi;
                                const unsigned m = __ballot_sync(0xffffffffu, pass);
                                if (pass) {
                                    const int at = qn[q] + __popc(m & ((1u << lane) - 1u));
                                    sm.qk[q][at] = kp;
                                    sm.qs[q][at] = (uint8_t)(w0 + slot);
                                }
                                qn[q] += __popc(m);
                                full = full || qn[q] > kNbQueue - 32;
                            }
                        }
                    }
                    __syncwarp();
                    if (lane == 0) {
#pragma unroll
                        for (int q = 0; q < NA; ++q) sm.qn[q] = qn[q];
                    }
                    __syncwarp();
                    if (full || last)  // warp-uniform: every queue through the exact test
                        for (int q = 0; q < A; ++q)
                            nb_drain<SLOTS, NA>(sm, st, q, cell_atoms[kr + q], o0, noff, wa, wu, xw, xfc, xloc, cell_atoms, P, lane);
                } while (cb < total);
                __syncwarp();
            }
        }
        if (P.GS > noff)
            for (int q = 0; q < A; ++q) {
                const int cnt = sm.cnt[q];
                int* gs = P.gstart + (size_t)cell_atoms[kr + q] * P.GS;
                for (int o = sm.last[q] + 1 + lane; o <= noff; o += 32) gs[o] = cnt;
            }
        if (lane < A) {
            const int cnt = sm.cnt[lane];
            P.count[ia] = cnt;
            if (cnt > P.M) atomicOr(err, ERRBIT_CAPACITY);
            most = max(most, cnt);
        }
        kr += A;
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0 && most > 0) atomicMax(max_count, most);
}

// Stencil cells held at a time and atoms per warp as template arguments of one launch.
template <int SLOTS, int NA>
static cudaError_t launch_nb(const StructDev* S, const int* sid, const double* xw, const float4* xfc, const float4* xloc,
                             const int* cell_of, const int* cell_start, const int* cell_atoms, int n, int warps,
                             const PairBufs& P, int* err, int* max_count, cudaStream_t st) {
    const size_t smem = warps * sizeof(NbWarp<SLOTS, NA>);
    const cudaError_t e = allow_smem(k_neighbors<SLOTS, NA>, smem);
    if (e != cudaSuccess) return e;
    const dim3 grid((unsigned)((n + warps * NA - 1) / (warps * NA))), block(32 * warps);
    // the kernels before have no shared memory: with many atoms each SM takes its split anew
    // (1048573 atoms 7159 -> 7078 us, 488206 5393 -> 5387, fewer the same)
    if (NA == 8)
        return launch_after(k_neighbors<SLOTS, NA>, grid, block, smem, st, S, sid, xw, xfc, xloc, cell_of, cell_start,
                            cell_atoms, n, P, err, max_count);
    return launch_pdl(k_neighbors<SLOTS, NA>, grid, block, smem, st, S, sid, xw, xfc, xloc, cell_of, cell_start, cell_atoms,
                      n, P, err, max_count);
}

cudaError_t launch_neighbors(const StructDev* S, const int* sid, const double* xw, const float4* xfc, const float4* xloc,
                             const int* cell_of, const int* cell_start, const int* cell_atoms, int n, int max_off,
                             int warps, int sms, const PairBufs& P, int* err, int* max_count, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    // atoms per warp: 8 where that leaves each SM 48 warps, two rounds of the resident ones,
    // halved until it does.  The stage with 1, 2, 4 and 8 atoms per warp: 4000 atoms 63, 66, 73,
    // 83 us; 25000 atoms 122, 122, 124, 131; 32000 atoms 141, 136, 130, 137 (half-width cells
    // 258, 230, 219, 244); 1M atoms 3163, 2858, 2497, 2293
    int chunk = kNbAtoms;
    while (chunk > 1 && n < chunk * 48 * sms) chunk >>= 1;
    const bool wide = max_off > 32;
#define NB_CASE(N_)                                                                                                     \
    if (chunk == N_)                                                                                                    \
        return wide ? launch_nb<128, N_>(S, sid, xw, xfc, xloc, cell_of, cell_start, cell_atoms, n, warps, P, err,      \
                                         max_count, st)                                                                 \
                    : launch_nb<32, N_>(S, sid, xw, xfc, xloc, cell_of, cell_start, cell_atoms, n, warps, P, err,       \
                                        max_count, st);
    NB_CASE(8) NB_CASE(4) NB_CASE(2)
    return wide ? launch_nb<128, 1>(S, sid, xw, xfc, xloc, cell_of, cell_start, cell_atoms, n, warps, P, err, max_count, st)
                : launch_nb<32, 1>(S, sid, xw, xfc, xloc, cell_of, cell_start, cell_atoms, n, warps, P, err, max_count, st);
#undef NB_CASE
}

// Mirror index: for entry (i -> j, image n) the position of (j -> i, image -n) in j's row.
// Rows are ordered by (cell-offset group, atom index); the mirrored entry lies in group
// noff-1-g of j's row (the negated cell offset).  With group starts kept, it is found
// in that group: halved by atom number to a few entries (a small box has tens of one image),
// which are read two at a time; otherwise by binary search on (group, atom).  One warp per row.
// Bound: the chain of dependent loads.  Reading a group's entries one after another took 14 us
// at 33 atoms and 549 on the 1M-atom glass, now 7 and 529 (1024-structure batch 402 -> 335).
__global__ void k_mirror(const StructDev* __restrict__ S, const int* __restrict__ sid, PairBufs P, int n,
                         int* __restrict__ err) {
    pdl_enter();
    const int i = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= n) return;
    const int M = P.M;
    const int ci = min(P.count[i], M);
    const StructDev& st = S[sid[i]];
    const int noff = (2 * st.R[0] + 1) * (2 * st.R[1] + 1) * (2 * st.R[2] + 1);
    const bool groups = P.GS > noff;
    for (int k = lane; k < ci; k += 32) {
        const size_t e = (size_t)i * M + k;
        const uint64_t key = P.key[e];
        const int j = (int)(key >> 32);
        const int want_g = noff - 1 - P.grp[e];
        int na, nb, nc;
        unpack_img((uint32_t)key, na, nb, nc);
        const uint64_t target = pair_key(i, pack_img(-na, -nb, -nc));
        const int cj = min(P.count[j], M);
        const uint64_t* row = P.key + (size_t)j * M;
        int found = -1;
        if (groups) {
            const int* gs = P.gstart + (size_t)j * P.GS;
            int lo = min(gs[want_g], cj);
            const int hi = min(gs[want_g + 1], cj);
            int len = hi - lo;
            while (len > 4) {  // the first entry whose atom is not below i stays within [lo, lo + len]
                const int half = len >> 1;
                const bool below = (int)(row[lo + half] >> 32) < i;
                lo = below ? lo + half + 1 : lo;
                len = below ? len - half - 1 : half;
            }
            for (int q = lo; q < hi && found < 0; q += 2) {
                const uint64_t v0 = row[q], v1 = q + 1 < hi ? row[q + 1] : 0;
                if (v0 == target) found = q;
                if (v1 == target) found = q + 1;
            }
        } else {
            const uint16_t* grow = P.grp + (size_t)j * M;
            const uint64_t want = ((uint64_t)(uint32_t)want_g << 32) | (uint32_t)i;
            int lo = 0, hi = cj;  // first q with composite(q) >= want
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                const uint64_t c = ((uint64_t)grow[mid] << 32) | (uint32_t)(row[mid] >> 32);
                if (c < want) lo = mid + 1; else hi = mid;
            }
            if (lo < cj && row[lo] == target) found = lo;
        }
        if (found >= 0) {
            P.rev[e] = (int)((size_t)j * M + found);
        } else {
            atomicOr(err, ERRBIT_NO_MIRROR);
            P.rev[e] = (int)e;
        }
    }
}

// ----------------------------------------------------------------- species sort
constexpr int kSortBlock = 256;

__global__ void k_type_hist(const int* __restrict__ type, int n, int T, int* __restrict__ block_counts) {
    pdl_enter();
    __shared__ int h[kMaxTypes];
    if (threadIdx.x < kMaxTypes) h[threadIdx.x] = 0;
    __syncthreads();
    const int i = blockIdx.x * kSortBlock + threadIdx.x;
    if (i < n) {
        const int t = type[i] - 1;
        if (t >= 0 && t < T) atomicAdd(&h[t], 1);
    }
    __syncthreads();
    if (threadIdx.x < T) block_counts[blockIdx.x * T + threadIdx.x] = h[threadIdx.x];
}

// In place: block_counts -> exclusive offsets in (type, block) order; type_start[T+1].
__global__ void k_type_offsets(int* __restrict__ block_counts, int nb, int T, int* __restrict__ type_start) {
    pdl_enter();
    __shared__ int warp_tot[32];
    __shared__ int carry;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid == 0) carry = 0;
    __syncthreads();
    for (int t = 0; t < T; ++t) {
        if (tid == 0) type_start[t] = carry;
        __syncthreads();
        for (int base = 0; base < nb; base += 1024) {
            const int b = base + tid;
            const int v = b < nb ? block_counts[b * T + t] : 0;
            int s = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                int u = __shfl_up_sync(0xffffffffu, s, o);
                if (lane >= o) s += u;
            }
            if (lane == 31) warp_tot[w] = s;
            __syncthreads();
            if (w == 0) {
                int q = warp_tot[lane];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    int u = __shfl_up_sync(0xffffffffu, q, o);
                    if (lane >= o) q += u;
                }
                warp_tot[lane] = q;
            }
            __syncthreads();
            const int before = (w ? warp_tot[w - 1] : 0) + carry;
            if (b < nb) block_counts[b * T + t] = before + s - v;
            __syncthreads();
            if (tid == 1023) carry = before + s;
            __syncthreads();
        }
    }
    if (tid == 0) type_start[T] = carry;
}

// Stable scatter: slot = offset(type, block) + rank of the atom among same-type atoms of its block.
__global__ void k_type_scatter(const int* __restrict__ type, int n, int T, const int* __restrict__ block_offsets,
                               int* __restrict__ perm) {
    pdl_enter();
    __shared__ int wc[kSortBlock / 32][kMaxTypes];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = blockIdx.x * kSortBlock + threadIdx.x;
    const int t = i < n ? type[i] - 1 : -1;
    unsigned mine = 0;
    for (int q = 0; q < T; ++q) {
        const unsigned m = __ballot_sync(0xffffffffu, t == q);
        if (lane == 0) wc[w][q] = __popc(m);
        if (t == q) mine = m;
    }
    __syncthreads();
    if (t < 0 || t >= T) return;
    int rank = __popc(mine & ((1u << lane) - 1u));
    for (int q = 0; q < w; ++q) rank += wc[q][t];
    perm[block_offsets[blockIdx.x * T + t] + rank] = i;
}

// ----------------------------------------------------------------- gather
// kGatherLanes lanes per atom a: F_a = sum_k (g[mirror(a,k)] - g[a,k]);
// W_a = sum_k dx[mirror(a,k)] (x) g[mirror(a,k)], with dx[mirror(a,k)] = -dx[a,k] (the
// mirrored displacement is the negated one; both are the same exact value rounded to
// nearest, which is symmetric under negation).  Each lane sums every kGatherLanes-th entry
// of the row as float-float pairs (exact products, error-free additions); the partial sums
// are combined by a fixed xor butterfly, so the result does not depend on timing.
// Own-row loads are coalesced; only g of the mirrored entry is a scattered load.  Four
// lanes per atom (eight atoms per warp) beat eight: 0.416 -> 0.347 ms on the batch's scatter
// stage.  Bound: HBM (the row, its mirror index and two gradients per entry); for few atoms the
// chain of loads and the instruction fetch, so the loop holds one entry and loads ahead:
// 286 -> 267 us on the batch, 455 -> 437 on the 1M-atom glass, 25 -> 18 on 4000 copper atoms.
constexpr int kGatherLanes = 4;

__device__ __forceinline__ void ff_merge(float& h, float& l, unsigned mask, int off) {
    const float oh = __shfl_xor_sync(mask, h, off), ol = __shfl_xor_sync(mask, l, off);
    float s, e;
    two_sum(h, oh, s, e);
    h = s;
    l = (l + ol) + e;
}

// orig: the atom of each row (rows in cell order), or NULL (rows are atoms).
__global__ void k_gather(PairBufs P, int n, const int* __restrict__ orig, double* __restrict__ forces,
                         double* __restrict__ virials) {
    pdl_enter();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int a = t / kGatherLanes, sub = t & (kGatherLanes - 1);
    if (a >= n) return;  // all lanes of an atom leave together
    const unsigned mask = ((1u << kGatherLanes) - 1u) << ((threadIdx.x & 31) & ~(kGatherLanes - 1));
    const int M = P.M;
    const int cnt = min(P.count[a], M);
    float fh[3] = {0.f, 0.f, 0.f}, fl[3] = {0.f, 0.f, 0.f};
    float vh[9], vl[9];
#pragma unroll
    for (int d = 0; d < 9; ++d) { vh[d] = 0.f; vl[d] = 0.f; }
    const size_t row = (size_t)a * M;
    // one entry per step, the next one's three loads and the mirror index of the one after it in
    // flight meanwhile
    constexpr int S = kGatherLanes;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 gr = zero, go = zero, dn = zero;
    int rn = 0;
    if (sub < cnt) {
        gr = P.g[P.rev[row + sub]];
        go = P.g[row + sub];
        dn = P.dx[row + sub];
        if (sub + S < cnt) rn = P.rev[row + sub + S];
    }
#pragma unroll 1
    for (int k = sub; k < cnt; k += S) {
        const float4 cr = gr, co = go, cd = dn;
        if (k + S < cnt) {
            gr = P.g[rn];
            go = P.g[row + k + S];
            dn = P.dx[row + k + S];
            if (k + 2 * S < cnt) rn = P.rev[row + k + 2 * S];
        }
        const float dx = -cd.x, dy = -cd.y, dz = -cd.z;
        ff_acc(fh[0], fl[0], cr.x); ff_acc(fh[0], fl[0], -co.x);
        ff_acc(fh[1], fl[1], cr.y); ff_acc(fh[1], fl[1], -co.y);
        ff_acc(fh[2], fl[2], cr.z); ff_acc(fh[2], fl[2], -co.z);
        ff_acc_prod(vh[0], vl[0], dx, cr.x);
        ff_acc_prod(vh[1], vl[1], dy, cr.y);
        ff_acc_prod(vh[2], vl[2], dz, cr.z);
        ff_acc_prod(vh[3], vl[3], dx, cr.y);
        ff_acc_prod(vh[4], vl[4], dx, cr.z);
        ff_acc_prod(vh[5], vl[5], dy, cr.z);
        ff_acc_prod(vh[6], vl[6], dy, cr.x);
        ff_acc_prod(vh[7], vl[7], dz, cr.x);
        ff_acc_prod(vh[8], vl[8], dz, cr.y);
    }
#pragma unroll
    for (int off = kGatherLanes / 2; off > 0; off >>= 1) {
#pragma unroll
        for (int d = 0; d < 3; ++d) ff_merge(fh[d], fl[d], mask, off);
#pragma unroll
        for (int d = 0; d < 9; ++d) ff_merge(vh[d], vl[d], mask, off);
    }
    if (sub == 0) {
        const size_t o = orig ? (size_t)orig[a] : (size_t)a;
#pragma unroll
        for (int d = 0; d < 3; ++d) forces[3 * o + d] = (double)fh[d] + (double)fl[d];
#pragma unroll
        for (int d = 0; d < 9; ++d) virials[9 * o + d] = (double)vh[d] + (double)vl[d];
    }
}

// ----------------------------------------------------------------- per-structure totals
// chunk c covers atoms [cb[c], ce[c]); partial[c][0] = sum E, partial[c][1..9] = sum W.  Where
// every structure is one chunk, energy and virial (else NULL) receive the totals at once.
constexpr int kRedBlock = 256;

__global__ void k_reduce_chunks(const int* __restrict__ cb, const int* __restrict__ ce,
                                const double* __restrict__ e_atom, const double* __restrict__ virials,
                                double* __restrict__ partial, double* __restrict__ energy,
                                double* __restrict__ virial) {
    pdl_enter();
    __shared__ double sm[10][kRedBlock / 32];
    const int c = blockIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double s[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int a = cb[c] + threadIdx.x; a < ce[c]; a += kRedBlock) {
        s[0] += e_atom[a];
#pragma unroll
        for (int d = 0; d < 9; ++d) s[1 + d] += virials[9 * (size_t)a + d];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int d = 0; d < 10; ++d) s[d] += __shfl_xor_sync(0xffffffffu, s[d], o);
    if (lane == 0)
#pragma unroll
        for (int d = 0; d < 10; ++d) sm[d][w] = s[d];
    __syncthreads();
    if (threadIdx.x < 10) {
        double t = 0.0;
        for (int q = 0; q < kRedBlock / 32; ++q) t += sm[threadIdx.x][q];
        if (!energy) partial[10 * (size_t)c + threadIdx.x] = t;
        else if (threadIdx.x == 0) energy[c] = t;
        else virial[9 * (size_t)c + threadIdx.x - 1] = t;
    }
}

// structure s owns chunks [sc[s], sc[s+1]); one warp per structure: lane q adds chunks q, q + 32,
// .., then a butterfly adds the lanes, a fixed order.  (Ten lanes that each added one total over
// all chunks took 107 us for the 1024 chunks of 1M atoms, now 32.)
__global__ void k_reduce_structs(const int* __restrict__ sc, int nstruct, const double* __restrict__ partial,
                                 double* __restrict__ energy, double* __restrict__ virial) {
    pdl_enter();
    const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (s >= nstruct) return;
    double t[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    const int c1 = sc[s + 1];
    for (int c = sc[s] + lane; c < c1; c += 32)
#pragma unroll
        for (int d = 0; d < 10; ++d) t[d] += partial[10 * (size_t)c + d];
    if (c1 - sc[s] > 1) {  // one chunk: lane 0 has the totals
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int d = 0; d < 10; ++d) t[d] += __shfl_xor_sync(0xffffffffu, t[d], o);
    }
    if (lane == 0) {
        energy[s] = t[0];
#pragma unroll
        for (int d = 1; d < 10; ++d) virial[9 * (size_t)s + d - 1] = t[d];
    }
}

}  // namespace nnapgb

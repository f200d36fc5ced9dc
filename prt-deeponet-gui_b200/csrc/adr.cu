// adr.cu -- the transport step of PRT-LB (solve_adr, prtlb_3d.py:781-1595)
// for sm_100a: finite-volume advection (MUSCL/minmod), harmonic-mean
// diffusion, the C div(u) correction, the inlet Dirichlet feed, the reaction
// source terms, forward Euler and the clip, fused into one launch per step.
//
// This file is compiled with -fmad=false.  The reference integrates in
// float32 with numpy, one rounding per operation; with no fused multiply-add
// and the reference's operation order kept below, every voxel of every step
// is bit-identical to it, and so are the convergence means (numpy's float32
// pairwise summation is replayed by adr_means_*), the stop step and the
// snapshots.
#include "adr_core.cuh"

namespace prt {

// 128-thread blocks: at 64^3 (117 164 solute voxels, 148 SMs) the finer
// blocks balance the SMs better than 256 (5.30 -> 5.01 us per step; the
// same at 128^3; 64 threads 5.08 us).
constexpr int kAdrThreads = 128;

// One transport step n = n_base + kstep + 1 over every solute voxel (one
// thread each; rock voxels are not in the state).
//
// Bound by instruction issue (about 370 warp instructions per 32 voxels with
// one Monod chemical) up to the L2's size, by DRAM beyond it.  Neighbour
// distances instead of flags and positions on dense grids, one set of
// differences per axis for diffusion and both limiters, no division for a cap
// that is certainly not met: 64^3 / 128^3 / 192^3 Monod 3.96 / 16.6 / 67.4 ->
// 3.3 / 11.8 / 54.1 us a step, four chemicals 7.8 / 45.5 -> 4.9 / 26.9, with
// biofilm 10.3 / 65.5 -> 5.7 / 34.1.  Places instead of 16-bit distances take
// 24 B more a voxel: 3.4 / 12.4 / 60.7.
// Launched with programmatic stream serialisation: what does not change
// during a run (the neighbours' places and the face velocities) is read while
// the previous step drains; the control block and the concentrations only
// after griddepcontrol.wait.
// late: the next step is let in after this one's stores (see pdl_late).
template <int ND, int NS, bool BF, bool WIDE>
__global__ void __launch_bounds__(kAdrThreads) adr_step_kernel(AdrDev d, prt_adr_params p,
                                                               const AdrCtrl* __restrict__ ctrl,
                                                               int kstep, int late, int turn) {
    if (!late) griddep_launch_dependents();
    // turn (a grid of more than half a wave): every other step walks the voxels
    // downwards, so it starts on what the step before left in the L2
    const unsigned b = (kstep & 1) && turn ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
    const unsigned k = b * kAdrThreads + threadIdx.x;
    const bool live = k < (unsigned)d.nm;
    VoxelSetup<ND> s;
    if (live) s = voxel_setup<ND, BF, WIDE>(d, p, k);
    griddep_wait();
    const long long n = ctrl->n_base + kstep + 1;
    if (ctrl->done || n > ctrl->n_stop) return;  // uniform over the grid
    if (!live) return;
    adr_voxel_step<ND, NS, BF>(d, p, n, k, s);
    if (late) griddep_launch_dependents();
}

// ---------------------------------------------------------------------------
// set-up (solve_adr 9.1-9.8, prtlb_3d.py:831-1158, 1425-1440)
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool is_m(const uint8_t* mat, long long c, int pore, int bf) {
    const int v = mat[c];
    return v == pore || (bf >= 0 && v == bf);
}
__device__ __forceinline__ bool is_bf(const uint8_t* mat, long long c, int bf) {
    return bf >= 0 && mat[c] == bf;
}

__global__ void adr_flags_kernel(const uint8_t* __restrict__ mat, Grid g, int nd, int pore,
                                 int bfc, uint32_t* __restrict__ flags, uint8_t* __restrict__ mflag) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.n) return;
    const VoxelPos v = voxel_pos(c, g);
    const bool m = is_m(mat, c, pore, bfc);
    uint32_t fl = 0;
    if (m) fl |= F_M;
    if (is_bf(mat, c, bfc)) fl |= F_BF;
    if (m && v.p[0] == 0) fl |= F_X0;
    for (int i = 0; i < nd; ++i) {
        const int a = (nd == 3) ? i : (i == 0 ? 0 : 2);
        const int p = v.p[a];
        const int n = extent(g, a);
        const long long s = stride(g, a);
        const int pm1 = p > 0 ? p - 1 : 0, pm2 = p > 1 ? p - 2 : 0;
        const int pp1 = p < n - 1 ? p + 1 : n - 1, pp2 = p < n - 2 ? p + 2 : n - 1;
        const long long cm1 = c + (long long)(pm1 - p) * s, cm2 = c + (long long)(pm2 - p) * s;
        const long long cp1 = c + (long long)(pp1 - p) * s, cp2 = c + (long long)(pp2 - p) * s;
        const bool oL = m && is_m(mat, cm1, pore, bfc);
        const bool oH = m && is_m(mat, cp1, pore, bfc);
        const bool fL = oL && is_m(mat, cm2, pore, bfc);
        const bool fH = oH && is_m(mat, cp2, pore, bfc);
        if (oL) fl |= f_open_lo(a);
        if (oH) fl |= f_open_hi(a);
        if (fL) fl |= f_far_lo(a);
        if (fH) fl |= f_far_hi(a);
        if (is_bf(mat, cm1, bfc)) fl |= f_nbf_lo(a);
        if (is_bf(mat, cp1, bfc)) fl |= f_nbf_hi(a);
    }
    flags[c] = fl;
    mflag[c] = m ? 1 : 0;
}

// map[idx[k]] = k.
__global__ void adr_map_kernel(const int* __restrict__ idx, long long nm, int* __restrict__ map) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < nm) map[idx[k]] = (int)k;
}

// The neighbours of solute voxel k along axis i as AdrDev has them (far low,
// low, high, far high), from the open / far flags at clamped positions.
__device__ __forceinline__ int4 neighbours(const AdrDev& d, const int* __restrict__ map, int k,
                                           int i, uint32_t fl, const VoxelPos& v) {
    const int a = (d.nd == 3) ? i : (i == 0 ? 0 : 2);
    const int p = v.p[a], n = extent(d.g, a), s = stride(d.g, a), c = v.c;
    const int pm1 = p > 0 ? 1 : 0, pm2 = p > 1 ? 2 : pm1;
    const int pp1 = p < n - 1 ? 1 : 0, pp2 = p < n - 2 ? 2 : pp1;
    int4 q;
    q.y = (fl & f_open_lo(a)) ? map[c - pm1 * s] : k;
    q.z = (fl & f_open_hi(a)) ? map[c + pp1 * s] : k;
    q.x = (fl & f_far_lo(a)) ? map[c - pm2 * s] : q.y;
    q.w = (fl & f_far_hi(a)) ? map[c + pp2 * s] : q.z;
    return q;
}

// *reach = the largest distance between a voxel and its neighbours.
__global__ void adr_reach_kernel(AdrDev d, const int* __restrict__ map, unsigned* reach) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned far = 0;
    if (k < d.nm) {
        const int c = d.idx[k];
        const VoxelPos v = voxel_pos(c, d.g);
        for (int i = 0; i < d.nd; ++i) {
            const int4 q = neighbours(d, map, (int)k, i, d.flags[c], v);
            far = max(far, (unsigned)max((int)k - q.x, q.w - (int)k));
        }
    }
    far = __reduce_max_sync(0xffffffffu, far);
    if ((threadIdx.x & 31) == 0 && far) atomicMax(reach, far);
}

// The run's fixed data of each solute voxel.  Face velocities u_f = 1/2 (u_lo +
// u_hi) on open faces, 0 on closed ones, from u = vel / u_scale (float32
// division) at the clamped positions of the face's two voxels
// (prtlb_3d.py:860-865, 1092-1135).
__global__ void adr_tables_kernel(const float* __restrict__ vel, AdrDev d, float u_scale,
                                  const int* __restrict__ map, uint2* __restrict__ near,
                                  int4* __restrict__ nb, float2* __restrict__ face,
                                  uint32_t* __restrict__ cflags) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= d.nm) return;
    const Grid& g = d.g;
    const int c = d.idx[k];
    const uint32_t fl = d.flags[c];
    cflags[k] = fl;
    const VoxelPos v = voxel_pos(c, g);
    for (int i = 0; i < d.nd; ++i) {
        const int a = (d.nd == 3) ? i : (i == 0 ? 0 : 2);
        const size_t at = axis_place<true>(i, (unsigned)k, d.nm);
        const int4 q = neighbours(d, map, (int)k, i, fl, v);
        if (near) {
            const unsigned u = (unsigned)k;
            near[at] = make_uint2((u - (unsigned)q.x) | ((u - (unsigned)q.y) << 16),
                                  ((unsigned)q.z - u) | (((unsigned)q.w - u) << 16));
        } else {
            nb[at] = q;
        }
        // velocity component of storage axis a: 3D -> a; 2D -> x: 0, y (stored as z): 1
        const float* vc = vel + (long long)((d.nd == 3) ? a : (a == 0 ? 0 : 1)) * g.n;
        const int s = stride(g, a);
        const float u = vc[c] / u_scale;
        float2 f = make_float2(0.f, 0.f);
        if (fl & f_open_lo(a)) f.x = 0.5f * (vc[v.p[a] > 0 ? c - s : c] / u_scale + u);
        if (fl & f_open_hi(a))
            f.y = 0.5f * (u + vc[v.p[a] < extent(g, a) - 1 ? c + s : c] / u_scale);
        face[at] = f;
    }
}

// Initial state (initial(), prtlb_3d.py:1425-1440) into buffer 0.
__global__ void adr_init_kernel(AdrDev d, prt_adr_params p, float* __restrict__ buf0) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= d.nm) return;
    const uint32_t fl = d.flags[d.idx[k]];
    for (int j = 0; j < p.ns; ++j) {
        float v = 0.f;
        if (p.init_mode[j] == 1 && (fl & F_M)) v = p.init_value[j];
        if (p.init_mode[j] == 2 && (fl & F_BF)) v = p.init_value[j];
        float* row = buf0 + (long long)j * d.ms;
        row[solute_place((unsigned)k, (unsigned)d.n0, (unsigned)d.nm)] = v;
        if (k < d.n0) row[k] = ((p.pinned_mask >> j) & 1u) ? p.feed[j] : v;
    }
}

// Ladder rows (stride nm) from the state's.
__global__ void adr_rows_kernel(AdrDev d, const float* __restrict__ buf, float* __restrict__ rows) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= d.nm) return;
    const unsigned at = solute_place((unsigned)k, (unsigned)d.n0, (unsigned)d.nm);
    for (int j = 0; j < d.ns; ++j) rows[j * d.nm + k] = buf[(long long)j * d.ms + at];
}

// out[j * n + idx[k]] = rows[j * nm + k].
__global__ void adr_expand_kernel(const float* __restrict__ rows, const int* __restrict__ idx,
                                  long long nm, long long n, int ns, float* __restrict__ out) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nm) return;
    const int c = idx[k];
    for (int j = 0; j < ns; ++j) out[(long long)j * n + c] = rows[(long long)j * nm + k];
}

// *n0 = how many of the nm voxel indices lie below `plane` (they ascend).
__global__ void adr_inlet_count_kernel(const int* __restrict__ idx, long long nm, int plane,
                                       int* __restrict__ n0) {
    long long lo = 0, hi = nm;
    while (lo < hi) {
        const long long mid = (lo + hi) / 2;
        if (idx[mid] < plane) lo = mid + 1;
        else hi = mid;
    }
    *n0 = (int)lo;
}

// Order-preserving compaction of the solute voxels (C order), in three passes.
constexpr int kScanBlock = 1024;
__global__ void count_kernel(const uint8_t* __restrict__ mflag, long long n, int* __restrict__ cnt) {
    const long long c = (long long)blockIdx.x * kScanBlock + threadIdx.x;
    int v = (c < n && mflag[c]) ? 1 : 0;
    v = __syncthreads_count(v);
    if (threadIdx.x == 0) cnt[blockIdx.x] = v;
}
// The counts to exclusive sums, in place, and their total; one block.  (One
// thread walking them took 0.4 us a count: 0.8 ms at 128^3, 2.8 ms at 192^3.)
__global__ void __launch_bounds__(kScanBlock)
    scan_counts_kernel(int* __restrict__ cnt, int nb, long long* __restrict__ total) {
    __shared__ int warp_sum[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int carry = 0;
    for (int at = 0; at < nb; at += kScanBlock) {
        const int i = at + threadIdx.x;
        const int v = i < nb ? cnt[i] : 0;
        int s = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += t;
        }
        if (lane == 31) warp_sum[w] = s;
        __syncthreads();
        int ws = warp_sum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, ws, o);
            if (lane >= o) ws += t;
        }
        const int before = w ? __shfl_sync(0xffffffffu, ws, w - 1) : 0;
        if (i < nb) cnt[i] = carry + before + s - v;
        carry += __shfl_sync(0xffffffffu, ws, 31);
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}
__global__ void scatter_kernel(const uint8_t* __restrict__ mflag, long long n,
                               const int* __restrict__ off, int* __restrict__ idx) {
    __shared__ int warp_tot[kScanBlock / 32];
    const long long c = (long long)blockIdx.x * kScanBlock + threadIdx.x;
    const int v = (c < n && mflag[c]) ? 1 : 0;
    const unsigned bal = __ballot_sync(0xffffffffu, v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int before = __popc(bal & ((1u << lane) - 1u));
    if (lane == 0) warp_tot[w] = __popc(bal);
    __syncthreads();
    int base = 0;
    for (int i = 0; i < w; ++i) base += warp_tot[i];
    if (v) idx[off[blockIdx.x] + base + before] = (int)c;
}

// ---------------------------------------------------------------------------
// numpy float32 pairwise means (the stop rule's `C[j][m].mean()`), per
// species: leaf sums (warp_leaf_sum) then the tree levels (tree_means)
// ---------------------------------------------------------------------------
constexpr int kLeafThreads = 256;
constexpr int kTreeThreads = 512;

// One warp per leaf and chemical.
__device__ __forceinline__ void block_of_leaves(const float* __restrict__ src, long long row,
                                                unsigned n0, unsigned nm, const PairTree& t,
                                                int ns, float* __restrict__ vals) {
    __shared__ float sh[kLeafThreads / 32][128];
    const int w = threadIdx.x >> 5;
    const long long item = (long long)blockIdx.x * (kLeafThreads / 32) + w;
    if (item >= (long long)t.nleaf * ns) return;  // whole warps
    const int leaf = (int)(item % t.nleaf);
    const int j = (int)(item / t.nleaf);
    const float v = warp_leaf_sum(src + j * row, n0, nm, t.leaf_start[leaf], t.leaf_len[leaf], sh[w]);
    if ((threadIdx.x & 31) == 0) vals[(long long)j * (t.nleaf + t.ninner) + leaf] = v;
}

__global__ void __launch_bounds__(kLeafThreads)
    means_leaf_kernel(const float* __restrict__ src, long long row, long long nm, PairTree t, int ns,
                      float* __restrict__ vals) {
    block_of_leaves(src, row, 0u, (unsigned)nm, t, ns, vals);
}

__global__ void __launch_bounds__(kTreeThreads)
    means_tree_kernel(PairTree t, long long nm, int ns, float* __restrict__ vals,
                      float* __restrict__ means) {
    tree_means(t, nm, ns, vals, means);
}

// The leaves of the state at the end of the current segment, when its means
// are due.
__global__ void __launch_bounds__(kLeafThreads)
    chunk_leaf_kernel(const AdrCtrl* __restrict__ ctrl, AdrDev d) {
    if (ctrl->done) return;
    const long long end = ctrl->n_stop;
    if (end % ctrl->check != 0) return;
    block_of_leaves(d.buf[end & 1], d.ms, (unsigned)d.n0, (unsigned)d.nm, d.tree, d.ns, d.tree_vals);
}

// The tree levels and means, where due, then the stop rule, the step count and
// the while-graph's condition.
__global__ void __launch_bounds__(kTreeThreads)
    chunk_end_kernel(AdrCtrl* ctrl, AdrDev d, float* __restrict__ means,
                     cudaGraphConditionalHandle h, int use_handle) {
    if (ctrl->done) {
        if (use_handle && threadIdx.x == 0) cudaGraphSetConditional(h, 0);
        return;
    }
    const long long end = ctrl->n_stop;
    const bool due = end > ctrl->n_base && end % ctrl->check == 0;
    if (due) tree_means(d.tree, d.nm, d.ns, d.tree_vals, means);
    __syncthreads();  // the means are written, and every thread has read ctrl
    if (threadIdx.x != 0) return;
    if (due) adr_check(ctrl, means, end, d.log, d.log_cap);
    ctrl->n_base = end;
    ctrl->n_stop = segment_end(end, ctrl->segment, ctrl->check, ctrl->limit);
    if (end >= ctrl->limit) ctrl->done = 1;
    const int go = (!ctrl->done && end < ctrl->n_pause) ? 1 : 0;
    if (use_handle) cudaGraphSetConditional(h, go);
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
// Blocks of `kern` the device holds at once (128 threads each).
template <class K>
static long long resident_blocks(K kern) {
    int per_sm = 0, dev = 0, sms = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kAdrThreads, 0) !=
            cudaSuccess ||
        cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return (long long)per_sm * sms;
}

// Steps go out with programmatic stream serialisation.  A step whose blocks
// exceed one resident wave lets the next step launch at its start (128^3
// Monod: 11.8 us a step against 12.6 at the end), and so does one that fills
// at most half a wave, because the next step's blocks then find room beside
// it (24^3: 2.35 -> 2.02, 40^3 2.43 -> 2.11, 128^2 first order 2.36 -> 2.05);
// between the two only after its stores (pdl_late), or the next step's blocks
// would slow the running one (64^3, four chemicals: 4.85 against 5.55).
// PRT_PDL=0 launches every step plainly.  The first step after a chunk's end
// always goes out plainly (in a loop's graph it is the first node and so does
// anyway): the control block is then in place before any step of the chunk is
// resident, and the steps may take it as read-only.
template <int ND, int NS>
static cudaError_t step_t(const AdrDev& d, const prt_adr_params& p, AdrCtrl* ctrl, int k,
                          cudaStream_t s) {
    if (d.nm <= 0) return cudaSuccess;
    auto kern = d.near ? (d.has_bf ? adr_step_kernel<ND, NS, true, false>
                                   : adr_step_kernel<ND, NS, false, false>)
                       : (d.has_bf ? adr_step_kernel<ND, NS, true, true>
                                   : adr_step_kernel<ND, NS, false, true>);
    const long long nb = (d.nm + kAdrThreads - 1) / kAdrThreads;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)nb);
    cfg.blockDim = dim3(kAdrThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    const long long resident = resident_blocks(kern);
    const int late = pdl_late(nb <= resident && 2 * nb > resident) ? 1 : 0;
    cfg.numAttrs = pdl_enabled() && k > 0 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, d, p, ctrl, k, late, 2 * nb > resident ? 1 : 0);
}

template <int ND>
static cudaError_t step_nd(const AdrDev& d, const prt_adr_params& p, AdrCtrl* ctrl, int k,
                           cudaStream_t s) {
    switch (d.ns) {
        case 1: return step_t<ND, 1>(d, p, ctrl, k, s);
        case 2: return step_t<ND, 2>(d, p, ctrl, k, s);
        case 3: return step_t<ND, 3>(d, p, ctrl, k, s);
        case 4: return step_t<ND, 4>(d, p, ctrl, k, s);
        case 5: return step_t<ND, 5>(d, p, ctrl, k, s);
        case 6: return step_t<ND, 6>(d, p, ctrl, k, s);
        case 7: return step_t<ND, 7>(d, p, ctrl, k, s);
        case 8: return step_t<ND, 8>(d, p, ctrl, k, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t adr_launch_step(const AdrDev& d, const prt_adr_params& p, AdrCtrl* ctrl, int kstep,
                            cudaStream_t s) {
    return d.nd == 3 ? step_nd<3>(d, p, ctrl, kstep, s) : step_nd<2>(d, p, ctrl, kstep, s);
}

// The axial velocity (which 0) or the float32 speed sqrt((v0^2 + v1^2) [+ v2^2])
// the way numpy forms it (which 1) of each solute voxel.
__global__ void vel_rows_kernel(const float* __restrict__ vel, const int* __restrict__ idx,
                                long long nm, long long n, int nd, int which,
                                float* __restrict__ row) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nm) return;
    const long long c = idx[k];
    const float v0 = vel[c];
    if (which == 0) {
        row[k] = v0;
        return;
    }
    const float v1 = vel[n + c];
    float s = v0 * v0 + v1 * v1;
    if (nd == 3) {
        const float v2 = vel[2 * n + c];
        s = s + v2 * v2;
    }
    row[k] = sqrtf(s);
}

// max |vel[a]| over the solute voxels (order-free: max is exact)
__global__ void vmax_kernel(const float* __restrict__ vel, const int* __restrict__ idx, long long nm,
                            long long n, int nd, unsigned* __restrict__ out) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    float m[3] = {0.f, 0.f, 0.f};
    if (t < nm) {
        const long long c = idx[t];
        for (int a = 0; a < nd; ++a) m[a] = fabsf(vel[(long long)a * n + c]);
    }
    for (int a = 0; a < 3; ++a) {
        float v = m[a];
        for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_down_sync(0xffffffffu, v, o));
        if ((threadIdx.x & 31) == 0 && v > 0.f) atomicMax(out + a, __float_as_uint(v));
    }
}

__global__ void count_bf_kernel(const uint32_t* __restrict__ flags, long long n,
                                unsigned long long* out) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int v = (c < n && (flags[c] & F_BF)) ? 1 : 0;
    v = __syncthreads_count(v);
    if (threadIdx.x == 0 && v) atomicAdd(out, (unsigned long long)v);
}

cudaError_t adr_launch_flags(const uint8_t* mat, const Grid& g, int nd, int pore, int bfc,
                             uint32_t* flags, uint8_t* mflag, cudaStream_t s) {
    const unsigned nb = (unsigned)((g.n + 255) / 256);
    adr_flags_kernel<<<nb, 256, 0, s>>>(mat, g, nd, pore, bfc, flags, mflag);
    return cudaGetLastError();
}

static unsigned leaf_blocks(const PairTree& t, int ns) {
    return (unsigned)(((long long)t.nleaf * ns + kLeafThreads / 32 - 1) / (kLeafThreads / 32));
}

// mean_axial, mean_speed (numpy float32 pairwise means over the solute
// voxels) into means[0..1]; max |v_a| bits into vmax_bits[0..2]; biofilm
// voxel count into *nbf, the inlet plane's solute voxels into *n0.  tmp: n
// floats of scratch.
cudaError_t adr_launch_vel_stats(const float* vel, const AdrDev& d, float* tmp, float* means,
                                 unsigned* vmax_bits, unsigned long long* nbf, int* n0, cudaStream_t s) {
    const Grid& g = d.g;
    const unsigned nb = (unsigned)((g.n + 255) / 256);
    cudaError_t e;
    for (int which = 0; which < 2; ++which) {
        if (d.nm > 0) {
            vel_rows_kernel<<<(unsigned)((d.nm + 255) / 256), 256, 0, s>>>(
                vel, d.idx, d.nm, g.n, d.nd, which, tmp);
            means_leaf_kernel<<<leaf_blocks(d.tree, 1), kLeafThreads, 0, s>>>(tmp, 0, d.nm, d.tree,
                                                                             1, d.tree_vals);
        }
        means_tree_kernel<<<1, kTreeThreads, 0, s>>>(d.tree, d.nm, 1, d.tree_vals, means + which);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    if (d.nm > 0)
        vmax_kernel<<<(unsigned)((d.nm + 255) / 256), 256, 0, s>>>(vel, d.idx, d.nm, g.n, d.nd,
                                                                  vmax_bits);
    count_bf_kernel<<<nb, 256, 0, s>>>(d.flags, g.n, nbf);
    adr_inlet_count_kernel<<<1, 1, 0, s>>>(d.idx, d.nm, g.ny * g.nz, n0);
    return cudaGetLastError();
}

cudaError_t adr_launch_map(const AdrDev& d, int* map, unsigned* reach, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(reach, 0, sizeof(*reach), s);
    if (e != cudaSuccess || d.nm <= 0) return e;
    const unsigned nb = (unsigned)((d.nm + 255) / 256);
    adr_map_kernel<<<nb, 256, 0, s>>>(d.idx, d.nm, map);
    adr_reach_kernel<<<nb, 256, 0, s>>>(d, map, reach);
    return cudaGetLastError();
}

cudaError_t adr_launch_setup(const float* vel, const prt_adr_params& p, const AdrDev& d,
                             const int* map, cudaStream_t s) {
    if (d.nm <= 0) return cudaSuccess;
    const unsigned nb = (unsigned)((d.nm + 255) / 256);
    adr_tables_kernel<<<nb, 256, 0, s>>>(vel, d, p.u_scale, map, const_cast<uint2*>(d.near),
                                         const_cast<int4*>(d.nb), const_cast<float2*>(d.face),
                                         const_cast<uint32_t*>(d.cflags));
    adr_init_kernel<<<nb, 256, 0, s>>>(d, p, d.buf[0]);
    return cudaGetLastError();
}

cudaError_t adr_launch_rows(const AdrDev& d, const float* buf, float* rows, cudaStream_t s) {
    if (d.nm <= 0) return cudaSuccess;
    adr_rows_kernel<<<(unsigned)((d.nm + 255) / 256), 256, 0, s>>>(d, buf, rows);
    return cudaGetLastError();
}

cudaError_t adr_launch_expand(const AdrDev& d, const float* rows, float* out, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(out, 0, (size_t)d.g.n * d.ns * sizeof(float), s);
    if (e != cudaSuccess || d.nm <= 0) return e;
    adr_expand_kernel<<<(unsigned)((d.nm + 255) / 256), 256, 0, s>>>(rows, d.idx, d.nm, d.g.n, d.ns,
                                                                    out);
    return cudaGetLastError();
}

cudaError_t adr_launch_count(const uint8_t* mflag, long long n, int* cnt, long long* total,
                             cudaStream_t s) {
    const int nb = (int)((n + kScanBlock - 1) / kScanBlock);
    count_kernel<<<nb, kScanBlock, 0, s>>>(mflag, n, cnt);
    scan_counts_kernel<<<1, kScanBlock, 0, s>>>(cnt, nb, total);
    return cudaGetLastError();
}

cudaError_t adr_launch_scatter(const uint8_t* mflag, long long n, const int* cnt, int* idx,
                               cudaStream_t s) {
    const int nb = (int)((n + kScanBlock - 1) / kScanBlock);
    scatter_kernel<<<nb, kScanBlock, 0, s>>>(mflag, n, cnt, idx);
    return cudaGetLastError();
}

cudaError_t adr_launch_means(const AdrDev& d, int slot, float* means_out, cudaStream_t s) {
    // the means of ladder slot `slot`, outside the time loop
    const float* src = d.ladder + (long long)slot * d.ns * d.nm;
    if (d.tree.nleaf > 0)
        means_leaf_kernel<<<leaf_blocks(d.tree, d.ns), kLeafThreads, 0, s>>>(
            src, d.nm, d.nm, d.tree, d.ns, d.tree_vals);
    means_tree_kernel<<<1, kTreeThreads, 0, s>>>(d.tree, d.nm, d.ns, d.tree_vals, means_out);
    return cudaGetLastError();
}

cudaError_t adr_launch_chunk_end(const AdrDev& d, AdrCtrl* ctrl, float* means,
                                 cudaGraphConditionalHandle h, int use_handle, cudaStream_t s) {
    if (d.tree.nleaf > 0)
        chunk_leaf_kernel<<<leaf_blocks(d.tree, d.ns), kLeafThreads, 0, s>>>(ctrl, d);
    chunk_end_kernel<<<1, kTreeThreads, 0, s>>>(ctrl, d, means, h, use_handle);
    return cudaGetLastError();
}

}  // namespace prt

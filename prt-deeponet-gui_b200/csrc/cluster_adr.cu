// cluster_adr.cu -- the transport loop of a small grid in one kernel of one
// thread-block cluster (see cluster.cuh): both copies of the state stay in the
// cluster's shared memory and a voxel's neighbours and faces in its thread's
// registers.  Compiled with -fmad=false like adr.cu, whose arithmetic
// (adr_core.cuh), means and stop rule it runs, so steps, snapshots and stop
// are bit-identical to the launches of adr_step_kernel.
//
// Bound by the barrier and shared-memory latency (0.85 us a step on the
// smallest grids), then by the arithmetic of the voxels a block holds.  us a
// step, launches -> cluster: Monod 16^3 2.02 -> 0.97, 24^3 2.01 -> 1.20, 28^3
// 1.99 -> 1.39; four chemicals 24^3 3.12 -> 2.44, 28^3 3.19 -> 3.00; 2D first
// order 64^2 1.94 -> 0.88, 128^2 1.99 -> 1.13.
#include "adr_core.cuh"
#include "cluster.cuh"

namespace prt {

namespace {

// Voxels per block: the registers of that many threads (102 each), and about
// where the launches catch up.
constexpr int T = 640;
// Chemicals: more take too many registers.
constexpr int kClusterSpecies = 4;

// Reads where u >= 0 (UP), or only where it is not, else 0.
template <bool UP>
__device__ __forceinline__ float ld_cluster_if(uint32_t a, float u) {
    float v;
    if (UP)
        asm volatile(
            "{\n.reg .pred q;\nsetp.ge.f32 q, %2, 0f00000000;\nmov.f32 %0, 0f00000000;\n"
            "@q ld.shared::cluster.f32 %0, [%1];\n}"
            : "=&f"(v)
            : "r"(a), "f"(u)
            : "memory");
    else
        asm volatile(
            "{\n.reg .pred q;\nsetp.ltu.f32 q, %2, 0f00000000;\nmov.f32 %0, 0f00000000;\n"
            "@q ld.shared::cluster.f32 %0, [%1];\n}"
            : "=&f"(v)
            : "r"(a), "f"(u)
            : "memory");
    return v;
}

// A voxel's fixed data: its neighbours' elements of chemical 0 in copy 0 of the
// state (far low, low, high, far high), in the cluster's shared memory.
template <int ND>
struct ClusterVoxel {
    uint32_t nb[ND][4];
    float2 fc[ND];
    uint32_t fl;
};

// One step at one voxel from copy FROM of the state to the other; cn takes the
// voxel's own new values.
template <int ND, int NS, bool BF, int FROM>
__device__ __forceinline__ void cluster_step(float (*st)[NS][T], const ClusterVoxel<ND>& v,
                                             const prt_adr_params& p, bool inlet,
                                             float (&cn)[NS]) {
    const int t = threadIdx.x;
    float C[NS], tr[NS];
#pragma unroll
    for (int j = 0; j < NS; ++j) C[j] = st[FROM][j][t];
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        tr[j] = 0.f;
        if ((p.moving_mask >> j) & 1u) {
            constexpr uint32_t row = T * 4;
            const uint32_t at = (FROM * NS + j) * row;
            float m2[ND], m1[ND], p1[ND], p2[ND];
#pragma unroll
            for (int i = 0; i < ND; ++i) {
                ld_cluster(v.nb[i][1] + at, m1[i]);
                ld_cluster(v.nb[i][2] + at, p1[i]);
                m2[i] = ld_cluster_if<true>(v.nb[i][0] + at, v.fc[i].x);
                p2[i] = ld_cluster_if<false>(v.nb[i][3] + at, v.fc[i].y);
            }
            const float dj[3] = {p.dface[j][0], p.dface[j][1], p.dface[j][2]};
            tr[j] = transport_terms<ND, BF>(m2, m1, p1, p2, v.fc, v.fl, C[j], dj);
        }
    }
    adr_update<ND, NS>(C, tr, v.fl, p, cn);
#pragma unroll
    for (int j = 0; j < NS; ++j)
        st[FROM ^ 1][j][t] = (inlet && ((p.pinned_mask >> j) & 1u)) ? p.feed[j] : cn[j];
}

// Block r of the cluster holds the voxels [r span, (r + 1) span), one per
// thread.  Runs from the control block's step count to its pause, its stop or
// its limit; the state is read from and left in the global buffers.
template <int ND, int NS, bool BF>
__global__ void __launch_bounds__(T, 1)
    adr_cluster_kernel(AdrDev d, prt_adr_params p, AdrCtrl* ctrl, float* __restrict__ means,
                       int span) {
    __shared__ float st[2][NS][T];
    __shared__ float sh[T / 32][128];
    __shared__ int s_go;
    const int t = threadIdx.x;
    const unsigned rank = cluster_rank();
    const unsigned k = rank * span + t;
    const unsigned nm = (unsigned)d.nm, ms = d.ms;
    const bool live = k < nm;
    const bool inlet = k < (unsigned)d.n0;
    const long long limit = ctrl->limit, pause = ctrl->n_pause;
    const int check = ctrl->check;
    long long n = ctrl->n_base, next = (n / check + 1) * check;
    int go = !ctrl->done && n < pause;
    ClusterVoxel<ND> v;
    if (live) {
        const VoxelSetup<ND> s = d.near ? voxel_setup<ND, BF, false>(d, p, k)
                                        : voxel_setup<ND, BF, true, false>(d, p, k);
        v.fl = s.fl;
        const uint32_t base = shared_address(&st[0][0][0]);
        auto place = [&](unsigned q) { return in_block(base + (q % span) * 4, q / span); };
#pragma unroll
        for (int i = 0; i < ND; ++i) {
            v.fc[i] = s.fc[i];
            v.nb[i][0] = place(k - s.nb[i].x);
            v.nb[i][1] = place(k - s.nb[i].y);
            v.nb[i][2] = place(k + s.nb[i].z);
            v.nb[i][3] = place(k + s.nb[i].w);
        }
        const float* row = d.buf[n & 1];
#pragma unroll
        for (int j = 0; j < NS; ++j) st[n & 1][j][t] = row[j * ms + k];
    }
    cluster_sync();
    while (go) {
        // to the next check or the limit (a run that left a batch begins at any
        // step)
        const long long end = min(next, limit);
        const bool due = end == next;
        next += check;
        float cn[NS];
        for (++n; n <= end; ++n) {
            if (live) {
                const int slot = d.slot_of_step[n];
                if (n & 1) cluster_step<ND, NS, BF, 0>(st, v, p, inlet, cn);
                else cluster_step<ND, NS, BF, 1>(st, v, p, inlet, cn);
                if (slot >= 0) {
                    float* lad = d.ladder + (long long)slot * NS * nm;
#pragma unroll
                    for (int j = 0; j < NS; ++j) lad[j * nm + k] = cn[j];
                }
                if (n == end) {  // the state of the chunk's last step, as the launches leave it
                    float* out = d.buf[n & 1];
#pragma unroll
                    for (int j = 0; j < NS; ++j) {
                        out[j * ms + k] = st[n & 1][j][t];
                        if (inlet) out[j * ms + nm + k] = cn[j];
                    }
                }
            }
            cluster_sync();
        }
        n = end;
        if (due) {  // the leaves, over the warps of the cluster
            const int warps = blockDim.x / 32, w = t >> 5;
            const int items = d.tree.nleaf * NS;
            const int all = warps * (int)gridDim.x;
            for (int q = (int)rank * warps + w; q < items; q += all) {
                const int leaf = q % d.tree.nleaf, j = q / d.tree.nleaf;
                const float x = warp_leaf_sum(d.buf[n & 1] + j * ms, (unsigned)d.n0, nm,
                                              d.tree.leaf_start[leaf], d.tree.leaf_len[leaf], sh[w]);
                if ((t & 31) == 0) d.tree_vals[j * (d.tree.nleaf + d.tree.ninner) + leaf] = x;
            }
            cluster_sync();
        }
        if (rank == 0) {
            if (due) tree_means(d.tree, d.nm, NS, d.tree_vals, means);
            __syncthreads();
            if (t == 0) {
                if (due) adr_check(ctrl, means, n, d.log, d.log_cap);
                ctrl->n_base = n;
                ctrl->n_stop = segment_end(n, ctrl->segment, check, limit);
                if (n >= limit) ctrl->done = 1;
                s_go = !ctrl->done && n < pause;
            }
        }
        cluster_sync();
        ld_cluster(in_block(shared_address(&s_go), 0), go);
    }
    cluster_sync();  // no block leaves while another may read its s_go
}

template <int ND, int NS>
cudaError_t run(const AdrDev& d, const prt_adr_params& p, AdrCtrl* ctrl, float* means, int blocks,
                int span, cudaStream_t s) {
    auto kern = d.has_bf ? adr_cluster_kernel<ND, NS, true> : adr_cluster_kernel<ND, NS, false>;
    return launch_cluster(kern, blocks, span, 0, 0, s, d, p, ctrl, means, span);
}

}  // namespace

cudaError_t adr_launch_cluster(const AdrDev& d, const prt_adr_params& p, AdrCtrl* ctrl,
                               float* means, cudaStream_t s) {
    if (d.nm <= 0 || d.ns > kClusterSpecies) return cudaErrorNotSupported;
    const int blocks = cluster_blocks(d.nm), span = cluster_span(d.nm, blocks);
    if (span > T) return cudaErrorNotSupported;
    if (d.nd == 3) {
        switch (d.ns) {
            case 1: return run<3, 1>(d, p, ctrl, means, blocks, span, s);
            case 2: return run<3, 2>(d, p, ctrl, means, blocks, span, s);
            case 3: return run<3, 3>(d, p, ctrl, means, blocks, span, s);
            default: return run<3, 4>(d, p, ctrl, means, blocks, span, s);
        }
    }
    switch (d.ns) {
        case 1: return run<2, 1>(d, p, ctrl, means, blocks, span, s);
        case 2: return run<2, 2>(d, p, ctrl, means, blocks, span, s);
        case 3: return run<2, 3>(d, p, ctrl, means, blocks, span, s);
        default: return run<2, 4>(d, p, ctrl, means, blocks, span, s);
    }
}

}  // namespace prt

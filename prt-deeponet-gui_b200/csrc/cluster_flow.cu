// cluster_flow.cu -- the whole flow loop of a small grid in one kernel of one
// thread-block cluster (see cluster.cuh): the lattice stays in the cluster's
// shared memory, the arithmetic is lb_core.cuh's and the in-place scheme
// lb_flow.cu's, so iterations, decisions and fields are bit-identical to the
// launches of lb_step_kernel.
//
// Bound by the barrier and shared-memory latency (0.75 us an iteration on the
// smallest grids) and then by the arithmetic of the slots a block holds, about
// 0.45 us for each further 128 slots of D3Q19 float64, 0.3 us of float32,
// which sets the largest size taken.  us an iteration, launches -> cluster:
// 16^3 float64 2.29 -> 1.02, 24^3 2.31 -> 1.75, 26^3 2.22 -> 1.93, 24^3 float32
// 2.15 -> 1.33;
// D2Q9 64^2 float64 1.79 -> 0.82, 128^2 1.81 -> 1.16, float32 1.69 ->
// 0.86, 150^2 float64 1.83 -> 1.61.
#include "cluster.cuh"
#include "lb_core.cuh"

namespace prt {

namespace {

// Threads, hence slots, per block at most: where the launches catch up (D3Q19
// float64 at 640 slots 2.68 against 2.32 us, at 512 1.93 against 2.22; float32
// at 640 1.81 against 2.15), or the registers of 1024 threads (D2Q9).
template <class L, class M>
constexpr int cluster_threads() {
    return L::Q == 19 ? (sizeof(typename M::RA) == 8 ? 512 : 640) : 1024;
}

template <class S>
__device__ __forceinline__ S ld_own(uint32_t a) {
    S v;
    if constexpr (sizeof(S) == 8) {
        double d;
        asm volatile("ld.shared.f64 %0, [%1];" : "=d"(d) : "r"(a) : "memory");
        v = d;
    } else if constexpr (sizeof(S) == 4) {
        float d;
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(d) : "r"(a) : "memory");
        v = d;
    } else {
        unsigned short d;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(d) : "r"(a) : "memory");
        v = __ushort_as_half(d);
    }
    return v;
}
__device__ __forceinline__ void st_own(uint32_t a, double v) {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void st_own(uint32_t a, float v) {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void st_own(uint32_t a, __half v) {
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"(__half_as_ushort(v)) : "memory");
}

// One iteration of one slot: `own` its element of row 0 in this block's shared
// memory, far[p] the far place's element of row 0 in the cluster's; rows are
// ROW bytes apart.  Returns |u_x|.
template <class L, class M, int ROW, bool ODD>
__device__ __forceinline__ double cluster_cell(uint32_t own, const uint32_t (&far)[L::NP],
                                               const LbParams& kc) {
    using S = typename M::S;
    using R = typename M::R;
    using RA = typename M::RA;
    constexpr int d = L::pb(0) - L::pa(0);
    constexpr int o = ODD ? 0 : d * ROW, f = ODD ? d * ROW : 0;  // see Lat
    typename Pop<S>::H h[L::Q];
#pragma unroll
    for (int p = 0; p < L::NP; ++p) {
        S v;
        ld_cluster(far[p] + L::pa(p) * ROW + f, v);
        h[L::pb(p)] = Pop<S>::dec(v, kc.inv_scale);
    }
    h[0] = Pop<S>::dec(ld_own<S>(own), kc.inv_scale);
#pragma unroll
    for (int p = 0; p < L::NP; ++p)
        h[L::pa(p)] = Pop<S>::dec(ld_own<S>(own + L::pa(p) * ROW + o), kc.inv_scale);
    const Moments<R, RA> m = moments<L, R, RA>(h, half_force<RA>(kc));
    collide_mode<L, M>(h, m, kc, [&](int i, int p, R v) {
        const S q = Pop<S>::enc(v, kc.scale);
        if (p < 0) st_own(own, q);
        else if (i == L::pa(p)) st_cluster(far[p] + i * ROW + f, q);
        else st_own(own + L::pa(p) * ROW + o, q);
    });
    return fabs((double)m.jx * (double)m.inv_rho);
}

// Block r of the cluster holds the slots [r span, (r + 1) span), one per
// thread; element t of row i is slot r span + t, element T + t the place of
// the thread's link of the pair (the row far places lie in).  The solve is at
// iteration 0, where the whole lattice is 0.
template <class L, class M, int T>
__global__ void __launch_bounds__(T, 1)
    lb_cluster_kernel(typename M::S* __restrict__ f, FlowMap fm, Grid g, LbParams kc, FlowCtrl* ctrl,
                      double* __restrict__ partials, int span, int nb) {
    using S = typename M::S;
    extern __shared__ __align__(16) unsigned char rows[];
    __shared__ double warp_sum[T / 32];
    __shared__ double sums[kFlowThreads];
    __shared__ int s_done;
    constexpr int ROW = 2 * T * (int)sizeof(S);
    const int t = threadIdx.x;
    const unsigned rank = cluster_rank();
    const int k = (int)rank * span + t;
    const bool live = k < fm.nf;
    for (int i = t; i < L::Q * ROW / 4; i += blockDim.x) reinterpret_cast<unsigned*>(rows)[i] = 0u;
    const uint32_t own = shared_address(rows) + t * (int)sizeof(S);
    uint32_t far[L::NP];
    int slot[L::NP];  // of the far places
    far_slots<L, Far::packed>(fm, g, k, slot);
#pragma unroll
    for (int p = 0; p < L::NP; ++p) {
        const bool link = slot[p] >= fm.nf;
        const unsigned b = link ? rank : (unsigned)(slot[p] / span);
        const int at = link ? T + t : slot[p] - (int)b * span;
        far[p] = in_block(shared_address(rows) + at * (int)sizeof(S), b);
    }
    // the control block is rank 0's thread 0's from here on
    const long long nit = ctrl->nit;
    const int every = ctrl->every;
    long long base = ctrl->it_base;
    int done = ctrl->done;
    cluster_sync();
    while (!done) {
        const int n = (int)min((long long)every, nit - base);
        const bool full = n == every;
        double acc = 0.0;
        for (int i = 0; i < n; ++i) {
            if (live)
                acc = (i & 1) ? cluster_cell<L, M, ROW, true>(own, far, kc)
                              : cluster_cell<L, M, ROW, false>(own, far, kc);
            cluster_sync();
        }
        // the chunk's last iteration: the sums of block_sum_store, one per
        // 128 slots, then block_sum_fixed over them in the first block
        if (full) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
            if ((t & 31) == 0) warp_sum[t >> 5] = acc;
            __syncthreads();
            constexpr int G = kFlowThreads / 32;
            const int grp = t >> 5;  // warp w forms the sum of the 128 slots w
            if (grp < (int)blockDim.x / kFlowThreads) {
                double v = (t & 31) < G ? warp_sum[grp * G + (t & 31)] : 0.0;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
                const int blk = (int)rank * (span / kFlowThreads) + grp;
                if ((t & 31) == 0 && blk < nb) partials[blk] = v;
            }
            cluster_sync();
        }
        if (rank == 0) {
            double s = 0.0;
            if (full) {
                if (t < kFlowThreads) {
                    double v = 0.0;
                    for (int i = t; i < nb; i += kFlowThreads) v += __ldcg(partials + i);
                    sums[t] = v;
                }
                __syncthreads();
                for (int w = kFlowThreads / 2; w > 0; w >>= 1) {
                    if (t < w) sums[t] += sums[t + w];
                    __syncthreads();
                }
                s = sums[0];
            }
            if (t == 0) {
                const long long end = base + n;
                flow_ctrl_advance(ctrl, end, full && (end % every) == 0, s);
                s_done = ctrl->done;
            }
        }
        cluster_sync();
        ld_cluster(in_block(shared_address(&s_done), 0), done);
        base += n;
    }
    // the lattice to where the launches keep it
    far_slots<L, Far::packed>(fm, g, k, slot);
    if (live) {
#pragma unroll
        for (int i = 0; i < L::Q; ++i) f[i * fm.rs + k] = ld_own<S>(own + i * ROW);
#pragma unroll
        for (int p = 0; p < L::NP; ++p) {
            if (slot[p] < fm.nf) continue;
            const uint32_t link = own + T * (int)sizeof(S);
            f[L::pa(p) * fm.rs + slot[p]] = ld_own<S>(link + L::pa(p) * ROW);
            f[L::pb(p) * fm.rs + slot[p]] = ld_own<S>(link + L::pb(p) * ROW);
        }
    }
    cluster_sync();  // no block leaves while another may read its s_done
}

template <class L, class M>
cudaError_t run(void* f, const FlowMap& fm, const Grid& g, const LbParams& k, FlowCtrl* ctrl,
                double* partials, int nb, cudaStream_t s) {
    constexpr int T = cluster_threads<L, M>();
    const int blocks = cluster_blocks(fm.nf), span = cluster_span(fm.nf, blocks);
    if (span > T) return cudaErrorNotSupported;
    const size_t smem = (size_t)L::Q * 2 * T * sizeof(typename M::S);
    return launch_cluster(lb_cluster_kernel<L, M, T>, blocks, span, smem, smem, s,
                          static_cast<typename M::S*>(f), fm, g, k, ctrl, partials, span, nb);
}

}  // namespace

cudaError_t flow_launch_cluster(int nd, int precision, void* f, const FlowMap& fm, const Grid& g,
                                const LbParams& k, FlowCtrl* ctrl, double* partials, int nb,
                                cudaStream_t s) {
    if (fm.nf <= 0) return cudaErrorNotSupported;
    if (nd == 3) {
        if (precision == PRT_FP64) return run<D3Q19, ModeF64>(f, fm, g, k, ctrl, partials, nb, s);
        if (precision == PRT_FP32) return run<D3Q19, ModeF32D>(f, fm, g, k, ctrl, partials, nb, s);
        if (precision == PRT_FP32_F32) return run<D3Q19, ModeF32>(f, fm, g, k, ctrl, partials, nb, s);
        return run<D3Q19, ModeF16>(f, fm, g, k, ctrl, partials, nb, s);
    }
    if (precision == PRT_FP64) return run<D2Q9, ModeF64>(f, fm, g, k, ctrl, partials, nb, s);
    if (precision == PRT_FP32) return run<D2Q9, ModeF32D>(f, fm, g, k, ctrl, partials, nb, s);
    if (precision == PRT_FP32_F32) return run<D2Q9, ModeF32>(f, fm, g, k, ctrl, partials, nb, s);
    return run<D2Q9, ModeF16>(f, fm, g, k, ctrl, partials, nb, s);
}

}  // namespace prt

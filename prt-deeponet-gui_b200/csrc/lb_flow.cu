// lb_flow.cu -- lattice-Boltzmann Stokes flow kernels (D2Q9 / D3Q19, TRT, Guo
// forcing, node bounce-back, periodic streaming) for sm_100a.
//
// What the reference does per iteration (prtlb_3d.py:427-445, prtlb_2d.py:449-474):
//   moments rho, u (u_x gets +g/2, u = 0 on solid)  -> feq
//   TRT collision (_trt_collide, prtlb_3d.py:142) + Guo term w_i(1-om-/2) 3 g e_ix
//   solid voxels: post-collision = the reversed ARRIVED populations
//   periodic streaming of every population (np.roll on every axis)
//
// Here one launch does one whole iteration in place, on one lattice: for each
// pair of opposite directions (a, b) a voxel reads f_a from its own place
// and f_b from the place of its neighbour x + e_a, and writes the collided
// f_b and f_a to the same two places, swapped (the storage order of
// "esoteric pull" streaming, M. Lehmann, Computation 10 (2022) 92).  The two
// places swap rows with the iteration parity, which completes the streaming.
// When x + e_a is rock, the reference rule "the solid voxel sends back what
// arrived there one iteration earlier" is what the place does by itself: it
// keeps the f_a written into it until the next iteration of the same parity
// reads it as f_b.  The same holds for the own place when x - e_a is rock.
// So rock voxels do no work, the transient is the reference's and not only
// the steady state, and an iteration reads and writes every population once.
// (Pulling from one lattice into another reads the two-iterations-old values
// from partly used sectors of the lattice it is about to overwrite, about
// one more lattice pass per iteration where the lattices exceed the L2.)
//
// Populations are stored shifted, h_i = f_i - w_i: the non-equilibrium part
// that carries the viscous stress is of the order of the force (1e-7) and
// would drown next to w_i ~ 0.3 in float32 (prtlb_2d.py:354-362).
#include <algorithm>
#include <cstdlib>

#include "lb_core.cuh"

namespace prt {

// One whole LB iteration t (ODD = t & 1); solid voxels do nothing.  late: the
// next iteration is let in after this one's stores (see pdl_late).  turn: odd
// iterations walk the slots downwards (a grid of several waves).
//
// Bound by the L2 and DRAM traffic where the lattice exceeds the L2 (192^3),
// by latency below; in place it reads and writes each population once and
// finds 9 places instead of 18.  Odd iterations walk the slots downwards when
// there are several waves, so an iteration starts on what the one before left in the L2: 128^3 float32
// 28.4 -> 26.8 us, float64 57.3 -> 48.3, 192^3 115 -> 105 and 174 -> 167.
// From one lattice into another (the form before): 40.3, 65.1, 126.6, 206.5;
// 96^3 float64 27.1 -> 16.2, float32 11.8 -> 10.7, 64^3 unchanged within 5 %.
// A grid of one wave whose threads overlap the next voxel's loads with this
// one's collision (two cp.async stages) was slower beyond the L2 (192^3 122).
enum class Form {
    wide,    // the mode's own
    four,    // D3Q19 float64 gathered into registers, four blocks an SM
    halves,  // the same with blocks of half the size, ten an SM (unsampled steps)
    narrow   // D2Q9 with fewer registers and more blocks an SM (see launch_step_one)
};
template <Form W>
__host__ __device__ constexpr int form_threads() {
    return W == Form::halves ? kFlowThreads / 2 : kFlowThreads;
}
template <class M, Form W>
__host__ __device__ constexpr int form_blocks() {
    return W == Form::four ? 4 : W == Form::halves ? 10 : W == Form::narrow ? M::narrow_blocks : M::min_blocks;
}

template <class L, class M, Far F, bool ODD, bool CHECK, Form W>
__global__ void __launch_bounds__(form_threads<W>(), form_blocks<M, W>())
    lb_step_kernel(typename M::S* __restrict__ f, FlowMap fm, Grid g, LbParams kc,
                   const FlowCtrl* __restrict__ ctrl, int kstep, double* __restrict__ partials,
                   int late, int turn) {
    if (!late) griddep_launch_dependents();
    const int b = ODD && turn ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
    const int k = b * form_threads<W>() + threadIdx.x;
    const Lat<typename M::S> lat = lattice<L>(f, fm.rs, ODD);
    // the pore maps never change during a solve: the far places are looked
    // up while the previous iteration may still be running
    int far[L::NP];
    far_slots<L, F>(fm, g, k, far);
    griddep_wait();
    const long long it = ctrl->it_base + kstep;
    if (ctrl->done || it >= ctrl->nit) return;  // uniform over the grid
    double acc = 0.0;
    if (k < fm.nf) {
        constexpr bool reg = W == Form::four || W == Form::halves;
        constexpr bool index = reg || (W == Form::narrow && sizeof(typename M::S) == 8);
        const double ux = lb_cell<L, M, M::staged && L::Q == 19 && !reg, index>(lat, kc, k, far);
        if (CHECK) acc = ux;
    }
    if (CHECK) block_sum_store(acc, partials + b);
    if (late) griddep_launch_dependents();
}

// FlowConvergence.done() at the end of a chunk, the next multiple of `every` or
// the cap (prtlb_3d.py:220-235).  Also decides whether the while-graph goes on.
__global__ void flow_check_kernel(FlowCtrl* ctrl, const double* __restrict__ partials, int nb,
                                  cudaGraphConditionalHandle h, int use_handle) {
    const int done_before = ctrl->done;
    const long long base = ctrl->it_base;
    const long long next = (base / ctrl->every + 1) * ctrl->every;
    const long long end = min(next, ctrl->nit);
    const bool sample = end == next;
    // the partials of the sampled iteration are summed for the convergence
    // mean and the non-finite stop
    double s = 0.0;
    if (!done_before && sample) s = block_sum_fixed(partials, nb);
    if (threadIdx.x != 0) return;
    if (done_before) {
        if (use_handle) cudaGraphSetConditional(h, 0);
        return;
    }
    flow_ctrl_advance(ctrl, end, sample, s);
    if (use_handle) cudaGraphSetConditional(h, ctrl->done ? 0 : 1);
}

// Final field (prtlb_3d.py:451-456): v = (sum e f + g/2 x) / rho on pore
// voxels, 0 in solid, cast to float32; plus FP64 reductions used by the
// refusals of _checked_flow (prtlb_3d.py:267-316) and the permeability.
// The state after `iters` iterations is gathered exactly as iteration
// `iters` would gather it.
// partials layout: 5 doubles per block: sum ux, sum rho, sum speed, max speed, nonfinite
template <class L, class M, bool ODD>
__global__ void __launch_bounds__(kFlowThreads, M::min_blocks)
    lb_moments_kernel(const typename M::S* __restrict__ f, FlowMap fm, Grid g, LbParams k,
                      float* __restrict__ vel, double* __restrict__ partials) {
    using S = typename M::S;
    using R = typename M::R;
    using RA = typename M::RA;
    const int kk = blockIdx.x * kFlowThreads + threadIdx.x;
    const Lat<S> lat = lattice<L>(const_cast<S*>(f), fm.rs, ODD);
    int far[L::NP];
    far_slots<L, Far::packed>(fm, g, kk, far);
    double sux = 0.0, srho = 0.0, ssp = 0.0, mx = 0.0, nonf = 0.0;
    if (kk < fm.nf) {
        // solid voxels of vel were zeroed before this launch
        int cx, cy, cz;
        unpack_cell((unsigned)fm.cells[kk], fm, cx, cy, cz);
        const long long c = ((long long)cx * g.ny + cy) * g.nz + cz;
        float vx = 0.f, vy = 0.f, vz = 0.f;
        {
            typename Pop<S>::H h[L::Q];
            gather<L, S>(lat, kk, far, k.inv_scale, h);
            const Moments<R, RA> m = moments<L, R, RA>(h, half_force<RA>(k));
            const RA ux = m.jx * m.inv_rho, uy = m.jy * m.inv_rho, uz = m.jz * m.inv_rho;
            vx = (float)ux;
            vy = (float)uy;
            vz = (float)uz;
            sux = (double)ux;
            srho = 1.0 + (double)m.drho;
            // speed the way _checked_flow computes it: float32, (x^2 + y^2) + z^2
            const float sp = sqrtf(__fadd_rn(__fadd_rn(__fmul_rn(vx, vx), __fmul_rn(vy, vy)),
                                             __fmul_rn(vz, vz)));
            nonf = (float)(!isfinite(vx)) + (float)(!isfinite(vy)) + (float)(!isfinite(vz));
            if (isfinite(sp)) {
                ssp = sp;
                mx = sp;
            }
        }
        // 2D grids: the reference returns (ux, uy, 0); our y is the storage z
        if (L::Q == 9) {
            vel[c] = vx;
            vel[g.n + c] = vz;
            vel[2 * g.n + c] = 0.f;
        } else {
            vel[c] = vx;
            vel[g.n + c] = vy;
            vel[2 * g.n + c] = vz;
        }
    }
    __shared__ double sh[5][kFlowThreads / 32];
    double v[5] = {sux, srho, ssp, mx, nonf};
#pragma unroll
    for (int q = 0; q < 5; ++q) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            double t = __shfl_down_sync(0xffffffffu, v[q], o);
            v[q] = (q == 3) ? fmax(v[q], t) : v[q] + t;
        }
        if ((threadIdx.x & 31) == 0) sh[q][threadIdx.x >> 5] = v[q];
    }
    __syncthreads();
    if (threadIdx.x < 32) {
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            double t = threadIdx.x < kFlowThreads / 32 ? sh[q][threadIdx.x] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                double u = __shfl_down_sync(0xffffffffu, t, o);
                t = (q == 3) ? fmax(t, u) : t + u;
            }
            if (threadIdx.x == 0) partials[(long long)blockIdx.x * 5 + q] = t;
        }
    }
}

__global__ void final_reduce_kernel(const double* __restrict__ partials, int nb, double* out) {
    __shared__ double sh[5][256];
    double v[5] = {0, 0, 0, 0, 0};
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            double t = partials[(long long)i * 5 + q];
            v[q] = (q == 3) ? fmax(v[q], t) : v[q] + t;
        }
    }
#pragma unroll
    for (int q = 0; q < 5; ++q) sh[q][threadIdx.x] = v[q];
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                double a = sh[q][threadIdx.x], b = sh[q][threadIdx.x + s];
                sh[q][threadIdx.x] = (q == 3) ? fmax(a, b) : a + b;
            }
        }
        __syncthreads();
    }
    if (threadIdx.x < 5) out[threadIdx.x] = sh[threadIdx.x][0];
}

// Pore flags (set-up of the compacted layout).
__global__ void fluid_flag_kernel(const uint8_t* __restrict__ mat, long long n, int pore,
                                  uint8_t* __restrict__ flag) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c < n) flag[c] = (mat[c] == pore) ? 1 : 0;
}

// imap[cells[k]] = k (imap was filled with -1 first); then cells[k] is
// rewritten from the voxel index to the packed coordinates.
__global__ void imap_scatter_kernel(int* __restrict__ cells, int nf, int* __restrict__ imap,
                                    Grid g, int ys, int xs) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nf) return;
    const int v = cells[k];
    imap[v] = k;
    const int z = v % g.nz;
    const int t = v / g.nz;
    const int y = t % g.ny;
    const int x = t / g.ny;
    cells[k] = (int)(((unsigned)x << xs) | ((unsigned)y << ys) | (unsigned)z);
}

// Links per warp of 32 slots and pair: cnt[p * nw + w] (nw warps).
template <class L>
__global__ void link_count_kernel(FlowMap fm, Grid g, int* __restrict__ cnt) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int nw = (fm.nf + 31) >> 5;
    int x = 0, y = 0, z = 0;
    if (k < fm.nf) unpack_cell((unsigned)fm.cells[k], fm, x, y, z);
#pragma unroll
    for (int p = 0; p < L::NP; ++p) {
        const int i = L::pa(p);
        int xx = x + L::c(i, 0), yy = y + L::c(i, 1), zz = z + L::c(i, 2);
        xx = xx < 0 ? g.nx - 1 : (xx == g.nx ? 0 : xx);
        yy = yy < 0 ? g.ny - 1 : (yy == g.ny ? 0 : yy);
        zz = zz < 0 ? g.nz - 1 : (zz == g.nz ? 0 : zz);
        const bool rock = k < fm.nf && fm.imap[(xx * g.ny + yy) * g.nz + zz] < 0;
        const unsigned links = __ballot_sync(0xffffffffu, rock);
        if ((threadIdx.x & 31) == 0 && k < fm.nf) cnt[p * nw + (k >> 5)] = __popc(links);
    }
}

// Each pair's counts to the rank of every warp's first link (exclusive sums,
// in place), and the pair's total to total[p]; one block per pair.
__global__ void __launch_bounds__(1024) link_scan_kernel(int* __restrict__ cnt, int nw,
                                                         int* __restrict__ total) {
    __shared__ int warp_sum[32];
    int* c = cnt + (long long)blockIdx.x * nw;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int carry = 0;
    for (int at = 0; at < nw; at += 1024) {
        const int i = at + threadIdx.x;
        const int v = i < nw ? c[i] : 0;
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
        if (i < nw) c[i] = carry + before + s - v;
        carry += __shfl_sync(0xffffffffu, ws, 31);
        __syncthreads();
    }
    if (threadIdx.x == 0) total[blockIdx.x] = carry;
}

// The packed table of far places (see FlowMap), one thread per slot.
template <class L>
__global__ void pack_fill_kernel(FlowMap fm, Grid g, unsigned* __restrict__ nbr) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int nfp = (fm.nf + 31) / 32 * 32;
    if (k >= nfp) return;  // whole warps
    int far[L::NP];
    far_slots_map<L>(fm, g, k, far);
    const bool live = k < fm.nf;
    const int lane = threadIdx.x & 31;
    constexpr int words = Packed<L>::words;
    unsigned w[words] = {};
    int mine = 0;  // this lane's share of the bases
    bool fits = true;
#pragma unroll
    for (int p = 0; p < L::NP; ++p) {
        const bool link = live && far[p] >= fm.nf;
        const int lo = __reduce_min_sync(0xffffffffu, live && !link ? far[p] : 0x7fffffff);
        const int hi = __reduce_max_sync(0xffffffffu, live && !link ? far[p] : -1);
        const int lbase = fm.nf + fm.link[p * (nfp / 32) + (k >> 5)];
        if (hi >= 0 && hi - lo > 255) fits = false;
        const int base = hi >= 0 ? lo : 0;
        if (lane == p) mine = base;
        if (lane == L::NP + p) mine = lbase;
        const unsigned d = live ? (unsigned)(far[p] - (link ? lbase : base)) & 0xffu : 0u;
        w[p / 4] |= d << (8 * (p % 4));
        if (link) w[words - 1] |= 1u << (8 + p);
    }
    if (!fits) w[words - 1] |= 1u << 31;  // uniform over the warp
    reinterpret_cast<uint2*>(nbr)[k] = make_uint2(w[0], w[1]);
    if (words > 2) nbr[2 * nfp + k] = w[words - 1];
    if (lane < 2 * L::NP) nbr[words * nfp + (k >> 5) * (2 * L::NP) + lane] = (unsigned)mine;
}

// The plain table of far places: nbr[p * nf + k].
template <class L>
__global__ void nbr_fill_kernel(FlowMap fm, Grid g, int* __restrict__ nbr) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    int far[L::NP];
    far_slots_map<L>(fm, g, k, far);
    if (k >= fm.nf) return;
#pragma unroll
    for (int p = 0; p < L::NP; ++p) nbr[p * fm.nf + k] = far[p];
}

// -------------------------------------------------------------------------
// launchers
// -------------------------------------------------------------------------
int flow_blocks(long long n) { return (int)((n + kFlowThreads - 1) / kFlowThreads); }

// Step kernels go out with programmatic stream serialisation: kernel t+1 starts
// launching while kernel t drains, finds its far places (the tables do not
// change during a solve) and waits in griddepcontrol.wait for t's results
// (launched plainly 64^3 float32 takes 4.52 us an iteration, 54^3 float64
// 4.20, against 4.03 and 3.92).  A grid of one resident wave releases the next
// step only after its stores (pdl_late).  The first step after a check goes out
// plainly (in a loop's graph it is the first node and so does anyway): the
// check's control block is then in place before any step of the chunk is
// resident, and the steps may take it as read-only.

// Blocks of `kern` the device holds at once.
template <class K>
static long long resident_blocks(K kern, int threads) {
    int per_sm = 0, dev = 0, sms = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, 0) !=
            cudaSuccess ||
        cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return (long long)per_sm * sms;
}

// Launches the step in form W and returns true if its blocks are resident at
// once (or ALWAYS), with the launch's error in *e.
template <class L, class M, bool ODD, bool CHECK, Form W, bool ALWAYS>
static bool launch_form(typename M::S* f, const FlowMap& fm, const Grid& g, const LbParams& k,
                        const FlowCtrl* ctrl, int kstep, double* partials, cudaStream_t s,
                        cudaError_t* e) {
    constexpr int threads = form_threads<W>();
    // both places' kernels are held to the same register budget
    static const long long resident =
        resident_blocks(lb_step_kernel<L, M, Far::table, ODD, CHECK, W>, threads);
    const long long nb = ((long long)fm.nf + threads - 1) / threads;
    const bool one_wave = nb <= resident;
    if (!ALWAYS && !one_wave) return false;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)nb);
    cfg.blockDim = dim3(threads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() && kstep > 0 ? 1 : 0;
    auto kern = lb_step_kernel<L, M, Far::table, ODD, CHECK, W>;
    if constexpr (ALWAYS)
        if (!fm.nbr) kern = lb_step_kernel<L, M, Far::packed, ODD, CHECK, W>;
    *e = cudaLaunchKernelEx(&cfg, kern, f, fm, g, k, ctrl, kstep, partials,
                            pdl_late(one_wave) ? 1 : 0, one_wave ? 0 : 1);
    return true;
}

// The waves that nb blocks of 128 take in form W.
template <class L, class M, Form W>
static long long waves(long long nb) {
    static const long long resident = std::max(
        resident_blocks(lb_step_kernel<L, M, Far::table, false, false, W>, kFlowThreads), 1ll);
    return (nb + resident - 1) / resident;
}

template <class L, class M, bool ODD, bool CHECK>
static cudaError_t launch_step_one(typename M::S* f, const FlowMap& fm, const Grid& g,
                                   const LbParams& k, const FlowCtrl* ctrl, int kstep,
                                   double* partials, cudaStream_t s) {
    cudaError_t e = cudaSuccess;
    // D3Q19 float64 stages its gather in shared memory, because in registers it
    // takes 118 of them; a solve whose blocks all fit at four an SM has the
    // registers (54^3: 4.16 -> 3.94 us an iteration, 44^3 3.23 -> 3.07).  One
    // that fits at five an SM gathers into 96 registers, in blocks of 64 that
    // spread evenly over the SMs (57^3 4.76 -> 4.54, 56^3 4.61 -> 4.51, 59^3
    // 4.77 -> 4.80; in blocks of 128 57^3 4.67); beyond, staging wins (60^3
    // 5.3 against 5.6).
    if constexpr (M::staged && L::Q == 19) {
        if (fm.nbr && launch_form<L, M, ODD, CHECK, Form::four, false>(f, fm, g, k, ctrl, kstep,
                                                                       partials, s, &e))
            return e;
        if constexpr (!CHECK)
            if (fm.nbr && launch_form<L, M, ODD, CHECK, Form::halves, false>(f, fm, g, k, ctrl, kstep,
                                                                             partials, s, &e))
                return e;
    }
    // D2Q9 takes the form of more blocks an SM where that saves a wave: us an
    // iteration, wide / narrow, float64 500^2 (1172 blocks, 1036 / 1332 at
    // once) 4.26 / 3.48, 530^2 4.45 / 3.84, 700^2 6.46 / 5.86, float32 560^2
    // (1469 blocks, 1332 / 1480) 3.59 / 3.20, float16 3.53 / 3.22; with as many
    // waves float32 600^2 3.72 / 3.81, 800^2 5.40 / 5.54, float16 400^2 2.37 /
    // 2.43.
    if constexpr (L::Q == 9 && M::narrow_blocks > 0) {
        const long long nb = flow_blocks(fm.nf);
        if (waves<L, M, Form::narrow>(nb) < waves<L, M, Form::wide>(nb)) {
            launch_form<L, M, ODD, CHECK, Form::narrow, true>(f, fm, g, k, ctrl, kstep, partials, s, &e);
            return e;
        }
    }
    launch_form<L, M, ODD, CHECK, Form::wide, true>(f, fm, g, k, ctrl, kstep, partials, s, &e);
    return e;
}

template <class L, class M>
static cudaError_t launch_step_t(bool odd, bool check, void* f, const FlowMap& fm,
                                 const Grid& g, const LbParams& k, const FlowCtrl* ctrl, int kstep,
                                 double* partials, cudaStream_t s) {
    if (fm.nf <= 0) return cudaSuccess;
    typename M::S* fs = static_cast<typename M::S*>(f);
    if (!odd && !check) return launch_step_one<L, M, false, false>(fs, fm, g, k, ctrl, kstep, partials, s);
    if (!odd && check) return launch_step_one<L, M, false, true>(fs, fm, g, k, ctrl, kstep, partials, s);
    if (odd && !check) return launch_step_one<L, M, true, false>(fs, fm, g, k, ctrl, kstep, partials, s);
    return launch_step_one<L, M, true, true>(fs, fm, g, k, ctrl, kstep, partials, s);
}

#define PRT_DISPATCH(FN, ...)                                                        \
    if (nd == 3) {                                                                   \
        if (precision == PRT_FP64) return FN<D3Q19, ModeF64>(__VA_ARGS__);           \
        if (precision == PRT_FP32) return FN<D3Q19, ModeF32D>(__VA_ARGS__);          \
        if (precision == PRT_FP32_F32) return FN<D3Q19, ModeF32>(__VA_ARGS__);       \
        return FN<D3Q19, ModeF16>(__VA_ARGS__);                                      \
    }                                                                                \
    if (precision == PRT_FP64) return FN<D2Q9, ModeF64>(__VA_ARGS__);                \
    if (precision == PRT_FP32) return FN<D2Q9, ModeF32D>(__VA_ARGS__);               \
    if (precision == PRT_FP32_F32) return FN<D2Q9, ModeF32>(__VA_ARGS__);            \
    return FN<D2Q9, ModeF16>(__VA_ARGS__);

cudaError_t flow_launch_step(int nd, int precision, bool odd, bool check, void* f,
                             const FlowMap& fm, const Grid& g, const LbParams& k,
                             const FlowCtrl* ctrl, int kstep, double* partials, cudaStream_t s) {
    PRT_DISPATCH(launch_step_t, odd, check, f, fm, g, k, ctrl, kstep, partials, s)
}

cudaError_t flow_launch_check(FlowCtrl* ctrl, const double* partials, int nblocks,
                              cudaGraphConditionalHandle h, int use_handle, cudaStream_t s) {
    flow_check_kernel<<<1, kFlowThreads, 0, s>>>(ctrl, partials, nblocks, h, use_handle);
    return cudaGetLastError();
}

template <class L, class M>
static cudaError_t launch_moments_t(bool odd, const void* f, const FlowMap& fm, const Grid& g,
                                    const LbParams& k, float* vel, double* partials, cudaStream_t s) {
    if (fm.nf <= 0) return cudaSuccess;
    const typename M::S* fs = static_cast<const typename M::S*>(f);
    if (odd) lb_moments_kernel<L, M, true><<<flow_blocks(fm.nf), kFlowThreads, 0, s>>>(fs, fm, g, k, vel, partials);
    else lb_moments_kernel<L, M, false><<<flow_blocks(fm.nf), kFlowThreads, 0, s>>>(fs, fm, g, k, vel, partials);
    return cudaGetLastError();
}

cudaError_t flow_launch_moments(int nd, int precision, bool odd, const void* f,
                                const FlowMap& fm, const Grid& g, const LbParams& k, float* vel,
                                double* partials, cudaStream_t s) {
    PRT_DISPATCH(launch_moments_t, odd, f, fm, g, k, vel, partials, s)
}

cudaError_t flow_launch_flags(const uint8_t* mat, long long n, int pore, uint8_t* flag,
                              cudaStream_t s) {
    fluid_flag_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(mat, n, pore, flag);
    return cudaGetLastError();
}

cudaError_t flow_launch_imap(int* cells, int nf, int* imap, const Grid& g, int ys, int xs,
                             cudaStream_t s) {
    if (nf <= 0) return cudaSuccess;
    imap_scatter_kernel<<<(unsigned)((nf + 255) / 256), 256, 0, s>>>(cells, nf, imap, g, ys, xs);
    return cudaGetLastError();
}

cudaError_t flow_launch_links(int nd, const FlowMap& fm, const Grid& g, int* link, int* total,
                              cudaStream_t s) {
    if (fm.nf <= 0) return cudaMemsetAsync(total, 0, 9 * sizeof(int), s);
    const unsigned nb = (unsigned)((fm.nf + 255) / 256);
    const int nw = (fm.nf + 31) / 32;
    if (nd == 3) link_count_kernel<D3Q19><<<nb, 256, 0, s>>>(fm, g, link);
    else link_count_kernel<D2Q9><<<nb, 256, 0, s>>>(fm, g, link);
    link_scan_kernel<<<nd == 3 ? D3Q19::NP : D2Q9::NP, 1024, 0, s>>>(link, nw, total);
    return cudaGetLastError();
}

cudaError_t flow_launch_nbr(int nd, const FlowMap& fm, const Grid& g, int* nbr, cudaStream_t s) {
    if (fm.nf <= 0) return cudaSuccess;
    const unsigned nb = (unsigned)((fm.nf + 255) / 256);
    if (nd == 3) nbr_fill_kernel<D3Q19><<<nb, 256, 0, s>>>(fm, g, nbr);
    else nbr_fill_kernel<D2Q9><<<nb, 256, 0, s>>>(fm, g, nbr);
    return cudaGetLastError();
}

cudaError_t flow_launch_pack(int nd, const FlowMap& fm, const Grid& g, int* pack, cudaStream_t s) {
    if (fm.nf <= 0) return cudaSuccess;
    const unsigned nb = (unsigned)((fm.nf + 255) / 256);
    unsigned* out = reinterpret_cast<unsigned*>(pack);
    if (nd == 3) pack_fill_kernel<D3Q19><<<nb, 256, 0, s>>>(fm, g, out);
    else pack_fill_kernel<D2Q9><<<nb, 256, 0, s>>>(fm, g, out);
    return cudaGetLastError();
}

cudaError_t flow_launch_final_reduce(const double* partials, int nb, double* out, cudaStream_t s) {
    final_reduce_kernel<<<1, 256, 0, s>>>(partials, nb, out);
    return cudaGetLastError();
}

// compile-time checks of the lattice tables
template <class L>
constexpr bool pairs_evenly_spaced() {
    for (int p = 0; p < L::NP; ++p)
        if (L::pb(p) - L::pa(p) != L::pb(0) - L::pa(0) || L::opp(L::pa(p)) != L::pb(p)) return false;
    return true;
}
static_assert(pairs_evenly_spaced<D3Q19>() && pairs_evenly_spaced<D2Q9>(), "Lat's row offsets");
static_assert(D3Q19::opp(7) == 8 && D3Q19::opp(18) == 17, "D3Q19 opposites");
static_assert(D3Q19::c(13, 0) == 1 && D3Q19::c(13, 2) == -1, "D3Q19 e_13");
static_assert(D3Q19::c(18, 1) == -1 && D3Q19::c(18, 2) == 1, "D3Q19 e_18");
static_assert(D2Q9::pa(0) == 1 && D2Q9::pb(0) == 3 && D2Q9::pa(3) == 6 && D2Q9::pb(3) == 8, "D2Q9 pairs");
static_assert(D2Q9::opp(1) == 3 && D2Q9::opp(2) == 4 && D2Q9::opp(3) == 1 && D2Q9::opp(4) == 2 &&
                  D2Q9::opp(5) == 7 && D2Q9::opp(6) == 8 && D2Q9::opp(7) == 5 && D2Q9::opp(8) == 6,
              "D2Q9 opposites");
static_assert(D2Q9::ex(6) == -1 && D2Q9::ey(6) == 1 && D2Q9::ex(8) == 1 && D2Q9::ey(8) == -1, "D2Q9 e");

}  // namespace prt

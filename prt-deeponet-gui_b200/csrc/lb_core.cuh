// lb_core.cuh -- lattices and the per-voxel TRT collision of the flow solve,
// shared by the single-solve and batched kernels.
#pragma once

#include <cuda_fp16.h>

#include "prt_internal.h"

namespace prt {

// -------------------------------------------------------------------------
// Lattices, in the storage frame (x, y, z).  The direction order and weights
// are the reference's (prtlb_3d.py:370-375, prtlb_2d.py:391-394); a D2Q9
// direction (ex, ey) is stored as (ex, 0, ey) because 2D grids are kept as
// (nx, 1, ny).
// -------------------------------------------------------------------------
struct D3Q19 {
    static constexpr int Q = 19;
    static constexpr int NP = 9;
    __host__ __device__ static constexpr int c(int i, int a) {
        return (a == 0) ? (i == 1 || i == 7 || i == 9 || i == 11 || i == 13   ? 1
                           : i == 2 || i == 8 || i == 10 || i == 12 || i == 14 ? -1
                                                                                : 0)
             : (a == 1) ? (i == 3 || i == 7 || i == 10 || i == 15 || i == 17   ? 1
                           : i == 4 || i == 8 || i == 9 || i == 16 || i == 18  ? -1
                                                                                : 0)
                        : (i == 5 || i == 11 || i == 14 || i == 15 || i == 18  ? 1
                           : i == 6 || i == 12 || i == 13 || i == 16 || i == 17 ? -1
                                                                                 : 0);
    }
    // pairs (a, b) with e_b = -e_a
    __host__ __device__ static constexpr int pa(int p) { return 2 * p + 1; }
    __host__ __device__ static constexpr int pb(int p) { return 2 * p + 2; }
    __host__ __device__ static constexpr int opp(int i) {
        return i == 0 ? 0 : ((i & 1) ? i + 1 : i - 1);
    }
    __host__ __device__ static constexpr double w(int i) {
        return i == 0 ? 1.0 / 3.0 : (i < 7 ? 1.0 / 18.0 : 1.0 / 36.0);
    }
};

struct D2Q9 {
    static constexpr int Q = 9;
    static constexpr int NP = 4;
    // reference order: (0,0) (1,0) (0,1) (-1,0) (0,-1) (1,1) (-1,1) (-1,-1) (1,-1)
    __host__ __device__ static constexpr int ex(int i) {
        return (i == 1 || i == 5 || i == 8) ? 1 : ((i == 3 || i == 6 || i == 7) ? -1 : 0);
    }
    __host__ __device__ static constexpr int ey(int i) {
        return (i == 2 || i == 5 || i == 6) ? 1 : ((i == 4 || i == 7 || i == 8) ? -1 : 0);
    }
    __host__ __device__ static constexpr int c(int i, int a) {
        return a == 0 ? ex(i) : (a == 1 ? 0 : ey(i));
    }
    __host__ __device__ static constexpr int pa(int p) { return p < 2 ? p + 1 : p + 3; }
    __host__ __device__ static constexpr int pb(int p) { return p < 2 ? p + 3 : p + 5; }
    __host__ __device__ static constexpr int opp(int i) {
        return i == 0 ? 0 : (i < 5 ? ((i + 1) % 4) + 1 : ((i - 3) % 4) + 5);
    }
    __host__ __device__ static constexpr double w(int i) {
        return i == 0 ? 4.0 / 9.0 : (i < 5 ? 1.0 / 9.0 : 1.0 / 36.0);
    }
};

// storage conversions ------------------------------------------------------
// Pop<S>::H is the register type a stored population is held in; enc() rounds
// the collision result to the storage type once.
template <class S>
struct Pop;
template <>
struct Pop<double> {
    using H = double;
    __device__ static double dec(double v, float) { return v; }
    template <class R>
    __device__ static double enc(R v, float) { return (double)v; }
};
template <>
struct Pop<float> {
    using H = float;
    __device__ static float dec(float v, float) { return v; }
    template <class R>
    __device__ static float enc(R v, float) { return (float)v; }
};
template <>
struct Pop<__half> {
    using H = float;
    __device__ static float dec(__half v, float inv) { return __half2float(v) * inv; }
    template <class R>
    __device__ static __half enc(R v, float scale) {
        float s = (float)v * scale;
        s = fminf(fmaxf(s, -65504.f), 65504.f);
        return __float2half_rn(s);
    }
};

// Whether the collision forms its store addresses again instead of keeping
// those of the loads, which use the same places: 2 (Q - 1) registers that
// spill in D3Q19's float64 arithmetic.  index: again from the slot numbers,
// base: again from the lattice's address.  Measured on 128^3 / 64^3 packs (us
// an iteration, none / index / base): float64 72.8 / 57.3 / 56.9 and 8.3 /
// 6.6 / 6.1, float32 with float64 momentum 32.1 / 28.6 / 29.3 and 4.8 / 4.7 /
// 4.9, float16 22.4 / 20.1 / 20.8 and - / 3.8 / 4.3; float32 alone without it
// spills 88 bytes (4.97 against 3.91 at 64^3).
enum class Fresh { none, index, base };

// Precision modes: storage type S, arithmetic R for the symmetric part and
// RA for the momentum and the antisymmetric non-equilibrium part (a small
// difference of two O(u) numbers), and the resident blocks of kFlowThreads
// per SM the register budget is cut for (single-solve and batched steps;
// narrow: D2Q9 single solves that save a wave by it, 0 where none does).
// `fresh`: see Fresh; `regrouped`: see collide_regrouped.
// `staged`: D3Q19's arrived populations go to shared memory by cp.async, so no
// register waits on a gather load.  Only float64 gains by it (80^3 9.8 against
// 12.1 us in registers, which spill); in float32 the 57 shared-memory accesses
// a voxel cost more than they save: us an iteration, staged -> in registers,
// 64^3 4.27 -> 3.91 (float64 momentum 4.73 -> 4.35), 128^3 23.8 -> 23.2 (26.5
// -> 25.6), 192^3 104 -> 93 (106 -> 100); D2Q9 256^2 float64 2.34 -> 2.14.
struct ModeF64 {  // the reference's arithmetic
    using S = double;
    using R = double;
    using RA = double;
    static constexpr int min_blocks = 7;
    static constexpr int narrow_blocks = 9;
    static constexpr Fresh fresh = Fresh::base;
    static constexpr bool regrouped = true;
    static constexpr int batch_min_blocks = 6;
    static constexpr bool staged = true;
};
struct ModeF32 {  // float32 populations, float32 collision
    using S = float;
    using R = float;
    using RA = float;
    // 64 registers (8 blocks per SM)
    static constexpr int min_blocks = 8;
    static constexpr int narrow_blocks = 10;
    static constexpr Fresh fresh = Fresh::index;
    static constexpr bool regrouped = true;
    static constexpr int batch_min_blocks = 8;
    static constexpr bool staged = false;
};
struct ModeF32D {  // float32 populations, float64 momentum
    using S = float;
    using R = float;
    using RA = double;
    // 64 registers: at 48 (10 blocks) the step kernel spills, and 64^3
    // (917 blocks) still fits one wave at 8 blocks per SM (5.67 -> 5.41 us
    // per iteration; 128^3 unchanged)
    static constexpr int min_blocks = 8;
    static constexpr int narrow_blocks = 0;
    static constexpr Fresh fresh = Fresh::index;
    static constexpr bool regrouped = false;
    static constexpr int batch_min_blocks = 8;
    static constexpr bool staged = false;
};
struct ModeF16 {  // scaled float16 populations, float32 collision
    using S = __half;
    using R = float;
    using RA = float;
    static constexpr int min_blocks = 6;
    static constexpr int narrow_blocks = 10;
    static constexpr Fresh fresh = Fresh::index;
    static constexpr bool regrouped = false;
    static constexpr int batch_min_blocks = 6;
    static constexpr bool staged = false;
};

// One lattice, updated in place (see the file comment of lb_flow.cu).  Row i
// holds one population of every pore slot (elements [0, nf)) and, behind
// them, the pair's rock links; row i starts at element i * rs.  In an
// iteration the pair (a, b), e_b = -e_a, of the voxel in slot k uses two
// places: its own element k of row `b` (even iterations) or `a` (odd), and
// element far of the other row, far being the slot of the voxel x + e_a or,
// when that is rock, the link's own element.  f_a is read from the own place
// and f_b written there; f_b is read from the far place and f_a written
// there.  No other thread touches either place in the iteration.
// Offsets are unsigned 32-bit: rs is at most the voxel count (a direction
// has no more links than the grid has rock voxels) and at most 2 nf, and
// 2 Q nf < 2^31 is checked at set-up.
template <class S>
struct Lat {
    S* f;
    unsigned rs, own, far;  // far / own: element offset of the rows of the two places
    __device__ S* at_own(int a, unsigned k) const { return f + (a * rs + own + k); }
    __device__ S* at_far(int a, unsigned slot) const { return f + (a * rs + far + slot); }
};

template <class L, class S>
__device__ __forceinline__ Lat<S> lattice(S* f, unsigned rs, bool odd) {
    constexpr unsigned d = L::pb(0) - L::pa(0);  // the same for every pair
    return Lat<S>{f, rs, odd ? 0u : d * rs, odd ? d * rs : 0u};
}

// The far places of slot k (see Lat), one per pair, from the packed cell and
// the voxel map: the slot of x + e_a (periodic), or nf + the rank of this
// link among the pair's links, which the warp forms from its first link's
// rank (fm.link) and the lanes below.  Every lane of the warp calls it;
// lanes beyond the last slot get nothing.
template <class L>
__device__ __forceinline__ void far_slots_map(const FlowMap& fm, const Grid& g, int k,
                                              int (&far)[L::NP]) {
    const bool live = k < fm.nf;
    int x = 0, y = 0, z = 0;
    if (live) unpack_cell((unsigned)fm.cells[k], fm, x, y, z);
    // the candidate coordinates per axis are formed once; a direction then
    // costs one index and one map load
    const int X[3] = {x == 0 ? g.nx - 1 : x - 1, x, x == g.nx - 1 ? 0 : x + 1};
    const int Y[3] = {y == 0 ? g.ny - 1 : y - 1, y, y == g.ny - 1 ? 0 : y + 1};
    const int Z[3] = {z == 0 ? g.nz - 1 : z - 1, z, z == g.nz - 1 ? 0 : z + 1};
#pragma unroll
    for (int p = 0; p < L::NP; ++p) {
        const int i = L::pa(p);
        far[p] = 0;
        if (live)
            far[p] = fm.imap[(X[1 + L::c(i, 0)] * g.ny + Y[1 + L::c(i, 1)]) * g.nz +
                             Z[1 + L::c(i, 2)]];
    }
    const unsigned below = (1u << (threadIdx.x & 31)) - 1u;
    const int nw = (fm.nf + 31) >> 5;
#pragma unroll
    for (int p = 0; p < L::NP; ++p) {
        const unsigned links = __ballot_sync(0xffffffffu, far[p] < 0);
        if (far[p] < 0) far[p] = fm.nf + fm.link[p * nw + (k >> 5)] + __popc(links & below);
    }
}

// The packed table of far places (fm.pack, see FlowMap) as one thread of a warp
// holds it: its own words and its lane's share of the warp's bases.
template <class L>
struct Packed {
    static constexpr int words = L::NP > 4 ? 3 : 2;
    unsigned w[words];
    int base;
};

// Ints before the bases of the packed table of nf slots.
template <class L>
__host__ __device__ inline long long packed_words(int nf) {
    return (long long)Packed<L>::words * ((nf + 31) / 32 * 32);
}

template <class L>
__device__ __forceinline__ Packed<L> load_packed(const FlowMap& fm, int k) {
    Packed<L> q;
    const unsigned nfp = (unsigned)(fm.nf + 31) / 32 * 32;
    const int lane = threadIdx.x & 31;
    q.base = 0;
    if ((unsigned)k < nfp) {  // uniform over the warp
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(fm.pack) + k);
        q.w[0] = v.x;
        q.w[1] = v.y;
        if (Packed<L>::words > 2) q.w[Packed<L>::words - 1] = __ldg(fm.pack + (2 * nfp + k));
        if (lane < 2 * L::NP)
            q.base = __ldg(fm.pack + (Packed<L>::words * nfp + (k >> 5) * (2 * L::NP) + lane));
    } else {
#pragma unroll
        for (int i = 0; i < Packed<L>::words; ++i) q.w[i] = 0;
    }
    return q;
}

// The far places of slot k from its packed words; a warp whose places do not
// fit the packed form looks them up in the maps.  Every lane of the warp
// calls it.
template <class L>
__device__ __forceinline__ void far_slots_packed(const FlowMap& fm, const Grid& g, int k,
                                                 const Packed<L>& q, int (&far)[L::NP]) {
    const unsigned last = q.w[Packed<L>::words - 1];
    if ((int)last < 0) {  // uniform over the warp
        far_slots_map<L>(fm, g, k, far);
        return;
    }
#pragma unroll
    for (int p = 0; p < L::NP; ++p) {
        const int src = p + ((last >> (8 + p)) & 1u) * L::NP;
        const unsigned d = (q.w[p / 4] >> (8 * (p % 4))) & 0xffu;
        far[p] = __shfl_sync(0xffffffffu, q.base, src) + (int)d;
    }
}

// How a launch finds its far places: from the plain table (one coalesced load
// per pair and 36 B a slot in D3Q19), or from the packed table (14.3 B) and
// the maps.  The plain table's chain is the shortest and wins while it and
// the lattice stay in the L2 (flow_use_nbr): us an iteration, plain / packed
// / maps alone, 64^3 float32 4.2 / 4.6 / 5.0, 96^3 float64 16.2 / 17.6 / 23.6,
// 128^3 float16 20.3 / 21.7 / 26.2; beyond it the bytes decide: 128^3 float32
// 26.7 / 24.9 / 30.7, 192^3 112 / 104 / 126 (populations staged, see below).
enum class Far { table, packed };

template <class L, Far F>
__device__ __forceinline__ void far_slots(const FlowMap& fm, const Grid& g, int k,
                                          int (&far)[L::NP]) {
    if constexpr (F == Far::table) {
#pragma unroll
        for (int p = 0; p < L::NP; ++p) far[p] = k < fm.nf ? __ldg(fm.nbr + p * fm.nf + k) : 0;
    } else {
        far_slots_packed<L>(fm, g, k, load_packed<L>(fm, k), far);
    }
}

// The populations that arrive at slot k in this iteration.
template <class L, class S>
__device__ __forceinline__ void gather(const Lat<S>& lat, int k, const int (&far)[L::NP],
                                       float inv, typename Pop<S>::H (&h)[L::Q]) {
    h[0] = Pop<S>::dec(lat.f[k], inv);
#pragma unroll
    for (int p = 0; p < L::NP; ++p) {
        h[L::pa(p)] = Pop<S>::dec(*lat.at_own(L::pa(p), k), inv);
        h[L::pb(p)] = Pop<S>::dec(*lat.at_far(L::pa(p), far[p]), inv);
    }
}

// 128-thread blocks: at 64^3 (458 blocks of 256 for 148 SMs) finer blocks
// balance the SMs better and cut an iteration from 6.25 to 5.73 us.
constexpr int kFlowThreads = 128;

// cp.async of one 4- or 8-byte population into this thread's shared slot.
template <class S>
__device__ __forceinline__ void cp_async_pop(S* dst, const S* src) {
    static_assert(sizeof(S) == 4 || sizeof(S) == 8, "cp.async copies 4 or 8 bytes here");
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if (sizeof(S) == 4)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}

__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// The arrived populations of one thread in shared memory: element i of the
// thread's column (stride kFlowThreads).
template <class S>
struct Staged {
    const S* col;
    __device__ S operator[](int i) const { return col[i * kFlowThreads]; }
};

// The gather with the population loads issued as cp.async into `col` (this
// thread's column of a [Q][kFlowThreads] shared array): the same sources,
// but no register is held while a load is in flight.
template <class L, class S>
__device__ __forceinline__ void gather_staged(const Lat<S>& lat, int k, const int (&far)[L::NP],
                                              S* col) {
    cp_async_pop(col, lat.f + k);
#pragma unroll
    for (int p = 0; p < L::NP; ++p) {
        cp_async_pop(col + L::pa(p) * kFlowThreads, lat.at_own(L::pa(p), k));
        cp_async_pop(col + L::pb(p) * kFlowThreads, lat.at_far(L::pa(p), far[p]));
    }
    cp_async_commit();
}

template <class RA>
__device__ __forceinline__ RA half_force(const LbParams& kc) {
    if constexpr (sizeof(RA) == 8) return kc.half_g;
    else return kc.half_g_f;
}

template <class R, class RA>
struct Moments {
    R drho, jsq;    // density deviation, rho u^2
    RA jx, jy, jz;  // J = rho u (with the half force on x)
    RA inv_rho;
};

// Moments of the arrived (shifted) populations (prtlb_3d.py:428-433):
// drho = sum h, J = rho u = sum e h + g/2 x.
template <class L, class R, class RA, class HA>
__device__ __forceinline__ Moments<R, RA> moments(const HA& h, RA half_g) {
    Moments<R, RA> m;
    RA s = RA(h[0]);
    RA jx = RA(0), jy = RA(0), jz = RA(0);
#pragma unroll
    for (int p = 0; p < L::NP; ++p) {
        const int a = L::pa(p), b = L::pb(p);
        s += RA(h[a]) + RA(h[b]);
        const RA d = RA(h[a]) - RA(h[b]);
        if (L::c(a, 0) == 1) jx += d;
        if (L::c(a, 0) == -1) jx -= d;
        if (L::c(a, 1) == 1) jy += d;
        if (L::c(a, 1) == -1) jy -= d;
        if (L::c(a, 2) == 1) jz += d;
        if (L::c(a, 2) == -1) jz -= d;
    }
    jx += half_g;
    m.jx = jx;
    m.jy = jy;
    m.jz = jz;
    const RA rho = RA(1) + s;
    m.inv_rho = RA(1) / rho;
    m.drho = R(s);
    m.jsq = R((jx * jx + jy * jy + jz * jz) * m.inv_rho);  // rho u^2 = |J|^2 / rho
    return m;
}

// TRT collision (_trt_collide, prtlb_3d.py:142-154) + Guo forcing in the
// shifted variables, written with J = rho u so that rho cancels in the
// antisymmetric equilibrium (w rho 3 e.u = 3 w e.J) and rho u u = J J / rho in
// the symmetric one.  The new population is h + delta with delta summed
// first, so the stored result rounds once.  put(i, p, v) takes the new
// population i, of pair p (-1: the rest population).
template <class L, class R, class RA, class HA, class Put>
__device__ __forceinline__ void collide(const HA& h, const Moments<R, RA>& m, const LbParams& kc,
                                        Put put) {
    const R omp = R(kc.omp);
    const R inv_rho = R(m.inv_rho);
    const R heq0 = R(L::w(0)) * (m.drho - R(1.5) * m.jsq);
    const R h0 = R(h[0]);
    put(0, -1, h0 - omp * (h0 - heq0));
#pragma unroll
    for (int p = 0; p < L::NP; ++p) {
        const int a = L::pa(p), b = L::pb(p);
        RA eJ = RA(0);
        if (L::c(a, 0) == 1) eJ += m.jx;
        if (L::c(a, 0) == -1) eJ -= m.jx;
        if (L::c(a, 1) == 1) eJ += m.jy;
        if (L::c(a, 1) == -1) eJ -= m.jy;
        if (L::c(a, 2) == 1) eJ += m.jz;
        if (L::c(a, 2) == -1) eJ -= m.jz;
        const R eJr = R(eJ);
        const R heq_p = R(L::w(a)) * (m.drho + (R(4.5) * eJr * eJr * inv_rho - R(1.5) * m.jsq));
        const R ha = R(h[a]), hb = R(h[b]);
        const R dp = omp * (R(0.5) * (ha + hb) - heq_p);
        const RA dma = RA(kc.omm) * (RA(0.5) * (RA(h[a]) - RA(h[b])) - RA(3.0 * L::w(a)) * eJ);
        const R dm = R(dma);
        const R gp = R(kc.guo[p]);
        put(a, p, ha + ((gp - dp) - dm));
        put(b, p, hb + ((dm - dp) - gp));
    }
}

// The same collision with its constants folded and the pair's symmetric and
// antisymmetric changes formed as one fused sum each, the two members as h +
// (A - B) and h + (A + B): 12 operations a pair where collide takes 18, and
// no conversion of constants.  Its rounding errors are of the same size (a
// sum of the same terms, fewer roundings); the modes whose collision has one
// arithmetic type and whose results are not tied to another rounding take it.
template <class L, class R, class HA, class Put>
__device__ __forceinline__ void collide_regrouped(const HA& h, const Moments<R, R>& m,
                                                  const Regrouped<R>& kc, Put put) {
    const R base = m.drho - R(1.5) * m.jsq;
    const R h0 = R(h[0]);
    put(0, -1, h0 + (kc.w0 * base - kc.omp * h0));
    const R b[2] = {kc.wp[0] * base, kc.wp[1] * base};
    const R q[2] = {kc.w45[0] * m.inv_rho, kc.w45[1] * m.inv_rho};
#pragma unroll
    for (int p = 0; p < L::NP; ++p) {
        const int a = L::pa(p), bb = L::pb(p);
        constexpr int axis_pairs = L::Q == 19 ? 3 : 2;
        const int c = p < axis_pairs ? 0 : 1;
        R eJ = R(0);
        if (L::c(a, 0) == 1) eJ += m.jx;
        if (L::c(a, 0) == -1) eJ -= m.jx;
        if (L::c(a, 1) == 1) eJ += m.jy;
        if (L::c(a, 1) == -1) eJ -= m.jy;
        if (L::c(a, 2) == 1) eJ += m.jz;
        if (L::c(a, 2) == -1) eJ -= m.jz;
        const R ha = R(h[a]), hb = R(h[bb]);
        const R A = (q[c] * eJ * eJ + b[c]) - kc.half_omp * (ha + hb);
        R B = kc.half_omm * (ha - hb) - kc.wm[c] * eJ;
        if (L::c(a, 0) != 0) B -= kc.guo[p];
        put(a, p, ha + (A - B));
        put(bb, p, hb + (A + B));
    }
}

// The mode's collision.
template <class L, class M, class HA, class Put>
__device__ __forceinline__ void collide_mode(const HA& h,
                                             const Moments<typename M::R, typename M::RA>& m,
                                             const LbParams& kc, Put put) {
    if constexpr (M::regrouped) {
        if constexpr (sizeof(typename M::R) == 8) collide_regrouped<L>(h, m, kc.d, put);
        else collide_regrouped<L>(h, m, kc.f, put);
    } else {
        collide<L, typename M::R, typename M::RA>(h, m, kc, put);
    }
}

// The collision of slot k with its results stored in the lattice: f_a to the
// pair's far place and f_b to its own (see Lat).
template <class L, class M, bool INDEX, class HA>
__device__ __forceinline__ void collide_store(const Lat<typename M::S>& lat0, int k,
                                              const int (&far)[L::NP], const HA& h,
                                              const Moments<typename M::R, typename M::RA>& m,
                                              const LbParams& kc) {
    using S = typename M::S;
    constexpr Fresh F = INDEX ? Fresh::index : L::Q == 19 ? M::fresh : Fresh::none;
    Lat<S> lat = lat0;
    int to[L::NP];
    if (F == Fresh::base) asm volatile("" : "+l"(lat.f));
    if (F == Fresh::index) asm volatile("" : "+r"(k));
#pragma unroll
    for (int p = 0; p < L::NP; ++p) {
        to[p] = far[p];
        if (F == Fresh::index) asm volatile("" : "+r"(to[p]));
    }
    collide_mode<L, M>(h, m, kc, [&](int i, int p, typename M::R v) {
        const S q = Pop<S>::enc(v, kc.scale);
        if (p < 0) lat.f[k] = q;
        else if (i == L::pa(p)) *lat.at_far(i, to[p]) = q;
        else *lat.at_own(L::pa(p), k) = q;
    });
}

// One pore voxel (slot k) of one LB iteration, its far places already found:
// gather, moments, collision, store; returns |u_x| for the convergence mean.
// INDEX: the store addresses from the slot numbers whatever the mode's Fresh.
template <class L, class M, bool STAGED = M::staged && L::Q == 19, bool INDEX = false>
__device__ __forceinline__ double lb_cell(const Lat<typename M::S>& lat, const LbParams& kc, int k,
                                          const int (&far)[L::NP]) {
    using S = typename M::S;
    using R = typename M::R;
    using RA = typename M::RA;
    if constexpr (STAGED) {
        __shared__ S stage[L::Q * kFlowThreads];
        S* col = stage + threadIdx.x;
        gather_staged<L, S>(lat, k, far, col);
        cp_async_wait<0>();
        const Staged<S> h{col};
        const Moments<R, RA> m = moments<L, R, RA>(h, half_force<RA>(kc));
        collide_store<L, M, INDEX>(lat, k, far, h, m, kc);
        return fabs((double)m.jx * (double)m.inv_rho);
    } else {
        typename Pop<S>::H h[L::Q];
        gather<L, S>(lat, k, far, kc.inv_scale, h);
        const Moments<R, RA> m = moments<L, R, RA>(h, half_force<RA>(kc));
        collide_store<L, M, INDEX>(lat, k, far, h, m, kc);
        return fabs((double)m.jx * (double)m.inv_rho);
    }
}

// Block sum of one double per thread (warp shuffles, then the warp sums in
// order), stored by thread 0.  Both the single-solve and the batched step
// kernels reduce |u_x| with it, so their per-block partials agree bit for
// bit.  Every thread of the block must call it.
__device__ __forceinline__ void block_sum_store(double acc, double* out) {
    __shared__ double sh[kFlowThreads / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x < 32) {
        double v = threadIdx.x < kFlowThreads / 32 ? sh[threadIdx.x] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (threadIdx.x == 0) *out = v;
    }
    __syncthreads();
}

// Deterministic sum of n per-block partials by one block of kFlowThreads
// threads (fixed order: strided per thread, then a shared-memory tree).
// Loads bypass L1 because in the batched kernel other blocks of the same
// launch wrote the partials.
__device__ __forceinline__ double block_sum_fixed(const double* p, int n) {
    __shared__ double sh[kFlowThreads];
    double v = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) v += __ldcg(p + i);
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    const double r = sh[0];
    __syncthreads();
    return r;
}

// FlowConvergence bookkeeping (prtlb_3d.py:220-235) once the iterations up
// to `end` are done; `sample` says whether the mean |u_x| of iteration end-1
// (sum s over the pore) was taken at this point (every `every` iterations).
// A sampled sum that is not finite stops the solve at once: the reference
// would run on to its cap (a NaN change never meets the tolerance) and then
// refuse the field, so stopping early changes only how long a doomed solve
// takes, never a finite result.
__device__ __forceinline__ void flow_ctrl_advance(FlowCtrl* c, long long end, bool sample,
                                                  double s) {
    c->iters = end;
    if (sample && !isfinite(s)) {
        c->nonfinite = 1;
    } else if (sample && c->tol > 0) {
        const double u = c->nfluid > 0 ? s / (double)c->nfluid : 0.0;
        if (c->has_prev) {
            c->change = fabs(u - c->prev) / fmax(fabs(u), 1e-30);
            if (c->change <= c->tol) c->converged = 1;
        }
        c->prev = u;
        c->has_prev = 1;
    }
    c->it_base = end;
    if (c->converged || c->nonfinite || end >= c->nit) c->done = 1;
}

}  // namespace prt

// adr_core.cuh -- per-voxel arithmetic of the transport step (solve_adr,
// prtlb_3d.py:1182-1413), shared by the single-solve and batched kernels.
// Every translation unit that includes it is compiled with -fmad=false: the
// reference integrates in float32 with numpy, one rounding per operation,
// and the operation order below is the reference's, so results are
// bit-identical to it.
#pragma once

#include "prt_internal.h"

namespace prt {

// numpy's elementwise semantics ---------------------------------------------
__device__ __forceinline__ float np_min(float a, float b) { return (a <= b || a != a) ? a : b; }
__device__ __forceinline__ float np_max(float a, float b) { return (a >= b || a != a) ? a : b; }

// min of two values that is NaN when either is (as np_min's value; the NaN
// may carry another payload).
__device__ __forceinline__ float min_nan(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// The upwind face value of _muscl (prtlb_3d.py:650-705), up + 1/2 minmod(down -
// up, up - upup), from the two differences along the axis, taken upwards: for
// flow up the axis they are (down - up, up - upup) themselves and s = 1, for
// flow down it both are negated, which negates the slope exactly, and s = -1.
// The reference forms minmod as 1/2 (sgn a + sgn b) min(|a|, |b|) and halves
// it; (1/4 sgn a + 1/4 sgn b) min rounds the same once (1/2 min or 0), and s
// x is exact inside the fused add.  The signs are taken from the sign bits,
// which differs from numpy's sign() only at +-0; there the product is a zero,
// and up + zero is up exactly unless up is -0.  No concentration is ever -0
// (states start at +0 or above, a sum is -0 only of two -0 operands, and the
// clip keeps its operand), so the result is numpy's bit for bit; NaN and
// infinities reach it through the min and the product.
__device__ __forceinline__ float limited(float up, float a, float b, float s) {
    const float q = copysignf(0.25f, a) + copysignf(0.25f, b);
    const float x = q * min_nan(fabsf(a), fabsf(b));
    return __fmaf_rn(s, x, up);
}

template <int ND>
struct Axes;
template <>
struct Axes<3> {
    static constexpr int n = 3;
    __host__ __device__ static constexpr int ax(int i) { return i; }
};
template <>
struct Axes<2> {  // a 2D grid (nx, ny) is stored as (nx, 1, ny)
    static constexpr int n = 2;
    __host__ __device__ static constexpr int ax(int i) { return i == 0 ? 0 : 2; }
};

// Index arithmetic is 32-bit: a transport grid holds fewer than 2^31
// values per buffer (ns x voxels, checked when the run begins).
struct VoxelPos {
    int p[3];
    int c;
};

// Coordinates of voxel c.
__device__ __forceinline__ VoxelPos voxel_pos(int c, const Grid& g) {
    VoxelPos v;
    v.c = c;
    unsigned t = (unsigned)c;
    v.p[2] = (int)(t % (unsigned)g.nz);
    t /= (unsigned)g.nz;
    v.p[1] = (int)(t % (unsigned)g.ny);
    v.p[0] = (int)(t / (unsigned)g.ny);
    return v;
}

__device__ __forceinline__ int extent(const Grid& g, int a) {
    return a == 0 ? g.nx : (a == 1 ? g.ny : g.nz);
}
__device__ __forceinline__ int stride(const Grid& g, int a) {
    return a == 0 ? g.ny * g.nz : (a == 1 ? g.nz : 1);
}

// p + B * n bytes as one multiply-add (B may be negative).
template <int B>
__device__ __forceinline__ const float* apart(const float* p, int n) {
    const float* q;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(q) : "r"(n), "n"(B), "l"(p));
    return q;
}

// A load of the state, issued where it stands; and the same only where u >= 0,
// or only where it is not, else 0: the far value that the upwind side does not
// need is not read.  Not through the read-only path (.nc): with programmatic
// launch a step's blocks are resident while the step before writes what they
// will read.
__device__ __forceinline__ float ld_early(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_if_up(const float* p, float u) {
    float v;
    asm volatile(
        "{\n.reg .pred q;\nsetp.ge.f32 q, %2, 0f00000000;\nmov.f32 %0, 0f00000000;\n"
        "@q ld.global.f32 %0, [%1];\n}"
        : "=&f"(v)
        : "l"(p), "f"(u));
    return v;
}
__device__ __forceinline__ float ld_if_down(const float* p, float u) {
    float v;
    asm volatile(
        "{\n.reg .pred q;\nsetp.ltu.f32 q, %2, 0f00000000;\nmov.f32 %0, 0f00000000;\n"
        "@q ld.global.f32 %0, [%1];\n}"
        : "=&f"(v)
        : "l"(p), "f"(u));
    return v;
}

// What one transport step needs of solute voxel k that does not change during
// a run: per axis the distances to its neighbours (x, y down to the far low and
// the low, z, w up to the high and the far high) and its low and high face velocity, and its flags where the run
// reads them.  WIDE: from AdrDev::nb instead of AdrDev::near.  BIG: the tables
// may exceed 32-bit places.
template <int ND>
struct VoxelSetup {
    int4 nb[ND];
    float2 fc[ND];
    uint32_t fl;
};

template <int ND, bool BF, bool WIDE, bool BIG = WIDE>
__device__ __forceinline__ VoxelSetup<ND> voxel_setup(const AdrDev& d, const prt_adr_params& p,
                                                      unsigned k) {
    VoxelSetup<ND> s;
#pragma unroll
    for (int i = 0; i < ND; ++i) {
        const size_t at = axis_place<BIG>(i, k, d.nm);
        if constexpr (WIDE) {
            const int4 q = __ldg(d.nb + at);
            s.nb[i] = make_int4((int)k - q.x, (int)k - q.y, q.z - (int)k, q.w - (int)k);
        } else {
            const uint2 q = __ldg(d.near + at);
            s.nb[i] = make_int4(q.x & 0xffffu, q.x >> 16, q.y & 0xffffu, q.y >> 16);
        }
        s.fc[i] = __ldg(d.face + at);
    }
    s.fl = (BF || (p.abio_on && p.surface_only)) ? __ldg(d.cflags + k) : 0u;
    return s;
}

// transport() of one chemical at one voxel (prtlb_3d.py:1182-1208): per axis
// the diffusion and advection are added to the sum in the reference's
// operation order.  The places of closed neighbours are the voxel's own (its
// near one for a far neighbour), so their differences vanish as the
// reference's replaced values do.  BF: the run has biofilm; without it every
// face takes the pore diffusivity.  Every transport kernel calls this, so
// they compute the same function bit for bit.  m2 is read only where the low
// face velocity is >= 0, p2 only where the high one is not.
template <int ND, bool BF>
__device__ __forceinline__ float transport_terms(const float (&m2)[ND], const float (&m1)[ND],
                                                 const float (&p1)[ND], const float (&p2)[ND],
                                                 const float2 (&fc)[ND], uint32_t fl, float Cc,
                                                 const float (&dj)[3]) {
    float out = 0.f;
    float divu = 0.f;
#pragma unroll
    for (int i = 0; i < ND; ++i) {
        const float uL = fc[i].x, uH = fc[i].y;
        float DL = dj[0], DH = dj[0];
        if constexpr (BF) {
            // face diffusivity by the biofilm count of its two voxels (0, 1,
            // 2); selected, not indexed, so the table stays in registers
            const int a = Axes<ND>::ax(i);
            const bool bf = fl & F_BF;
            const float pore = bf ? dj[1] : dj[0], film = bf ? dj[2] : dj[1];
            DL = (fl & f_nbf_lo(a)) ? film : pore;
            DH = (fl & f_nbf_hi(a)) ? film : pore;
        }
        // differences upwards along the axis
        const float below = Cc - m1[i], above = p1[i] - Cc;
        // out += D_hi (C+1 - C) + D_lo (C-1 - C)
        out = out + (DH * above - DL * below);
        const bool rH = uH >= 0.f, rL = uL >= 0.f;
        const float fh = limited(rH ? Cc : p1[i], above, rH ? below : p2[i] - p1[i],
                                 rH ? 1.f : -1.f);
        const float flo = limited(rL ? m1[i] : Cc, below, rL ? m1[i] - m2[i] : above,
                                  rL ? 1.f : -1.f);
        // out -= u_hi f_hi - u_lo f_lo
        out = out - (uH * fh - uL * flo);
        divu = divu + (uH - uL);
    }
    return out + Cc * divu;
}

// The same with the neighbours read from the row whose voxel k is at Ck.
template <int ND, bool BF>
__device__ __forceinline__ float transport_one(const float* __restrict__ Ck,
                                               const VoxelSetup<ND>& s, float Cc,
                                               const float (&dj)[3]) {
    float m2[ND], m1[ND], p1[ND], p2[ND];
#pragma unroll
    for (int i = 0; i < ND; ++i) {
        m1[i] = ld_early(apart<-4>(Ck, s.nb[i].y));
        p1[i] = ld_early(apart<4>(Ck, s.nb[i].z));
        m2[i] = ld_if_up(apart<-4>(Ck, s.nb[i].x), s.fc[i].x);
        p2[i] = ld_if_down(apart<4>(Ck, s.nb[i].w), s.fc[i].y);
    }
    return transport_terms<ND, BF>(m2, m1, p1, p2, s.fc, s.fl, Cc, dj);
}

// Whether r <= 1/2 (c / t) rounded as the reference rounds it is certain without
// the division (t > 0).  r t <= 0.49 c with c not tiny: the two roundings of
// the products and the two of the reference's cap move either side by less
// than 1e-6 of it, and the least product that passes, 4.9e-31, is far above
// the subnormal range.  r <= 0 <= c: the cap is at least +0.  A NaN fails both;
// an infinite r passes only with an infinite c, where the cap is infinite too.
__device__ __forceinline__ bool below_half(float r, float c, float t) {
    return (r * t <= 0.49f * c && c >= 1e-30f) || (r <= 0.f && c >= 0.f);
}

// a / b with the zero numerators of a front that has not arrived (b > 0: +0)
// kept out of the division's path for special operands.
__device__ __forceinline__ float ratio(float a, float b) {
    const bool none = a == 0.f && b > 0.f;
    const float q = (none ? b : a) / b;
    return none ? a : q;
}

// The reaction terms (rate_biotic, rate_abiotic, reaction: prtlb_3d.py:1224-1367)
// at one voxel, plus the reversible-sorption exchange (no reference counterpart).
template <int NS>
__device__ __forceinline__ void reaction(const float (&C)[NS], float surf,
                                         const prt_adr_params& p, float (&dC)[NS]) {
#pragma unroll
    for (int j = 0; j < NS; ++j) dC[j] = 0.f;
    float R = 0.f;
    if (p.biotic_on) {
        R = p.ks_donor_pos ? ratio(p.k * C[0], p.ks_donor + C[0]) : p.k * C[0];
        if (NS > 1) R = R * (p.ks_acceptor_pos
                                 ? ratio(C[NS > 1 ? 1 : 0], p.ks_acceptor + C[NS > 1 ? 1 : 0])
                                 : C[NS > 1 ? 1 : 0]);
        if (NS > 3 && p.coupled) R = (R * C[NS > 3 ? 3 : 0]) / p.c3_init;
        // caps: R <= 1/2 min(C0 / dt, C1 / (alpha dt))
        const bool c1 = NS > 1 && p.alpha_cap;
        if (!(below_half(R, C[0], p.dt) &&
              (!c1 || (p.alpha_dt > 0.f && below_half(R, C[NS > 1 ? 1 : 0], p.alpha_dt))))) {
            float lim = C[0] / p.dt;
            if (c1) lim = np_min(lim, C[NS > 1 ? 1 : 0] / p.alpha_dt);
            R = np_min(R, 0.5f * lim);
        }
    }
    float Ra = 0.f;
    if (p.abio_on) {
        float cj = 0.f;
#pragma unroll
        for (int j = 0; j < NS; ++j)
            if (j == p.j_ab) cj = C[j];
        Ra = p.surface_only ? (p.ka * cj) * surf : p.ka * cj;
        if (!below_half(Ra, cj, p.dt)) Ra = np_min(Ra, (0.5f * cj) / p.dt);
    }
    if (p.biotic_on) {
        dC[0] = -R;
        if (NS > 1) dC[NS > 1 ? 1 : 0] = p.neg_alpha * R;
        if (NS > 2) dC[NS > 2 ? 2 : 0] = p.prod_coef * R;
        if (NS > 3) dC[NS > 3 ? 3 : 0] = p.yield_ * R - p.kd * C[NS > 3 ? 3 : 0];
    } else {
        // R is the float32 scalar 0: -R, -alpha R, coef R are zeros, biomass 0
    }
    if (p.abio_on) {
#pragma unroll
        for (int j = 0; j < NS; ++j) {
            if (j == p.j_ab) dC[j] = dC[j] - Ra;
        }
#pragma unroll
        for (int j = 0; j < NS; ++j) {
            if (j == p.j_mk && p.j_mk != p.j_ab) dC[j] = dC[j] + Ra;
        }
    }
    if (p.sorp_on) {
        float c = 0.f, s = 0.f;
#pragma unroll
        for (int j = 0; j < NS; ++j) {
            if (j == p.j_c) c = C[j];
            if (j == p.j_s) s = C[j];
        }
        float r = p.k_sorp * (c - s * p.inv_kd_sorp);
        if (!(below_half(r, c, p.dt) && below_half(-r, s, p.dt))) {
            r = np_min(r, (0.5f * c) / p.dt);
            r = np_max(r, -((0.5f * s) / p.dt));
        }
#pragma unroll
        for (int j = 0; j < NS; ++j) {
            if (j == p.j_c) dC[j] = dC[j] - r;
            if (j == p.j_s) dC[j] = dC[j] + r;
        }
    }
}

// The rest of step() at one solute voxel (prtlb_3d.py:1392-1413) once the
// transport terms T of the moving chemicals are known: the reaction terms
// (with the surface weight of a surface-only abiotic reaction), forward
// Euler and the clip at zero.  C holds the voxel's values after the inlet
// pin.
template <int ND, int NS>
__device__ __forceinline__ void adr_update(const float (&C)[NS], const float (&T)[NS], uint32_t fl,
                                           const prt_adr_params& p, float (&cn)[NS]) {
    float surf = 0.f;
    if (p.abio_on && p.surface_only) {
        float nface = 0.f;
#pragma unroll
        for (int i = 0; i < ND; ++i) {
            const int a = Axes<ND>::ax(i);
            nface = nface + ((fl & f_open_lo(a)) ? 0.f : 1.f);
            nface = nface + ((fl & f_open_hi(a)) ? 0.f : 1.f);
        }
        surf = nface / (float)(2 * ND);
    }
    float dC[NS];
    reaction<NS>(C, surf, p, dC);
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        const bool mv = (p.moving_mask >> j) & 1u;
        const float rhs = mv ? (T[j] + dC[j]) : dC[j];
        const float v = C[j] + p.dt * rhs;
        cn[j] = np_max(v, 0.f);
    }
}

// One transport step of solute voxel k (compacted C order) at step n: reads the
// state after step n-1 from buf[(n-1)&1], writes the state after step n to
// buf[n&1] and, when n is a snapshot step, to its ladder slot.  On the inlet
// plane the pinned feed replaces a value before transport (step(),
// prtlb_3d.py:1392-1400), so that is what the next step is given; the value
// itself goes behind the row.
template <int ND, int NS, bool BF>
__device__ __forceinline__ void adr_voxel_step(const AdrDev& d, const prt_adr_params& p,
                                               long long n, unsigned k,
                                               const VoxelSetup<ND>& s) {
    const unsigned ms = d.ms;
    const float* __restrict__ Ck = d.buf[(n - 1) & 1] + k;
    float* __restrict__ Cout = d.buf[n & 1];
    float C[NS];
#pragma unroll
    for (int j = 0; j < NS; ++j) C[j] = Ck[j * ms];
    float T[NS];
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        T[j] = 0.f;
        if ((p.moving_mask >> j) & 1u) {
            const float dj[3] = {p.dface[j][0], p.dface[j][1], p.dface[j][2]};
            T[j] = transport_one<ND, BF>(Ck + j * ms, s, C[j], dj);
        }
    }
    float cn[NS];
    adr_update<ND, NS>(C, T, s.fl, p, cn);
    const int slot = d.slot_of_step[n];
    if (slot >= 0) {
        float* __restrict__ lad = d.ladder + (long long)slot * NS * d.nm;
#pragma unroll
        for (int j = 0; j < NS; ++j) lad[j * d.nm + k] = cn[j];
    }
    if (k < (unsigned)d.n0) {
#pragma unroll
        for (int j = 0; j < NS; ++j) {
            Cout[j * ms + (unsigned)d.nm + k] = cn[j];
            if ((p.pinned_mask >> j) & 1u) cn[j] = p.feed[j];
        }
    }
#pragma unroll
    for (int j = 0; j < NS; ++j) Cout[j * ms + k] = cn[j];
}

// The check of the time loop at step `end` (prtlb_3d.py:1499-1543), in
// float64 like the reference's arrays of Python floats: running scale,
// per-check change, geometric-tail remainder `rest`, the progress record,
// and the stop decision.
__device__ __forceinline__ double npd_max(double a, double b) { return (a >= b || a != a) ? a : b; }

__device__ inline void adr_check(AdrCtrl* ctrl, const float* __restrict__ means, long long end,
                                 ProgressRec* log, int log_cap) {
    const int ns = ctrl->ns;
    double cur[PRT_MAX_SPECIES], stepc[PRT_MAX_SPECIES];
    double change = 0.0, rest = 0.0;
    bool first = true;
    for (int j = 0; j < ns; ++j) {
        cur[j] = (double)means[j];
        ctrl->scale[j] = npd_max(ctrl->scale[j], fabs(cur[j]));
        stepc[j] = fabs(cur[j] - ctrl->prev[j]) / ctrl->scale[j];
        const double r = ctrl->prev_change[j] > 0 ? stepc[j] / ctrl->prev_change[j] : 0.0;
        double rj = (r < 1.0) ? stepc[j] * r / npd_max(1.0 - r, 1e-12) : INFINITY;
        if (!isfinite(rj)) rj = INFINITY;
        if (first) {
            change = stepc[j];
            rest = rj;
            first = false;
        } else {
            change = (change != change) ? change : ((stepc[j] != stepc[j]) ? stepc[j] : fmax(change, stepc[j]));
            rest = fmax(rest, rj);
        }
    }
    if (ctrl->nlog < log_cap) {
        ProgressRec& rec = log[ctrl->nlog];
        rec.n = end;
        rec.mean0 = cur[0];
        rec.value = isfinite(rest) ? rest : change;
    }
    ctrl->nlog += 1;
    ctrl->checks += 1;
    ctrl->last_rest = rest;
    if (ctrl->until_conv && end >= 10ll * ctrl->check && rest <= ctrl->tol) {
        ctrl->converged = 1;
        ctrl->done = 1;
    } else {
        for (int j = 0; j < ns; ++j) {
            ctrl->prev[j] = cur[j];
            ctrl->prev_change[j] = stepc[j];
        }
    }
}

// Sum of the leaf [start, start + len) (at most 128 values) of numpy's float32
// pairwise tree over the solute values of a row, by one warp: under 8 values
// sequentially from 0, otherwise eight interleaved accumulators
// ((r0+r1)+(r2+r3))+((r4+r5)+(r6+r7)) and a tail.  The lanes load the values
// into `sh` (through L2: other blocks of the launch may have written them),
// lanes 0-7 run the accumulators and every lane then combines them and adds
// the tail.  The result is the same in every lane.
__device__ __forceinline__ float warp_leaf_sum(const float* __restrict__ row, unsigned n0,
                                               unsigned nm, int start, int len, float* sh) {
    const int lane = threadIdx.x & 31;
    for (int i = lane; i < len; i += 32)
        sh[i] = __ldcg(row + solute_place((unsigned)(start + i), n0, nm));
    __syncwarp();
    float res;
    if (len < 8) {
        res = 0.f;
        for (int i = 0; i < len; ++i) res = res + sh[i];
    } else {
        const int body = len - (len % 8);
        float r = 0.f;
        if (lane < 8) {
            r = sh[lane];
            for (int i = 8 + lane; i < body; i += 8) r = r + sh[i];
        }
        float q[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) q[k] = __shfl_sync(0xffffffffu, r, k);
        res = ((q[0] + q[1]) + (q[2] + q[3])) + ((q[4] + q[5]) + (q[6] + q[7]));
        for (int i = body; i < len; ++i) res = res + sh[i];
    }
    __syncwarp();  // sh is reused by the warp's next leaf
    return res;
}

// The inner levels of the tree for ns chemicals at once (the whole block takes
// part; chemical j's node values at v + j * (nleaf + ninner)), then mean = (0
// + sum) / nm in float32 as ndarray.mean() does.  The leaves are read through
// L2 (other blocks may have written them).
__device__ inline void tree_means(const PairTree& t, long long nm, int ns, float* v,
                                  float* means) {
    const int nodes = t.nleaf + t.ninner;
    for (int h = 0; h < t.nlevel; ++h) {
        const int lo = t.level_off[h], width = t.level_off[h + 1] - lo;
        for (int q = threadIdx.x; q < width * ns; q += blockDim.x) {
            const int j = q / width, i = lo + q - j * width;
            float* w = v + (long long)j * nodes;
            w[t.nleaf + i] = __ldcg(w + t.inner_l[i]) + __ldcg(w + t.inner_r[i]);
        }
        __threadfence_block();
        __syncthreads();
    }
    if ((int)threadIdx.x < ns) {
        const float sum = t.root >= 0 ? 0.f + __ldcg(v + (long long)threadIdx.x * nodes + t.root) : 0.f;
        means[threadIdx.x] = sum / (float)nm;  // 0/0 -> NaN for an empty pore space, as numpy
    }
}

}  // namespace prt

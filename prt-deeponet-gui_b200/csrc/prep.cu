// prep.cu -- the walk from the inlet face through the pore space, for the
// geometry preparation done once per rock before its solves.
//
// What the reference does:
//   keep_inlet_connected (prtlb_3d.py:530-563): label the 6- (4-) connected
//     pore components with scipy, keep those touching the x = 0 face;
//   geodesic_steps (prt_core/conventions.py:72-115): a breadth-first walk
//     from the face, one Python queue step per voxel;
//   geodesic (build_practice_dataset.py:53-73): repeated relaxation sweeps
//     of d = min(d, neighbour + 1) until nothing changes.
// All three are one computation: the fewest face-neighbour steps from a pore
// voxel of the inlet face to every pore voxel (the reached set is exactly
// the union of the components touching the face).
//
// The same walk from any plane x_a = p (prt_walk_from_plane) serves the
// percolation checks of the dataset builders (build_dataset_3d.py:281-286,
// build_dataset_2d.py:290-294, build_geometry_3d.py:201-221): a component
// touches planes p and q exactly when the walk from p reaches plane q.
//
// Here the walk is level-synchronous and pulls.  A grid whose voxels, as bits,
// fit in the shared memory of one thread-block cluster (up to about 8.4
// million voxels in whole words of 32 along z) walks inside one kernel: the
// pore not reached yet and the last levels are bit masks, and a level ends
// with the cluster barrier: 2.4 us a level at 128^3, bound by the barrier
// behind the scattered stores of the steps, against 9 us for a launch that
// reads every voxel's step number (the whole call 2.58 -> 1.05 ms).
// A larger grid takes a launch per level, which visits every voxel
// once; a pore voxel not reached yet takes L + 1 if a face neighbour holds
// L.  There a voxel is written only by its own thread, and during launch L the
// values change only from "unreached" to L + 1, neither of which is L, so
// the result does not depend on the order threads run in.  The host enqueues
// a chunk of levels and stops after the first chunk whose last level reached
// nothing new (no level can reach anything after one that reached nothing).
#include <vector>

#include "cluster.cuh"
#include "runtime_internal.h"

namespace prt {

namespace {

constexpr int kWalkThreads = 256;
constexpr int kUnreached = 0x7fffffff;
constexpr int kLevelsPerChunk = 32;

struct WalkGrid {
    Grid g;
    FastDiv dz, dy;
    int axis;   // storage axis of the seed plane (0 x, 1 y, 2 z)
    int plane;  // its coordinate along that axis
};

__device__ __forceinline__ void coords(unsigned c, const WalkGrid& w, int& x, int& y, int& z) {
    const unsigned q = fast_div(c, w.dz);
    z = (int)(c - q * w.dz.d);
    const unsigned xx = fast_div(q, w.dy);
    y = (int)(q - xx * w.dy.d);
    x = (int)xx;
}

// steps = 0 on the pore of the seed plane, unreached on the other pore,
// -1 elsewhere; counts[0] += pore voxels.
__global__ void __launch_bounds__(kWalkThreads)
    walk_init_kernel(const uint8_t* __restrict__ mat, WalkGrid w, int code, int* __restrict__ steps,
                     unsigned long long* __restrict__ counts) {
    const unsigned c = blockIdx.x * kWalkThreads + threadIdx.x;
    int pore = 0;
    if (c < (unsigned)w.g.n) {
        pore = mat[c] == code;
        int x, y, z;
        coords(c, w, x, y, z);
        const int along = w.axis == 0 ? x : (w.axis == 1 ? y : z);
        steps[c] = pore ? (along == w.plane ? 0 : kUnreached) : -1;
    }
    const int nb = __syncthreads_count(pore);
    if (threadIdx.x == 0 && nb) atomicAdd(counts, (unsigned long long)nb);
}

// One level: unreached pore voxels next to a voxel at `level` take level + 1;
// *flag = 1 when any did.
__global__ void __launch_bounds__(kWalkThreads)
    walk_level_kernel(int* __restrict__ steps, WalkGrid w, int level, int* __restrict__ flag) {
    const unsigned c = blockIdx.x * kWalkThreads + threadIdx.x;
    bool reached = false;
    if (c < (unsigned)w.g.n && steps[c] == kUnreached) {
        int x, y, z;
        coords(c, w, x, y, z);
        const int sz = 1, sy = w.g.nz, sx = w.g.ny * w.g.nz;
        bool hit = false;
        if (z > 0) hit |= steps[c - sz] == level;
        if (z < w.g.nz - 1) hit |= steps[c + sz] == level;
        if (y > 0) hit |= steps[c - sy] == level;
        if (y < w.g.ny - 1) hit |= steps[c + sy] == level;
        if (x > 0) hit |= steps[c - sx] == level;
        if (x < w.g.nx - 1) hit |= steps[c + sx] == level;
        if (hit) {
            steps[c] = level + 1;
            reached = true;
        }
    }
    if (__syncthreads_or(reached) && threadIdx.x == 0) *flag = 1;
}

// Unreached pore -> -2; counts[1] += reached pore voxels.
__global__ void __launch_bounds__(kWalkThreads)
    walk_final_kernel(int* __restrict__ steps, long long n, unsigned long long* __restrict__ counts) {
    const unsigned c = blockIdx.x * kWalkThreads + threadIdx.x;
    int reached = 0;
    if (c < (unsigned)n) {
        const int s = steps[c];
        if (s == kUnreached) steps[c] = -2;
        reached = s >= 0 && s != kUnreached;
    }
    const int nb = __syncthreads_count(reached);
    if (threadIdx.x == 0 && nb) atomicAdd(counts + 1, (unsigned long long)nb);
}

// ---------------------------------------------------------------------------
// the walk on bit masks inside one cluster
// ---------------------------------------------------------------------------
// A row is a line of nz voxels along z, in wpr words of 32.  A walk's front is
// much of a plane at a time, so the rows are dealt out to the 16 blocks
// diagonally, (x + y) mod 16 (by the row number when ny < 16), and a front
// across any axis is spread over all of them: with whole planes to a block a
// level took 6.1 us at 128^3.
struct BitWalk {
    int nx, ny, nz, wpr;
    int nyc;   // rows of one x in a block (diagonal dealing), 0: by row number
    int rows;  // rows of a block
    FastDiv by_word, by_nyc, by_ny;
};
constexpr int kBitThreads = 512;
constexpr int kBitWords = 16384;  // words of a block: three masks and a queue in 224 KB
constexpr int kLevelsPerVote = 16;

inline BitWalk make_bit_walk(const Grid& g) {
    BitWalk b;
    b.nx = g.nx;
    b.ny = g.ny;
    b.nz = g.nz;
    b.wpr = (g.nz + 31) / 32;
    b.nyc = g.ny >= kClusterMax ? (g.ny + kClusterMax - 1) / kClusterMax : 0;
    const long long rows = b.nyc ? (long long)g.nx * b.nyc
                                 : ((long long)g.nx * g.ny + kClusterMax - 1) / kClusterMax;
    b.rows = (int)std::min<long long>(rows, kBitWords + 1);  // more is refused below
    b.by_word = make_fastdiv((unsigned)b.wpr);
    b.by_nyc = make_fastdiv((unsigned)std::max(b.nyc, 1));
    b.by_ny = make_fastdiv((unsigned)g.ny);
    return b;
}

// Row (x, y): its block and its number there; and back.
__device__ __forceinline__ void row_place(const BitWalk& b, int x, int y, int& blk, int& lr) {
    const int row = x * b.ny + y;
    blk = (b.nyc ? x + y : row) & (kClusterMax - 1);
    lr = b.nyc ? x * b.nyc + y / kClusterMax : row / kClusterMax;
}
__device__ __forceinline__ void place_row(const BitWalk& b, int blk, int lr, int& x, int& y) {
    if (b.nyc) {
        x = (int)fast_div((unsigned)lr, b.by_nyc);
        y = (lr - x * b.nyc) * kClusterMax + ((blk - x) & (kClusterMax - 1));
    } else {
        const int row = lr * kClusterMax + blk;
        x = (int)fast_div((unsigned)row, b.by_ny);
        y = row - x * b.ny;
    }
}

// One warp per word: steps = 0 on the pore of the seed plane, -2 on the other
// pore, -1 elsewhere; seed and rest (zeroed before): the bits of the first
// two, block by block; counts[0] += pore voxels.
__global__ void __launch_bounds__(kWalkThreads)
    bit_init_kernel(const uint8_t* __restrict__ mat, WalkGrid w, BitWalk b, int code,
                    int* __restrict__ steps, unsigned* __restrict__ seed,
                    unsigned* __restrict__ rest, unsigned long long* __restrict__ counts) {
    const unsigned word = blockIdx.x * (kWalkThreads / 32) + (threadIdx.x >> 5);
    int pore = 0;
    if (word < (unsigned)(b.nx * b.ny * b.wpr)) {  // whole warps
        const unsigned row = fast_div(word, b.by_word);
        const int q = (int)(word - row * b.wpr), z = q * 32 + (threadIdx.x & 31);
        const int x = (int)fast_div(row, b.by_ny), y = (int)row - x * b.ny;
        bool start = false;
        if (z < b.nz) {
            const long long c = (long long)row * b.nz + z;
            pore = mat[c] == code;
            start = pore && (w.axis == 0 ? x : (w.axis == 1 ? y : z)) == w.plane;
            steps[c] = pore ? (start ? 0 : -2) : -1;
        }
        const unsigned s = __ballot_sync(0xffffffffu, start);
        const unsigned r = __ballot_sync(0xffffffffu, pore && !start);
        if ((threadIdx.x & 31) == 0) {
            int blk, lr;
            row_place(b, x, y, blk, lr);
            const long long at = ((long long)blk * b.rows + lr) * b.wpr + q;
            seed[at] = s;
            rest[at] = r;
        }
    }
    const int n = __syncthreads_count(pore);
    if (threadIdx.x == 0 && n) atomicAdd(counts, (unsigned long long)n);
}

// The whole walk from the masks; steps of the reached voxels, counts[1] +=
// reached pore voxels.  A level: every thread looks through its words for bits
// that the level before sent (few have any), what of them is still open is
// the level's pore and its words are queued; then the queued words' bits are
// sent on, to their own word shifted by one voxel, and to the words of the
// neighbouring rows in their blocks.
__global__ void __launch_bounds__(kBitThreads, 1)
    bit_walk_kernel(BitWalk b, const unsigned* __restrict__ seed, const unsigned* __restrict__ rest,
                    int* __restrict__ steps, unsigned long long* __restrict__ counts) {
    extern __shared__ unsigned masks[];  // open, sent to even and to odd levels, queue
    __shared__ int votes[kClusterMax];
    __shared__ int queued[2];
    const int t = threadIdx.x;
    const int rank = (int)cluster_rank();
    const int mine = b.rows * b.wpr;
    unsigned* open = masks;
    unsigned* sent[2] = {masks + mine, masks + 2 * mine};
    unsigned short* queue = reinterpret_cast<unsigned short*>(masks + 3 * mine);
    const uint32_t sent_at[2] = {shared_address(sent[0]), shared_address(sent[1])};
    for (int i = t; i < mine; i += kBitThreads) {
        const long long at = (long long)rank * mine + i;
        const unsigned s = seed[at];
        open[i] = rest[at] | s;
        sent[0][i] = s;
        sent[1][i] = 0u;
    }
    if (t < 2) queued[t] = 0;
    unsigned long long reached = 0;
    cluster_sync();
    for (int lv = 0;; ++lv) {
        unsigned* now = sent[lv & 1];
        unsigned* next = sent[(lv & 1) ^ 1];
        int* n = queued + (lv & 1);
        for (int i = t; i < mine; i += kBitThreads) {
            if (now[i] == 0u) continue;
            const unsigned o = open[i], f = now[i] & o;
            now[i] = f;
            if (f == 0u) continue;
            open[i] = o ^ f;
            reached += __popc(f);
            queue[atomicAdd(n, 1)] = (unsigned short)i;
        }
        __syncthreads();
        const int nq = *n;
        if (t == 0) queued[(lv & 1) ^ 1] = 0;
        for (int e = t; e < nq; e += kBitThreads) {
            const int i = queue[e];
            const unsigned f = now[i];
            now[i] = 0u;
            const int lr = (int)fast_div((unsigned)i, b.by_word), q = i - lr * b.wpr;
            int x, y;
            place_row(b, rank, lr, x, y);
            auto send = [&](int xn, int yn) {  // f to the same word of row (xn, yn)
                int blk, r;
                row_place(b, xn, yn, blk, r);
                const uint32_t a =
                    in_block(sent_at[(lv & 1) ^ 1] + (r * b.wpr + q) * 4, (unsigned)blk);
                asm volatile("red.relaxed.cluster.shared::cluster.or.b32 [%0], %1;" ::"r"(a), "r"(f)
                             : "memory");
            };
            if (y > 0) send(x, y - 1);
            if (y < b.ny - 1) send(x, y + 1);
            if (x > 0) send(x - 1, y);
            if (x < b.nx - 1) send(x + 1, y);
            atomicOr(next + i, (f << 1) | (f >> 1));
            if (q > 0 && (f & 1u)) atomicOr(next + (i - 1), 1u << 31);
            if (q < b.wpr - 1 && (f >> 31)) atomicOr(next + (i + 1), 1u);
            int* out = steps + ((long long)(x * b.ny + y) * b.nz + q * 32);
            for (unsigned m = f; m; m &= m - 1) out[__ffs(m) - 1] = lv;
        }
        // no level can reach anything after one that reached nothing
        const bool vote = lv % kLevelsPerVote == kLevelsPerVote - 1;
        if (vote && t == 0) {
            const uint32_t a = in_block(shared_address(votes + rank), 0);
            asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(a), "r"(nq) : "memory");
        }
        cluster_sync();
        if (vote) {
            int v = 0;
            if (t < kClusterMax) ld_cluster(in_block(shared_address(votes + t), 0), v);
            if (!__syncthreads_or(v)) break;
        }
    }
    for (int o = 16; o > 0; o >>= 1) reached += __shfl_down_sync(0xffffffffu, reached, o);
    if ((t & 31) == 0 && reached) atomicAdd(counts + 1, reached);
    cluster_sync();  // no block leaves while another may read its votes or words
}

// label_materials (build_geometry_3d.py:224-239): pore 2, solid with a
// pore face neighbour 1, other solid 0; positions beyond the grid's faces
// count as solid (no wrap).  One thread per voxel, six neighbour reads
// through the cache; 2D grids are (nx, 1, ny).
__global__ void label_materials_kernel(const uint8_t* __restrict__ solid, WalkGrid w,
                                       uint8_t* __restrict__ out) {
    const long long n = w.g.n;
    const unsigned c = blockIdx.x * kWalkThreads + threadIdx.x;
    if (c >= (unsigned)n) return;
    if (!solid[c]) {
        out[c] = 2;
        return;
    }
    int x, y, z;
    coords(c, w, x, y, z);
    const Grid& g = w.g;
    const int sy = g.nz, sx = g.ny * g.nz;
    bool touch = false;
    if (x > 0) touch |= !solid[c - sx];
    if (x < g.nx - 1) touch |= !solid[c + sx];
    if (y > 0) touch |= !solid[c - sy];
    if (y < g.ny - 1) touch |= !solid[c + sy];
    if (z > 0) touch |= !solid[c - 1];
    if (z < g.nz - 1) touch |= !solid[c + 1];
    out[c] = touch ? 1 : 0;
}

}  // namespace

}  // namespace prt

using namespace prt;

extern "C" int prt_label_materials(prt_ctx* ctx, const uint8_t* solid, int32_t nd,
                                   const int32_t* dims, uint8_t* mat_out) {
    if (!ctx || !solid || !dims || !mat_out) return fail(ctx, PRT_E_INVALID, "null argument");
    if (nd != 2 && nd != 3) return fail(ctx, PRT_E_INVALID, "nd must be 2 or 3");
    for (int i = 0; i < nd; ++i)
        if (dims[i] <= 0) return fail(ctx, PRT_E_INVALID, "grid dimensions must be positive");
    const Grid g = make_grid(nd, dims);
    if (g.n >= (1ll << 31))
        return fail(ctx, PRT_E_INVALID, "grids of 2^31 voxels or more are not supported");
    CK(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    PrepState& P = ctx->prep;
    CK(P.mat.ensure((size_t)g.n * 2));  // the solid grid, then the codes
    P.staged_mat = -1;
    uint8_t* d_solid = P.mat.as<uint8_t>();
    uint8_t* d_out = d_solid + g.n;
    CK(copy_in(ctx, d_solid, solid, (size_t)g.n));
    WalkGrid w;
    w.g = g;
    w.dz = make_fastdiv((unsigned)g.nz);
    w.dy = make_fastdiv((unsigned)g.ny);
    w.axis = 0;
    w.plane = 0;
    const unsigned nb = (unsigned)((g.n + kWalkThreads - 1) / kWalkThreads);
    label_materials_kernel<<<nb, kWalkThreads, 0, s>>>(d_solid, w, d_out);
    CK(cudaGetLastError());
    ctx->launches += 1;
    CK(copy_out(ctx, mat_out, d_out, (size_t)g.n));
    return PRT_OK;
}

// PRT_CLUSTER=0: a launch per level whatever the size (the same steps).
static bool bit_walk_enabled() {
    const char* v = std::getenv("PRT_CLUSTER");
    return !(v && v[0] == '0');
}

extern "C" int prt_walk_from_plane(prt_ctx* ctx, const uint8_t* mat, int32_t nd,
                                   const int32_t* dims, int32_t pore_code, int32_t axis,
                                   int32_t plane, int32_t* steps_out, int64_t* n_reached,
                                   int64_t* n_pore) {
    if (!ctx || !mat || !dims || !steps_out) return fail(ctx, PRT_E_INVALID, "null argument");
    if (nd != 2 && nd != 3) return fail(ctx, PRT_E_INVALID, "nd must be 2 or 3");
    for (int i = 0; i < nd; ++i)
        if (dims[i] <= 0) return fail(ctx, PRT_E_INVALID, "grid dimensions must be positive");
    if (axis < 0 || axis >= nd)
        return fail(ctx, PRT_E_INVALID, "the walk's axis must be one of the grid's axes");
    if (plane < 0 || plane >= dims[axis])
        return fail(ctx, PRT_E_INVALID, "the seed plane lies outside the grid");
    const Grid g = make_grid(nd, dims);
    // levels stay below the unreached marker: at most one per pore voxel,
    // plus one chunk
    if (g.n >= (1ll << 31) - 2 * kLevelsPerChunk)
        return fail(ctx, PRT_E_INVALID, "grids of 2^31 voxels or more are not supported");
    CK(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    PrepState& P = ctx->prep;
    CK(P.mat.ensure((size_t)g.n));
    CK(P.steps.ensure((size_t)g.n * 4));
    CK(P.flags.ensure(kLevelsPerChunk * sizeof(int)));
    CK(P.counts.ensure(2 * sizeof(unsigned long long)));
    CK(copy_in(ctx, P.mat.p, mat, (size_t)g.n));
    P.staged_mat = -1;  // the buffer now holds the walk's grid
    CK(cudaMemsetAsync(P.counts.p, 0, 2 * sizeof(unsigned long long), s));
    WalkGrid w;
    w.g = g;
    w.dz = make_fastdiv((unsigned)g.nz);
    w.dy = make_fastdiv((unsigned)g.ny);
    w.axis = nd == 3 ? axis : (axis == 0 ? 0 : 2);  // 2D (nx, ny) is (nx, 1, ny)
    w.plane = plane;
    const unsigned nb = (unsigned)((g.n + kWalkThreads - 1) / kWalkThreads);
    int* steps = P.steps.as<int>();
    int* flags = P.flags.as<int>();
    unsigned long long* counts = P.counts.as<unsigned long long>();
    bool walked = false;
    const BitWalk b = make_bit_walk(g);
    if (bit_walk_enabled() && (long long)b.rows * b.wpr <= kBitWords) {
        const size_t words = (size_t)kClusterMax * b.rows * b.wpr;
        CK(P.bits.ensure(words * 2 * sizeof(unsigned)));
        CK(cudaMemsetAsync(P.bits.p, 0, words * 2 * sizeof(unsigned), s));
        unsigned* seed = P.bits.as<unsigned>();
        unsigned* rest = seed + words;
        const unsigned used = (unsigned)(b.nx * b.ny * b.wpr);
        bit_init_kernel<<<(used + kWalkThreads / 32 - 1) / (kWalkThreads / 32), kWalkThreads, 0,
                          s>>>(P.mat.as<uint8_t>(), w, b, pore_code, steps, seed, rest, counts);
        CK(cudaGetLastError());
        constexpr size_t word = 3 * sizeof(unsigned) + sizeof(unsigned short);
        const cudaError_t e = launch_cluster(bit_walk_kernel, kClusterMax, kBitThreads,
                                             (size_t)b.rows * b.wpr * word, kBitWords * word, s, b,
                                             (const unsigned*)seed, (const unsigned*)rest, steps,
                                             counts);
        walked = e != cudaErrorNotSupported;
        if (walked) CK(e);
        ctx->launches += 1 + walked;
        if (!walked) CK(cudaMemsetAsync(P.counts.p, 0, 2 * sizeof(unsigned long long), s));
    }
    if (!walked) {
        walk_init_kernel<<<nb, kWalkThreads, 0, s>>>(P.mat.as<uint8_t>(), w, pore_code, steps, counts);
        CK(cudaGetLastError());
        ctx->launches += 1;
        // at most one level per pore voxel, so the loop ends; in practice after
        // the longest shortest path
        std::vector<int> h(kLevelsPerChunk);
        for (long long base = 0; base <= g.n; base += kLevelsPerChunk) {
            CK(cudaMemsetAsync(flags, 0, kLevelsPerChunk * sizeof(int), s));
            for (int i = 0; i < kLevelsPerChunk; ++i)
                walk_level_kernel<<<nb, kWalkThreads, 0, s>>>(steps, w, (int)(base + i), flags + i);
            CK(cudaGetLastError());
            ctx->launches += kLevelsPerChunk;
            CK(cudaMemcpyAsync(h.data(), flags, kLevelsPerChunk * sizeof(int), cudaMemcpyDeviceToHost, s));
            CK(cudaStreamSynchronize(s));
            if (h[kLevelsPerChunk - 1] == 0) break;
        }
        walk_final_kernel<<<nb, kWalkThreads, 0, s>>>(steps, g.n, counts);
        CK(cudaGetLastError());
        ctx->launches += 1;
    }
    unsigned long long hc[2];
    CK(cudaMemcpyAsync(hc, counts, sizeof(hc), cudaMemcpyDeviceToHost, s));
    CK(copy_out(ctx, steps_out, steps, (size_t)g.n * 4));  // waits for both
    if (n_pore) *n_pore = (int64_t)hc[0];
    if (n_reached) *n_reached = (int64_t)hc[1];
    return PRT_OK;
}

extern "C" int prt_inlet_walk(prt_ctx* ctx, const uint8_t* mat, int32_t nd, const int32_t* dims,
                              int32_t pore_code, int32_t inlet_axis, int32_t* steps_out,
                              int64_t* n_reached, int64_t* n_pore) {
    return prt_walk_from_plane(ctx, mat, nd, dims, pore_code, inlet_axis, 0, steps_out, n_reached,
                               n_pore);
}

// The inner FP32 PCG of a small board as one cooperative kernel.
//
// A board of up to some 220 thousand nodes is bound by latency, not by bytes:
// on a 128 x 128 x 8 board (150 k nodes) an iteration of the graph-captured
// kernels takes 31 us with the two-level preconditioner and 15 us with Jacobi,
// of which moving its vectors would be one.  The rest is kernel boundaries,
// the z-march of the operator's few tiles, and after each reduction a ticket,
// a last block and a scalar read back by the next kernel.  Here one block per
// SM keeps its share of the nodes, their operator rows and vectors in
// registers for many iterations (with two nodes a thread, above 113 thousand
// padded nodes, some 100 bytes a thread of them spill to local memory).
// Measured (12-slab boards of 64 .. 118 cells a side, 55 .. 220 thousand nodes):
// 13.0 .. 16.0 us an iteration against 30 .. 31 with the two-level
// preconditioner, 6.7 .. 8.7 against 15 .. 19 with Jacobi; 128 x 128 x 8: 16.9
// against 32, and 8.3 against 18.
// What is left is the round trips: about 1.5 us for each of the two exchanges
// and 1 us for each of the words of the direction, the patch sums and c.
//
// One launch has the whole device, so solves of several host threads follow one
// another where the graph-captured kernels overlap.  Milliseconds per solve with
// 1 / 2 / 3 / 4 / 8 threads, this kernel and the graph-captured ones:
//   64 x 64 x 8 two-level     19.6 17.1 17.2 16.7 17.3     46.5 24.3 16.9 14.2 10.7
//   120 x 120 x 8 two-level   49.7 47.8 45.8 43.9 45.0     93.5 55.3 42.9 36.0 33.0
//   96 x 80 x 8 Jacobi        61.3 60.7 59.9 57.9 59.5     135  81.2 55.2 45.5 33.1
//   24 x 24 x 8 two-level      4.4  3.5  2.6  2.6  2.3     12.5 10.2  7.2  5.9  4.2
// Which kernels a solve takes does not depend on what else runs, so that its bits
// do not; a program with four or more such solves at a time sets a launch plan
// (tb_set_apply_plan), or hands its boards to a batch engine.
//
// What the blocks tell each other travels in 64-bit words that carry their own
// tag (the iteration) beside the FP32 value, so that no fence or flag has to
// follow the data and a reader needs one round trip: the direction (each
// block stages its nodes' neighbourhood in shared memory), the patch sums and
// the coarse solution, and, twice an iteration, the partial sums of a
// reduction, which every block reads from all the others and merges in the
// same order (so the scalars need no broadcast).  A word is written again only
// after an exchange that its readers had joined after reading it: the
// direction, patch sums and coarse solution of the next iteration follow the
// exchange of p.q or of r.z, and the two exchanges alternate.
//
// Operator.  A node's row of A is 27 coefficients, built in FP64 from the
// element conductivities and rounded once (resident_rows).  The action is
// taken on differences, along z first:
//     y_i = R_i p_i + sum_d s_d (u_d - p_i)
//                   + sum_d a_d+ (u_d+ - u_d) + a_d- (u_d- - u_d),
// d over the nine columns around the node, u_d, u_d+, u_d- the free part of p
// on the node's plane and the planes above and below, a_d+, a_d- the couplings
// to those planes and s_d = a_d- + a_d0 + a_d+.  A thin slab's couplings through
// it are some fifty times those along it and cancel in s_d, so that they act
// on z differences alone, as the Haar form of the tile kernels has it; on plain
// differences p_j - p_i their parts in a_d0 and a_d+ would meet only after
// rounding.  A fixed row is the identity.
//
// Two-level step.  A block sums its nodes' residuals by patch and posts the
// sums (`part`: one slot per block that touches a patch).  The coarse inverse
// is cut into tiles, one per block, that stay in shared memory; a block adds
// the slots of its tile's columns to R and posts its part of c = Minv R for the
// tile's rows, and each block adds up the parts of the patches it touches.  (A
// tile per block, not a row of tiles: a block then reads some 500 words of R
// instead of 6,000, which took 7 us an iteration.)
//
// Every wait is bounded: a block whose wait runs out sets the error word, which
// the host reads after every launch, and leaves; the others, which then miss its
// next words, do the same.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "tb_coarse.cuh"
#include "tb_reduce.cuh"
#include "tb_types.h"
#include "tb_vec.cuh"

namespace tb {

constexpr int kResThreads = 768;   // 80 registers a thread: most of two nodes' rows of 27 coefficients
constexpr int kResNodes = 2;       // nodes per thread at most
constexpr int kResRow = 27;        // s_d (8 columns), a_d- and a_d+ (9 each), and the Robin term
constexpr int kResMaxBlocks = 160; // blocks whose posts one exchange reads (five warps)
constexpr int kResTileCols = 16;   // tiles of the coarse inverse side by side at most
constexpr int kResTouched = 1024;  // patches a block touches at most
constexpr int kResSlots = 16;      // blocks that touch one patch row at most
constexpr int kResPolls = 1 << 22; // polls of a post before a block gives up (seconds)

// The kinds of words the blocks post (ResidentParams::mute).
enum { kResDirection = 1, kResPq = 2, kResPatchSums = 4, kResCoarse = 8, kResRz = 16 };

struct ResidentParams {
    float *p, *x, *r;
    const float* dinv;
    unsigned long long* halo;   // [L] the direction as the neighbours read it
    const float* rows;   // [kResRow][L] operator rows
    Layout lay;
    int pstride;
    SolveCtl* ctl;
    KernelClock* clock;
    unsigned long long* posts;  // partial sums: kResCopies copies, p.q then r.r and r.z
    unsigned int* tag;          // tag of the next iteration
    int* err;
    int chunk;  // nodes of a block
    int limit;  // iterations of one launch
    int polls;
    // test only: words (kResDirection ..) that block `mute_block` does not post,
    // so that the waits for them run out
    int mute, mute_block;
    // two-level (null minv: Jacobi)
    CoarseLayout cl;
    const float* minv;
    unsigned long long* part;  // [slots][ld] patch sums by the blocks that touch the patch
    unsigned long long* c;     // [tile columns][ld] the coarse solution's parts
    int slots;
    int tiles_x, tiles_y;      // tiles of the inverse along its columns and rows
    int trows, tcols;          // rows and columns of a tile (multiples of 4)
};

// Operator rows of every node: a_d- (9), s_d without the centre (8), a_d+ (9),
// columns in the order (dy, dx) ascending, then the Robin term (1 on a fixed
// row).  Both ends of a coupling add its elements in the same order, so the
// stored operator is exactly symmetric.
__global__ void resident_rows(float* __restrict__ rows, const double* __restrict__ kin, const double* __restrict__ kz,
                              const double* __restrict__ rf, const double* __restrict__ thick,
                              const double* __restrict__ px, const double* __restrict__ py, Layout lay) {
    const int stride = gridDim.x * blockDim.x;
    const long long plane = (long long)(lay.R + 1) * lay.Xp;
    for (long long i = blockIdx.x * blockDim.x + threadIdx.x; i < lay.L; i += stride) {
        const int z = (int)(i / plane);
        const int rem = (int)(i - z * plane);
        const int y = rem / lay.Xp, x = rem - (rem / lay.Xp) * lay.Xp;
        double a[27];
#pragma unroll
        for (int o = 0; o < 27; ++o) a[o] = 0.0;
        double robin = (x <= lay.C && rf[i] < 0.0) ? 1.0 : 0.0;
        if (x <= lay.C && !(rf[i] < 0.0)) {
#pragma unroll
            for (int c = 0; c < 8; ++c) {  // elements in ascending (z, y, x)
                const int oz = c >> 2, oy = (c >> 1) & 1, ox = c & 1;
                const int ez = z - 1 + oz, ey = y - 1 + oy, ex = x - 1 + ox;
                if (ez < 0 || ez >= lay.S || ey < 0 || ey >= lay.R || ex < 0 || ex >= lay.C) continue;
                const long long e = ((long long)ez * lay.R + ey) * lay.Xe + ex;
                const double hz = thick[ez], hy = py[ey], hx = px[ex];
                const double ax = kin[e] * hy * hz / hx, ay = kin[e] * hx * hz / hy, az = kz[e] * hx * hy / hz;
#pragma unroll
                for (int b = 1; b < 8; ++b) {  // the corner that differs in the axes of b
                    const int bz = b >> 2, by = (b >> 1) & 1, bx = b & 1;
                    const double mz = bz ? 1.0 / 6.0 : 2.0 / 6.0, my = by ? 1.0 / 6.0 : 2.0 / 6.0;
                    const double mx = bx ? 1.0 / 6.0 : 2.0 / 6.0;
                    const double sz = bz ? -1.0 : 1.0, sy = by ? -1.0 : 1.0, sx = bx ? -1.0 : 1.0;
                    const double k = ax * (mz * my * sx) + ay * (mz * sy * mx) + az * (sz * my * mx);
                    const int dz = bz ? 2 * oz - 1 : 0, dy = by ? 2 * oy - 1 : 0, dx = bx ? 2 * ox - 1 : 0;
                    a[(dz + 1) * 9 + (dy + 1) * 3 + dx + 1] += k;
                }
            }
            robin = rf[i];
#pragma unroll
            for (int k = 0; k < 9; ++k) a[9 + k] += a[k] + a[18 + k];
        }
#pragma unroll
        for (int o = 0; o < 27; ++o)
            if (o != 13) rows[(long long)(o < 13 ? o : o - 1) * lay.L + i] = (float)a[o];
        rows[26LL * lay.L + i] = (float)robin;
    }
}

__device__ __forceinline__ void res_post(unsigned long long* w, unsigned int tag, float v) {
    const unsigned long long word = ((unsigned long long)tag << 32) | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(w), "l"(word) : "memory");
}
__device__ __forceinline__ unsigned long long res_peek(const unsigned long long* w) {
    unsigned long long word;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(word) : "l"(w) : "memory");
    return word;
}
// The words at(0) .. at(N-1) (null: reads as 0) once each carries `tag`: all
// are asked for at once, those not there yet again.
template <int N, class At>
__device__ __forceinline__ bool res_take(At&& at, unsigned int tag, int polls, float (&v)[N]) {
    unsigned long long word[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const unsigned long long* const w = at(k);
        word[k] = w != nullptr ? res_peek(w) : ((unsigned long long)tag << 32);
    }
    for (int i = 0;; ++i) {
        bool all = true;
#pragma unroll
        for (int k = 0; k < N; ++k) all = all && (unsigned int)(word[k] >> 32) == tag;
        if (all || i >= polls) {
#pragma unroll
            for (int k = 0; k < N; ++k) v[k] = __uint_as_float((unsigned int)word[k]);
            return all;
        }
#pragma unroll
        for (int k = 0; k < N; ++k)  // one round trip for all that are missing
            if ((unsigned int)(word[k] >> 32) != tag) word[k] = res_peek(at(k));
    }
}

// Words of 48 bits of an FP64 value (rounded to 37 bits) and the tag's low 16:
// enough to tell a word from the iteration before, the only older one it can
// hold.  The blocks' parts of a patch sum keep more than FP32 on the way to
// their sum, which alone is rounded to FP32.
__device__ __forceinline__ void res_post48(unsigned long long* w, unsigned int tag, double v) {
    const unsigned long long bits = (unsigned long long)__double_as_longlong(v) + 0x8000ull;
    const unsigned long long word = (bits & ~0xffffull) | (tag & 0xffffu);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(w), "l"(word) : "memory");
}
// The words at(0) .. at(N-1) (null: reads as 0), as res_take.
template <int N, class At>
__device__ __forceinline__ bool res_take48(At&& at, unsigned int tag, int polls, double (&v)[N]) {
    const unsigned int mark = tag & 0xffffu;
    unsigned long long word[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const unsigned long long* const w = at(k);
        word[k] = w != nullptr ? res_peek(w) : (unsigned long long)mark;
    }
    for (int i = 0;; ++i) {
        bool all = true;
#pragma unroll
        for (int k = 0; k < N; ++k) all = all && ((unsigned int)word[k] & 0xffffu) == mark;
        if (all || i >= polls) {
#pragma unroll
            for (int k = 0; k < N; ++k) v[k] = __longlong_as_double((long long)(word[k] & ~0xffffull));
            return all;
        }
#pragma unroll
        for (int k = 0; k < N; ++k)
            if (((unsigned int)word[k] & 0xffffu) != mark) word[k] = res_peek(at(k));
    }
}

// A pair of words side by side (16 bytes, each word with its own tag).
__device__ __forceinline__ void res_post2(unsigned long long* w, unsigned int tag, float a, float b) {
    const unsigned long long t = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(w), "l"(t | __float_as_uint(a)),
                 "l"(t | __float_as_uint(b))
                 : "memory");
}
// N pairs (null: reads as 0), as res_take.
template <int N, class At>
__device__ __forceinline__ bool res_take2(At&& at, unsigned int tag, int polls, float (&a)[N], float (&b)[N]) {
    unsigned long long u[N], v[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
        u[k] = (unsigned long long)(tag - 1u) << 32;
        v[k] = u[k];
        if (at(k) == nullptr) u[k] = v[k] = (unsigned long long)tag << 32;
    }
    for (int i = 0;; ++i) {
        bool all = true;
#pragma unroll
        for (int k = 0; k < N; ++k)
            all = all && (unsigned int)(u[k] >> 32) == tag && (unsigned int)(v[k] >> 32) == tag;
        if (all || i > polls) {
#pragma unroll
            for (int k = 0; k < N; ++k) {
                a[k] = __uint_as_float((unsigned int)u[k]);
                b[k] = __uint_as_float((unsigned int)v[k]);
            }
            return all;
        }
#pragma unroll
        for (int k = 0; k < N; ++k)
            if ((unsigned int)(u[k] >> 32) != tag || (unsigned int)(v[k] >> 32) != tag)
                asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(u[k]), "=l"(v[k]) : "l"(at(k)) : "memory");
    }
}

__device__ __forceinline__ double res_warp_sum(double v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// MUTE: the instantiations of the test switch (a test in the loop of the others
// costs a tenth of a small board's iteration).
template <bool MUTE>
__device__ __forceinline__ bool res_muted(const ResidentParams& P, const int kind) {
    return MUTE && (P.mute & kind) != 0 && (int)blockIdx.x == P.mute_block;
}

// One exchange of NA sums.  Warp k merges the block's warps for sum k, posts
// it (FP64, as two FP32 words: the sum rounded and what is left) and gathers
// every block's, five posts a lane; warp 0 then runs fin(totals) on all its
// lanes while the other warps wait at the closing barrier.  False: a wait ran
// out.
constexpr int kResGather = kResMaxBlocks / 32;
constexpr int kResCopies = 8;  // copies of the posts, each polled by an eighth of the blocks
struct ResShared {
    double red[3][kResThreads / 32], tot[3];
    int ok[3], go;
};
template <int NA, bool MUTE, class Fin>
__device__ __forceinline__ bool res_exchange(const ResidentParams& P, unsigned long long* posts, int kind,
                                             unsigned int tag, const Acc32 (&acc)[NA], ResShared& sh, Fin&& fin) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, blocks = gridDim.x;
#pragma unroll
    for (int k = 0; k < NA; ++k) {
        const double v = res_warp_sum(acc[k].value());
        if (lane == 0) sh.red[k][warp] = v;
    }
    __syncthreads();
    if (warp < NA) {
        const double mine = res_warp_sum(lane < kResThreads / 32 ? sh.red[warp][lane] : 0.0);
        // copy c of this sum's posts: [block] pairs
        auto column = [&](const int c) { return posts + ((size_t)c * blocks * NA + warp) * 2; };
        if (lane < kResCopies && !res_muted<MUTE>(P, kind)) {
            const float hi = (float)mine;
            res_post2(column(lane) + (size_t)blockIdx.x * 2 * NA, tag, hi, (float)(mine - (double)hi));
        }
        float hi[kResGather], lo[kResGather];
        const unsigned long long* const mycopy = column(blockIdx.x % kResCopies);
        const bool ok = __all_sync(0xffffffffu, res_take2(
            [&](const int g) -> const unsigned long long* {
                const int b = lane + 32 * g;
                return b < blocks ? mycopy + (size_t)b * 2 * NA : nullptr;
            },
            tag, P.polls, hi, lo));
        double sum = 0.0;
#pragma unroll
        for (int g = 0; g < kResGather; ++g) sum += (double)hi[g] + (double)lo[g];
        double tot[NA];
        tot[0] = res_warp_sum(sum);
        bool all = ok;
        if (NA > 1) {
            if (lane == 0) {
                sh.tot[warp] = tot[0];
                sh.ok[warp] = ok ? 1 : 0;
            }
            asm volatile("bar.sync 1, %0;" ::"n"(32 * NA) : "memory");  // the NA warps
#pragma unroll
            for (int k = 0; k < NA; ++k) {
                tot[k] = sh.tot[k];
                all = all && sh.ok[k] != 0;
            }
        }
        if (warp == 0) {
            if (all) fin(tot);
            __syncwarp();
            if (lane == 0) sh.go = all ? 1 : 0;
        }
    }
    __syncthreads();
    return sh.go != 0;
}

// Shared memory of a block: the staged direction (three plane segments of its
// nodes with a row and a node on both sides), and for the two-level form its
// tile of the inverse (by columns, whose stride is an odd multiple of four
// floats so that lanes on successive columns meet no bank conflict), R for the
// tile's rows and columns, the masked residuals of its nodes and the c of the
// patches it touches.
__host__ __device__ inline int resident_segment(int chunk, int Xp) { return chunk + 2 * Xp + 2; }
__host__ __device__ inline int resident_tile_stride(int trows) { return (trows / 4) % 2 ? trows : trows + 4; }
inline size_t resident_smem(int trows, int tcols, int chunk, int Xp) {
    const size_t tl = trows > 0 ? (size_t)tcols * resident_tile_stride(trows) + trows + tcols + chunk + kResTouched : 0;
    return sizeof(float) * (tl + 3 * (size_t)resident_segment(chunk, Xp));
}

template <int NODES, bool TL, bool MUTE>
__global__ void __launch_bounds__(kResThreads, 1) resident_pcg(const __grid_constant__ ResidentParams P) {
    constexpr int NA = TL ? 3 : 2;
    __shared__ ResShared sh;
    __shared__ float s_alpha, s_beta;
    __shared__ int s_state;
    __shared__ double s_above;  // r.r above this is above the tolerance
    __shared__ SolveCtl s_ctl;  // the block's copy of the scalars (the same in every block), kept by warp 0
    __shared__ unsigned long long s_op_ns;  // block 0: time from the posted direction to the merged p.q
    extern __shared__ __align__(16) float res_sm[];
    const int mstride = TL ? resident_tile_stride(P.trows) : 0;
    float* const s_m = res_sm;                                 // [tcols][mstride]
    float* const s_R = s_m + (TL ? P.tcols * mstride : 0);     // [tcols] of the tile's columns, [trows] of its rows
    float* const s_res = s_R + (TL ? P.tcols + P.trows : 0);   // [chunk]
    float* const s_c = s_res + (TL ? P.chunk : 0);             // [kResTouched]
    float* const s_h = s_c + (TL ? kResTouched : 0);           // [3][seg]
    const int t = threadIdx.x, blk = blockIdx.x;
    const int ps = P.pstride, Xp = P.lay.Xp, L = (int)P.lay.L, seg = resident_segment(P.chunk, Xp);
    if (P.ctl->state != ST_RUNNING) return;  // uniform across the grid
    unsigned int tag = *P.tag;

    // this thread's nodes
    const int base = blk * P.chunk;
    bool own[NODES];
    float a[NODES][26], e[NODES], p[NODES], r[NODES], d[NODES];
    int patch[NODES];  // the patch that corrects the node, counted from the block's first patch row; -1: none
    // the patch rows (node layer z, patch row) this block's lines touch
    auto patch_row = [&](const int line) {
        const int z = line / (P.lay.R + 1), y = line - z * (P.lay.R + 1);
        return z * P.cl.nby + y / P.cl.b;
    };
    const int prow_first = TL ? patch_row(base / Xp) : 0;
    const int prow_count = TL ? patch_row((min(base + P.chunk, L) - 1) / Xp) - prow_first + 1 : 0;
#pragma unroll
    for (int k = 0; k < NODES; ++k) {
        const int at = t + k * kResThreads, node = base + at;
        own[k] = at < P.chunk && node < L;
#pragma unroll
        for (int o = 0; o < 26; ++o) a[k][o] = own[k] ? P.rows[(size_t)o * L + node] : 0.f;
        e[k] = own[k] ? P.rows[(size_t)26 * L + node] : 0.f;
        p[k] = own[k] ? P.p[node] : 0.f;
        r[k] = own[k] ? P.r[node] : 0.f;
        d[k] = own[k] ? P.dinv[node] : 0.f;
        patch[k] = -1;
        if (TL && d[k] > 0.f) {
            const int z = node / ps, rem = node - z * ps, y = rem / Xp, x = rem - y * Xp;
            if (x <= P.lay.C) patch[k] = (z * P.cl.nby + y / P.cl.b - prow_first) * P.cl.nbx + x / P.cl.b;
        }
    }
    // this block's tile of the inverse, transposed; blocks beyond the tiles have none
    const int tile_y = TL ? blk / P.tiles_x : 0, tile_x = TL ? blk - tile_y * P.tiles_x : 0;
    const bool tiled = TL && tile_y < P.tiles_y;
    const int row0 = tile_y * P.trows, col0 = tile_x * P.tcols;
    const int nrow = tiled ? max(0, min(P.trows, P.cl.nc - row0)) : 0, ncol = tiled ? max(0, min(P.tcols, P.cl.nc - col0)) : 0;
    if (TL && tiled) {
        for (int k = t; k < P.trows * P.tcols; k += kResThreads) {
            const int row = k / P.tcols, col = k - row * P.tcols;
            s_m[col * mstride + row] =
                (row < nrow && col < ncol) ? __ldg(P.minv + (size_t)(row0 + row) * P.cl.ld + col0 + col) : 0.f;
        }
    }
    // the entry of R this thread adds up (a column of the tile, then a row) and
    // its slots: the blocks from the one with its patch row's first node to the
    // one with its last
    int entry = -1, nslots = 0;
    if (TL && tiled && t < P.tcols + P.trows) {
        const int I = t < P.tcols ? col0 + t : row0 + t - P.tcols;
        if (t < P.tcols ? t < ncol : t - P.tcols < nrow) {
            const int pr = I / P.cl.nbx, z = pr / P.cl.nby, y0 = (pr - z * P.cl.nby) * P.cl.b;
            const int first = (z * (P.lay.R + 1) + y0) * Xp;
            nslots = (first + min(P.cl.b, P.lay.R + 1 - y0) * Xp - 1) / P.chunk - first / P.chunk + 1;
            entry = I;
        }
    }
    if (t == 0) {
        s_ctl = *P.ctl;
        s_state = ST_RUNNING;
        s_op_ns = 0;
        const double limit = s_ctl.tol * s_ctl.bnorm;
        s_above = limit * limit * (1.0 + 1e-9);
    }

    bool ok = true;
    for (int n = 0; n < P.limit; ++n, ++tag) {
        if (t == 0 && blk == 0) s_op_ns -= global_ns();
        // post the direction and stage the neighbourhood of this block's nodes
#pragma unroll
        for (int k = 0; k < NODES; ++k) {
            const int at = t + k * kResThreads;
            if (own[k]) {
                const float u = d[k] > 0.f ? p[k] : 0.f;  // the free part
                if (!res_muted<MUTE>(P, kResDirection)) res_post(P.halo + base + at, tag, u);
                s_h[seg + Xp + 1 + at] = u;
            }
        }
        constexpr int AHEAD = 6;
        for (int w0 = t; w0 < 3 * seg; w0 += AHEAD * kResThreads) {
            float v[AHEAD];
            ok = res_take(
                     [&](const int u) -> const unsigned long long* {
                         const int at = w0 + u * kResThreads, dz = at < seg ? -1 : (at < 2 * seg ? 0 : 1);
                         const int j = at - (dz + 1) * seg;
                         const int node = base + dz * ps + j - Xp - 1;
                         const bool mine = dz == 0 && j > Xp && j <= Xp + P.chunk;  // written above, or beyond the board
                         return (at < 3 * seg && !mine && node >= 0 && node < L) ? P.halo + node : nullptr;
                     },
                     tag, P.polls, v) &&
                 ok;
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
                const int at = w0 + u * kResThreads;
                const bool mine = at >= seg + Xp + 1 && at < seg + Xp + 1 + P.chunk && base + at - seg - Xp - 1 < L;
                if (at < 3 * seg && !mine) s_h[at] = v[u];
            }
        }
        if (!__syncthreads_and(ok)) {
            ok = false;
            break;
        }
        // q = A p and p.q
        float q[NODES];
        Acc32 apq[1];
#pragma unroll
        for (int k = 0; k < NODES; ++k) {
            q[k] = 0.f;
            if (!own[k]) continue;
            const float* const h = s_h + seg + Xp + 1 + t + k * kResThreads;
            float s0 = 0.f, s1 = 0.f, s2 = e[k] * p[k];
#pragma unroll
            for (int c = 0; c < 9; ++c) {
                const float* const hc = h + (c / 3 - 1) * Xp + c % 3 - 1;
                const float u = hc[0];
                s0 = fmaf(a[k][c], hc[-seg] - u, s0);
                s1 = fmaf(a[k][17 + c], hc[seg] - u, s1);
                if (c != 4) s2 = fmaf(a[k][c < 4 ? 9 + c : 8 + c], u - p[k], s2);
            }
            q[k] = (s0 + s1) + s2;
            apq[0].add_product(p[k], q[k]);
        }
        ok = res_exchange<1, MUTE>(P, P.posts, kResPq, tag, apq, sh, [&](const double (&tot)[1]) {
            const double alpha = s_ctl.rz / tot[0];
            if (t != 0) return;
            s_ctl.pq = tot[0];
            s_ctl.applications += 1;
            if (!(isfinite(tot[0]) && tot[0] > 0.0)) s_state = ST_NOT_SPD;
            else s_ctl.alpha = alpha;
            s_alpha = (float)s_ctl.alpha;
        });
        if (t == 0 && blk == 0) s_op_ns += global_ns();
        if (!ok || s_state != ST_RUNNING) break;
        const float alpha = s_alpha;
        // r -= alpha q; r.r and sum r^2 / d
        Acc32 au[NA];
#pragma unroll
        for (int k = 0; k < NODES; ++k) {
            r[k] = fmaf(-alpha, q[k], r[k]);
            au[0].add_product(r[k], r[k]);
            au[1].add_product(r[k], r[k] * fabsf(d[k]));
            if (TL && own[k]) s_res[t + k * kResThreads] = patch[k] >= 0 ? r[k] : 0.f;
        }
        if (TL) {
            // sums of the block's part of each patch it touches, in FP64: 16 lanes
            // per patch
            __syncthreads();
            const int lane = t & 15, pairs = prow_count * P.cl.nbx;
            for (int w = t >> 4; w < (pairs + 1) / 2 * 2; w += kResThreads / 16) {
                const bool real = w < pairs;
                const int pr = prow_first + w / P.cl.nbx, pc = w % P.cl.nbx;
                const int z = pr / P.cl.nby, y0 = (pr - z * P.cl.nby) * P.cl.b, x0 = pc * P.cl.b;
                const int bw = min(P.cl.b, P.lay.C + 1 - x0), bh = min(P.cl.b, P.lay.R + 1 - y0);
                const int first = (z * (P.lay.R + 1) + y0) * Xp, origin = first + x0 - base;
                double v = 0.0;  // lane: every fourth column of every fourth row
                for (int yy = lane >> 2; real && yy < bh; yy += 4)
                    for (int xx = lane & 3; xx < bw; xx += 4) {
                        const int at = origin + yy * Xp + xx;
                        if (at >= 0 && at < P.chunk) v += (double)s_res[at];
                    }
#pragma unroll
                for (int off = 8; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off, 16);
                if (real && lane == 0 && !res_muted<MUTE>(P, kResPatchSums))
                    res_post48(P.part + (size_t)(blk - first / P.chunk) * P.cl.ld + (size_t)pr * P.cl.nbx + pc, tag, v);
            }
            // R of the tile's columns and rows
            double sum = 0.0;
            for (int s0 = 0; s0 < P.slots; s0 += 4) {
                double v[4];
                ok = res_take48(
                         [&](const int k) -> const unsigned long long* {
                             return s0 + k < nslots ? P.part + (size_t)(s0 + k) * P.cl.ld + entry : nullptr;
                         },
                         tag, P.polls, v) &&
                     ok;
                sum += (v[0] + v[1]) + (v[2] + v[3]);
            }
            if (t < P.tcols + P.trows) s_R[t] = (float)sum;
            if (!__syncthreads_and(ok)) {
                ok = false;
                break;
            }
            // the tile's part of c: four rows and every sixteenth column a thread
            const int cg = t & 15;
            for (int rq = t >> 4; rq < (P.trows / 4 + 1) / 2 * 2 && tiled; rq += kResThreads / 16) {
                const bool real = rq < P.trows / 4;
                float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
                for (int col = cg; real && col < P.tcols; col += 16) {
                    const float4 mm = *reinterpret_cast<const float4*>(s_m + col * mstride + 4 * rq);
                    const float x = s_R[col];
                    m.x = fmaf(mm.x, x, m.x);
                    m.y = fmaf(mm.y, x, m.y);
                    m.z = fmaf(mm.z, x, m.z);
                    m.w = fmaf(mm.w, x, m.w);
                }
                // sums over the 16 lanes, a lane left with row 2 bit3 + bit2 of its number
                const bool h8 = (cg & 8) != 0, h4 = (cg & 4) != 0;
                float u0 = (h8 ? m.z : m.x) + __shfl_xor_sync(0xffffffffu, h8 ? m.x : m.z, 8);
                float u1 = (h8 ? m.w : m.y) + __shfl_xor_sync(0xffffffffu, h8 ? m.y : m.w, 8);
                float u = (h4 ? u1 : u0) + __shfl_xor_sync(0xffffffffu, h4 ? u0 : u1, 4);
                u += __shfl_xor_sync(0xffffffffu, u, 2);
                u += __shfl_xor_sync(0xffffffffu, u, 1);
                const int row = 4 * rq + (h8 ? 2 : 0) + (h4 ? 1 : 0);
                if (real && (cg & 3) == 0 && row < nrow) {
                    if (!res_muted<MUTE>(P, kResCoarse)) res_post(P.c + (size_t)tile_x * P.cl.ld + row0 + row, tag, u);
                    au[NA - 1].add_product(s_R[P.tcols + row], u);
                }
            }
        }
        ok = res_exchange<NA, MUTE>(P, P.posts + 2 * kResCopies * gridDim.x, kResRz, tag, au, sh, [&](const double (&tot)[NA]) {
            if (t != 0) return;
            const double rzn = TL ? tot[1] + tot[NA - 1] : tot[1], ratio = rzn / s_ctl.rz;
            s_ctl.iterations += 1;
            s_ctl.rr = tot[0];
            s_ctl.rdr = tot[1];
            // the root and the quotient only where r.r is not far above the
            // limit (their latency is on every block's way)
            if (!(tot[0] > s_above) && sqrt(tot[0]) / s_ctl.bnorm <= s_ctl.tol) {
                s_state = ST_CONVERGED;
            } else if (!isfinite(rzn) || s_ctl.rz == 0.0) {
                s_state = ST_BREAKDOWN;
            } else {
                s_ctl.beta = ratio;
                s_ctl.rz = rzn;
                if (s_ctl.iterations >= s_ctl.max_it) s_state = ST_MAXIT;
            }
            s_beta = (float)s_ctl.beta;
        });
        if (!ok || s_state != ST_RUNNING) break;
        const float beta = s_beta;
        if (TL) {  // c of the patches this block touches: four lanes each, four parts a lane at most
            const int count = prow_count * P.cl.nbx;
            for (int i = t >> 2; i < (count + 7) / 8 * 8; i += kResThreads / 4) {
                float v[4];
                ok = res_take(
                         [&](const int k) -> const unsigned long long* {
                             const int part = (t & 3) + 4 * k;
                             return i < count && part < P.tiles_x
                                        ? P.c + (size_t)part * P.cl.ld + (size_t)prow_first * P.cl.nbx + i
                                        : nullptr;
                         },
                         tag, P.polls, v) &&
                     ok;
                float sum = (v[0] + v[1]) + (v[2] + v[3]);
                sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                if ((t & 3) == 0 && i < count) s_c[i] = sum;
            }
            __syncthreads();  // ok is voted on with the next iteration's neighbourhood
        }
#pragma unroll
        for (int k = 0; k < NODES; ++k) {
            const int at = t + k * kResThreads;
            if (own[k]) P.x[base + at] = fmaf(alpha, p[k], P.x[base + at]);
            float z = r[k] * fabsf(d[k]);
            if (TL && patch[k] >= 0) z += s_c[patch[k]];
            p[k] = fmaf(beta, p[k], z);
        }
    }
    ok = __syncthreads_and(ok);
#pragma unroll
    for (int k = 0; k < NODES; ++k) {
        const int at = t + k * kResThreads;
        if (own[k]) {
            P.r[base + at] = r[k];
            P.p[base + at] = p[k];
        }
    }
    if (t != 0) return;
    if (!ok) {
        atomicExch(P.err, 1);
    } else if (blk == 0) {
        P.clock->total_ns += s_op_ns;
        P.clock->count += (unsigned long long)(s_ctl.applications - P.ctl->applications);
        s_ctl.state = s_state;
        if (s_ctl.iterations != P.ctl->iterations) s_ctl.rel = sqrt(s_ctl.rr) / s_ctl.bnorm;
        *P.ctl = s_ctl;
        *P.tag = tag + 1;
    }
}

}  // namespace tb

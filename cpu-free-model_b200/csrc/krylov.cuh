// Persistent Krylov solvers on one GPU, templated on the operator.
//
// Operators (one row per thread, tiles of CG_TILE consecutive rows):
//   CsrOp        CSR SpMV, row order, one fma per nonzero (CG/src/common.cu:150-168)
//   ClassOp      the same sums for matrices whose rows fall into few classes
//   StencilOp<D> matrix-free cell-centred -div(k grad u), 5-point (D = 2) or
//                7-point (D = 3): t = d_i u_i, then one fma(-w, u_nb, t) per
//                neighbour in the order x-1, x+1, y-1, y+1, z-1, z+1
// Each operator also applies in FP32 (applyN32) from FP32 copies of its
// coefficients, for the inner solve of the mixed-precision method.
//
// Solvers, each one cooperative launch for the whole solve:
//   cg_std_kernel    standard CG, 3 grid barriers per iteration
//                    (CG/src/common.cu:399-538, CG/src/single-stream/standard.cu:158-299)
//   cg_pipe_kernel   pipelined CG (CG/src/single-stream/pipelined.cu:176-330): the
//                    SpMV q = A w and every vector recurrence of an iteration fused
//                    into one pass, double-buffered w and dot partials, 1 grid
//                    barrier per iteration
//   cg_mixed_kernel  FP32 CG with FP64 reliable updates: the true residual, the
//                    correction x += |b| d and the dot reductions (FP64 sums of
//                    exact FP32 products) stay FP64
// Every dot is a fixed tree (1024-row tiles, xor butterflies, then the tile
// partials in lane order), so results do not depend on the launch shape and
// the CPU oracle reproduces them bit for bit.  Scalar arithmetic is written
// with explicit-rounding intrinsics where the compiler could otherwise fuse a
// multiply into an add.
#pragma once

#include "barrier.cuh"

namespace cfm {

constexpr int CG_TILE = 1024;  // rows per tile == threads per block
constexpr unsigned CG_FULL = 0xffffffffu;

// Partial-sum slots (each ntiles doubles) in KArgs::part.
enum : int { SL_G0 = 0, SL_D0 = 1, SL_TT = 2, SL_B = 3, SL_G1 = 4, SL_D1 = 5, NSLOTS = 6 };

struct CgResult {
    long long iters;
    int status;
    int restarts;  // restarts (standard, pipelined) or FP64 reliable updates (mixed)
    double gamma;
    double bnorm;
};

__device__ __forceinline__ double warp_xor_sum(double v) {
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) v = __dadd_rn(v, __shfl_xor_sync(CG_FULL, v, off));
    return v;
}

// Tree sum over the 1024 threads of the block; every thread gets the result (each
// warp adds the 32 warp sums for itself, which costs no second hand-over).
__device__ __forceinline__ double block_sum(double v, double *sm /* 32 doubles */) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_xor_sum(v);
    if (lane == 0) sm[warp] = v;
    __syncthreads();
    const double out = warp_xor_sum(sm[lane]);
    __syncthreads();
    return out;
}

// One or two sums of tile partials in the fixed order (thread t of 1024 adds part[t],
// part[t+1024], ..., then the tree of block_sum) behind one block barrier: every warp
// adds the 32 warp sums for itself.  Blocks of NW < 32 warps take several of the 32 warps'
// parts per warp.  sm: N x 32 doubles that no thread still reads.
template <int N, int NW = 32>
__device__ __forceinline__ void partial_sums(const double *p, const double *p2, int ntiles, double *sm, double *out,
                                             double *out2) {
    static_assert(32 % NW == 0, "whole turns");
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int warp = threadIdx.x >> 5; warp < 32; warp += NW) {
        double v = 0.0, v2 = 0.0;
        for (int i = warp * 32 + lane; i < ntiles; i += CG_TILE) {
            v = __dadd_rn(v, p[i]);
            if (N > 1) v2 = __dadd_rn(v2, p2[i]);
        }
        v = warp_xor_sum(v);
        if (N > 1) v2 = warp_xor_sum(v2);
        if (lane == 0) {
            sm[warp] = v;
            if (N > 1) sm[32 + warp] = v2;
        }
    }
    __syncthreads();
    *out = warp_xor_sum(sm[lane]);
    if (N > 1) *out2 = warp_xor_sum(sm[32 + lane]);
}

// Sum of tile partials in the fixed order: thread t adds part[t], part[t+1024], ...
__device__ __forceinline__ double sum_partials(const double *part, int ntiles, double *sm) {
    double acc = 0.0;
    for (int i = threadIdx.x; i < ntiles; i += CG_TILE) acc = __dadd_rn(acc, part[i]);
    return block_sum(acc, sm);
}

// Per-tile sums of a tile loop without a block barrier per tile.  Each
// warp reduces its 32 rows at once (the xor butterfly of block_sum) and
// parks the warp sum in shared memory; every TS_TILES tiles, and at the end,
// one barrier, then warp w reduces parked entry w (the 32 warp sums of one
// tile, in warp order: again block_sum's tree) into dst[k][tile].  The
// partials are bit for bit block_sum's, while the warps of a block run ahead
// of each other from tile to tile.  The block's tiles are t0, t0 + stride,
// ...; every thread of the block calls add() for every tile, and flush()
// after the loop.
constexpr int TS_TILES = 16;
constexpr int TS_SMEM = TS_TILES * 2 * 32;  // doubles (also >= 33 for block_sum)

template <int K>
struct TileSums {
    double *sm;
    double *dst[K];
    int stride, t0 = 0, g = 0;
    __device__ __forceinline__ TileSums(double *s, int step, double *d0, double *d1 = nullptr)
        : sm(s), stride(step) {
        dst[0] = d0;
        if (K > 1) dst[K - 1] = d1;
    }
    __device__ __forceinline__ void add(int tile, double v0, double v1 = 0.0) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        if (g == 0) t0 = tile;
        v0 = warp_xor_sum(v0);
        if (lane == 0) sm[(g * K) * 32 + warp] = v0;
        if (K > 1) {
            v1 = warp_xor_sum(v1);
            if (lane == 0) sm[(g * K + K - 1) * 32 + warp] = v1;
        }
        if (++g == TS_TILES) flush();
    }
    __device__ __forceinline__ void flush() {
        if (g == 0) return;
        __syncthreads();
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        if (warp < g * K) {
            const double v = warp_xor_sum(sm[warp * 32 + lane]);
            double *d = dst[0];
            if (K > 1 && (warp & 1)) d = dst[K - 1];  // a select: no indexed local array
            if (lane == 0) d[t0 + (warp / K) * stride] = v;
        }
        __syncthreads();
        g = 0;
    }
};

// Exact product of two FP32 values, as FP64.
__device__ __forceinline__ double xprod(float a, float b) { return __dmul_rn((double)a, (double)b); }

// U of the block's tiles per step (t0 + u gridDim.x, u < U), the FP32
// passes' form of the tile pairs.  Mixed, us per iteration on B200 for U = 1, 2, 4: 128^3
// 7-point with row classes 34.2 / 32.7 / 35.7, renumbered so that it has none 58.9 / 51.5 / 62.4.
constexpr int INNER_U = 2;
template <int U>
struct TileGroup {
    int tile[U], row[U];
    bool has[U], ok[U];
    __device__ __forceinline__ TileGroup(int ntiles, int n, int t0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            tile[u] = t0 + u * (int)gridDim.x;
            has[u] = tile[u] < ntiles;
            row[u] = tile[u] * CG_TILE + (int)threadIdx.x;
            ok[u] = has[u] && row[u] < n;
        }
    }
};
template <int U>
struct Vals32 {
    float v[U];
};

// ------------------------------------------------------------- operators
// CSR entries per row whose loads a thread issues together (CsrOp::apply2_t,
// the FP64 passes).  Standard CG on 128^3 7-point renumbered so that it has no row
// classes, us per iteration for 1, 4, 8: 73.3 / 71.4 / 71.1 (bit-identical); the same form
// in the FP32 passes was no faster, so those keep one entry per step.
constexpr int CSR_Q = 4;
struct CsrOp {
    static constexpr bool ROW_FIRST = false;  // phase_pipe_step (its registers would spill)
    const int *rowptr, *col;
    const double *val;
    const float *val32;
    __device__ __forceinline__ double apply(const double *x, int i) const {
        double acc = 0.0;
        const int j1 = rowptr[i + 1];
        for (int j = rowptr[i]; j < j1; ++j) acc = __fma_rn(val[j], x[col[j]], acc);
        return acc;
    }
    // apply for rows i (if v1) and i2 (if v2), their entries interleaved so
    // that both rows' loads are in flight together; 0 for an absent row.
    template <class T>
    __device__ __forceinline__ void apply2_t(const T *v, const T *x, int i, bool v1, int i2,
                                             bool v2, T &y1, T &y2) const {
        int j1 = 0, e1 = 0, j2 = 0, e2 = 0;
        if (v1) {
            j1 = rowptr[i];
            e1 = rowptr[i + 1];
        }
        if (v2) {
            j2 = rowptr[i2];
            e2 = rowptr[i2 + 1];
        }
        T a1 = T(0), a2 = T(0);
        // CSR_Q entries of each row per step: all their col / val loads,
        // then all their x gathers, then the FMAs in entry order (the sum is
        // the one-entry-at-a-time one, bit for bit), so up to 4 CSR_Q
        // independent loads are in flight per thread instead of two chains
        while (j1 < e1 || j2 < e2) {
            int c1[CSR_Q], c2[CSR_Q];
            T w1[CSR_Q], w2[CSR_Q], g1[CSR_Q], g2[CSR_Q];
#pragma unroll
            for (int q = 0; q < CSR_Q; ++q) {
                c1[q] = j1 + q < e1 ? col[j1 + q] : -1;
                c2[q] = j2 + q < e2 ? col[j2 + q] : -1;
                w1[q] = j1 + q < e1 ? v[j1 + q] : T(0);
                w2[q] = j2 + q < e2 ? v[j2 + q] : T(0);
            }
#pragma unroll
            for (int q = 0; q < CSR_Q; ++q) {
                g1[q] = c1[q] >= 0 ? x[c1[q]] : T(0);
                g2[q] = c2[q] >= 0 ? x[c2[q]] : T(0);
            }
#pragma unroll
            for (int q = 0; q < CSR_Q; ++q) {
                if (c1[q] >= 0) a1 = fma_rn(w1[q], g1[q], a1);
                if (c2[q] >= 0) a2 = fma_rn(w2[q], g2[q], a2);
            }
            j1 += CSR_Q;
            j2 += CSR_Q;
        }
        y1 = a1;
        y2 = a2;
    }
    __device__ __forceinline__ static double fma_rn(double u, double w, double c) {
        return __fma_rn(u, w, c);
    }
    __device__ __forceinline__ static float fma_rn(float u, float w, float c) {
        return __fmaf_rn(u, w, c);
    }
    __device__ __forceinline__ void apply2(const double *x, int i, bool v1, int i2, bool v2,
                                           double &y1, double &y2) const {
        apply2_t(val, x, i, v1, i2, v2, y1, y2);
    }
    // What a row's loads begin with, for a caller that has time to load it ahead.
    __device__ __forceinline__ int key(int i) const { return rowptr[i]; }
    // FP32 apply for the rows of a tile group (0 for an absent row), their
    // entries interleaved; key: key() of the rows.
    template <int U>
    __device__ __forceinline__ Vals32<U> applyN32(const float *x, const TileGroup<U> &g, const int (&key)[U]) const {
        int j[U], e[U];
        Vals32<U> y;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            j[u] = g.ok[u] ? key[u] : 0;
            e[u] = g.ok[u] ? rowptr[g.row[u] + 1] : 0;
            y.v[u] = 0.f;
        }
        bool more = true;
        while (more) {
            more = false;
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (j[u] < e[u]) {
                    y.v[u] = __fmaf_rn(val32[j[u]], x[col[j[u]]], y.v[u]);
                    ++j[u];
                    more = true;
                }
        }
        return y;
    }
    // A x0 with x0 = 0, summed like apply (always +0)
    __device__ __forceinline__ double apply_zero(int i) const {
        double acc = 0.0;
        const int j1 = rowptr[i + 1];
        for (int j = rowptr[i]; j < j1; ++j) acc = __fma_rn(val[j], 0.0, acc);
        return acc;
    }
};

// CSR matrix whose rows fall into at most 256 classes (cfm_csr_create finds
// them): rows of a class have the same column offsets col - i and, with VALS, the
// same values bit for bit (a constant-coefficient grid operator has one class per
// kind of boundary).  A row then costs one byte and a table entry that stays in L1
// instead of its column indices (and values) from L2 or HBM, and its gathers wait
// for that byte instead of rowptr and col in turn.  Entries are taken in row order,
// so the sums are CsrOp's bit for bit.  Table rows are L entries (a multiple of 4).
template <bool VALS>
struct ClassOp {
    static constexpr bool ROW_FIRST = true;
    const int *rowptr;
    const double *val;
    const float *val32;
    const unsigned char *cls;
    const int *len, *off;  // per class: entries, offsets
    const double *tval;    // VALS: per class values
    const float *tval32;
    int L;
    __device__ __forceinline__ static double fma_rn(double u, double w, double c) { return __fma_rn(u, w, c); }
    __device__ __forceinline__ static float fma_rn(float u, float w, float c) { return __fmaf_rn(u, w, c); }
    // 16 bytes of a value row, and as many offsets
    __device__ __forceinline__ static void load(const double *p, double (&v)[2]) {
        const double2 a = __ldg(reinterpret_cast<const double2 *>(p));
        v[0] = a.x, v[1] = a.y;
    }
    __device__ __forceinline__ static void load(const float *p, float (&v)[4]) {
        const float4 a = __ldg(reinterpret_cast<const float4 *>(p));
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
    }
    __device__ __forceinline__ static void load(const int *p, int (&v)[2]) {
        const int2 a = __ldg(reinterpret_cast<const int2 *>(p));
        v[0] = a.x, v[1] = a.y;
    }
    __device__ __forceinline__ static void load(const int *p, int (&v)[4]) {
        const int4 a = __ldg(reinterpret_cast<const int4 *>(p));
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
    }
    // Row i's class, for a caller that has time to load it ahead of the row.
    __device__ __forceinline__ int key(int i) const { return cls[i]; }
    // The rows of a group (those with ok; c: their classes), C entries of each at a time,
    // their gathers (and, without VALS, values) in flight together; 0 for an absent row.
    // With VALS the values come from the table (L1) only as they are used, which leaves
    // the registers to the gathers: a 7-point row takes one step in FP32, two in FP64.
    template <int U, class T>
    __device__ __forceinline__ void rows(const T *v, const T *tv, const T *x, const int (&row)[U],
                                         const bool (&ok)[U], const int (&c)[U], T (&y)[U]) const {
        constexpr int Q = 16 / sizeof(T), C = Q;
        int m[U], at[U], src[U], most = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            m[u] = ok[u] ? __ldg(len + c[u]) : 0;
            at[u] = c[u] * L;
            src[u] = !VALS && ok[u] ? rowptr[row[u]] : 0;
            most = max(most, m[u]);
            y[u] = T(0);
        }
#pragma unroll 1
        for (int k = 0; k < most; k += C) {
            T w[U][VALS ? 1 : C], g[U][C];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int h = 0; h < C; h += Q) {
                    if (k + h >= m[u]) continue;
                    int o[Q];
                    load(off + at[u] + k + h, o);
#pragma unroll
                    for (int q = 0; q < Q; ++q) {
                        const bool in = k + h + q < m[u];
                        if (!VALS) w[u][VALS ? 0 : h + q] = in ? v[src[u] + k + h + q] : T(0);
                        g[u][h + q] = in ? x[row[u] + o[q]] : T(0);
                    }
                }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int h = 0; h < C; h += Q) {
                    if (k + h >= m[u]) continue;
                    T t[Q];
                    if (VALS) load(tv + at[u] + k + h, t);
#pragma unroll
                    for (int q = 0; q < Q; ++q)
                        if (k + h + q < m[u]) y[u] = fma_rn(VALS ? t[q] : w[u][VALS ? 0 : h + q], g[u][h + q], y[u]);
                }
        }
    }
    __device__ __forceinline__ double apply(const double *x, int i) const {
        const int row[1] = {i}, c[1] = {cls[i]};
        const bool ok[1] = {true};
        double y[1];
        rows<1>(val, tval, x, row, ok, c, y);
        return y[0];
    }
    __device__ __forceinline__ void apply2(const double *x, int i, bool v1, int i2, bool v2, double &y1,
                                           double &y2) const {
        const int row[2] = {i, i2}, c[2] = {v1 ? cls[i] : 0, v2 ? cls[i2] : 0};
        const bool ok[2] = {v1, v2};
        double y[2];
        rows<2>(val, tval, x, row, ok, c, y);
        y1 = y[0];
        y2 = y[1];
    }
    template <int U>
    __device__ __forceinline__ Vals32<U> applyN32(const float *x, const TileGroup<U> &g, const int (&key)[U]) const {
        Vals32<U> y;
        rows<U>(val32, tval32, x, g.row, g.ok, key, y.v);
        return y;
    }
    // A x0 with x0 = 0, summed like apply (always +0)
    __device__ __forceinline__ double apply_zero(int i) const {
        const int c = cls[i], m = __ldg(len + c);
        double acc = 0.0;
        for (int k = 0; k < m; ++k) acc = __fma_rn(VALS ? __ldg(tval + c * L + k) : val[rowptr[i] + k], 0.0, acc);
        return acc;
    }
};

template <int D>
struct StencilOp {
    static constexpr bool ROW_FIRST = true;
    int nx, ny, nz;
    const double *we, *wn, *wt, *dg;
    const float *we32, *wn32, *wt32, *dg32;
    __device__ __forceinline__ double apply(const double *x, int i) const {
        const int q = i / nx, ix = i - q * nx, iy = D == 3 ? q % ny : q;
        double t = __dmul_rn(dg[i], x[i]);
        if (ix > 0) t = __fma_rn(-we[i - 1], x[i - 1], t);
        if (ix < nx - 1) t = __fma_rn(-we[i], x[i + 1], t);
        if (iy > 0) t = __fma_rn(-wn[i - nx], x[i - nx], t);
        if (iy < ny - 1) t = __fma_rn(-wn[i], x[i + nx], t);
        if (D == 3) {
            const int iz = q / ny, P = nx * ny;
            if (iz > 0) t = __fma_rn(-wt[i - P], x[i - P], t);
            if (iz < nz - 1) t = __fma_rn(-wt[i], x[i + P], t);
        }
        return t;
    }
    __device__ __forceinline__ float apply32(const float *x, int i) const {
        const int q = i / nx, ix = i - q * nx, iy = D == 3 ? q % ny : q;
        float t = __fmul_rn(dg32[i], x[i]);
        if (ix > 0) t = __fmaf_rn(-we32[i - 1], x[i - 1], t);
        if (ix < nx - 1) t = __fmaf_rn(-we32[i], x[i + 1], t);
        if (iy > 0) t = __fmaf_rn(-wn32[i - nx], x[i - nx], t);
        if (iy < ny - 1) t = __fmaf_rn(-wn32[i], x[i + nx], t);
        if (D == 3) {
            const int iz = q / ny, P = nx * ny;
            if (iz > 0) t = __fmaf_rn(-wt32[i - P], x[i - P], t);
            if (iz < nz - 1) t = __fmaf_rn(-wt32[i], x[i + P], t);
        }
        return t;
    }
    __device__ __forceinline__ double apply_zero(int) const { return 0.0; }
    __device__ __forceinline__ void apply2(const double *x, int i, bool v1, int i2, bool v2,
                                           double &y1, double &y2) const {
        y1 = v1 ? apply(x, i) : 0.0;
        y2 = v2 ? apply(x, i2) : 0.0;
    }
    __device__ __forceinline__ int key(int) const { return 0; }
    template <int U>
    __device__ __forceinline__ Vals32<U> applyN32(const float *x, const TileGroup<U> &g, const int (&)[U]) const {
        Vals32<U> y;
#pragma unroll
        for (int u = 0; u < U; ++u) y.v[u] = g.ok[u] ? apply32(x, g.row[u]) : 0.f;
        return y;
    }
};

template <class Op>
struct KArgs {
    Op op;
    int n;
    int ntiles;
    const double *b;  // nullptr: ones
    double *x, *r, *p, *s, *t;
    double *z, *w0, *w1;           // pipelined
    float *r32, *p32, *s32, *d32;  // mixed inner
    double *part;                  // NSLOTS * ntiles
    CgResult *res;
    BarrierState *bar;
    int maxiter;
    double tol;
    int inner_maxiter;
    double inner_tol;
    // standard CG only: copy x after every snap_every-th iteration into
    // snap[(k / snap_every - 1) * n ...] while fewer than snap_max are taken
    double *snap;
    int snap_every, snap_max;
};

#define CFM_TILES(a) for (int tile = blockIdx.x; tile < (a).ntiles; tile += gridDim.x)
#define CFM_ROW(a) const int i = tile * CG_TILE + threadIdx.x
// Two of the block's tiles per step (tile, tile2 = tile + gridDim.x): the
// loads of both rows go out before either row's arithmetic, halving the
// chains of dependent memory round trips a warp waits on.
#define CFM_TILE_GROUPS(a, U) for (int tile = blockIdx.x; tile < (a).ntiles; tile += (U) * (int)gridDim.x)
#define CFM_TILE_PAIRS(a) for (int tile = blockIdx.x; tile < (a).ntiles; tile += 2 * (int)gridDim.x)
#define CFM_ROW_PAIR(a)                                                      \
    const int tile2 = tile + (int)gridDim.x;                                 \
    const bool has2 = tile2 < (a).ntiles;                                    \
    const int i = tile * CG_TILE + threadIdx.x, i2 = tile2 * CG_TILE + threadIdx.x; \
    const bool v1 = i < (a).n, v2 = has2 && i2 < (a).n

template <class Op>
__device__ __forceinline__ double *slot(const KArgs<Op> &a, int s) {
    return a.part + (size_t)s * a.ntiles;
}

// A persistent solver's barriers and grid-wide sums: a sum is a barrier, after which
// every block adds the tile partials of a slot (or two) in sum_partials' order.  Each
// returns false once a wait ran out.
template <class Op>
struct CgGrid {
    const KArgs<Op> &a;
    double *red;  // 4 x 32 doubles of shared memory, used by turns
    int site = 0, par = 0;
    __device__ __forceinline__ CgGrid(const KArgs<Op> &args, double *r) : a(args), red(r) {}
    __device__ __forceinline__ bool barrier() { return grid_barrier(a.bar, gridDim.x, site++); }
    __device__ __forceinline__ bool sum(int s, double *out) {
        if (!barrier()) return false;
        sums<1>(slot(a, s), nullptr, out, nullptr);
        return true;
    }
    __device__ __forceinline__ bool sum2(int s, double *out, int s2, double *out2) {
        if (!barrier()) return false;
        sums<2>(slot(a, s), slot(a, s2), out, out2);
        return true;
    }
    template <int N>
    __device__ __forceinline__ void sums(const double *p, const double *p2, double *out, double *out2) {
        partial_sums<N>(p, p2, a.ntiles, red + 64 * (par ^= 1), out, out2);
    }
};

// -------------------------------------------------------- standard phases
template <class Op>
__device__ void phase_init(const KArgs<Op> &a, double *sm) {
    TileSums<2> ts(sm, gridDim.x, slot(a, SL_G0), slot(a, SL_B));
    CFM_TILES(a) {
        CFM_ROW(a);
        double g = 0.0, bb = 0.0;
        if (i < a.n) {
            const double bi = a.b ? a.b[i] : 1.0;
            const double ri = __fma_rn(-1.0, a.op.apply_zero(i), bi);  // r0 = b - A x0, x0 = 0
            a.x[i] = 0.0;
            a.r[i] = ri;
            a.p[i] = ri;
            g = __dmul_rn(ri, ri);
            bb = __dmul_rn(bi, bi);
        }
        ts.add(tile, g, bb);
    }
    ts.flush();
}

template <class Op>
__device__ void phase_spmv_dot(const KArgs<Op> &a, double *sm) {
    TileSums<1> ts(sm, gridDim.x, slot(a, SL_D0));
    CFM_TILE_PAIRS(a) {
        CFM_ROW_PAIR(a);
        double p1 = 0.0, p2 = 0.0, s1, s2;
        if (v1) p1 = a.p[i];
        if (v2) p2 = a.p[i2];
        a.op.apply2(a.p, i, v1, i2, v2, s1, s2);
        if (v1) a.s[i] = s1;
        if (v2) a.s[i2] = s2;
        ts.add(tile, v1 ? __dmul_rn(p1, s1) : 0.0);
        if (has2) ts.add(tile2, v2 ? __dmul_rn(p2, s2) : 0.0);
    }
    ts.flush();
}

template <class Op>
__device__ void phase_update(const KArgs<Op> &a, double alpha, double *sm) {
    TileSums<1> ts(sm, gridDim.x, slot(a, SL_G0));
    CFM_TILE_PAIRS(a) {
        CFM_ROW_PAIR(a);
        double x1 = 0.0, p1 = 0.0, r1 = 0.0, s1 = 0.0, x2 = 0.0, p2 = 0.0, r2 = 0.0, s2 = 0.0;
        if (v1) {
            x1 = a.x[i];
            p1 = a.p[i];
            r1 = a.r[i];
            s1 = a.s[i];
        }
        if (v2) {
            x2 = a.x[i2];
            p2 = a.p[i2];
            r2 = a.r[i2];
            s2 = a.s[i2];
        }
        double g1 = 0.0, g2 = 0.0;
        if (v1) {
            a.x[i] = __fma_rn(alpha, p1, x1);
            const double ri = __fma_rn(-alpha, s1, r1);
            a.r[i] = ri;
            g1 = __dmul_rn(ri, ri);
        }
        if (v2) {
            a.x[i2] = __fma_rn(alpha, p2, x2);
            const double ri = __fma_rn(-alpha, s2, r2);
            a.r[i2] = ri;
            g2 = __dmul_rn(ri, ri);
        }
        ts.add(tile, g1);
        if (has2) ts.add(tile2, g2);
    }
    ts.flush();
}

// t = b - A x (FP64) and its squared norm into SL_TT
template <class Op>
__device__ void phase_true_residual(const KArgs<Op> &a, double *sm) {
    TileSums<1> ts(sm, gridDim.x, slot(a, SL_TT));
    CFM_TILES(a) {
        CFM_ROW(a);
        double q = 0.0;
        if (i < a.n) {
            const double bi = a.b ? a.b[i] : 1.0;
            const double ti = __dsub_rn(bi, a.op.apply(a.x, i));
            a.t[i] = ti;
            q = __dmul_rn(ti, ti);
        }
        ts.add(tile, q);
    }
    ts.flush();
}

template <class Op>
__device__ void phase_snap(const KArgs<Op> &a, int slot_i) {
    double *dst = a.snap + (size_t)slot_i * a.n;
    CFM_TILES(a) {
        CFM_ROW(a);
        if (i < a.n) dst[i] = a.x[i];
    }
}

template <class Op>
__device__ void phase_restart(const KArgs<Op> &a) {
    CFM_TILES(a) {
        CFM_ROW(a);
        if (i < a.n) {
            a.r[i] = a.t[i];
            a.p[i] = a.t[i];
        }
    }
}

template <class Op>
__device__ void phase_p(const KArgs<Op> &a, double beta) {
    CFM_TILE_PAIRS(a) {
        CFM_ROW_PAIR(a);
        double p1 = 0.0, r1 = 0.0, p2 = 0.0, r2 = 0.0;
        if (v1) {
            p1 = a.p[i];
            r1 = a.r[i];
        }
        if (v2) {
            p2 = a.p[i2];
            r2 = a.r[i2];
        }
        if (v1) a.p[i] = __fma_rn(beta, p1, r1);
        if (v2) a.p[i2] = __fma_rn(beta, p2, r2);
    }
}

__device__ __forceinline__ void write_result(CgResult *res, long long k, int status, int restarts,
                                             double gamma, double bnorm) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        res->iters = k;
        res->status = status;
        res->restarts = restarts;
        res->gamma = gamma;
        res->bnorm = bnorm;
    }
}

// Standard CG; tol > 0 stops when the recursive residual reaches tol ||b||
// and the FP64 true residual confirms it (a restart from the true residual
// otherwise); tol <= 0 runs exactly maxiter iterations (reference -niter).
template <class Op>
__global__ void __launch_bounds__(CG_TILE, 1) cg_std_kernel(KArgs<Op> a) {
    __shared__ double sm[TS_SMEM], red[128];
    CgGrid<Op> grid(a, red);
    phase_init(a, sm);
    double gamma0, bb;
    if (!grid.sum2(SL_G0, &gamma0, SL_B, &bb)) return;
    const double bnorm = sqrt(bb);
    const bool use_tol = a.tol > 0.0;
    const double target = a.tol * bnorm;
    int status = use_tol ? CFM_NOT_CONVERGED : CFM_OK;
    int restarts = 0;
    long long k = 0;
    if (use_tol && sqrt(gamma0) <= target) status = CFM_OK;
    while (k < a.maxiter && !(use_tol && status == CFM_OK)) {
        phase_spmv_dot(a, sm);
        double delta;
        if (!grid.sum(SL_D0, &delta)) return;
        const double alpha = gamma0 / delta;
        if (use_tol && !(delta > 0.0 && isfinite(alpha))) {
            status = CFM_BREAKDOWN;
            break;
        }
        phase_update(a, alpha, sm);
        double gamma1;
        if (!grid.sum(SL_G0, &gamma1)) return;
        ++k;
        if (a.snap && k % a.snap_every == 0 && k / a.snap_every <= a.snap_max)
            phase_snap(a, (int)(k / a.snap_every) - 1);  // x is stable until the next update
        if (use_tol && sqrt(gamma1) <= target) {
            phase_true_residual(a, sm);
            double tt;
            if (!grid.sum(SL_TT, &tt)) return;
            if (sqrt(tt) <= target) {
                status = CFM_OK;
                gamma0 = gamma1;
                break;
            }
            phase_restart(a);
            ++restarts;
            gamma0 = tt;
            if (!grid.barrier()) return;
            continue;
        }
        const double beta = gamma1 / gamma0;
        if (use_tol && !isfinite(beta)) {
            status = CFM_BREAKDOWN;
            break;
        }
        phase_p(a, beta);
        if (!grid.barrier()) return;
        gamma0 = gamma1;
    }
    write_result(a.res, k, status, restarts, gamma0, bnorm);
}

// ------------------------------------------------------- pipelined phases
// r0 = b - A x0 with x0 = 0 (into t), and ||b||^2.
template <class Op>
__device__ void phase_pipe_init(const KArgs<Op> &a, double *sm) {
    TileSums<1> ts(sm, gridDim.x, slot(a, SL_B));
    CFM_TILES(a) {
        CFM_ROW(a);
        double bb = 0.0;
        if (i < a.n) {
            const double bi = a.b ? a.b[i] : 1.0;
            a.x[i] = 0.0;
            a.t[i] = __fma_rn(-1.0, a.op.apply_zero(i), bi);
            bb = __dmul_rn(bi, bi);
        }
        ts.add(tile, bb);
    }
    ts.flush();
}

// r = v, w = A v, z = s = p = 0; partials <r, r> -> G[par], <w, r> -> D[par].
// v is the initial residual, or the true residual t at a restart.
template <class Op>
__device__ void phase_pipe_start(const KArgs<Op> &a, const double *v, double *w, int par,
                                 double *sm) {
    TileSums<2> ts(sm, gridDim.x, slot(a, par ? SL_G1 : SL_G0), slot(a, par ? SL_D1 : SL_D0));
    CFM_TILES(a) {
        CFM_ROW(a);
        double g = 0.0, d = 0.0;
        if (i < a.n) {
            const double ri = v[i];
            const double wi = a.op.apply(v, i);
            a.r[i] = ri;
            w[i] = wi;
            a.z[i] = 0.0;
            a.s[i] = 0.0;
            a.p[i] = 0.0;
            g = __dmul_rn(ri, ri);
            d = __dmul_rn(wi, ri);
        }
        ts.add(tile, g, d);
    }
    ts.flush();
}

// One pipelined iteration, row-local once q = A w is known:
//   z = q + beta z; s = w + beta s; p = r + beta p
//   x += alpha p; r -= alpha s; w' = w - alpha z
// and the next iteration's partials <r', r'>, <w', r'> into slot parity `nxt`.
template <class Op>
__device__ void phase_pipe_step(const KArgs<Op> &a, const double *w, double *wn, double alpha,
                                double beta, int nxt, double *sm) {
    TileSums<2> ts(sm, gridDim.x, slot(a, nxt ? SL_G1 : SL_G0), slot(a, nxt ? SL_D1 : SL_D0));
    CFM_TILES(a) {
        CFM_ROW(a);
        double g = 0.0, d = 0.0;
        if (i < a.n) {
            // ROW_FIRST: the row's own entries are in flight while the operator's chain of
            // loads runs
            double wi, z0, s0, p0, r0, x0, q;
            if (!Op::ROW_FIRST) q = a.op.apply(w, i);
            wi = w[i], z0 = a.z[i], s0 = a.s[i], p0 = a.p[i], r0 = a.r[i], x0 = a.x[i];
            if (Op::ROW_FIRST) q = a.op.apply(w, i);
            const double zi = __fma_rn(beta, z0, q);
            const double si = __fma_rn(beta, s0, wi);
            const double pi = __fma_rn(beta, p0, r0);
            a.x[i] = __fma_rn(alpha, pi, x0);
            const double ri = __fma_rn(-alpha, si, r0);
            const double wni = __fma_rn(-alpha, zi, wi);
            a.z[i] = zi;
            a.s[i] = si;
            a.p[i] = pi;
            a.r[i] = ri;
            wn[i] = wni;
            g = __dmul_rn(ri, ri);
            d = __dmul_rn(wni, ri);
        }
        ts.add(tile, g, d);
    }
    ts.flush();
}

// Residual replacement, first half: t = b - A x, s = A p.
template <class Op>
__device__ void phase_replace_a(const KArgs<Op> &a) {
    CFM_TILES(a) {
        CFM_ROW(a);
        if (i < a.n) {
            const double bi = a.b ? a.b[i] : 1.0;
            a.t[i] = __dsub_rn(bi, a.op.apply(a.x, i));
            a.s[i] = a.op.apply(a.p, i);
        }
    }
}

// Residual replacement, second half: r = t, w = A t, z = A s and the
// partials <r, r> -> G[par], <w, r> -> D[par].
template <class Op>
__device__ void phase_replace_b(const KArgs<Op> &a, double *w, int par, double *sm) {
    TileSums<2> ts(sm, gridDim.x, slot(a, par ? SL_G1 : SL_G0), slot(a, par ? SL_D1 : SL_D0));
    CFM_TILES(a) {
        CFM_ROW(a);
        double g = 0.0, d = 0.0;
        if (i < a.n) {
            const double ri = a.t[i];
            const double wi = a.op.apply(a.t, i);
            a.r[i] = ri;
            w[i] = wi;
            a.z[i] = a.op.apply(a.s, i);
            g = __dmul_rn(ri, ri);
            d = __dmul_rn(wi, ri);
        }
        ts.add(tile, g, d);
    }
    ts.flush();
}

// Iterations between residual replacements in pipelined CG.
constexpr long long PIPE_REPLACE = 50;

// Pipelined CG.  Scalars follow the reference's recurrence
// (CG/src/single-stream/pipelined.cu:262-272): with rr = <r, r>, wr = <w, r>,
//   beta = rr / rr_prev, alpha = rr / (wr - (beta / alpha_prev) rr)
// from the third step of a run on, and beta = 0, alpha = rr / wr on the
// first two (the reference tests `k > 1`).  Convergence as cg_std_kernel.
// The pipelined recurrences let the recursive residual drift from b - A x on
// ill-conditioned systems, so with tol > 0 every PIPE_REPLACE iterations the
// vectors r, w, s, z are recomputed from x and p (residual replacement: two
// extra barriers, four operator applications); the scalar recurrence goes on.
template <class Op>
__global__ void __launch_bounds__(CG_TILE, 1) cg_pipe_kernel(KArgs<Op> a) {
    __shared__ double sm[TS_SMEM], red[128];
    CgGrid<Op> grid(a, red);
    phase_pipe_init(a, sm);
    double bb;
    if (!grid.sum(SL_B, &bb)) return;
    const double bnorm = sqrt(bb);
    phase_pipe_start(a, a.t, a.w0, 0, sm);
    const bool use_tol = a.tol > 0.0;
    const double target = a.tol * bnorm;
    int status = use_tol ? CFM_NOT_CONVERGED : CFM_OK;
    int restarts = 0, cur = 0;
    long long k = 0, kk = 0, replaced = -1;
    double rr = 0.0, rr_prev = 0.0, alpha = 0.0;
    while (true) {
        double *w = cur ? a.w1 : a.w0;
        double wr;
        if (!grid.sum2(cur ? SL_G1 : SL_G0, &rr, cur ? SL_D1 : SL_D0, &wr)) return;
        if (use_tol && sqrt(rr) <= target) {
            phase_true_residual(a, sm);
            double tt;
            if (!grid.sum(SL_TT, &tt)) return;
            if (sqrt(tt) <= target) {
                status = CFM_OK;
                break;
            }
            phase_pipe_start(a, a.t, w, cur, sm);  // restart from the true residual
            ++restarts;
            kk = 0;
            replaced = k;  // a restart needs no replacement at this count
            continue;
        }
        if (k >= a.maxiter) break;
        if (use_tol && k > 0 && k % PIPE_REPLACE == 0 && replaced != k) {
            phase_replace_a(a);
            if (!grid.barrier()) return;
            phase_replace_b(a, w, cur, sm);
            replaced = k;
            ++restarts;
            continue;
        }
        double beta;
        if (kk > 1) {
            beta = rr / rr_prev;
            alpha = rr / __dsub_rn(wr, __dmul_rn(beta / alpha, rr));
        } else {
            beta = 0.0;
            alpha = rr / wr;
        }
        if (use_tol && !(isfinite(alpha) && alpha > 0.0 && isfinite(beta))) {
            status = CFM_BREAKDOWN;
            break;
        }
        phase_pipe_step(a, w, cur ? a.w0 : a.w1, alpha, beta, cur ^ 1, sm);
        rr_prev = rr;
        cur ^= 1;
        ++k;
        ++kk;
    }
    write_result(a.res, k, status, restarts, rr, bnorm);
}

// ----------------------------------------------------------- mixed phases
// x = 0, t = b - A x0, partials ||t||^2 (SL_TT) and ||b||^2 (SL_B).
template <class Op>
__device__ void phase_mixed_init(const KArgs<Op> &a, double *sm) {
    TileSums<2> ts(sm, gridDim.x, slot(a, SL_TT), slot(a, SL_B));
    CFM_TILES(a) {
        CFM_ROW(a);
        double q = 0.0, bb = 0.0;
        if (i < a.n) {
            const double bi = a.b ? a.b[i] : 1.0;
            const double ti = __fma_rn(-1.0, a.op.apply_zero(i), bi);
            a.x[i] = 0.0;
            a.t[i] = ti;
            q = __dmul_rn(ti, ti);
            bb = __dmul_rn(bi, bi);
        }
        ts.add(tile, q, bb);
    }
    ts.flush();
}

// Start of the FP32 iteration: r32 = fl32(t * scale), p32 = r32, d32 = 0;
// <r32, r32> -> G0.
template <class Op>
__device__ void phase_inner_start(const KArgs<Op> &a, double scale, double *sm) {
    TileSums<1> ts(sm, gridDim.x, slot(a, SL_G0));
    CFM_TILES(a) {
        CFM_ROW(a);
        double g = 0.0;
        if (i < a.n) {
            const float ri = __double2float_rn(__dmul_rn(a.t[i], scale));
            a.r32[i] = ri;
            a.p32[i] = ri;
            a.d32[i] = 0.f;
            g = xprod(ri, ri);
        }
        ts.add(tile, g);
    }
    ts.flush();
}

// The FP32 passes load a group's own values while the group before it is worked on:
// a block has few groups (seven at 128^3), and each otherwise waits out a round trip.
template <class Op>
__device__ void phase_inner_spmv(const KArgs<Op> &a, double *sm) {
    constexpr int U = INNER_U;
    TileSums<1> ts(sm, gridDim.x, slot(a, SL_D0));
    float p[U];
    int key[U];
    auto load = [&](const TileGroup<U> &g, float (&pv)[U], int (&kv)[U]) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            pv[u] = g.ok[u] ? a.p32[g.row[u]] : 0.f;
            kv[u] = g.ok[u] ? a.op.key(g.row[u]) : 0;
        }
    };
    load(TileGroup<U>(a.ntiles, a.n, blockIdx.x), p, key);
    CFM_TILE_GROUPS(a, U) {
        const TileGroup<U> g(a.ntiles, a.n, tile);
        float pn[U];
        int kn[U];
        load(TileGroup<U>(a.ntiles, a.n, tile + U * (int)gridDim.x), pn, kn);
        const Vals32<U> y = a.op.template applyN32<U>(a.p32, g, key);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (g.ok[u]) a.s32[g.row[u]] = y.v[u];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (g.has[u]) ts.add(g.tile[u], g.ok[u] ? xprod(p[u], y.v[u]) : 0.0);
#pragma unroll
        for (int u = 0; u < U; ++u) p[u] = pn[u], key[u] = kn[u];
    }
    ts.flush();
}

template <class Op>
__device__ void phase_inner_update(const KArgs<Op> &a, float af, double *sm) {
    constexpr int U = INNER_U;
    TileSums<1> ts(sm, gridDim.x, slot(a, SL_G0));
    struct Own {
        float d[U], p[U], r[U], s[U];
    } cur, nxt;
    auto load = [&](const TileGroup<U> &g, Own &v) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            v.d[u] = v.p[u] = v.r[u] = v.s[u] = 0.f;
            if (g.ok[u]) {
                v.d[u] = a.d32[g.row[u]];
                v.p[u] = a.p32[g.row[u]];
                v.r[u] = a.r32[g.row[u]];
                v.s[u] = a.s32[g.row[u]];
            }
        }
    };
    load(TileGroup<U>(a.ntiles, a.n, blockIdx.x), cur);
    CFM_TILE_GROUPS(a, U) {
        const TileGroup<U> g(a.ntiles, a.n, tile);
        load(TileGroup<U>(a.ntiles, a.n, tile + U * (int)gridDim.x), nxt);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            double q = 0.0;
            if (g.ok[u]) {
                a.d32[g.row[u]] = __fmaf_rn(af, cur.p[u], cur.d[u]);
                const float ri = __fmaf_rn(-af, cur.s[u], cur.r[u]);
                a.r32[g.row[u]] = ri;
                q = xprod(ri, ri);
            }
            if (g.has[u]) ts.add(g.tile[u], q);
        }
        cur = nxt;
    }
    ts.flush();
}

template <class Op>
__device__ void phase_inner_p(const KArgs<Op> &a, float bf) {
    constexpr int U = 2 * INNER_U;
    CFM_TILE_GROUPS(a, U) {
        const TileGroup<U> g(a.ntiles, a.n, tile);
        float p[U], r[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            p[u] = r[u] = 0.f;
            if (g.ok[u]) {
                p[u] = a.p32[g.row[u]];
                r[u] = a.r32[g.row[u]];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (g.ok[u]) a.p32[g.row[u]] = __fmaf_rn(bf, p[u], r[u]);
    }
}

// Reliable update, first half: x += |b| d32 in FP64, d32 = 0.
template <class Op>
__device__ void phase_correct(const KArgs<Op> &a, double norm) {
    CFM_TILES(a) {
        CFM_ROW(a);
        if (i < a.n) {
            a.x[i] = __fma_rn(norm, (double)a.d32[i], a.x[i]);
            a.d32[i] = 0.f;
        }
    }
}

// Reliable update, second half: t = b - A x (FP64) with |t|^2 -> TT, and
// r32 = fl32(t / |b|) with <r32, r32> -> G0.
template <class Op>
__device__ void phase_replace32(const KArgs<Op> &a, double scale, double *sm) {
    TileSums<2> ts(sm, gridDim.x, slot(a, SL_TT), slot(a, SL_G0));
    CFM_TILES(a) {
        CFM_ROW(a);
        double q = 0.0, g = 0.0;
        if (i < a.n) {
            const double bi = a.b ? a.b[i] : 1.0;
            const double ti = __dsub_rn(bi, a.op.apply(a.x, i));
            const float ri = __double2float_rn(__dmul_rn(ti, scale));
            a.t[i] = ti;
            a.r32[i] = ri;
            q = __dmul_rn(ti, ti);
            g = xprod(ri, ri);
        }
        ts.add(tile, q, g);
    }
    ts.flush();
}

// Mixed-precision CG with reliable updates.  The iteration runs in FP32
// (FP32 SpMV and axpys; the dots are FP64 sums of the exact FP32 products;
// alpha, beta in FP64, applied rounded to FP32) on r32 = fl32(r / |b|) and
// gathers its steps in an FP32 correction d32.  When <r32, r32> falls to
// tol^2, below inner_tol^2 times its largest value since the last update,
// or after inner_maxiter steps (0: no cap), a reliable update adds |b| d32
// to x in FP64 and replaces r32 by fl32((b - A x) / |b|) from the FP64 true
// residual; the search direction p32 is kept, so the recurrence goes on
// (beta from the replaced residual) instead of restarting (Sleijpen and van
// der Vorst's reliable updated residuals).  Stops when the FP64 true
// residual |b - A x| <= tol |b|; maxiter caps the FP32 steps.
template <class Op>
__global__ void __launch_bounds__(CG_TILE, 1) cg_mixed_kernel(KArgs<Op> a) {
    __shared__ double sm[TS_SMEM], red[128];
    CgGrid<Op> grid(a, red);
    phase_mixed_init(a, sm);
    double bb, tt;
    if (!grid.sum2(SL_B, &bb, SL_TT, &tt)) return;
    const double bnorm = sqrt(bb);
    const double target = a.tol * bnorm;
    int status = CFM_NOT_CONVERGED, updates = 0;
    long long k = 0;
    if (sqrt(tt) <= target || bnorm == 0.0) {
        write_result(a.res, 0, sqrt(tt) <= target ? CFM_OK : CFM_NOT_CONVERGED, 0, tt, bnorm);
        return;
    }
    const double scale = 1.0 / bnorm, tol2 = a.tol * a.tol;
    const double delta2 = a.inner_tol * a.inner_tol;
    phase_inner_start(a, scale, sm);
    double g0;
    if (!grid.sum(SL_G0, &g0)) return;
    double gmax = g0;
    int since = 0;
    while (k < a.maxiter) {
        phase_inner_spmv(a, sm);
        double delta;
        if (!grid.sum(SL_D0, &delta)) return;
        const double alpha = g0 / delta;
        if (!(delta > 0.0 && isfinite(alpha))) {
            status = CFM_BREAKDOWN;
            break;
        }
        phase_inner_update(a, __double2float_rn(alpha), sm);
        double g1;
        if (!grid.sum(SL_G0, &g1)) return;
        ++k;
        ++since;
        if (g1 <= tol2 || g1 < delta2 * gmax || k >= a.maxiter ||
            (a.inner_maxiter > 0 && since >= a.inner_maxiter)) {
            phase_correct(a, bnorm);
            if (!grid.barrier()) return;
            phase_replace32(a, scale, sm);
            if (!grid.sum2(SL_TT, &tt, SL_G0, &g1)) return;
            ++updates;
            since = 0;
            gmax = g1;
            if (sqrt(tt) <= target) {
                status = CFM_OK;
                break;
            }
            if (k >= a.maxiter) break;
        } else if (g1 > gmax) {
            gmax = g1;
        }
        const double beta = g1 / g0;
        phase_inner_p(a, __double2float_rn(beta));
        if (!grid.barrier()) return;
        g0 = g1;
    }
    if (since > 0) phase_correct(a, bnorm);  // a breakdown left steps in d32
    write_result(a.res, k, status, updates, tt, bnorm);
}

// ------------------------------------------------ host-controlled pieces
// One kernel per operation (the comparator of CG/src/common.cu:458-531).
template <class Op>
__global__ void __launch_bounds__(CG_TILE) k_init(KArgs<Op> a) {
    __shared__ double sm[TS_SMEM];
    phase_init(a, sm);
}
template <class Op>
__global__ void __launch_bounds__(CG_TILE) k_spmv_dot(KArgs<Op> a) {
    __shared__ double sm[TS_SMEM];
    phase_spmv_dot(a, sm);
}
template <class Op>
__global__ void __launch_bounds__(CG_TILE) k_update(KArgs<Op> a, double alpha) {
    __shared__ double sm[TS_SMEM];
    phase_update(a, alpha, sm);
}
template <class Op>
__global__ void __launch_bounds__(CG_TILE) k_true_residual(KArgs<Op> a) {
    __shared__ double sm[TS_SMEM];
    phase_true_residual(a, sm);
}
template <class Op>
__global__ void __launch_bounds__(CG_TILE) k_restart(KArgs<Op> a) {
    phase_restart(a);
}
template <class Op>
__global__ void __launch_bounds__(CG_TILE) k_p(KArgs<Op> a, double beta) {
    phase_p(a, beta);
}
// Single block: reduce partial slot `which` into out[which].
template <class Op>
__global__ void __launch_bounds__(CG_TILE) k_reduce(KArgs<Op> a, int which, double *out) {
    __shared__ double sm[TS_SMEM];
    const double v = sum_partials(slot(a, which), a.ntiles, sm);
    if (threadIdx.x == 0) out[which] = v;
}

// y = A x, one row per thread.
template <class Op>
__global__ void k_apply(Op op, int n, const double *x, double *y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = op.apply(x, i);
}

#undef CFM_TILES
#undef CFM_ROW

}  // namespace cfm

// 3D 7-point sweeps, two per pass over global memory.
//
// One sweep at a time is bound by HBM: 16 bytes (FP64) or 8 (FP32) per cell and
// sweep, at 512^3 FP64 0.78 to 0.90 of the copy rate.  Here a pass reads and
// writes the grid once for two sweeps.
//
// Work unit: a tile of 32 V columns by CW R rows (one 16-byte vector of V columns per
// lane, R rows per consumer warp) over a chunk of z planes, the outermost two
// rows and the outermost vector of columns on either inner side overlapping
// the neighbouring tiles.  A producer warp copies the planes of the unit, one after the
// other, into a ring of S shared-memory stages: one tensor copy (TMA) per plane, or
// cp.async row by row where the window wraps around in y or the rows are not a multiple
// of 16 bytes (the first form of this kernel, 512^3 FP64, 100 sweeps: 30.4 ms with every plane by
// cp.async, 29.1 with the tensor copies); rows and planes wrap as
// the periodic images do, so the halo planes (and rows, with PY) are read only by the
// single sweeps.  Consumer warps march along z with everything they own in
// registers: as plane s arrives, sweep 1 makes plane s - 1 from the planes s - 2,
// s - 1, s, and sweep 2 makes plane s - 2 from sweep 1's planes s - 3, s - 2, s - 1.
// Five register planes rotate through these roles (five steps unrolled, no
// moves).  x neighbours come by shuffle; the rows above and below a warp come from
// the ring for sweep 1, and for sweep 2 from a small exchange in shared memory,
// published one step before it is read, with waits on the two adjacent warps
// only.
//
// 512^3, 100 sweeps on B200, the best one-sweep shape against this: FP64 36.8 to 41 ms, now
// 26.8 (495 GLUP/s, 4.0 TB/s: 0.62 of the measured copy); FP32 20.6, now 17.3 (767 GLUP/s).
// What bounds it now is the consumers' latency: eight warps, two per scheduler, at 1.6
// instructions per clock and SM, waiting on fixed latencies and shared memory.  168
// registers per thread (three warps to one scheduler) leave no room for more warps of this
// shape; two blocks per SM at 96 registers spill or overlap too much (8 x 2 rows 33.1 ms,
// 8 x 3 38.5, 8 x 4 61.8).
//
// Overlap cells are computed from the same inputs by the same operations as by
// their owners, so the grid is the one-sweep grid bit for bit
// (Stencil/jacobi3D/src/common.cu:31-57).  The first sweep of a run runs alone, since
// it reads the halo planes as they are (they need not be images yet), and so
// does the last one of an odd rest.
#pragma once

#include <type_traits>

#include "j2d_temporal.cuh"
#include "tma.cuh"

namespace cfm {

template <typename T, int CW, int R, int S>
struct J3PairGeom {
    static constexpr int V = 16 / sizeof(T), W = 32 * V, ROWS = CW * R;
    static constexpr int OX = W - 2 * V, OY = ROWS - 4;  // own columns (inner tiles) and rows
    static constexpr size_t STAGE = (size_t)ROWS * W * sizeof(T);
    static constexpr size_t EDGES = (size_t)4 * CW * 2 * 32 * 16;  // 4 steps x warp x (first, last)
    static constexpr size_t SMEM = S * STAGE + EDGES + sizeof(uint64_t) * (2 * S + 4 * CW) + 16;
};

// Tiles in x: the first has no overlap on its left.  Tiles in y: even split.
template <typename G>
__host__ __device__ inline int j3p_tiles_x(int nx) {
    return nx <= G::W ? 1 : 1 + (nx - (G::W - G::V) + G::OX - 1) / G::OX;
}
template <typename G>
__host__ __device__ inline int j3p_tiles_y(int ny) {
    return (ny - 2 + G::OY - 1) / G::OY;
}

template <typename T>
struct J3Op;
template <>
struct J3Op<double> : J2Op<double> {
    static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
};
template <>
struct J3Op<float> : J2Op<float> {
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
};

// One row of a sweep in a lane's V columns: c the row, n / s the rows at y+1 / y-1, t / b
// the planes z+1 / z-1.  EDGE: some cells of the window are fixed.
template <typename T, int V, bool EDGE>
__device__ __forceinline__ void j3_row(const T (&c)[V], const T (&n)[V], const T (&s)[V], const T (&t)[V],
                                       const T (&b)[V], const J2Edge &ed, bool fixed_row, T (&o)[V]) {
    using O = J3Op<T>;
    const T w0 = __shfl_up_sync(J2_FULL, c[V - 1], 1);
    const T eV = __shfl_down_sync(J2_FULL, c[0], 1);
    const T c6 = T(1) / T(6);
#pragma unroll
    for (int j = 0; j < V; ++j) {
        const T e = j + 1 < V ? c[j + 1 < V ? j + 1 : 0] : eV;
        const T w = j > 0 ? c[j > 0 ? j - 1 : 0] : w0;
        T v = O::mul(c6, O::add(O::add(O::add(O::add(O::add(e, w), n[j]), s[j]), t[j]), b[j]));
        if (EDGE && (fixed_row || j == ed.first || j == ed.last)) v = c[j];
        o[j] = v;
    }
}

// A consumer warp's view of the block's ring and of its current work unit.  VEC: rows are a
// multiple of 16 bytes.
template <typename T, int CW, int R, int S, bool PY, bool VEC>
struct J3PairWarp {
    using G = J3PairGeom<T, CW, R, S>;
    static constexpr int V = G::V, ROWS = G::ROWS;
    using Plane = T[R][V];
    using Row = T[V];

    float4 (*ring)[ROWS][32];
    float4 (*edge)[CW][2][32];
    uint64_t *full, *empty, *ready;  // ready[step & 3][warp]
    BarrierState *bar;
    unsigned long long budget;
    int lane, warp, nx, ny, nz;
    int slot, prev;  // ring stages of the next plane and the one before it
    unsigned turn;   // parity of the turns around the ring so far
    unsigned steps;  // two-sweep steps so far
    bool ok;  // (rows that are not a multiple of 16 bytes) no wait has run out
    // the unit
    T *out;
    int x0, ya, h, zb;
    bool own;
    J2Edge ed;

    // Set once a wait of a block has run out for good.
    __device__ __forceinline__ static int &dead() {
        __shared__ int d;
        return d;
    }
    __device__ __forceinline__ void wait(uint64_t *b, unsigned parity) {
        if (!VEC) {
            // after a timeout nothing waits any more and the next grid barrier, before which the
            // producer's cp.async have landed, ends the run
            if (ok && !mbar_wait_bounded(b, parity, budget)) {
                ok = false;
                if (atomicCAS(&bar->error, 0, 1) == 0) bar->where = (int)steps;
            }
            return;
        }
        // A wait beyond its budget is an error, which ends the run at the next grid barrier, but goes
        // on (bounded): no stage may be handed on, and the block may not give up its shared memory,
        // while a tensor copy into it is in flight.  All of it in one loop and without a flag in a
        // register: this stands fifteen times in the march, where instructions and registers are
        // short (512^3, 100 sweeps, ms: an `ok` that every wait tests, as above, FP64 27.75, FP32 17.5; this
        // 26.8 and 17.3; waiting on in a second loop 28.1 and 19.8, in a call 28.9 and 17.5).
        if (mbar_try_wait(b, parity)) return;
        const unsigned long long t0 = global_ns();
        while (!mbar_try_wait(b, parity)) {
            const unsigned long long t = global_ns() - t0;
            if (t <= budget) continue;
            *(volatile int *)&bar->where = (int)steps;
            *(volatile int *)&bar->error = 1;
            if (t > budget + DRAIN_NS || *(volatile int *)&dead()) {
                dead() = 1;
                return;
            }
        }
    }
    __device__ __forceinline__ static void unpack(const float4 &t, Row &v) {
        const T *e = reinterpret_cast<const T *>(&t);
#pragma unroll
        for (int j = 0; j < V; ++j) v[j] = e[j];
    }
    __device__ __forceinline__ void give(int side, const Row &v) {
        float4 t;
        T *e = reinterpret_cast<T *>(&t);
#pragma unroll
        for (int j = 0; j < V; ++j) e[j] = v[j];
        edge[steps & 3][warp][side][lane] = t;
    }
    // Row r of the warp at p (the lane's first column of its row 0); the images are
    // written at the end of the run.
    __device__ __forceinline__ void store(T *p, int r, const Row &o) const {
        const int l = warp * R + r;
        if (l < 2 || l >= h + 2 || !own) return;
        p += (size_t)r * nx;
        if (VEC) {
            float4 t;
            T *e = reinterpret_cast<T *>(&t);
#pragma unroll
            for (int j = 0; j < V; ++j) e[j] = o[j];
            *reinterpret_cast<float4 *>(p) = t;
        } else {
#pragma unroll
            for (int j = 0; j < V; ++j)
                if (x0 + j < nx) p[j] = o[j];
        }
    }
    __device__ __forceinline__ T *target(int z) const {
        return out + ((ptrdiff_t)z * ny + (ya - 2 + warp * R)) * nx + x0;
    }
    // Row r of the plane after one sweep, from the planes a, b (its own), c.
    template <bool EDGE>
    __device__ __forceinline__ void row(int r, const Plane &a, const Plane &b, const Plane &c, const Row &up,
                                        const Row &dn, Row &o) const {
        const int y = ya - 2 + warp * R + r;
        const bool fixed = EDGE && !PY && (y <= 0 || y >= ny - 1);
        if (r == 0)
            j3_row<T, V, EDGE>(b[0], b[1], up, c[0], a[0], ed, fixed, o);
        else if (r == R - 1)
            j3_row<T, V, EDGE>(b[R - 1], dn, b[R - 2], c[R - 1], a[R - 1], ed, fixed, o);
        else
            j3_row<T, V, EDGE>(b[r], b[r + 1 < R ? r + 1 : r], b[r > 0 ? r - 1 : r], c[r], a[r], ed, fixed, o);
    }
    // Ring row beside the warp (above, or below) of the plane before the newest.
    __device__ __forceinline__ void beside(bool first, bool below, Row &v) const {
        if (first) {  // the unit's first plane has none: what is computed from it is not used
#pragma unroll
            for (int j = 0; j < V; ++j) v[j] = T(0);
            return;
        }
        const int l = below ? min(warp * R + R, ROWS - 1) : max(warp * R - 1, 0);
        unpack(ring[prev][l][lane], v);
    }
    // The stage of the plane before the newest is done with.
    __device__ __forceinline__ void release(bool first) {
        if (VEC) fence_proxy_async_shared();  // the reads of the stage before the next tensor copy
        __syncwarp();
        if (!first && lane == 0) mbar_arrive(&empty[prev]);
        next();
    }
    __device__ __forceinline__ void next() {
        prev = slot;
        if (++slot == S) {
            slot = 0;
            turn ^= 1;
        }
    }
    // One sweep: plane s in, plane s - 1 out.
    __device__ __forceinline__ void single(int s, Plane &a, Plane &b, Plane &c) {
        const bool first = s == zb - 1;
        wait(&full[slot], turn);
        T *p = target(s - 1);
        Row up, dn;
        beside(first, false, up);
        beside(first, true, dn);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            unpack(ring[slot][warp * R + r][lane], c[r]);
            Row o;
            row<true>(r, a, b, c, up, dn, o);
            if (s - 1 >= zb) store(p, r, o);
        }
        release(first);
    }
    // Two sweeps: plane s into c; sweep 1's plane s - 1, from a, b, c, takes the place of
    // plane s - 2 in a; sweep 2's plane s - 2, from sweep 1's planes d, e, a, goes out.
    // Row by row, so that four planes and a few rows are live at a time.
    template <bool EDGE>
    __device__ __forceinline__ void twice(int s, Plane &a, Plane &b, Plane &c, Plane &d, Plane &e) {
        const bool first = s == zb - 2, emit = s - 2 >= zb;
        wait(&full[slot], turn);
        T *out_row = target(s - 2);
        // The neighbour warps' outer rows of sweep 1's plane s - 2, from their last step.
        // Every step waits for that step of theirs, so adjacent warps are never two
        // steps apart: of the four copies and mbarriers no two in use coincide.
        const unsigned p = steps - 1;
        const int wu = warp > 0 ? warp - 1 : 0, wd = warp + 1 < CW ? warp + 1 : CW - 1;
        if (steps > 0) {
            wait(&ready[(p & 3) * CW + wu], (p >> 2) & 1);
            wait(&ready[(p & 3) * CW + wd], (p >> 2) & 1);
        }
        Row up0, dn0, up1, dn1;
        beside(first, false, up0);
        unpack(edge[p & 3][wu][1][lane], up1);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            unpack(ring[slot][warp * R + r][lane], c[r]);
            if (r == R - 1) {
                beside(first, true, dn0);
                unpack(edge[p & 3][wd][0][lane], dn1);
            }
            row<EDGE>(r, a, b, c, up0, dn0, a[r]);
            Row o;
            row<EDGE>(r, d, e, a, up1, dn1, o);
            if (emit) store(out_row, r, o);
        }
        give(0, a[0]);
        give(1, a[R - 1]);
        release(first);  // (its __syncwarp also orders the rows given above)
        if (lane == 0) mbar_arrive(&ready[(steps & 3) * CW + warp]);
        ++steps;
    }
    __device__ __forceinline__ void march1(int ze, Plane (&q)[5]) {
#pragma unroll 1
        for (int s = zb - 1; s < ze + 1; s += 3) {
            single(s, q[0], q[1], q[2]);
            if (s + 1 < ze + 1) single(s + 1, q[1], q[2], q[0]);
            if (s + 2 < ze + 1) single(s + 2, q[2], q[0], q[1]);
        }
    }
    template <bool EDGE>
    __device__ __forceinline__ void march2(int ze, Plane (&q)[5]) {
#pragma unroll 1
        for (int s = zb - 2; s < ze + 2; s += 5) {
            twice<EDGE>(s, q[0], q[1], q[2], q[3], q[4]);
            if (s + 1 < ze + 2) twice<EDGE>(s + 1, q[1], q[2], q[3], q[4], q[0]);
            if (s + 2 < ze + 2) twice<EDGE>(s + 2, q[2], q[3], q[4], q[0], q[1]);
            if (s + 3 < ze + 2) twice<EDGE>(s + 3, q[3], q[4], q[0], q[1], q[2]);
            if (s + 4 < ze + 2) twice<EDGE>(s + 4, q[4], q[0], q[1], q[2], q[3]);
        }
    }
};

template <typename T, int CW, int R, int S, bool PY, bool VEC>
__global__ void __launch_bounds__(32 * (CW + 1), 1)
    j3d_pair_kernel(const __grid_constant__ CUtensorMap map0, const __grid_constant__ CUtensorMap map1, T *g0, T *g1,
                    int nx, int ny, int nz, int niter, int zchunk, BarrierState *bar) {
    using G = J3PairGeom<T, CW, R, S>;
    constexpr int V = G::V, W = G::W;
    extern __shared__ __align__(128) unsigned char j3p_smem[];
    J3PairWarp<T, CW, R, S, PY, VEC> w;
    w.ring = reinterpret_cast<float4(*)[G::ROWS][32]>(j3p_smem);
    w.edge = reinterpret_cast<float4(*)[CW][2][32]>(j3p_smem + S * G::STAGE);
    w.full = reinterpret_cast<uint64_t *>(j3p_smem + S * G::STAGE + G::EDGES);
    w.empty = w.full + S;
    w.ready = w.empty + S;
    w.bar = bar;
    w.budget = bar->timeout_ns;
    w.lane = threadIdx.x & 31;
    w.warp = threadIdx.x >> 5;
    w.nx = nx;
    w.ny = ny;
    w.nz = nz;
    w.slot = 0;
    w.prev = S - 1;
    w.turn = w.steps = 0;
    w.ok = true;
    const bool producer = w.warp == CW;
    const size_t plane = (size_t)nx * ny;
    const int PZ = nz - 2, PR = ny - 2;  // periods of the planes and (PY) rows
    const int ntx = j3p_tiles_x<G>(nx), nty = j3p_tiles_y<G>(ny);
    const int nch = (PZ + zchunk - 1) / zchunk;
    const long long units = (long long)ntx * nty * nch;
    if (threadIdx.x == 0) {
        for (int i = 0; i < S; ++i) {
            mbar_init(&w.full[i], 32);
            mbar_init(&w.empty[i], CW);
        }
        for (int i = 0; i < 4 * CW; ++i) mbar_init(&w.ready[i], 1);
        w.dead() = 0;
        mbar_fence_init();
    }
    __syncthreads();

    T q[5][R][V];  // the planes in registers; their roles rotate
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int j = 0; j < V; ++j) q[i][r][j] = T(0);
    int filled = 0;  // producer: stages that have been filled at least once
    T *in = g0, *out = g1;
    int site = 0;
    for (int left = niter; left > 0; ++site) {
        // this pass's tensor copies after the stores of the last (and of earlier kernels)
        if (producer) fence_proxy_async_global();
        const bool pair = site > 0 && left >= 2;
        const int H = pair ? 2 : 1;  // planes (and, of the two overlap rows, rows) around the unit that feed it
        for (long long u = blockIdx.x; u < units; u += gridDim.x) {
            const int ch = (int)(u / (ntx * nty)), tile = (int)(u - (long long)ch * ntx * nty);
            const int tx = tile % ntx, ty = tile / ntx;
            const int xa = tx == 0 ? 0 : (W - V) + (tx - 1) * G::OX;
            const int xb = tx + 1 == ntx ? nx : (W - V) + tx * G::OX;
            const int xs = tx == 0 ? 0 : xa - V, x0 = xs + w.lane * V;
            const int ya = 1 + (int)((long long)ty * PR / nty);
            const int h = 1 + (int)((long long)(ty + 1) * PR / nty) - ya;
            const int zb = 1 + ch * zchunk, ze = min(PZ + 1, zb + zchunk);
            if (producer) {
                // window row l is grid row ya - 2 + l; off-grid columns read as 0
                const bool on = x0 < nx;
                const size_t pitch = on ? nx : 0;
                // rows of 16-byte multiples that do not wrap come as one tensor copy per plane
                const bool box = VEC && (site == 0 || !PY || (ya > 2 && ya + h + 1 <= PR));
                const CUtensorMap *map = in == g0 ? &map0 : &map1;
                for (int s = zb - H; s < ze + H; ++s, w.next()) {
                    const int slot = w.slot;
                    if (filled >= S) w.wait(&w.empty[slot], w.turn ^ 1);
                    filled = min(filled + 1, S);
                    int z = s;
                    if (site > 0) {  // ring of the planes 1 .. nz-2
                        z = (s - 1) % PZ;
                        z = (z < 0 ? z + PZ : z) + 1;
                    }
                    if (box) {
                        if (w.lane == 0) {
                            mbar_arrive_expect_tx(&w.full[slot], (unsigned)G::STAGE);
                            tma_load_3d(&w.ring[slot][0][0], map, xs, ya - 2, z, &w.full[slot]);
                        } else {
                            mbar_arrive(&w.full[slot]);
                        }
                        continue;
                    }
                    int l = 2 - H, y = ya - 2 + l, end = h + 2 + H;
                    if (PY && site > 0) {
                        y = (y - 1) % PR;
                        y = (y < 0 ? y + PR : y) + 1;
                    } else {
                        if (y < 0) l -= y, y = 0;
                        end = min(end, l + ny - y);
                    }
                    // runs of rows that follow one another in memory (one, but for the wrap)
                    while (l < end) {
                        const int n = PY && site > 0 ? min(end - l, PR + 1 - y) : end - l;
                        const T *p = on ? in + (size_t)z * plane + (size_t)y * nx + x0 : in;
                        uint32_t d = smem_u32(&w.ring[slot][l][w.lane]);
                        if (VEC) {
#pragma unroll 8
                            for (int r = 0; r < n; ++r, p += pitch, d += 512u) cp_async16(d, p, on);
                        } else {
#pragma unroll 4
                            for (int r = 0; r < n; ++r, p += pitch, d += 512u)
#pragma unroll
                                for (int j = 0; j < V; ++j) {
                                    const bool in_row = x0 + j < nx;
                                    cp_async_small<(int)sizeof(T)>(d + j * (uint32_t)sizeof(T), in_row ? p + j : p,
                                                                   in_row);
                                }
                        }
                        l += n;
                        y = 1;
                    }
                    // counts as this lane's arrival once its copies above have landed
                    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(
                                     smem_u32(&w.full[slot]))
                                 : "memory");
                }
                continue;
            }
            w.out = out;
            w.x0 = x0;
            w.ya = ya;
            w.h = h;
            w.zb = zb;
            w.own = x0 >= xa && x0 < xb;
            w.ed = j2_edge(x0, V, nx);
            if (!pair)
                w.march1(ze, q);
            else if (xs == 0 || xs + W >= nx || (!PY && (ya <= 2 || ya + h + 2 >= ny)))
                w.template march2<true>(ze, q);
            else
                w.template march2<false>(ze, q);
            if (VEC) fence_proxy_async_shared();
            __syncwarp();
            if (w.lane == 0) mbar_arrive(&w.empty[w.prev]);  // the unit's last plane
        }
        left -= pair ? 2 : 1;
        if (producer) cp_async_wait_all();
        if (!grid_barrier(bar, gridDim.x, site)) return;
        T *t = in;
        in = out;
        out = t;
    }
    // The result's halo cells (nothing above read any after the first sweep): full
    // rows of the planes 0 and nz-1, and with PY the rows 0 and ny-1 of the others.
    const int warps = gridDim.x * (CW + 1);
    const int nplane = 2 * ny, nrows = nplane + (PY ? 2 * PZ : 0);
    for (int i = blockIdx.x * (CW + 1) + w.warp; i < nrows; i += warps) {
        int z, y;
        if (i < nplane) {
            z = i < ny ? 0 : nz - 1;
            y = i < ny ? i : i - ny;
        } else {
            z = 1 + (i - nplane) / 2;
            y = (i - nplane) & 1 ? ny - 1 : 0;
        }
        const int sz = z == 0 ? nz - 2 : z == nz - 1 ? 1 : z;
        const int sy = !PY ? y : y == 0 ? ny - 2 : y == ny - 1 ? 1 : y;
        const T *src = in + ((size_t)sz * ny + sy) * nx;
        T *dst = in + ((size_t)z * ny + y) * nx;
        for (int x = w.lane; x < nx; x += 32) dst[x] = __ldcg(src + x);
    }
}

// The compiled shapes (j3d_pair.cu).  fn and tiles by whether the rows are a multiple of 16
// bytes; one geometry serves the other rows in every shape.
struct J3PairShape {
    int cw, rpw, stages;
    const void *fn[2][2];  // [precision][periodic_y]
    size_t smem;
    int tx[2];  // [precision]: tile columns
    long long (*tiles)(int precision, int nx, int ny);
};
const J3PairShape &j3d_pair_shape(int i, bool vec);
constexpr int J3_PAIR_SHAPES = 4;

// Passes for niter sweeps: the first alone, pairs, and one more for an odd rest.
inline int j3p_passes(int niter) { return niter <= 0 ? 0 : 1 + (niter - 1) / 2 + ((niter - 1) & 1); }

}  // namespace cfm

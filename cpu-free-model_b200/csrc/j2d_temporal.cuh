// 2D 5-point sweeps with several sweeps per pass over global memory.
//
//   j2d_tile_kernel    the grid on chip: each block keeps one tile in registers
//                      for all sweeps and exchanges a K-cell rim with its eight
//                      neighbours every K sweeps
//   j2d_stream_kernel  grids beyond the chip: every warp marches down a column
//                      strip with TS sweeps in flight, so a pass over HBM does TS
//                      sweeps
//
// Both compute every cell with the reference's sum order (Stencil/jacobi2D/src/
// common.cu:28-42, and :44-66 for the mirror boundary), overlap cells
// recomputed from the same inputs with the same operations, so the grid is the
// one-sweep-at-a-time grid bit for bit.  The rows 1 .. ny-2 form a ring (rows
// 0 and ny-1 are the images of ny-2 and 1 after any sweep); only the first
// sweep reads the two halo rows as they are, so it runs by itself.
#pragma once

#include <type_traits>

#include "barrier.cuh"
#include "tma.cuh"

namespace cfm {

constexpr unsigned J2_FULL = 0xffffffffu;

template <typename T>
struct J2Op;
template <>
struct J2Op<double> {
    static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
    static __device__ __forceinline__ double quarter(double s) { return __dmul_rn(0.25, s); }
};
template <>
struct J2Op<float> {
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    // a power of two: one rounding, as the reference's double product stored to float
    static __device__ __forceinline__ float quarter(float s) { return __fmul_rn(0.25f, s); }
};

// Which of a lane's V columns x0 .. x0 + V - 1 are the grid's first and last.
struct J2Edge {
    int first, last;  // index of column 0 / nx-1 in the lane's vector, or -1
    bool out;         // the whole vector lies outside the grid
};

// One row of the sweep in a lane's V columns.  c: the row, n: the row below it in
// memory, s: the row above.  EDGE: the warp's window touches column 0 or nx-1.
template <typename T, int V, bool MIRROR, bool EDGE>
__device__ __forceinline__ void j2_row(const T (&c)[V], const T (&n)[V], const T (&s)[V],
                                       const J2Edge &ed, T (&o)[V]) {
    using O = J2Op<T>;
    const T w0 = __shfl_up_sync(J2_FULL, c[V - 1], 1);
    const T eV = __shfl_down_sync(J2_FULL, c[0], 1);
#pragma unroll
    for (int j = 0; j < V; ++j) {
        T e = j + 1 < V ? c[j + 1 < V ? j + 1 : 0] : eV;
        T w = j > 0 ? c[j > 0 ? j - 1 : 0] : w0;
        if (EDGE && MIRROR) {
            if (j == ed.last) e = c[j];
            if (j == ed.first) w = c[j];
        }
        T v;
        if (MIRROR)
            v = O::quarter(O::add(O::add(O::add(n[j], s[j]), e), w));
        else
            v = O::quarter(O::add(O::add(O::add(e, w), n[j]), s[j]));
        if (EDGE && !MIRROR && (j == ed.first || j == ed.last)) v = c[j];
        if (EDGE && ed.out) v = T(0);
        o[j] = v;
    }
}

__device__ __forceinline__ J2Edge j2_edge(int x0, int V, int nx) {
    J2Edge e;
    e.first = x0 == 0 ? 0 : -1;
    e.last = (nx - 1 >= x0 && nx - 1 < x0 + V) ? nx - 1 - x0 : -1;
    e.out = x0 >= nx || x0 + V <= 0;
    return e;
}

// Lane's V columns of a row <-> global memory.  vec: nx and x0 are multiples of
// 16 bytes.  Columns outside [0, nx) read as 0 and are not written.  Loads go to
// L2: other blocks write these cells during the kernel.
template <typename T, int V>
__device__ __forceinline__ void j2_load(const T *row, int x0, int nx, bool vec, T (&v)[V]) {
    constexpr int VL = 16 / sizeof(T);
    if (vec) {
#pragma unroll
        for (int q = 0; q < V / VL; ++q) {
            const int x = x0 + q * VL;
            float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
            if (x >= 0 && x < nx) t = __ldcg(reinterpret_cast<const float4 *>(row + x));
            const T *e = reinterpret_cast<const T *>(&t);
#pragma unroll
            for (int j = 0; j < VL; ++j) v[q * VL + j] = e[j];
        }
    } else {
#pragma unroll
        for (int j = 0; j < V; ++j) {
            const int x = x0 + j;
            v[j] = x >= 0 && x < nx ? __ldcg(row + x) : T(0);
        }
    }
}
template <typename T, int V>
__device__ __forceinline__ void j2_store(T *row, int x0, int nx, bool vec, const T (&v)[V]) {
    constexpr int VL = 16 / sizeof(T);
    if (vec) {
#pragma unroll
        for (int q = 0; q < V / VL; ++q) {
            const int x = x0 + q * VL;
            float4 t;
            T *e = reinterpret_cast<T *>(&t);
#pragma unroll
            for (int j = 0; j < VL; ++j) e[j] = v[q * VL + j];
            if (x >= 0 && x < nx) *reinterpret_cast<float4 *>(row + x) = t;
        }
    } else {
#pragma unroll
        for (int j = 0; j < V; ++j)
            if (x0 + j >= 0 && x0 + j < nx) row[x0 + j] = v[j];
    }
}

// ------------------------------------------------------------ grids on chip
// Tile decomposition: tx x ty blocks.  Block (bx, by) owns the columns
// [xa, xb) and ring rows [ya, ya + h) and computes a window of 32 V columns by
// WARPS R rows around them: K cells beyond its own on every inner side.
struct J2Tiling {
    int tx, ty, ux, k;  // ux: columns between inner tile boundaries
};
constexpr int J2T_V = 4, J2T_W = 32 * J2T_V;
__host__ __device__ inline int j2_xbound(const J2Tiling &t, int i, int nx) {
    return i == 0 ? 0 : i == t.tx ? nx : t.k + i * t.ux;
}

// Each warp holds R consecutive window rows, V columns per lane, in registers.
// A sweep: every warp puts its first and last row in shared memory (two
// copies, by turns, so one block barrier per sweep), and updates its rows in place,
// the x neighbours by shuffle.  After K sweeps the block's own cells are right and
// the rest of the window is stale: own cells within K of the border go out to
// the grid buffer of the exchange's parity, the block's counter is released,
// the (at most eight) neighbours' counters are awaited (bounded), and the rim
// is read back.  A neighbour can be at most one exchange ahead, and writes the
// other buffer then.  The counters go on counting from run to run (`base`: exchanges before
// this run, which all blocks have made), so no run begins with setting them to zero.
//
// Bound: FP64 issue (16 operations per warp and row of 128) or FP32 issue while
// a sweep runs, and per exchange the latency of store - release - acquire -
// load (about 2.5 us), divided by K.
template <typename T, int WARPS>
constexpr size_t j2_tile_smem() {
    return (size_t)2 * WARPS * 2 * J2T_W * sizeof(T);
}
template <typename T, int R, int WARPS, bool MIRROR>
__global__ void __launch_bounds__(32 * WARPS, 1)
    j2d_tile_kernel(T *in, T *other, int nx, int ny, int niter, J2Tiling tl, unsigned int *flags,
                    unsigned int base, BarrierState *bar) {
    constexpr int V = J2T_V, W = J2T_W, Q = V * sizeof(T) / 16;  // 16-byte pieces per lane
    // edge rows of each warp: [parity][warp][first, last][piece][lane]
    extern __shared__ __align__(16) unsigned char j2t_smem[];
    auto edge = reinterpret_cast<float4(*)[WARPS][2][Q][32]>(j2t_smem);
    __shared__ int s_ok;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int K = tl.k, P = ny - 2;
    const int bx = blockIdx.x % tl.tx, by = blockIdx.x / tl.tx;
    const int xa = j2_xbound(tl, bx, nx), xb = j2_xbound(tl, bx + 1, nx);
    const int xs = bx == 0 ? 0 : xa - K;
    const int ya = 1 + (int)((long long)by * P / tl.ty), h = 1 + (int)((long long)(by + 1) * P / tl.ty) - ya;
    const int x0 = xs + lane * V;
    const int r0 = warp * R;  // first window row of the warp; window row l is ring row ya - K + l
    const bool vec = nx % (16 / (int)sizeof(T)) == 0;
    const bool touches = xs == 0 || xs + W >= nx;
    const J2Edge ed = j2_edge(x0, V, nx);
    // the lane's columns are the block's own / lie within K of an inner side (xa, xb
    // and K are multiples of V except xb = nx)
    const bool own_x = x0 >= xa && x0 < xb;
    const bool rim_x = own_x && ((bx > 0 && x0 < xa + K) || (bx + 1 < tl.tx && x0 >= xb - K));
    auto ring = [&](int y) { return y < 1 ? y + P : y > P ? y - P : y; };

    // Row r sits in a[r + 1] (phase 0) or a[r] (phase 1).  A sweep in phase 0 goes
    // down: the row above the warp comes into a[0] and row r's new value takes the
    // place of the old row above it, a[r]; in phase 1 it goes up, the row below
    // into a[R], new values into a[r + 1].  No row is ever moved.
    T a[R + 1][V];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int l = r0 + r, y = ya - K + l;
        // the first sweep reads the halo rows 0 and ny-1 as they are
        const int yy = y == 0 || y == ny - 1 ? y : ring(y);
        if (l < h + 2 * K)
            j2_load<T, V>(in + (size_t)yy * nx, x0, nx, vec, a[r + 1]);
        else
#pragma unroll
            for (int j = 0; j < V; ++j) a[r + 1][j] = T(0);
    }
    float4 *const mine = &edge[0][warp][0][0][lane];  // + parity, side and piece strides, all constants
    const float4 *const above = &edge[0][warp > 0 ? warp - 1 : 0][1][0][lane];
    const float4 *const below = &edge[0][warp + 1 < WARPS ? warp + 1 : warp][0][0][lane];
    constexpr int PARITY = WARPS * 2 * Q * 32, SIDE = Q * 32;
    auto put = [&](float4 *p, const T(&v)[V]) {
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            float4 t;
            T *e = reinterpret_cast<T *>(&t);
#pragma unroll
            for (int j = 0; j < V / Q; ++j) e[j] = v[q * (V / Q) + j];
            p[q * 32] = t;
        }
    };
    auto get = [&](const float4 *p, T(&v)[V]) {
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const float4 t = p[q * 32];
            const T *e = reinterpret_cast<const T *>(&t);
#pragma unroll
            for (int j = 0; j < V / Q; ++j) v[q * (V / Q) + j] = e[j];
        }
    };
    // (the window's outermost rows get a wrong neighbour, and go stale either way)
    auto sweep = [&](auto ph_c, auto edge_c) {
        constexpr bool EDGE = decltype(edge_c)::value;
        constexpr int PH = decltype(ph_c)::value;
        put(mine + PH * PARITY, a[PH ? 0 : 1]);
        put(mine + PH * PARITY + SIDE, a[PH ? R - 1 : R]);
        __syncthreads();
        T far[V];
        if (PH) {
            get(below + PH * PARITY, a[R]);
            get(above + PH * PARITY, far);
#pragma unroll
            for (int r = R - 1; r >= 1; --r) j2_row<T, V, MIRROR, EDGE>(a[r], a[r + 1], a[r - 1], ed, a[r + 1]);
            j2_row<T, V, MIRROR, EDGE>(a[0], a[1], far, ed, a[1]);
        } else {
            get(above + PH * PARITY, a[0]);
            get(below + PH * PARITY, far);
#pragma unroll
            for (int r = 0; r + 1 < R; ++r) j2_row<T, V, MIRROR, EDGE>(a[r + 1], a[r + 2], a[r], ed, a[r]);
            j2_row<T, V, MIRROR, EDGE>(a[R], far, a[R - 1], ed, a[R - 1]);
        }
    };
    // n sweeps from phase 0 to phase 0
    auto run = [&](int n, auto edge_c) {
        for (int i = 0; i + 1 < n; i += 2) {
            sweep(std::integral_constant<int, 0>(), edge_c);
            sweep(std::integral_constant<int, 1>(), edge_c);
        }
        if (n & 1) {
            sweep(std::integral_constant<int, 0>(), edge_c);
#pragma unroll
            for (int r = R; r > 0; --r)
#pragma unroll
                for (int j = 0; j < V; ++j) a[r][j] = a[r - 1][j];
        }
    };

    unsigned e = 0;  // exchanges so far
    for (int left = niter, step = 1; left > 0;) {
        const int n = min(step, left);
        if (touches)
            run(n, std::true_type());
        else
            run(n, std::false_type());
        left -= n;
        step = K;
        if (left == 0) break;
        ++e;
        T *xg = (e & 1) ? other : in;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int l = r0 + r - K;  // own row index
            if (l >= 0 && l < h && own_x && (rim_x || l < K || l >= h - K))
                j2_store<T, V>(xg + (size_t)(ya + l) * nx, x0, nx, vec, a[r + 1]);
        }
        __syncthreads();
        if (warp == 0) {
            if (lane == 0) st_release_u32(flags + blockIdx.x, base + e);
            bool ok = true;
            if (lane < 9) {
                const int qx = bx + lane % 3 - 1, qy = (by + lane / 3 - 1 + tl.ty) % tl.ty;
                if (qx >= 0 && qx < tl.tx && lane != 4) {
                    const unsigned int *f = flags + qy * tl.tx + qx;
                    const unsigned long long t0 = global_ns(), budget = bar->timeout_ns;
                    for (unsigned it = 1; (int)(ld_acquire_u32(f) - (base + e)) < 0; ++it) {
                        if ((it & 63) != 0) continue;
                        if (ld_relaxed_i32(&bar->error)) {
                            ok = false;
                            break;
                        }
                        if (global_ns() - t0 > budget) {
                            if (atomicCAS(&bar->error, 0, 1) == 0) bar->where = (int)e;
                            ok = false;
                            break;
                        }
                    }
                }
            }
            ok = __all_sync(J2_FULL, ok);
            if (lane == 0) s_ok = ok;
        }
        __syncthreads();
        if (!s_ok) return;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int l = r0 + r - K;
            if (l < h + K && x0 < xb + K && !(own_x && l >= 0 && l < h))
                j2_load<T, V>(xg + (size_t)ring(ya + l) * nx, x0, nx, vec, a[r + 1]);
        }
    }
    // The buffer of the exchange before last has no readers left: a neighbour
    // that published exchange e had read exchange e - 1.
    T *fin = (e & 1) ? in : other;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int l = r0 + r - K, y = ya + l;
        if (l < 0 || l >= h || !own_x) continue;
        j2_store<T, V>(fin + (size_t)y * nx, x0, nx, vec, a[r + 1]);
        if (y == 1) j2_store<T, V>(fin + (size_t)(ny - 1) * nx, x0, nx, vec, a[r + 1]);
        if (y == ny - 2) j2_store<T, V>(fin, x0, nx, vec, a[r + 1]);
    }
}

// ------------------------------------------------------- grids beyond the chip
// Work unit: a strip of 32 V columns (H = the sweeps rounded up to V columns
// of overlap on either inner side) by a chunk of rows, one warp each.  Rows of
// the ring enter at sweep level 0; every step computes one row of each level
// from the last three rows of the level below, which each lane keeps for its V
// columns in registers; the finished row leaves at level TS.  Rows come
// through a ring of J2S_D slots in shared memory per warp, each lane copying
// (cp.async) and reading its own 16-byte pieces, so no lane waits for another
// and no barrier is needed inside a pass.
//
// Bound: a pass of one sweep by HBM (0.41 ms at 16384^2 FP32, 0.8 of the copy rate); one of
// eight (0.58 ms) by issue, 18 instructions per row of 128 columns and level, of which 16
// are the cell's additions and multiplications.
constexpr int J2S_D = 8;        // rows in flight per warp (a power of two)
constexpr int J2S_WARPS = 4;    // warps per block
// Sweeps per pass.  Eight: 16384^2 FP32 91 us per sweep in long runs (one per pass 394, four 127,
// twelve 157), FP64 194 (one per pass 797).  Six is 1 to 10% faster in long FP32 runs (100 sweeps in us, six
// against eight: 2048^2 334 / 367, 4096^2 739 / 786, 8192^2 2411 / 2471, 16384^2 8422 / 8625, mirror boundary
// alike) and leaves more rest passes in short ones (9 sweeps are two passes with eight, three with six);
// in FP64, two columns per lane, it is slower from 16384^2 on (20104 / 18347; 4096^2 1281 / 1272).  FP64 with
// four columns per lane takes at most six (262 us per sweep at 16384^2; more do not fit the registers).
constexpr int J2S_SWEEPS = 8;

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool on) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(on ? 16 : 0)
                 : "memory");
}
template <int BYTES>
__device__ __forceinline__ void cp_async_small(uint32_t dst, const void *src, bool on) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(BYTES),
                 "r"(on ? BYTES : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// One pass of TS sweeps from `in` to `out`, rows 1 .. ny-2.  RAW: the halo rows 0 and
// ny-1 are read as they are (only with TS = 1: the run's first sweep).  VEC: rows are a
// multiple of 16 bytes.
template <typename T, int V, int TS, bool MIRROR, bool RAW, bool VEC>
__device__ void j2_stream_pass(const T *in, T *out, int nx, int ny, T *slots) {
    constexpr int W = 32 * V, H = (TS + V - 1) / V * V, U = W - 2 * H, Q = V * sizeof(T) / 16;
    constexpr int VL = V / Q;
    static_assert(!RAW || TS == 1, "the raw halo rows serve one sweep");
    const int lane = threadIdx.x & 31;
    const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    const int P = ny - 2;
    // strips: inner boundaries every U columns; the first strip has no overlap
    // on its left
    const int ns = nx <= W ? 1 : 1 + (nx - (W - H) + U - 1) / U;
    // as many chunks as give every warp one unit (more would add 2 TS rows each)
    int nch = (int)max(1LL, min((long long)P, nw / ns));
    const int rc = (P + nch - 1) / nch;
    nch = (P + rc - 1) / rc;
    // the lane's pieces of slot s: piece q at ((s * Q + q) * 32 + lane) * 16 bytes
    const float4 *const ring = reinterpret_cast<const float4 *>(slots) + lane;
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(ring);
    for (long long u = gw; u < (long long)ns * nch; u += nw) {
        const int st = (int)(u % ns), ch = (int)(u / ns);
        const int xa = st == 0 ? 0 : (W - H) + (st - 1) * U;            // own columns [xa, xb)
        const int xb = st + 1 == ns ? nx : (W - H) + st * U;
        const int xs = st == 0 ? 0 : xa - H, x0 = xs + lane * V;
        const int yb = 1 + ch * rc, ye = min(P + 1, yb + rc);
        const bool touches = xs == 0 || xs + W >= nx;
        const J2Edge ed = j2_edge(x0, V, nx);
        const bool own = x0 >= xa && x0 < xb;
        // next row to fetch (RAW rows need no wrap), rows left, and the row it sits in
        int fy = yb - TS, fleft = ye - yb + 2 * TS;
        if (!RAW) {
            fy = (yb - TS - 1) % P;
            fy = (fy < 0 ? fy + P : fy) + 1;
        }
        const T *src = in + (size_t)fy * nx + x0;
        auto fetch = [&](int slot) {
            if (fleft > 0) {
                const uint32_t d = sbase + (uint32_t)slot * (Q * 512u);
                if (VEC) {
#pragma unroll
                    for (int q = 0; q < Q; ++q) {
                        const bool on = x0 + q * VL < nx;
                        cp_async16(d + q * 512u, on ? src + q * VL : in, on);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < V; ++j) {
                        const bool on = x0 + j < nx;
                        cp_async_small<(int)sizeof(T)>(
                            d + (uint32_t)(j / VL) * 512u + (uint32_t)(j % VL) * (uint32_t)sizeof(T),
                            on ? src + j : in, on);
                    }
                }
                --fleft;
                src += nx;
                if (!RAW && ++fy > P) {
                    fy = 1;
                    src -= (size_t)P * nx;
                }
            }
            cp_async_commit();
        };
        // The last three rows of each level below TS.  In the step of phase PH a
        // level's slots PH, PH + 1, PH + 2 (mod 3) hold its rows in order, and slot
        // PH, its oldest, takes the next one: three steps bring every register back
        // to its role, so no row is ever moved, and the levels of a step (deepest
        // first, each from rows of earlier steps) do not wait for one another.
        T lv[TS][3][V];
#pragma unroll
        for (int l = 0; l < TS; ++l)
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < V; ++j) lv[l][i][j] = T(0);
#pragma unroll 1
        for (int i = 0; i < J2S_D - 1; ++i) fetch(i);
        int slot = 0;
        // The step that takes row yb - TS + n in at level 0: level l gets its row
        // yb - TS + n - 2 l, and level TS leaves from n = 3 TS on.
        T *dst = out + (ptrdiff_t)(yb - 3 * TS) * nx + x0;
        auto step = [&](auto ph_c, auto edge_c, int n) {
            constexpr int A = decltype(ph_c)::value, B = (A + 1) % 3, C = (A + 2) % 3;
            constexpr bool EDGE = decltype(edge_c)::value;
            {
                T o[V];
                j2_row<T, V, MIRROR, EDGE>(lv[TS - 1][B], lv[TS - 1][C], lv[TS - 1][A], ed, o);
                if (n >= 3 * TS && own) {
                    if (VEC) {
#pragma unroll
                        for (int q = 0; q < Q; ++q) {
                            float4 t;
                            T *e = reinterpret_cast<T *>(&t);
#pragma unroll
                            for (int j = 0; j < VL; ++j) e[j] = o[q * VL + j];
                            if (!EDGE || x0 + q * VL < nx) *reinterpret_cast<float4 *>(dst + q * VL) = t;
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < V; ++j)
                            if (!EDGE || x0 + j < nx) dst[j] = o[j];
                    }
                }
                dst += nx;
            }
#pragma unroll
            for (int l = TS - 2; l >= 0; --l)
                j2_row<T, V, MIRROR, EDGE>(lv[l][B], lv[l][C], lv[l][A], ed, lv[l + 1][A]);
            cp_async_wait<J2S_D - 2>();
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const float4 t = ring[(slot * Q + q) * 32];
                const T *e = reinterpret_cast<const T *>(&t);
#pragma unroll
                for (int j = 0; j < VL; ++j) lv[0][A][q * VL + j] = e[j];
            }
            fetch((slot + J2S_D - 1) & (J2S_D - 1));
            slot = (slot + 1) & (J2S_D - 1);
        };
        auto march = [&](auto edge_c) {
            const int steps = ye - yb + 3 * TS;
#pragma unroll 1
            for (int n = 0; n < steps; n += 3) {
                step(std::integral_constant<int, 0>(), edge_c, n);
                if (n + 1 < steps) step(std::integral_constant<int, 1>(), edge_c, n + 1);
                if (n + 2 < steps) step(std::integral_constant<int, 2>(), edge_c, n + 2);
            }
        };
        if (touches)
            march(std::true_type());
        else
            march(std::false_type());
        cp_async_wait<0>();
    }
}

// All sweeps of a run: the first alone, then passes of TS, what remains in passes of
// 4, 2 and 1, and the result's two halo rows (which no pass after the first reads).
template <typename T, int V, int TS, bool MIRROR, bool VEC>
__global__ void __launch_bounds__(32 * J2S_WARPS, sizeof(T) == 4 ? 4 : 3)
    j2d_stream_kernel(T *g0, T *g1, int nx, int ny, int niter, BarrierState *bar) {
    extern __shared__ __align__(16) unsigned char j2s_smem[];
    T *slots = reinterpret_cast<T *>(j2s_smem) + (size_t)(threadIdx.x >> 5) * J2S_D * 32 * V;
    T *in = g0, *out = g1;
    int site = 0;
    for (int left = niter; left > 0; ++site) {
        int n;
        if (site == 0) {
            j2_stream_pass<T, V, 1, MIRROR, true, VEC>(in, out, nx, ny, slots);
            n = 1;
        } else if (left >= TS) {
            j2_stream_pass<T, V, TS, MIRROR, false, VEC>(in, out, nx, ny, slots);
            n = TS;
        } else if (TS > 4 && left >= 4) {
            j2_stream_pass<T, V, 4, MIRROR, false, VEC>(in, out, nx, ny, slots);
            n = 4;
        } else if (TS > 2 && left >= 2) {
            j2_stream_pass<T, V, 2, MIRROR, false, VEC>(in, out, nx, ny, slots);
            n = 2;
        } else {
            j2_stream_pass<T, V, 1, MIRROR, false, VEC>(in, out, nx, ny, slots);
            n = 1;
        }
        left -= n;
        if (!grid_barrier(bar, gridDim.x, site)) return;
        T *t = in;
        in = out;
        out = t;
    }
    const int stride = gridDim.x * blockDim.x;
    for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < nx; x += stride) {
        in[x] = __ldcg(in + (size_t)(ny - 2) * nx + x);
        in[(size_t)(ny - 1) * nx + x] = __ldcg(in + (size_t)nx + x);
    }
}

// Passes that j2d_stream_kernel makes for niter sweeps (the buffers swap per pass).
inline int j2s_passes(int niter, int ts) {
    if (niter <= 0) return 0;
    int left = niter - 1, n = 1 + left / ts;
    left %= ts;
    if (ts > 4) {
        n += left / 4;
        left %= 4;
    }
    if (ts > 2) {
        n += left / 2;
        left %= 2;
    }
    return n + left;
}

}  // namespace cfm

// Standard CG on a stencil operator with the system on chip, for systems of at
// most a few 1024-row tiles per SM.
//
// cg_std_kernel (krylov.cuh) streams every vector through L2 in three passes
// per iteration, each behind a grid barrier; on a 512^2 grid a pass is a few
// hundred nanoseconds of work and the barriers and round trips are the rest.
// Here a block keeps T consecutive tiles: x and r in registers, p and the
// operator's coefficients in shared memory, one row per thread and tile.  Only
// the rows that another block's stencil reaches go through global memory, and an
// iteration has two grid barriers, those of the two dots:
//   p = r + beta p       own rows; a neighbour block's value of p is formed from
//                        its published r and previous p by the same operation
//   s = A p, <p, s>      sum 1
//   x += alpha p, r -= alpha s, <r, r>     r published, sum 2
// Arithmetic, dot trees, stopping and restarts are cg_std_kernel's, so x and
// the iteration count are the same bit for bit.
#pragma once

#include "krylov.cuh"

namespace cfm {

// Doubles of shared memory: p and the coefficients of T tiles, the coefficients
// of the rows before the first (north faces, and in 3D top faces), the reductions.
template <int D>
__host__ __device__ inline size_t cgr_smem_doubles(int T, int nx, int ny) {
    const size_t rows = (size_t)T * CG_TILE;
    return rows * (D + 2) + 1 + nx + (D == 3 ? (size_t)nx * ny : 0) + 32 * T + 128;
}

template <int D, int T>
__global__ void __launch_bounds__(CG_TILE, 1)
    cg_std_res_kernel(KArgs<StencilOp<D>> a) {
    extern __shared__ double cgr_sm[];
    constexpr int ROWS = T * CG_TILE;
    const int nx = a.op.nx, ny = a.op.ny, P = nx * ny, n = a.n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tile0 = blockIdx.x * T, lo = tile0 * CG_TILE, hi = min(n, lo + ROWS);
    double *ps = cgr_sm;                  // p, own rows
    double *sdg = ps + ROWS;              // diagonal, own rows
    double *swe = sdg + ROWS + 1;         // swe[q]: east face of row lo + q, q >= -1
    double *swn = swe + ROWS + nx;        // swn[q]: north face, q >= -nx
    double *swt = swn + ROWS + (D == 3 ? P : 0);  // 3D: top face, q >= -P
    double *sums = (D == 3 ? swt : swn) + ROWS;   // T x 32 warp sums
    double *red = sums + 32 * T;          // 4 x 32
    double *pbuf0 = a.p, *pbuf1 = a.s;    // published p by iteration parity
    const int reach = D == 3 ? P : nx;

    for (int q = threadIdx.x; q < hi - lo; q += CG_TILE) sdg[q] = a.op.dg[lo + q];
    for (int q = (int)threadIdx.x - 1; q < hi - lo; q += CG_TILE) swe[q] = lo + q >= 0 ? a.op.we[lo + q] : 0.0;
    for (int q = (int)threadIdx.x - nx; q < hi - lo; q += CG_TILE) swn[q] = lo + q >= 0 ? a.op.wn[lo + q] : 0.0;
    if (D == 3)
        for (int q = (int)threadIdx.x - P; q < hi - lo; q += CG_TILE) swt[q] = lo + q >= 0 ? a.op.wt[lo + q] : 0.0;

    double x[T], r[T], s[T];
    unsigned nb[T];  // 1: the row exists; 2, 4, 8, ...: it has the neighbour x-1, x+1, y-1, ...
#pragma unroll
    for (int t = 0; t < T; ++t) {
        const int i = lo + t * CG_TILE + (int)threadIdx.x;
        nb[t] = 0;
        if (i < n) {
            const int ix = i % nx, q = i / nx, iy = q % ny;
            nb[t] = 1u | (ix > 0 ? 2u : 0u) | (ix < nx - 1 ? 4u : 0u) | (iy > 0 ? 8u : 0u) | (iy < ny - 1 ? 16u : 0u);
            if (D == 3) nb[t] |= (q >= ny ? 32u : 0u) | (i + P < n ? 64u : 0u);
        }
    }

    CgGrid<StencilOp<D>> grid(a, red);
    // The block's tile partials of a slot: its warp sums in shared memory, then one
    // warp per tile (callers put a block barrier between two of these).
    auto publish = [&](int s, const double (&v)[T]) {
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const double w = warp_xor_sum(v[t]);
            if (lane == 0) sums[t * 32 + warp] = w;
        }
        __syncthreads();
        if (warp < T && tile0 + warp < a.ntiles) {
            const double w = warp_xor_sum(sums[warp * 32 + lane]);
            if (lane == 0) slot(a, s)[tile0 + warp] = w;
        }
    };
    auto rim = [&](int i) { return i - lo < reach || hi - i <= reach; };

    {
        double g[T], bb[T];
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const int i = lo + t * CG_TILE + (int)threadIdx.x;
            x[t] = r[t] = g[t] = bb[t] = 0.0;
            if (nb[t]) {
                const double bi = a.b ? a.b[i] : 1.0;
                r[t] = __fma_rn(-1.0, 0.0, bi);  // b - A x0, x0 = 0
                if (rim(i)) a.r[i] = r[t];
                g[t] = __dmul_rn(r[t], r[t]);
                bb[t] = __dmul_rn(bi, bi);
            }
        }
        publish(SL_G0, g);
        __syncthreads();
        publish(SL_B, bb);
    }
    double gamma0, bb;
    if (!grid.sum2(SL_G0, &gamma0, SL_B, &bb)) return;
    const double bnorm = sqrt(bb);
    const bool use_tol = a.tol > 0.0;
    const double target = a.tol * bnorm;
    int status = use_tol ? CFM_NOT_CONVERGED : CFM_OK;
    int restarts = 0;
    long long k = 0;
    double beta = 0.0;
    bool fresh = true;  // p = r (the start, and after a restart)
    if (use_tol && sqrt(gamma0) <= target) status = CFM_OK;
    while (k < a.maxiter && !(use_tol && status == CFM_OK)) {
        const double *pold = (k & 1) ? pbuf0 : pbuf1;
        double *pnew = (k & 1) ? pbuf1 : pbuf0;
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const int q = t * CG_TILE + (int)threadIdx.x;
            if (nb[t]) {
                const double pv = fresh ? r[t] : __fma_rn(beta, ps[q], r[t]);
                ps[q] = pv;
                if (rim(lo + q)) pnew[lo + q] = pv;
            }
        }
        __syncthreads();
        // p of this iteration at the neighbour row lo + q (on: it exists).  The loads for a
        // row of another block are predicated, so all of a row's are in flight together.
        const double *rg = a.r + lo, *pg = pold + lo;
        auto pat = [&](bool on, int q) -> double {
            const bool mine = (unsigned)q < (unsigned)(hi - lo), far = on && !mine;
            const double rj = far ? __ldcg(rg + q) : 0.0;
            const double pj = far && !fresh ? __ldcg(pg + q) : 0.0;
            const double v = fresh ? rj : __fma_rn(beta, pj, rj);
            return mine ? ps[q] : v;
        };
        double d[T];
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const int q = t * CG_TILE + (int)threadIdx.x;
            const unsigned m = nb[t];
            d[t] = s[t] = 0.0;
            if (m) {
                const double pv = ps[q];
                const double yl = pat(m & 8u, q - nx), yh = pat(m & 16u, q + nx);
                double zl = 0.0, zh = 0.0;
                if (D == 3) {
                    zl = pat(m & 32u, q - P);
                    zh = pat(m & 64u, q + P);
                }
                const double xl = pat(m & 2u, q - 1), xh = pat(m & 4u, q + 1);
                double v = __dmul_rn(sdg[q], pv);
                if (m & 2u) v = __fma_rn(-swe[q - 1], xl, v);
                if (m & 4u) v = __fma_rn(-swe[q], xh, v);
                if (m & 8u) v = __fma_rn(-swn[q - nx], yl, v);
                if (m & 16u) v = __fma_rn(-swn[q], yh, v);
                if (D == 3) {
                    if (m & 32u) v = __fma_rn(-swt[q - P], zl, v);
                    if (m & 64u) v = __fma_rn(-swt[q], zh, v);
                }
                s[t] = v;
                d[t] = __dmul_rn(pv, v);
            }
        }
        publish(SL_D0, d);
        double delta;
        if (!grid.sum(SL_D0, &delta)) return;
        const double alpha = gamma0 / delta;
        if (use_tol && !(delta > 0.0 && isfinite(alpha))) {
            status = CFM_BREAKDOWN;
            break;
        }
        double g[T];
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const int q = t * CG_TILE + (int)threadIdx.x;
            g[t] = 0.0;
            if (nb[t]) {
                x[t] = __fma_rn(alpha, ps[q], x[t]);
                r[t] = __fma_rn(-alpha, s[t], r[t]);
                if (rim(lo + q)) a.r[lo + q] = r[t];
                g[t] = __dmul_rn(r[t], r[t]);
            }
        }
        publish(SL_G0, g);
        double gamma1;
        if (!grid.sum(SL_G0, &gamma1)) return;
        ++k;
        if (a.snap && k % a.snap_every == 0 && k / a.snap_every <= a.snap_max) {
            double *dst = a.snap + (size_t)(k / a.snap_every - 1) * n;
#pragma unroll
            for (int t = 0; t < T; ++t)
                if (nb[t]) dst[lo + t * CG_TILE + (int)threadIdx.x] = x[t];
        }
        if (use_tol && sqrt(gamma1) <= target) {
            // the FP64 true residual decides: t = b - A x from x in global memory
            double tr[T], q2[T];
#pragma unroll
            for (int t = 0; t < T; ++t)
                if (nb[t]) a.x[lo + t * CG_TILE + (int)threadIdx.x] = x[t];
            if (!grid.barrier()) return;
#pragma unroll
            for (int t = 0; t < T; ++t) {
                const int i = lo + t * CG_TILE + (int)threadIdx.x;
                tr[t] = q2[t] = 0.0;
                if (nb[t]) {
                    tr[t] = __dsub_rn(a.b ? a.b[i] : 1.0, a.op.apply(a.x, i));
                    q2[t] = __dmul_rn(tr[t], tr[t]);
                    if (rim(i)) a.r[i] = tr[t];  // nobody reads r until the next iteration
                }
            }
            publish(SL_TT, q2);
            double tt;
            if (!grid.sum(SL_TT, &tt)) return;
            if (sqrt(tt) <= target) {
                status = CFM_OK;
                gamma0 = gamma1;
                break;
            }
#pragma unroll
            for (int t = 0; t < T; ++t) r[t] = tr[t];
            fresh = true;
            ++restarts;
            gamma0 = tt;
            continue;
        }
        beta = gamma1 / gamma0;
        if (use_tol && !isfinite(beta)) {
            status = CFM_BREAKDOWN;
            break;
        }
        fresh = false;
        gamma0 = gamma1;
    }
#pragma unroll
    for (int t = 0; t < T; ++t)
        if (nb[t]) a.x[lo + t * CG_TILE + (int)threadIdx.x] = x[t];
    write_result(a.res, k, status, restarts, gamma0, bnorm);
}

}  // namespace cfm

// cg_kernels.cuh -- the persistent CG kernels of libcgb (sm_100a).
//
// One cooperative, persistent kernel runs a whole outer step of the inverse
// power iteration (GMAP/NPB-GPU CUDA/CG/cg.cu:500-520): the conj_grad
// iterations (cg.cu:653-801), the explicit residual ||x - A z||, and the
// zeta / normalisation update (cg.cu:508-519).  The reference spreads the
// same work over 157 launches and 54 blocking device-to-host copies per
// outer step (kernels one..eleven, cg.cu:848-1265); here the reductions
// finish on the device and every phase boundary is a bounded grid barrier.
//
// Work split: CTA c owns rows [row_split[c], row_split[c+1]), chosen on the
// host so every CTA holds about the same number of stored entries.  A CTA
// computes the SpMV rows it owns and all vector updates of those rows, so
// only the gathers of p (or z) cross CTA boundaries.  Reductions: each CTA
// writes one partial per quantity; after the barrier every CTA sums the
// partials in the same fixed order, so all CTAs take identical control
// decisions and results are run-to-run deterministic.
//
// Bodies:
//   outer_step_body        FP64 CG: the reference algorithm (fixed cgitmax
//                          steps from z = 0) or stopped at a relative
//                          residual;
//   outer_step_mixed_body  FP32 SpMV (values and search vector in FP32,
//                          FP32 row sums) inside FP64 CG: dot products,
//                          alpha/beta, the z/r/p updates, zeta and a
//                          periodic true-residual replacement r = x - A z
//                          computed with the FP64 matrix stay in FP64.
#pragma once

#include "galerkin.cuh"
#include "spmv_policies.cuh"

namespace cgb {


// Partial-sum slots (each holds `gpad` doubles, one per CTA).
enum Slot { kSlotRho = 0, kSlotD = 1, kSlotXX = 2, kSlotRes = 3, kSlotXZ = 4, kSlotZZ = 5,
            kSlotGram = 6, kSlotCount = kSlotGram + kGramValues };

// Per-step trace record written by CTA 0.
struct StepTrace {
    double zeta;
    double rnorm;
    double inner;     // CG steps taken
    double rho;       // final recursive residual norm squared
    double refresh;   // true-residual replacements (mixed mode)
    double spare[3];
};

struct OuterArgs {
    int n;
    MatrixView M;
    double *x, *z, *p, *q, *r;
    float *p32;                         // FP32 search vector (mixed modes)
    float *r32;                         // FP32 residual (preconditioned mode, row plan)
    __nv_bfloat16 *r16, *t16;           // BF16 residual and F r (preconditioned mode, sliced plan)
    double *y;                          // preconditioned residual (preconditioned mode)
    MatrixView F, FT;                   // preconditioner factor F (lower) and F^T (FP32 CSR;
                                        // BF16 sliced copies)
    const int *__restrict__ row_split;  // gridDim.x + 1 entries
    double *part;                       // kSlotCount * gpad
    int gpad;
    GridBarrier gb;
    double shift;
    int cgitmax;        // fixed mode: exact count; tolerance modes: cap
    int fixed;          // 1: reference semantics (no tolerance test, z0 = 0)
    double tol;         // tolerance modes: stop when ||r|| <= tol * ||x||
    int refresh_every;  // mixed mode: replace r by x - A z at least every k steps
    int step;           // outer step index (trace slot)
    int finish;         // 1: zeta + x update (power iteration); 0: conj_grad only
    StepTrace *trace;
    // Galerkin start (tolerance modes): ring of the last `recycle` iterates
    // x_j and A x_j, slot j % recycle, `hstride` doubles a vector
    double *hx, *hw;
    size_t hstride;
    int recycle;        // 0: off; 1..kMaxRecycle
};

// Writes this CTA's share of a reduction into slot `slot`.
__device__ __forceinline__ void put_partial(const OuterArgs &A, int slot, double v, double *scratch)
{
    const double s = block_sum(v, scratch);
    if (threadIdx.x == 0) A.part[slot * A.gpad + blockIdx.x] = s;
}

__device__ __forceinline__ double get_total(const OuterArgs &A, int slot, double *bcast)
{
    return all_partials(A.part + slot * A.gpad, gridDim.x, bcast);
}

// Leaves the kernel when a barrier or an SpMV wait failed.
#define CGB_BARRIER_OR_RETURN(A) \
    do {                         \
        if (!grid_barrier((A).gb)) return; \
    } while (0)
#define CGB_OK_OR_RETURN(ok) \
    do {                     \
        if (!(ok)) return;   \
    } while (0)

template <class Spmv, typename VT>
__device__ __forceinline__ double spmv(Spmv &sp, const OuterArgs &A, const VT *v, double *out,
                                       const double *dotv, bool &ok)
{
    return sp.template apply<VT>(A.M, v, out, dotv, A.n, A.gb.limit_ns, A.gb.status, ok);
}

// Row j of the product just computed (to `out`), once every CTA is past a
// barrier: by column parts the sum of the row's parts, in part order.
template <class Spmv>
__device__ __forceinline__ double product_at(const OuterArgs &A, const double *out, int j)
{
    if constexpr (Spmv::kParts) {
        double t = 0.0;
        for (int k = 0; k < A.M.parts; k++) t += __ldcg(A.M.part_out + k * A.M.part_stride + j);
        return t;
    }
    return out[j];
}

// Makes a product's rows readable by product_at where no reduction follows it:
// a grid barrier where rows have parts of other CTAs, else the CTA's own.
template <class Spmv>
__device__ __forceinline__ bool product_ready(const OuterArgs &A)
{
    if constexpr (Spmv::kParts) return grid_barrier(A.gb);
    __syncthreads();
    return true;
}

// Start of a solve (shared by the bodies): z0 = 0, r0 = x, p0 = r0 (the
// mixed body also fills p32); leaves the partial of r.r = x.x.  (CG's first
// iterate from z0 = 0 is already the best multiple of x, the Galerkin
// solution on span{x}, so no other starting guess built from x saves work.)
template <class Spmv>
__device__ __forceinline__ void start_solve(const OuterArgs &A, int row0, int vend, bool fill32,
                                            double *scratch)
{
    double acc = 0.0;
    for (int j = row0 + threadIdx.x; j < vend; j += blockDim.x) {
        const double xv = A.x[j];
        A.q[j] = 0.0;
        A.z[j] = 0.0;
        A.r[j] = xv;
        A.p[j] = xv;
        if (fill32) A.p32[j] = float(xv);
        if (j < A.n) acc = fma(xv, xv, acc);
    }
    put_partial(A, kSlotRho, acc, scratch);
}

// End of a solve (shared): r = A z (FP64), rnorm = ||x - r|| (cg.cu:777-800),
// x.z and z.z (cg.cu:508-511), zeta, the trace record and, when finishing
// an outer step, x = z / ||z|| (cg.cu:517-519).
// When `r_true` the caller's r already holds x - A z computed in FP64 (a
// true-residual replacement right before), so the residual SpMV is skipped
// and r is left as the residual instead of A z.
template <class Spmv>
__device__ __forceinline__ void end_solve(Spmv &sp, const OuterArgs &A, int row0, int row1, int it,
                                          double rho, int refreshes, bool r_true, double *scratch,
                                          double *bcast, double rsign = 1.0)
{
    if (!r_true) {
        bool ok = true;
        spmv<Spmv, double>(sp, A, A.z, A.r, nullptr, ok);
        if (!ok || !product_ready<Spmv>(A)) return;
    }
    double res = 0.0, xz = 0.0, zz = 0.0;
    for (int j = row0 + threadIdx.x; j < row1; j += blockDim.x) {
        const double xv = A.x[j], zv = A.z[j];
        double rv = A.r[j];
        if constexpr (Spmv::kParts) {
            if (!r_true) {
                rv = product_at<Spmv>(A, A.r, j);
                A.r[j] = rv;
            }
        }
        const double dv = r_true ? rv : xv - rv;
        res = fma(dv, dv, res);
        xz = fma(xv, zv, xz);
        zz = fma(zv, zv, zz);
    }
    put_partial(A, kSlotRes, res, scratch);
    put_partial(A, kSlotXZ, xz, scratch);
    put_partial(A, kSlotZZ, zz, scratch);
    if (!grid_barrier(A.gb)) return;
    const double sum = get_total(A, kSlotRes, &bcast[4]);
    const double t1 = get_total(A, kSlotXZ, &bcast[5]);
    const double t2 = get_total(A, kSlotZZ, &bcast[6]);
    const double rnorm = sqrt(sum);
    const double zeta = A.shift + 1.0 / t1;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        StepTrace &t = A.trace[A.step];
        t.zeta = zeta;
        t.rnorm = rnorm;
        t.inner = double(it);
        t.rho = rho;
        t.refresh = double(refreshes);
        if (!isfinite(zeta) || !isfinite(rnorm)) raise_status(A.gb.status, kDevNonFinite);
    }
    if (A.finish) {
        const double norm = 1.0 / sqrt(t2);
        if (A.recycle > 0 && !A.fixed) {
            // the next iterate and A times it, for the next step's Galerkin
            // start: A x' = norm A z, with A z = r (SpMV above) or, when r
            // is the true residual rsign (x - A z), A z = x - rsign r
            const size_t slot = size_t((A.step + 1) % A.recycle) * A.hstride;
            for (int j = row0 + threadIdx.x; j < row1; j += blockDim.x) {
                const double az = r_true ? A.x[j] - rsign * A.r[j] : A.r[j];
                const double xn = norm * A.z[j];
                A.hx[slot + j] = xn;
                A.hw[slot + j] = norm * az;
                A.x[j] = xn;
            }
        } else {
            for (int j = row0 + threadIdx.x; j < row1; j += blockDim.x) A.x[j] = norm * A.z[j];
        }
    }
}

// ---------------------------------------------------------- Galerkin start
// Iterates of the power iteration span a Krylov space of A: x_{j+1} is
// A^-1 x_j scaled, so A x_{j+1} is x_j scaled.  At outer step k the ring
// holds x_j and A x_j for j = k, ..., k-v+1 (v = min(k, recycle); A x_j
// came from the end-of-step product A z at no extra cost).  The start
// vector z0 is the Galerkin solution of A z = x on their span:
//   (V^T A V) y = V^T x,   z0 = V y,   A z0 = W y   (W = A V),
// which for v = 1 is CG's first iterate from z = 0 and for larger v
// removes the slowly converging eigen-directions the previous solves met.
// The v x v system is solved by every CTA identically (Cholesky of -V^T A V,
// SPD for negative definite A; a direction whose pivot falls below tau
// times the first is left out, tau raised until the coefficients stay
// small so that W y is accurate to ~1e-14 of x).

// What the Galerkin start reads and writes (passed by value to the outlined
// function, so the kernel's argument block is not copied to local memory).
struct GalerkinArgs {
    const double *hx, *hw;
    size_t hstride;
    int recycle, step;
    const double *x;
    double *z, *q;
    double *part;
    int gpad;
    GridBarrier gb;
};

__device__ __forceinline__ GalerkinArgs galerkin_args(const OuterArgs &A)
{
    GalerkinArgs G;
    G.hx = A.hx;
    G.hw = A.hw;
    G.hstride = A.hstride;
    G.recycle = A.recycle;
    G.step = A.step;
    G.x = A.x;
    G.z = A.z;
    G.q = A.q;
    G.part = A.part;
    G.gpad = A.gpad;
    G.gb = A.gb;
    return G;
}

// Per-CTA sums of nq per-thread values into slots [slot0, slot0 + nq).
// Four values a round keep the static shared memory small (the sliced
// kernels give nearly all of it to staging).
__device__ __forceinline__ void put_partials_multi(const GalerkinArgs &A, int slot0,
                                                   const double *vals, int nq)
{
    constexpr int kRound = 4;
    __shared__ double red[32][kRound];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
    for (int q0 = 0; q0 < kGramValues; q0 += kRound) {
        if (q0 < nq) {
#pragma unroll
            for (int k = 0; k < kRound; k++) {
                if (q0 + k < nq && q0 + k < kGramValues) {
                    const double v = warp_sum(vals[q0 + k < kGramValues ? q0 + k : 0]);
                    if (l == 0) red[w][k] = v;
                }
            }
            __syncthreads();
            if (threadIdx.x < kRound && q0 + int(threadIdx.x) < nq) {
                double t = 0.0;
                for (int i = 0; i < int(blockDim.x >> 5); i++) t += red[i][threadIdx.x];
                A.part[size_t(slot0 + q0 + threadIdx.x) * A.gpad + blockIdx.x] = t;
            }
            __syncthreads();
        }
    }
}

// Totals of slots [slot0, slot0 + nq) into out[] (shared), the same in
// every CTA: slot q summed by warp q % nwarps in a fixed order.
__device__ __forceinline__ void get_totals_multi(const GalerkinArgs &A, int slot0, int nq, double *out)
{
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int q = w; q < nq; q += nw) {
        double t = 0.0;
        for (int i = l; i < int(gridDim.x); i += 32) t += __ldcg(A.part + size_t(slot0 + q) * A.gpad + i);
        t = warp_sum(t);
        if (l == 0) out[q] = t;
    }
    __syncthreads();
}

// z0 and A z0 of the Galerkin start into A.z and A.q (own rows; entry n of
// the last CTA zero), and x.x into *xx (all CTAs).  v >= 1.  Returns false
// when a grid barrier failed.
static __device__ __noinline__ bool galerkin_start(const GalerkinArgs A, int row0, int row1, int vend,
                                                  int v, double *xx)
{
    __shared__ double g_sh[kGramValues];
    __shared__ double y_sh[kMaxRecycle];
    const int m = A.recycle;
    size_t off[kMaxRecycle];
#pragma unroll
    for (int a = 0; a < kMaxRecycle; a++) off[a] = size_t(((A.step - a) % m + m) % m) * A.hstride;
    const int npairs = v * (v + 1) / 2;
    double vals[kGramValues];
#pragma unroll
    for (int q = 0; q < kGramValues; q++) vals[q] = 0.0;
    for (int j = row0 + threadIdx.x; j < row1; j += blockDim.x) {
        double xa[kMaxRecycle], wa[kMaxRecycle];
#pragma unroll
        for (int a = 0; a < kMaxRecycle; a++) {
            if (a < v) {
                xa[a] = A.hx[off[a] + j];
                wa[a] = A.hw[off[a] + j];
            }
        }
        const double xv = A.x[j];
#pragma unroll
        for (int b = 0; b < kMaxRecycle; b++) {
#pragma unroll
            for (int a = 0; a <= b; a++)
                if (b < v) vals[gram_index(a, b)] = fma(xa[a], wa[b], vals[gram_index(a, b)]);
            if (b < v) vals[kGramPairs + b] =
                fma(xa[b], xv, vals[kGramPairs + b]);
        }
    }
    // pack: Gram pairs first, then the right-hand sides
    double packed[kGramValues];
#pragma unroll
    for (int q = 0; q < kGramValues; q++) packed[q] = 0.0;
#pragma unroll
    for (int q = 0; q < kGramPairs; q++)
        if (q < npairs) packed[q] = vals[q];
#pragma unroll
    for (int b = 0; b < kMaxRecycle; b++)
        if (b < v) packed[npairs + b] = vals[kGramPairs + b];
    put_partials_multi(A, kSlotGram, packed, npairs + v);
    if (!grid_barrier(A.gb)) return false;
    get_totals_multi(A, kSlotGram, npairs + v, g_sh);
    if (threadIdx.x == 0) {
        double g[kGramValues];
        for (int q = 0; q < kGramValues; q++) g[q] = 0.0;
        for (int q = 0; q < npairs; q++) g[q] = g_sh[q];
        for (int b = 0; b < v; b++) g[kGramPairs + b] = g_sh[npairs + b];
        double y[kMaxRecycle];
        galerkin_solve(g, v, y);
        for (int a = 0; a < kMaxRecycle; a++) y_sh[a] = a < v ? y[a] : 0.0;
    }
    __syncthreads();
    // x_k is the newest ring entry: x.x = its right-hand-side entry
    *xx = g_sh[npairs];
    for (int j = row0 + threadIdx.x; j < vend; j += blockDim.x) {
        double z0 = 0.0, az = 0.0;
        if (j < row1) {
#pragma unroll
            for (int a = 0; a < kMaxRecycle; a++) {
                if (a < v) {
                    z0 = fma(y_sh[a], A.hx[off[a] + j], z0);
                    az = fma(y_sh[a], A.hw[off[a] + j], az);
                }
            }
        }
        A.z[j] = z0;
        A.q[j] = az;
    }
    __syncthreads();
    return true;
}

// Iterates available for the Galerkin start of this outer step (0: start
// from z = 0).
__device__ __forceinline__ int recycle_depth(const OuterArgs &A)
{
    if (A.fixed || A.recycle <= 0 || !A.finish) return 0;
    return A.step < A.recycle ? A.step : A.recycle;
}

// FP64 CG (reference semantics when A.fixed).
template <class Spmv>
__device__ __forceinline__ void outer_step_body(const OuterArgs &A)
{
    __shared__ double scratch[32];
    __shared__ double bcast[8];
    const int row0 = A.row_split[blockIdx.x];
    const int row1 = A.row_split[blockIdx.x + 1];
    Spmv sp;
    sp.setup(A.M, row0, row1);
    bool ok = true;
    // the reference initialises n+1 vector entries (cg.cu:670-675); the
    // last CTA also owns entry n, which never enters a dot product
    const int vend = (blockIdx.x == gridDim.x - 1) ? row1 + 1 : row1;
    const int v = recycle_depth(A);
    double xx = 0.0;
    if (v > 0) {
        // tolerance mode: Galerkin start, r0 = x - A z0, p0 = r0
        if (!galerkin_start(galerkin_args(A), row0, row1, vend, v, &xx)) return;
        double acc = 0.0;
        for (int j = row0 + threadIdx.x; j < vend; j += blockDim.x) {
            const double rv = A.x[j] - A.q[j];
            A.r[j] = rv;
            A.p[j] = rv;
            if (j < A.n) acc = fma(rv, rv, acc);
        }
        put_partial(A, kSlotRho, acc, scratch);
    } else {
        start_solve<Spmv>(A, row0, vend, false, scratch);
    }
    CGB_BARRIER_OR_RETURN(A);
    double rho = get_total(A, kSlotRho, &bcast[0]);
    if (v == 0) xx = rho;                     // rho = x.x when z0 = 0
    const double stop2 = A.tol * A.tol * xx;

    // ---- CG iterations (cg.cu:678-768)
    int it = 0;
    for (; it < A.cgitmax; it++) {
        if (!A.fixed && rho <= stop2) break;
        // q = A p, d = p.q
        double acc = spmv<Spmv, double>(sp, A, A.p, A.q, A.p, ok);
        CGB_OK_OR_RETURN(ok);
        put_partial(A, kSlotD, acc, scratch);
        CGB_BARRIER_OR_RETURN(A);
        const double d = get_total(A, kSlotD, &bcast[2]);
        const double alpha = rho / d;
        const double rho0 = rho;
        // z += alpha p, r -= alpha q, rho = r.r
        acc = 0.0;
        for (int j = row0 + threadIdx.x; j < row1; j += blockDim.x) {
            const double qv = product_at<Spmv>(A, A.q, j);
            if constexpr (Spmv::kParts)
                if (!A.finish) A.q[j] = qv;  // conj_grad returns q
            A.z[j] = fma(alpha, A.p[j], A.z[j]);
            const double rv = fma(-alpha, qv, A.r[j]);
            A.r[j] = rv;
            acc = fma(rv, rv, acc);
        }
        put_partial(A, kSlotRho, acc, scratch);
        CGB_BARRIER_OR_RETURN(A);
        rho = get_total(A, kSlotRho, &bcast[3]);
        const double beta = rho / rho0;
        // p = r + beta p
        for (int j = row0 + threadIdx.x; j < row1; j += blockDim.x)
            A.p[j] = fma(beta, A.p[j], A.r[j]);
        CGB_BARRIER_OR_RETURN(A);
    }
    end_solve(sp, A, row0, row1, it, rho, 0, false, scratch, bcast);
}

// Mixed precision: q = A32 p32 in FP32, everything else FP64, as
// iterative refinement.  The recursive residual drifts from the true one by
// the FP32 rounding of each product, so r is replaced by x - A z (FP64
// matrix) and CG restarts from it (p = r) whenever the recursive residual
// has fallen kDrift2 below its value at the last replacement, after
// refresh_every steps, or when it claims convergence; the solve stops only
// on a true residual below tol.
constexpr double kDrift2 = 1e-12;  // (1e-6)^2: what one FP32-driven cycle can reliably gain

template <class Spmv>
__device__ __forceinline__ void outer_step_mixed_body(const OuterArgs &A)
{
    __shared__ double scratch[32];
    __shared__ double bcast[8];
    const int row0 = A.row_split[blockIdx.x];
    const int row1 = A.row_split[blockIdx.x + 1];
    Spmv sp;
    sp.setup(A.M, row0, row1);
    bool ok = true;
    const int vend = (blockIdx.x == gridDim.x - 1) ? row1 + 1 : row1;
    const int v = recycle_depth(A);
    double xx = 0.0;
    if (v > 0) {
        // Galerkin start: r0 = x - A z0 (a true residual), p0 = r0
        if (!galerkin_start(galerkin_args(A), row0, row1, vend, v, &xx)) return;
        double acc = 0.0;
        for (int j = row0 + threadIdx.x; j < vend; j += blockDim.x) {
            const double rv = A.x[j] - A.q[j];
            A.r[j] = rv;
            A.p[j] = rv;
            A.p32[j] = float(rv);
            if (j < A.n) acc = fma(rv, rv, acc);
        }
        put_partial(A, kSlotRho, acc, scratch);
    } else {
        start_solve<Spmv>(A, row0, vend, true, scratch);
    }
    CGB_BARRIER_OR_RETURN(A);
    double rho = get_total(A, kSlotRho, &bcast[0]);
    if (v == 0) xx = rho;                      // rho = x.x when z0 = 0
    const double stop2 = A.tol * A.tol * xx;
    double rho_cycle = rho;                    // rho at the last true residual

    int it = 0, since = 0, refreshes = 0;
    bool fresh = true;  // r is a true residual (and p = r)
    for (;;) {
        bool refresh = false;
        if (rho <= stop2) {
            if (fresh) break;
            refresh = true;
        } else if (!fresh && (since >= A.refresh_every || rho <= kDrift2 * rho_cycle)) {
            refresh = true;
        }
        if (!refresh && it >= A.cgitmax) break;
        if (refresh) {
            // r = x - A z with the FP64 matrix (z is complete: we are past a
            // barrier), then restart: p = r
            spmv<Spmv, double>(sp, A, A.z, A.r, nullptr, ok);
            CGB_OK_OR_RETURN(ok && product_ready<Spmv>(A));
            double acc = 0.0;
            for (int j = row0 + threadIdx.x; j < row1; j += blockDim.x) {
                const double rv = A.x[j] - product_at<Spmv>(A, A.r, j);
                A.r[j] = rv;
                A.p[j] = rv;
                A.p32[j] = float(rv);
                acc = fma(rv, rv, acc);
            }
            put_partial(A, kSlotRho, acc, scratch);
            CGB_BARRIER_OR_RETURN(A);
            rho = get_total(A, kSlotRho, &bcast[3]);
            rho_cycle = rho;
            refreshes++;
            since = 0;
            fresh = true;
            continue;
        }
        // q = A32 p32 (FP32 rows), d = p.q in FP64
        double acc = spmv<Spmv, float>(sp, A, A.p32, A.q, A.p, ok);
        CGB_OK_OR_RETURN(ok);
        put_partial(A, kSlotD, acc, scratch);
        CGB_BARRIER_OR_RETURN(A);
        const double d = get_total(A, kSlotD, &bcast[2]);
        const double alpha = rho / d;
        const double rho0 = rho;
        acc = 0.0;
        for (int j = row0 + threadIdx.x; j < row1; j += blockDim.x) {
            A.z[j] = fma(alpha, A.p[j], A.z[j]);
            const double rv = fma(-alpha, product_at<Spmv>(A, A.q, j), A.r[j]);
            A.r[j] = rv;
            acc = fma(rv, rv, acc);
        }
        put_partial(A, kSlotRho, acc, scratch);
        CGB_BARRIER_OR_RETURN(A);
        rho = get_total(A, kSlotRho, &bcast[3]);
        const double beta = rho / rho0;
        for (int j = row0 + threadIdx.x; j < row1; j += blockDim.x) {
            const double pv = fma(beta, A.p[j], A.r[j]);
            A.p[j] = pv;
            A.p32[j] = float(pv);
        }
        CGB_BARRIER_OR_RETURN(A);
        it++;
        since++;
        fresh = false;
    }
    end_solve(sp, A, row0, row1, it, rho, refreshes, fresh, scratch, bcast);
}

// Preconditioned mixed precision.  A is negative definite, so CG runs on
// A' = -A (SPD) with b' = -x, which has the same solution z; the
// preconditioner is M = F^T F (F lower triangular with a positive diagonal,
// e.g. the learned factor scaled by diag(A')^-1/2), applied as two FP32
// sparse products y = F^T (F r).  The refinement structure is the mixed
// body's (FP32 A-products, FP64 everything else, true-residual replacement
// with restart).  When the preconditioned iteration stalls -- no halving of
// |r|^2 in four steps, or a non-positive p.A'p or r.y -- the outer step
// falls back to unpreconditioned CG (counted in the trace).
// y = M r = F^T (F r) and the partial of r.y, then its total in rho_out.
//  - sliced policy: F and F^T have their own sliced copies with interleaved
//    row ownership (CTA c computes rows c, c+G, ...).  F is lower
//    triangular, so contiguous row ranges would leave the first CTAs almost
//    idle and the last ones with whole rows (and the reverse for F^T);
//    interleaving gives every CTA a fair sample of row lengths.  Their
//    values are stored in BF16 (4 bytes an entry with the 16-bit column;
//    products and sums in FP32): M = F~^T F~ of the rounded factor is still
//    SPD.  The vectors they gather (r, then F r) are staged in BF16 too, so
//    a 96 KB slot holds a 49152-column block (4 blocks at class C, not 7);
//    rounding them measured no extra iterations on these matrices.  The F^T product fuses
//    the r.y partial over the rows it computes.
//  - row policy: CSR rows of F and F^T with LPRG lanes per row over the
//    CTA's own rows.
template <class Spmv, int LPRG>
__device__ __forceinline__ bool apply_prec(Spmv &sp, const OuterArgs &A, int row0, int row1,
                                           bool use, double &rho_out, double *scratch,
                                           double *bcast)
{
    // r32 of every row is complete (caller passed a barrier)
    double acc = 0.0;
    if (use) {
        if constexpr (Spmv::kSliced) {
            bool ok = true;
            (void)sp.template apply<__nv_bfloat16, __nv_bfloat16>(
                A.F, A.r16, A.q, nullptr, A.n, A.gb.limit_ns, A.gb.status,
                ok);  // t = F r (interleaved rows)
            if (!ok) return false;
            const int G = gridDim.x, nr = interleaved_rows(A.n, blockIdx.x, G);
            for (int i = threadIdx.x; i < nr; i += blockDim.x) {
                const int j = blockIdx.x + G * i;
                A.t16[j] = __float2bfloat16_rn(float(A.q[j]));
            }
            if (!grid_barrier(A.gb)) return false;
            acc = sp.template apply<__nv_bfloat16, __nv_bfloat16>(
                A.FT, A.t16, A.y, A.r, A.n, A.gb.limit_ns, A.gb.status,
                ok);  // y = F^T t, r.y
            if (!ok) return false;
        } else {
            spmv_rows<LPRG, float>(A.F, A.r32, A.q, row0, row1, nullptr);  // t = F r
            __syncthreads();
            for (int j = row0 + threadIdx.x; j < row1; j += blockDim.x) A.p32[j] = float(A.q[j]);
            if (!grid_barrier(A.gb)) return false;
            spmv_rows<LPRG, float>(A.FT, A.p32, A.y, row0, row1, nullptr);  // y = F^T t
            __syncthreads();
            for (int j = row0 + threadIdx.x; j < row1; j += blockDim.x) acc = fma(A.r[j], A.y[j], acc);
        }
    } else {
        for (int j = row0 + threadIdx.x; j < row1; j += blockDim.x) {
            A.y[j] = A.r[j];
            acc = fma(A.r[j], A.r[j], acc);
        }
    }
    put_partial(A, kSlotD, acc, scratch);
    if (!grid_barrier(A.gb)) return false;
    rho_out = get_total(A, kSlotD, &bcast[2]);
    return true;
}

// r' in the precision the factor products gather: BF16 for the sliced
// copies (rounding the gathered vector to BF16 measured no extra
// iterations on these matrices), FP32 for the row plan.
template <class Spmv>
__device__ __forceinline__ void put_r_lowp(const OuterArgs &A, int j, double rv)
{
    if constexpr (Spmv::kSliced) A.r16[j] = __float2bfloat16_rn(float(rv));
    else A.r32[j] = float(rv);
}

// Solver state of the preconditioned body that does not need registers:
// thread 0 writes it after a reduction every thread already holds, and the
// CTA barriers of the next phase order the write before any read.  The
// stall test compares |r|^2 with its value four iterations earlier through
// a ring of five, so the slot read and the slot written in one iteration
// differ.
struct PcgShared {
    double stop2;       // (tol ||x||)^2
    double rr_cycle;    // |r|^2 at the last true residual
    double ring[5];     // |r|^2 after iteration k (k % 5; the refresh value at its own k)
};

template <class Spmv, int LPRG>
__device__ __forceinline__ void outer_step_pcg_body(const OuterArgs &A)
{
    __shared__ double scratch[32];
    __shared__ double bcast[8];
    __shared__ PcgShared st;
    const int row0 = A.row_split[blockIdx.x];
    const int row1 = A.row_split[blockIdx.x + 1];
    Spmv sp;
    sp.setup(A.M, row0, row1);
    bool ok = true;
    {
        const int vend = (blockIdx.x == gridDim.x - 1) ? row1 + 1 : row1;
        const int v = recycle_depth(A);
        double xx = 0.0;
        double acc = 0.0;
        if (v > 0) {
            // Galerkin start: r' = b' - A' z0 = A z0 - x
            if (!galerkin_start(galerkin_args(A), row0, row1, vend, v, &xx)) return;
            for (int j = row0 + threadIdx.x; j < vend; j += blockDim.x) {
                const double rv = A.q[j] - A.x[j];
                A.r[j] = rv;
                put_r_lowp<Spmv>(A, j, rv);
                if (j < A.n) acc = fma(rv, rv, acc);
            }
        } else {
            // z0 = 0, r' = b' = -x
            for (int j = row0 + threadIdx.x; j < vend; j += blockDim.x) {
                const double xv = A.x[j];
                A.q[j] = 0.0;
                A.z[j] = 0.0;
                A.r[j] = -xv;
                put_r_lowp<Spmv>(A, j, -xv);
                if (j < A.n) acc = fma(xv, xv, acc);
            }
        }
        put_partial(A, kSlotRho, acc, scratch);
        CGB_BARRIER_OR_RETURN(A);
        const double rr = get_total(A, kSlotRho, &bcast[3]);
        if (v == 0) xx = rr;
        if (threadIdx.x == 0) {
            st.stop2 = A.tol * A.tol * xx;
            st.rr_cycle = rr;
            st.ring[0] = rr;
        }
    }
    bool use_prec = true;
    int fallbacks = 0;
    double rho = 0.0;
    // p = y = M r'
    if (!apply_prec<Spmv, LPRG>(sp, A, row0, row1, use_prec, rho, scratch, bcast)) return;
    for (int j = row0 + threadIdx.x; j < row1; j += blockDim.x) {
        A.p[j] = A.y[j];
        A.p32[j] = float(A.y[j]);
    }
    CGB_BARRIER_OR_RETURN(A);

    int it = 0, since = 0, refreshes = 0;
    bool fresh = true;
    for (;;) {
        bool refresh = false;
        {
            const double rr = bcast[3];  // |r|^2 (every path leaves it there)
            if (rr <= st.stop2) {
                if (fresh) break;
                refresh = true;
            } else if (!fresh && (since >= A.refresh_every || rr <= kDrift2 * st.rr_cycle)) {
                refresh = true;
            }
        }
        if (!refresh && it >= A.cgitmax) break;
        bool restart = refresh;
        if (refresh) {
            // r' = b' - A' z = A z - x (FP64 matrix)
            spmv<Spmv, double>(sp, A, A.z, A.r, nullptr, ok);
            CGB_OK_OR_RETURN(ok && product_ready<Spmv>(A));
            double acc = 0.0;
            for (int j = row0 + threadIdx.x; j < row1; j += blockDim.x) {
                const double rv = product_at<Spmv>(A, A.r, j) - A.x[j];
                A.r[j] = rv;
                put_r_lowp<Spmv>(A, j, rv);
                acc = fma(rv, rv, acc);
            }
            put_partial(A, kSlotRho, acc, scratch);
            CGB_BARRIER_OR_RETURN(A);
            const double rr = get_total(A, kSlotRho, &bcast[3]);
            if (threadIdx.x == 0) {
                st.rr_cycle = rr;
                st.ring[it % 5] = rr;
            }
            refreshes++;
            since = 0;
            fresh = true;
            if (rr <= st.stop2) break;
        } else {
            // q = A32 p32; p.A'p = -p.q
            double acc = spmv<Spmv, float>(sp, A, A.p32, A.q, A.p, ok);
            CGB_OK_OR_RETURN(ok);
            put_partial(A, kSlotD, acc, scratch);
            CGB_BARRIER_OR_RETURN(A);
            const double pAp = -get_total(A, kSlotD, &bcast[2]);
            const double alpha = rho / pAp;
            acc = 0.0;
            for (int j = row0 + threadIdx.x; j < row1; j += blockDim.x) {
                A.z[j] = fma(alpha, A.p[j], A.z[j]);
                const double rv = fma(alpha, product_at<Spmv>(A, A.q, j), A.r[j]);  // r' -= alpha A'p
                A.r[j] = rv;
                put_r_lowp<Spmv>(A, j, rv);
                acc = fma(rv, rv, acc);
            }
            put_partial(A, kSlotRho, acc, scratch);
            CGB_BARRIER_OR_RETURN(A);
            const double rr = get_total(A, kSlotRho, &bcast[3]);
            it++;
            since++;
            fresh = false;
            // stall: no halving of |r|^2 over four steps (the ring slot of
            // it - 4, not the one written below), or lost positivity
            if (use_prec && (!(pAp > 0.0) || (since >= 4 && rr > 0.25 * st.ring[(it + 1) % 5]))) {
                use_prec = false;
                fallbacks++;
                restart = true;
            }
            if (threadIdx.x == 0) st.ring[it % 5] = rr;
        }
        // y = M r', new rho; p = y + beta p (beta = 0 on a restart)
        double rho_new = 0.0;
        if (!apply_prec<Spmv, LPRG>(sp, A, row0, row1, use_prec, rho_new, scratch, bcast)) return;
        if (use_prec && !(rho_new > 0.0)) {
            use_prec = false;
            fallbacks++;
            restart = true;
            if (!apply_prec<Spmv, LPRG>(sp, A, row0, row1, false, rho_new, scratch, bcast)) return;
        }
        const double beta = restart ? 0.0 : rho_new / rho;
        rho = rho_new;
        for (int j = row0 + threadIdx.x; j < row1; j += blockDim.x) {
            const double pv = fma(beta, A.p[j], A.y[j]);
            A.p[j] = pv;
            A.p32[j] = float(pv);
        }
        CGB_BARRIER_OR_RETURN(A);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) A.trace[A.step].spare[0] = double(fallbacks);
    end_solve(sp, A, row0, row1, it, bcast[3], refreshes, fresh, scratch, bcast, -1.0);
}

// Block shapes of the sliced kernels (one CTA per SM; each thread may use
// 65536 / block registers).  768 threads (80 registers) let the FP64 walk
// keep six step pairs a lane in flight without spilling -- at class B, whose
// column blocks hold short slices, that shortens each warp's chain of
// dependent loads; the preconditioned body holds the most live state and
// runs with 512 (128 registers).
constexpr int kSlicedBlock = 768;
constexpr int kSlicedMixedBlock = 768;
constexpr int kSlicedPcgBlock = 512;

template <int LPR>
__global__ void __launch_bounds__(512, 2) outer_step_fp64(OuterArgs A)
{
    outer_step_body<RowSpmv<LPR>>(A);
}

static __global__ void __launch_bounds__(kSlicedBlock, 1) outer_step_fp64_sliced(OuterArgs A)
{
    outer_step_body<SlicedSpmv>(A);
}

// the same with the L2 prefetch of each warp's next-block slices
static __global__ void __launch_bounds__(kSlicedBlock, 1) outer_step_fp64_sliced_pf(OuterArgs A)
{
    outer_step_body<SlicedSpmvPf>(A);
}

template <int LPR>
__global__ void __launch_bounds__(512, 2) outer_step_mixed(OuterArgs A)
{
    outer_step_mixed_body<RowSpmv<LPR>>(A);
}

static __global__ void __launch_bounds__(kSlicedMixedBlock, 1) outer_step_mixed_sliced(OuterArgs A)
{
    outer_step_mixed_body<SlicedSpmvMixed>(A);
}

static __global__ void __launch_bounds__(kSlicedMixedBlock, 1) outer_step_mixed_sliced_pf(OuterArgs A)
{
    outer_step_mixed_body<SlicedSpmvMixedPf>(A);
}

// Column-part instances (slice_shape)
static __global__ void __launch_bounds__(kSlicedBlock, 1) outer_step_fp64_parts(OuterArgs A)
{
    outer_step_body<PartSpmv64>(A);
}

static __global__ void __launch_bounds__(kSlicedMixedBlock, 1) outer_step_mixed_parts(OuterArgs A)
{
    outer_step_mixed_body<PartSpmvMixed>(A);
}

// Row-panel instances: the sliced plan of a matrix whose rows per CTA do
// not fit the shared accumulators (class D: 10 K rows a CTA).
static __global__ void __launch_bounds__(kSlicedBlock, 1) outer_step_fp64_sliced_pn(OuterArgs A)
{
    outer_step_body<SlicedSpmvPanels>(A);
}

static __global__ void __launch_bounds__(kSlicedMixedBlock, 1) outer_step_mixed_sliced_pn(OuterArgs A)
{
    outer_step_mixed_body<SlicedSpmvMixedPanels>(A);
}

// lanes per row of the preconditioner products (F has about half of A's
// entries per row)
constexpr int kLanesF = 16;

template <int LPR>
__global__ void __launch_bounds__(512, 2) outer_step_pcg(OuterArgs A)
{
    outer_step_pcg_body<RowSpmv<LPR>, kLanesF>(A);
}

static __global__ void __launch_bounds__(kSlicedPcgBlock, 1) outer_step_pcg_sliced(OuterArgs A)
{
    outer_step_pcg_body<SlicedSpmvPcg, kLanesF>(A);
}

static __global__ void __launch_bounds__(kSlicedPcgBlock, 1) outer_step_pcg_parts(OuterArgs A)
{
    outer_step_pcg_body<PartSpmvPcg, kLanesF>(A);
}

static __global__ void __launch_bounds__(kSlicedPcgBlock, 1) outer_step_pcg_sliced_pn(OuterArgs A)
{
    outer_step_pcg_body<SlicedSpmvPcgPanels, kLanesF>(A);
}

// Standalone q = A p with the p.q reduction fused (the work of reference
// kernels three and four, cg.cu:937-1004): per-CTA partials, the last CTA to
// finish (ticket counter) sums them in a fixed order into *dot.
struct SpmvArgs {
    OuterArgs A;
    unsigned *ticket;
    unsigned *group_ticket;  // column parts: one a group, zero between launches
    double *dot;
    int fp32;  // 1: q = A32 p32
};

// kPrec: 0 = FP64 or FP32 by S.fp32; 1 = FP64 only; 2 = FP32 only (a kernel
// per precision keeps each one's register allocation to itself).
template <class Spmv, int kPrec>
__device__ __forceinline__ void spmv_dot_body(const SpmvArgs &S)
{
    __shared__ double scratch[32];
    __shared__ bool last;
    const OuterArgs &A = S.A;
    Spmv sp;
    sp.setup(A.M, A.row_split[blockIdx.x], A.row_split[blockIdx.x + 1]);
    bool ok = true;
    double acc;
    if constexpr (kPrec == 1) acc = spmv<Spmv, double>(sp, A, A.p, A.q, A.p, ok);
    else if constexpr (kPrec == 2) acc = spmv<Spmv, float>(sp, A, A.p32, A.q, A.p, ok);
    else acc = S.fp32 ? spmv<Spmv, float>(sp, A, A.p32, A.q, A.p, ok)
                      : spmv<Spmv, double>(sp, A, A.p, A.q, A.p, ok);
    if (!ok) return;
    if constexpr (Spmv::kParts) {
        if (int(blockIdx.x) < A.M.part_ctas) {  // the group's last CTA adds its rows' parts
            __threadfence();
            __syncthreads();
            const int group = int(blockIdx.x) / A.M.parts;
            if (threadIdx.x == 0) last = atomicAdd(S.group_ticket + group, 1u) == unsigned(A.M.parts - 1);
            __syncthreads();
            if (last) {
                __threadfence();
                const int j1 = A.M.group_split[group + 1];
                for (int j = A.M.group_split[group] + threadIdx.x; j < j1; j += blockDim.x)
                    A.q[j] = product_at<Spmv>(A, A.q, j);
                if (threadIdx.x == 0) S.group_ticket[group] = 0u;
            }
        }
    }
    const double s = block_sum(acc, scratch);
    if (threadIdx.x == 0) {
        A.part[blockIdx.x] = s;
        __threadfence();
        last = (atomicAdd(S.ticket, 1u) == gridDim.x - 1);
    }
    __syncthreads();
    if (last) {
        __threadfence();
        if (threadIdx.x < 32) {
            double t = 0.0;
            for (int i = threadIdx.x; i < (int)gridDim.x; i += 32) t += __ldcg(A.part + i);
            t = warp_sum(t);
            if (threadIdx.x == 0) {
                *S.dot = t;
                *S.ticket = 0u;
            }
        }
    }
}

template <int LPR>
__global__ void __launch_bounds__(512, 2) spmv_dot_row(SpmvArgs S)
{
    spmv_dot_body<RowSpmv<LPR>, 0>(S);
}

static __global__ void __launch_bounds__(kSlicedBlock, 1) spmv_dot_sliced(SpmvArgs S)
{
    spmv_dot_body<SlicedSpmv, 1>(S);
}

static __global__ void __launch_bounds__(kSlicedBlock, 1) spmv_dot_sliced32(SpmvArgs S)
{
    spmv_dot_body<SlicedSpmv, 2>(S);
}

static __global__ void __launch_bounds__(kSlicedBlock, 1) spmv_dot_sliced_pf(SpmvArgs S)
{
    spmv_dot_body<SlicedSpmvPf, 1>(S);
}

static __global__ void __launch_bounds__(kSlicedBlock, 1) spmv_dot_sliced32_pf(SpmvArgs S)
{
    spmv_dot_body<SlicedSpmvPf, 2>(S);
}

static __global__ void __launch_bounds__(kSlicedBlock, 1) spmv_dot_parts(SpmvArgs S)
{
    spmv_dot_body<PartSpmv64, 1>(S);
}

static __global__ void __launch_bounds__(kSlicedBlock, 1) spmv_dot_parts32(SpmvArgs S)
{
    spmv_dot_body<PartSpmvMixed, 2>(S);
}

static __global__ void __launch_bounds__(kSlicedBlock, 1) spmv_dot_sliced_pn(SpmvArgs S)
{
    spmv_dot_body<SlicedSpmvPanels, 1>(S);
}

static __global__ void __launch_bounds__(kSlicedBlock, 1) spmv_dot_sliced32_pn(SpmvArgs S)
{
    spmv_dot_body<SlicedSpmvPanels, 2>(S);
}

// ------------------------------------------------------------- utilities
// Demotes the L2 lines of [p, p + bytes) to normal eviction priority: the
// lines a sliced walk kept at evict_last, so that whoever uses the L2 next
// starts from plain replacement.  Touches no data (a priority hint on lines
// that are cached, nothing for the others).
static __global__ void l2_demote(const char *p, size_t bytes)
{
    const size_t step = size_t(gridDim.x) * blockDim.x * 128;
    for (size_t o = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) * 128; o < bytes; o += step)
        asm volatile("applypriority.global.L2::evict_normal [%0], 128;" ::"l"(p + o) : "memory");
}

// x = 1 over n+1 entries (cg.cu:485-488).
static __global__ void fill_ones(double *x, int count)
{
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < count; j += gridDim.x * blockDim.x)
        x[j] = 1.0;
}

// out[i] = (float) in[i].
static __global__ void to_fp32(const double *__restrict__ in, float *__restrict__ out,
                               long long count)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count;
         i += (long long)gridDim.x * blockDim.x)
        out[i] = float(in[i]);
}

// Segment table of the column blocking: seg[b*stride + j] = first entry of
// row j whose column is >= b*width (b < nblk), seg[nblk*stride + j] = end of
// row j; *unsorted is set when some row's columns do not ascend.
static __global__ void build_segments(const int *__restrict__ rowstr,
                                      const int *__restrict__ colidx, int n, int nblk, int width,
                                      int *seg, int stride, int *unsorted)
{
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const int k0 = rowstr[j], k1 = rowstr[j + 1];
        int bad = 0;
        for (int k = k0 + 1; k < k1; k++) bad |= (colidx[k] <= colidx[k - 1]);
        if (bad) atomicOr(unsorted, 1);
        for (int b = 0; b < nblk; b++) {
            const int lo_col = b * width;
            int lo = k0, hi = k1;  // first k with colidx[k] >= lo_col
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (colidx[mid] < lo_col) lo = mid + 1;
                else hi = mid;
            }
            seg[size_t(b) * stride + j] = lo;
        }
        seg[size_t(nblk) * stride + j] = k1;
    }
}

// Sliced layout, step 1 -- one CTA per chunk (row panel k of CTA c of the
// solve grid, column block b; chunk (c*panels + k)*nblk + b): order the
// chunk's rows by descending segment length
// (counting sort on min(len, 255)), 32 to a slice; srow gets the local row of
// each (slice, lane), 0xffff for the tail; slice_width the longest segment,
// rounded up to even.
// Each row is summed by one lane in its CSR order wherever it lands; rows of a
// bin keep their order (below).
// Rows of CTA c: row_split[c] + i for i < row_split[c+1] - row_split[c], or
// (interleaved, grid G) c + G i for i < interleaved_rows(n, c, G).  Row
// panel k of `panels` takes the local rows [panel_begin(rows, k), panel_begin(
// rows, k+1)); pc = c*panels + k names the panel, local row i of a panel is
// i after its first.
__device__ __forceinline__ int cta_rows(const int *row_split, int interleave_grid, int n, int c)
{
    return interleave_grid ? interleaved_rows(n, c, interleave_grid) : row_split[c + 1] - row_split[c];
}
__device__ __forceinline__ int panel_rows(const int *row_split, int interleave_grid, int n,
                                          int panels, int pc)
{
    const int rows = cta_rows(row_split, interleave_grid, n, pc / panels), k = pc % panels;
    return panel_begin(rows, k + 1, panels) - panel_begin(rows, k, panels);
}
__device__ __forceinline__ int chunk_row(const int *row_split, int interleave_grid, int n, int panels,
                                         int pc, int i)
{
    const int c = pc / panels;
    const int li = panel_begin(cta_rows(row_split, interleave_grid, n, c), pc % panels, panels) + i;
    return interleave_grid ? c + interleave_grid * li : row_split[c] + li;
}

constexpr int kSortBlock = 256;
static __global__ void __launch_bounds__(kSortBlock) slice_sort_rows(const int *__restrict__ seg, int seg_stride, int nblk,
                                       const int *__restrict__ row_split, int interleave_grid,
                                       int panels, int n, const int *__restrict__ chunk_slice,
                                       unsigned short *srow, int *slice_width)
{
    __shared__ int hist[256], count[kSortBlock / 32][256];
    const int pc = blockIdx.x / nblk, b = blockIdx.x % nblk;
    const int nrows = panel_rows(row_split, interleave_grid, n, panels, pc);
    const int s0 = chunk_slice[blockIdx.x], ns = chunk_slice[blockIdx.x + 1] - s0;
    const int *lo = seg + size_t(b) * seg_stride;
    const int *hi = seg + size_t(b + 1) * seg_stride;
#define SEG_LEN(i) (hi[chunk_row(row_split, interleave_grid, n, panels, pc, (i))] - \
                    lo[chunk_row(row_split, interleave_grid, n, panels, pc, (i))])
    for (int i = threadIdx.x; i < 256; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < nrows; i += blockDim.x)
        atomicAdd(&hist[255 - min(SEG_LEN(i), 255)], 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int k = 0; k < 256; k++) {
            const int h = hist[k];
            hist[k] = run;
            run += h;
        }
    }
    __syncthreads();
    unsigned short *dst = srow + size_t(s0) * 32;
    // rows of one length stay in order, so that the slices -- and with column
    // parts the order in which p.q is summed -- are the same every time
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int t0 = 0; t0 < nrows; t0 += kSortBlock) {
        const int i = t0 + threadIdx.x;
        const int key = i < nrows ? 255 - min(SEG_LEN(i), 255) : 256;
#pragma unroll
        for (int w = 0; w < kSortBlock / 32; w++) count[w][threadIdx.x] = 0;
        __syncthreads();
        const unsigned same = __match_any_sync(~0u, key);
        const int before = __popc(same & ((1u << lane) - 1u));
        if (key < 256 && before == 0) count[warp][key] = __popc(same);
        __syncthreads();
        if (key < 256) {
            int pos = hist[key] + before;
            for (int w = 0; w < warp; w++) pos += count[w][key];
            dst[pos] = (unsigned short)i;
        }
        __syncthreads();
#pragma unroll
        for (int w = 0; w < kSortBlock / 32; w++) hist[threadIdx.x] += count[w][threadIdx.x];
    }
    for (int i = nrows + threadIdx.x; i < ns * 32; i += blockDim.x) dst[i] = 0xffffu;
    __syncthreads();
    for (int t = threadIdx.x; t < ns; t += blockDim.x) {
        int w = 0;
        for (int l = 0; l < 32; l++) {
            const unsigned short row = dst[t * 32 + l];
            if (row != 0xffffu) w = max(w, SEG_LEN(row));
        }
        slice_width[s0 + t] = (w + 1) & ~1;  // whole step pairs
    }
#undef SEG_LEN
}

// Step 2 -- one CTA: slice_off[s] = 32 * sum_{s' < s} width[s'];
// slice_off[total] = all entries.  Per-thread ranges, then a serial scan of
// the per-thread sums.
static __global__ void slice_offsets(const int *__restrict__ width, int total, unsigned *slice_off)
{
    __shared__ unsigned part[1024];
    const int per = (total + blockDim.x - 1) / blockDim.x;
    const int a = threadIdx.x * per, e = min(total, a + per);
    unsigned s = 0;
    for (int i = a; i < e; i++) s += 32u * unsigned(width[i]);
    part[threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned run = 0;
        for (int t = 0; t < (int)blockDim.x; t++) {
            const unsigned v = part[t];
            part[t] = run;
            run += v;
        }
        slice_off[total] = run;
    }
    __syncthreads();
    unsigned run = part[threadIdx.x];
    for (int i = a; i < e; i++) {
        slice_off[i] = run;
        run += 32u * unsigned(width[i]);
    }
}

// Step 3 -- one warp per slice: copy each lane's row segment in step-pair
// column-major order (entry k of lane i at off + 64 (k/2) + 2 i + k%2),
// values (from FP64 or FP32 source values; sval or sval32 may be null) and
// 16-bit local columns; padding steps get value 0, column 0.
template <typename ST>
__global__ void slice_fill(const int *__restrict__ seg, int seg_stride, int nblk, int width,
                           const int *__restrict__ row_split, int interleave_grid, int panels,
                           int n, const int *__restrict__ chunk_slice,
                           int nchunks, const int *__restrict__ colidx, const ST *__restrict__ a,
                           const unsigned short *__restrict__ srow,
                           const int *__restrict__ slice_width,
                           const unsigned *__restrict__ slice_off, int total, double *sval,
                           float *sval32, __nv_bfloat16 *sval16, unsigned short *scol)
{
    const int lane = threadIdx.x & 31;
    for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < total;
         s += (gridDim.x * blockDim.x) >> 5) {
        int lo = 0, hi = nchunks;  // chunk of slice s: last ch with chunk_slice[ch] <= s
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (chunk_slice[mid] <= s) lo = mid;
            else hi = mid;
        }
        const int pc = lo / nblk, b = lo % nblk;
        const unsigned short row = srow[size_t(s) * 32 + lane];
        int e0 = 0, e1 = 0;
        if (row != 0xffffu) {
            const int j = chunk_row(row_split, interleave_grid, n, panels, pc, row);
            e0 = seg[size_t(b) * seg_stride + j];
            e1 = seg[size_t(b + 1) * seg_stride + j];
        }
        const int w = slice_width[s];
        const unsigned off = slice_off[s] + 2u * lane;
        const int base = b * width;
        for (int k = 0; k < w; k++) {
            const int e = e0 + k;
            double v = 0.0;
            int col = 0;
            if (e < e1) {
                v = double(a[e]);
                col = colidx[e] - base;
            }
            const unsigned at = off + 64u * unsigned(k >> 1) + unsigned(k & 1);
            if (sval) sval[at] = v;
            if (sval32) sval32[at] = float(v);
            if (sval16) sval16[at] = __float2bfloat16_rn(float(v));
            scol[at] = (unsigned short)col;
        }
    }
}

// Self-test of the bounded wait: CTA 1 never arrives, so CTA 0's barrier
// wait runs into its limit and records kDevTimeout.
// `iters` grid barriers back to back: the barrier's cost (cgb_time_barrier).
static __global__ void barrier_loop(GridBarrier gb, int iters)
{
    for (int i = 0; i < iters; i++)
        if (!grid_barrier(gb)) return;
}

// An empty persistent kernel: launched with an outer step's shape (grid,
// block, dynamic shared memory, cooperative) it costs what a kernel
// boundary costs in the solve's graph -- launch, CTA dispatch, teardown --
// and nothing else (cgb_time_outer_steps).
static __global__ void __launch_bounds__(1024, 1) launch_probe(int) {}

static __global__ void barrier_timeout_probe(GridBarrier gb)
{
    if (blockIdx.x == 1) return;
    (void)grid_barrier(gb);
}

}  // namespace cgb

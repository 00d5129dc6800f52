// mg.cu -- the NPB MG benchmark's V-cycle on the GPU: a multigrid solve of
// the 3-D Poisson problem on a periodic 2^lt cube (GMAP/NPB-GPU
// CUDA/MG/mg.cu: main's timed loop :498-508, mg3P :1078-1133).
//
// Grids are cubes of side m = 2^k + 2 (one ghost layer a face), x fastest,
// one buffer per level for u and r, v on the finest level only.  The operators:
//   resid   r = v - A u       (:1572-1625)  27-point, a[1] = 0
//   psinv   u = u + C r       (:1395-1440)  27-point, c[3] = 0
//   rprj3   s = P^T r         (:1724-1790)  full weighting onto the coarse grid
//   interp  u (+)= P z        (:836-890)    trilinear prolongation
//   norm2u3                   (:1201-1230)  deterministic two-level reduction
// A V-cycle runs them fused: k_down (resid, rprj3) and k_up (interp, resid,
// psinv) walk a level along z and keep the intermediate grids on the SM;
// k_coarse runs every level up to 32^3 in one launch of a cluster.  Each
// operator is also a kernel of its own for cgb_mg_apply (k_rprj3 serves the
// levels between as well): the 27-point ones stage their input in shared
// memory, plane by plane along z (a ring of three planes of a 32 x 8 tile
// with its halo, the next plane loading while the current one is computed).
// The periodic ghost exchange (comm3, :687-716, which only copies interior
// values) is fused: the thread that writes an interior point also writes that
// value into each ghost cell that mirrors it.  On coarse levels the reference
// zeroes u and then adds the prolongation; here u' = 0 + P z in one pass.
//
// Arithmetic: every sum in the reference's order and no fused multiply-add
// (this file is compiled with -fmad=false), so each grid equals the serial
// reference's operation for operation; only the norm's sum runs in another
// (fixed) order.  The whole timed region is one CUDA graph.
//
// zran3 (:2175-2303): the LCG value of interior point (i1, i2, i3) is draw
// L + 1 of the stream seeded 314159265 with multiplier 5^13, L = (i1-1) +
// n (i2-1) + n^2 (i3-1).  Each thread jumps to its chunk's first draw and
// steps through the chunk, keeping the values above 1 - C/N and below C/N
// (a few hundred candidates); the host picks the ten largest and smallest
// among them -- the values are distinct, so that is the reference's choice.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <new>
#include <utility>
#include <vector>

#include "cgb_internal.h"

namespace cgb {
namespace mg {

constexpr int kMaxLevels = 11;   // lt <= 10: a 1024^3 grid (class D)
constexpr int kRows = 4;         // (y) rows of a restriction / prolongation CTA; x is a warp
constexpr int kNormBlocks = 1184;
constexpr int kNormThreads = 256;
constexpr int kCandCap = 8192;   // zran3 candidates kept per side
constexpr int kChunk = 64;       // zran3 draws a thread steps through
constexpr uint64_t kMask46 = (uint64_t(1) << 46) - 1;
constexpr uint64_t kMult = 1220703125ull;  // 5^13
constexpr uint64_t kSeed = 314159265ull;

struct Coef {
    double a0, a2, a3;  // resid: a[1] = 0 is left out, as the reference does
    double c0, c1, c2;  // psinv: c[3] = 0 is left out
};

// Launched with programmatic stream serialization, a kernel may start while
// its predecessor drains: it waits here before it touches what the
// predecessor wrote, and lets its own successor start at once.
__device__ __forceinline__ void wait_for_predecessor()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ size_t at(int m, int i3, int i2, int i1)
{
    return (size_t(i3) * m + i2) * m + i1;
}

// The indices along one axis that hold the value of interior index i: i
// itself and, at the two ends, the ghost that mirrors it (comm3's copies).
__device__ __forceinline__ int images(int m, int i, int *out)
{
    int k = 0;
    out[k++] = i;
    if (i == m - 2) out[k++] = 0;
    if (i == 1) out[k++] = m - 1;
    return k;
}

// g(i1, i2, i3) = val and every ghost cell that comm3 would fill from it.
__device__ __forceinline__ void store_periodic(double *g, int m, int i3, int i2, int i1, double val)
{
    int x[2], y[2], z[2];
    const int nx = images(m, i1, x), ny = images(m, i2, y), nz = images(m, i3, z);
    for (int c = 0; c < nz; c++)
        for (int b = 0; b < ny; b++)
            for (int a = 0; a < nx; a++) g[at(m, z[c], y[b], x[a])] = val;
}

// The 27-point operators (resid, psinv) stage their input grid in shared
// memory: a CTA owns a 32 x 8 (x, y) tile and walks kPlanes z planes,
// keeping planes z-1, z, z+1 of the tile plus a one-cell halo in a ring of
// three (34 x 10 doubles each), so each input value is read from L2/HBM
// about once instead of by nine threads; the next plane's loads are issued
// into registers before the current plane is computed.  A thread owns one
// x of two consecutive rows, so the four rows of each staged plane around
// them serve both points' column sums (12 shared reads for two points
// instead of 16, the centres with them).  A warp is 32 consecutive x: a
// lane takes its neighbours' column sums by shuffles.  kPsinv:
// u = u + C g (g = r); otherwise out = w - A g (g = u, w = v; out may be w).
constexpr int kPlanes = 16;
constexpr int kTileW = 34;

constexpr int kRB = 2;                    // rows a thread
constexpr int kWarpsRB = 4;
constexpr int kRowsRB = kRB * kWarpsRB;   // 8 rows a tile
constexpr int kTileRB = kTileW * (kRowsRB + 2);
constexpr int kThreadsRB = 32 * kWarpsRB;
constexpr int kStageRB = (kTileRB + kThreadsRB - 1) / kThreadsRB;  // cells a thread stages

template <bool kPsinv>
__global__ void __launch_bounds__(kThreadsRB) k_stencil_rb(const double *__restrict__ g, const double *w,
                                                           double *out, int m, Coef cf)
{
    __shared__ double ring[3][kTileRB];
    wait_for_predecessor();
    const int n = m - 2;
    const int tx = threadIdx.x, wy = threadIdx.y, t = wy * 32 + tx;
    const int x0 = 1 + int(blockIdx.x) * 32, y0 = 1 + int(blockIdx.y) * kRowsRB;
    const int z0 = 1 + int(blockIdx.z) * kPlanes, z1 = min(n, z0 + kPlanes - 1);
    const int x = x0 + tx, yb = y0 + wy * kRB;
    const size_t plane = size_t(m) * m;
    size_t off[kStageRB];
    bool inside[kStageRB];
#pragma unroll
    for (int q = 0; q < kStageRB; q++) {
        const int e = t + q * kThreadsRB;
        const int gx = x0 - 1 + e % kTileW, gy = y0 - 1 + e / kTileW;
        inside[q] = e < kTileRB && gx <= m - 1 && gy <= m - 1;
        off[q] = size_t(gy) * m + gx;
    }
    auto fetch = [&](int z, double *v) {
#pragma unroll
        for (int q = 0; q < kStageRB; q++) v[q] = inside[q] ? g[z * plane + off[q]] : 0.0;
    };
    auto put = [&](int z, const double *v) {
#pragma unroll
        for (int q = 0; q < kStageRB; q++) {
            const int e = t + q * kThreadsRB;
            if (e < kTileRB) ring[z % 3][e] = v[q];
        }
    };
    {
        double a[kStageRB], b[kStageRB], c[kStageRB];
        fetch(z0 - 1, a);
        fetch(z0, b);
        fetch(z0 + 1, c);
        put(z0 - 1, a);
        put(z0, b);
        put(z0 + 1, c);
    }
    __syncthreads();
    const int lx = tx + 1, lr = wy * kRB;  // the tile row above this thread's first row
    for (int z = z0; z <= z1; z++) {
        double next[kStageRB];
        if (z + 1 <= z1) fetch(z + 2, next);  // in flight during this plane
        double wc[kRB];
#pragma unroll
        for (int i = 0; i < kRB; i++) {
            const int y = yb + i;
            wc[i] = (x <= n && y <= n) ? (kPsinv ? out[at(m, z, y, x)] : w[at(m, z, y, x)]) : 0.0;
        }
        const double *Pm = ring[(z - 1) % 3], *P0 = ring[z % 3], *Pp = ring[(z + 1) % 3];
        // rows lr .. lr + kRB + 1 of column k in the three planes, and the
        // kRB rows' column sums (the reference's u1, u2) and centres
        auto column = [&](int k, double *s1, double *s2, double *ctr) {
            double a[kRB + 2], b[kRB + 2], c[kRB + 2];
#pragma unroll
            for (int j = 0; j < kRB + 2; j++) {
                a[j] = P0[(lr + j) * kTileW + k];
                b[j] = Pm[(lr + j) * kTileW + k];
                c[j] = Pp[(lr + j) * kTileW + k];
            }
#pragma unroll
            for (int i = 0; i < kRB; i++) {
                s1[i] = a[i] + a[i + 2] + b[i + 1] + c[i + 1];
                s2[i] = b[i] + b[i + 2] + c[i] + c[i + 2];
                ctr[i] = a[i + 1];
            }
        };
        double s1[kRB], s2[kRB], ctr[kRB], s1m[kRB], s2m[kRB], cm[kRB], s1p[kRB], s2p[kRB], cp[kRB];
        column(lx, s1, s2, ctr);
#pragma unroll
        for (int i = 0; i < kRB; i++) {
            s1m[i] = __shfl_up_sync(0xffffffffu, s1[i], 1);
            s2m[i] = __shfl_up_sync(0xffffffffu, s2[i], 1);
            s1p[i] = __shfl_down_sync(0xffffffffu, s1[i], 1);
            s2p[i] = __shfl_down_sync(0xffffffffu, s2[i], 1);
            cm[i] = __shfl_up_sync(0xffffffffu, ctr[i], 1);
            cp[i] = __shfl_down_sync(0xffffffffu, ctr[i], 1);
        }
        if (tx == 0) column(lx - 1, s1m, s2m, cm);
        if (tx == 31) column(lx + 1, s1p, s2p, cp);
#pragma unroll
        for (int i = 0; i < kRB; i++) {
            const int y = yb + i;
            if (x > n || y > n) continue;
            double val;
            if constexpr (kPsinv)
                val = wc[i] + cf.c0 * ctr[i] + cf.c1 * (cm[i] + cp[i] + s1[i]) +
                      cf.c2 * (s2[i] + s1m[i] + s1p[i]);
            else
                val = wc[i] - cf.a0 * ctr[i] - cf.a2 * (s2[i] + s1m[i] + s1p[i]) -
                      cf.a3 * (s2m[i] + s2p[i]);
            store_periodic(out, m, z, y, x, val);
        }
        __syncthreads();  // every read of plane z-1's slot is done
        if (z + 1 <= z1) put(z + 2, next);
        __syncthreads();
    }
}

// s (side mj) = restriction of r (side mk = 2 mj - 2).  A thread per coarse
// column j1 in [1, mj - 1]: its x1 / y1 (at fine i1 = 2 j1 - 1), the next
// lane's for i1 + 2; outputs for j1 <= mj - 2.
__global__ void __launch_bounds__(32 * kRows) k_rprj3(const double *__restrict__ r, int mk, double *s,
                                                      int mj)
{
    wait_for_predecessor();
    const int lane = threadIdx.x & 31;
    const int j1 = 1 + int(blockIdx.x) * 32 + int(threadIdx.x);
    const int j2 = 1 + int(blockIdx.y) * kRows + int(threadIdx.y);
    const int j3 = 1 + int(blockIdx.z);
    if (j2 > mj - 2) return;
    const int i1 = 2 * j1 - 1, i2 = 2 * j2 - 1, i3 = 2 * j3 - 1;
    auto xy1 = [&](int x, double &x1, double &y1) {
        x1 = r[at(mk, i3 + 1, i2, x)] + r[at(mk, i3 + 1, i2 + 2, x)] + r[at(mk, i3, i2 + 1, x)] +
             r[at(mk, i3 + 2, i2 + 1, x)];
        y1 = r[at(mk, i3, i2, x)] + r[at(mk, i3 + 2, i2, x)] + r[at(mk, i3, i2 + 2, x)] +
             r[at(mk, i3 + 2, i2 + 2, x)];
    };
    double x1 = 0.0, y1 = 0.0;
    if (j1 <= mj - 1) xy1(i1, x1, y1);
    double x1p = __shfl_down_sync(0xffffffffu, x1, 1);
    double y1p = __shfl_down_sync(0xffffffffu, y1, 1);
    if (j1 > mj - 2) return;
    if (lane == 31) xy1(i1 + 2, x1p, y1p);
    const double y2 = r[at(mk, i3, i2, i1 + 1)] + r[at(mk, i3 + 2, i2, i1 + 1)] +
                      r[at(mk, i3, i2 + 2, i1 + 1)] + r[at(mk, i3 + 2, i2 + 2, i1 + 1)];
    const double x2 = r[at(mk, i3 + 1, i2, i1 + 1)] + r[at(mk, i3 + 1, i2 + 2, i1 + 1)] +
                      r[at(mk, i3, i2 + 1, i1 + 1)] + r[at(mk, i3 + 2, i2 + 1, i1 + 1)];
    const double val = 0.5 * r[at(mk, i3 + 1, i2 + 1, i1 + 1)] +
                       0.25 * (r[at(mk, i3 + 1, i2 + 1, i1)] + r[at(mk, i3 + 1, i2 + 1, i1 + 2)] + x2) +
                       0.125 * (x1 + x1p + y2) + 0.0625 * (y1 + y1p);
    store_periodic(s, mj, j3, j2, j1, val);
}

// u (side mk = 2 mj - 2) += (or, assign: =) prolongation of z (side mj).
// A thread per coarse cell (i1, i2, i3) in [0, mj - 2]^3 writes its eight
// fine points as four pairs.  Covers every fine cell, ghosts included.
__global__ void __launch_bounds__(32 * kRows) k_interp(const double *__restrict__ z, int mj, double *u,
                                                       int mk, int assign)
{
    const int i1 = int(blockIdx.x) * 32 + int(threadIdx.x);
    const int i2 = int(blockIdx.y) * kRows + int(threadIdx.y);
    const int i3 = int(blockIdx.z);
    if (i1 > mj - 2 || i2 > mj - 2) return;
    const double z000 = z[at(mj, i3, i2, i1)], z001 = z[at(mj, i3, i2, i1 + 1)];
    const double z010 = z[at(mj, i3, i2 + 1, i1)], z011 = z[at(mj, i3, i2 + 1, i1 + 1)];
    const double z100 = z[at(mj, i3 + 1, i2, i1)], z101 = z[at(mj, i3 + 1, i2, i1 + 1)];
    const double z110 = z[at(mj, i3 + 1, i2 + 1, i1)], z111 = z[at(mj, i3 + 1, i2 + 1, i1 + 1)];
    // the reference's line buffers at i1 and i1 + 1
    const double z1a = z010 + z000, z1b = z011 + z001;
    const double z2a = z100 + z000, z2b = z101 + z001;
    const double z3a = z110 + z100 + z1a, z3b = z111 + z101 + z1b;
    const double add[4][2] = {{z000, 0.5 * (z001 + z000)},
                              {0.5 * z1a, 0.25 * (z1a + z1b)},
                              {0.5 * z2a, 0.25 * (z2a + z2b)},
                              {0.25 * z3a, 0.125 * (z3a + z3b)}};
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int f3 = 2 * i3 + (q >> 1), f2 = 2 * i2 + (q & 1);
        double2 *p = reinterpret_cast<double2 *>(u + at(mk, f3, f2, 2 * i1));
        double2 w;
        if (assign) {
            w.x = 0.0 + add[q][0];
            w.y = 0.0 + add[q][1];
        } else {
            const double2 o = *p;
            w.x = o.x + add[q][0];
            w.y = o.y + add[q][1];
        }
        *p = w;
    }
}

// ---------------------------------------------------- the fused z marches
// The V-cycle's operators on one level, fused so that a level's grids cross
// HBM once:
//   k_up     u' = u + P z;  r = v - A u';  out = u' + C r   (interp, resid, psinv)
//   k_down   r = v - A u;   s = P^T r                        (resid, rprj3)
// u' and r stay on the SM (k_down writes r when asked).  A warp owns 64
// consecutive x (two a lane) of two consecutive y, a CTA kW such warps; it
// walks z, and from plane to plane a thread keeps, for its four points, what
// the next planes' column sums need (Plane27).  Rows of neighbouring warps
// come through shared memory, neighbouring x by shuffles.  The rows and
// columns at the tile's edge are computed by both neighbours: of 64 x 2 kW
// points a plane, 60 x (2 kW - 4) are the CTA's own.
//
// Indices F run over [0, n) with F = 0 standing for index n, whose image the
// ghost at 0 holds, so tiles start at even F and all accesses are aligned
// pairs; reads wrap F modulo n.  An image of F <= 1 lies at F + n (comm3).
//
// Every point's sums are formed in the reference's order, like the single
// operators' above, so the grids stay bit-identical.  HBM-bound by its
// algorithmic bytes: k_up moves 3.1 grids where interp, resid and psinv apart
// move 8.1, k_down 2.1 (3.1 writing r) where resid and rprj3 move 4.1.  At
// 512^3: interp, resid and psinv 443 + 793 + 811 us -> k_up 1058 us (3.2
// TB/s); resid and rprj3 793 + 307 -> k_down 824 us, writing r.  Both now wait
// mostly on the chain of a plane's two barriers, shuffles and dependent FP64
// adds, at 12 to 16 warps an SM.
constexpr int kOwnX = 60;  // own columns of a warp's 64
// Warps a CTA (one CTA an SM), by registers: k_up holds about 160 a thread.
// 16 warps at 128 with spills: class C 56.4 ms; two CTAs of 8: 63.0; 12: 41.3.
constexpr int kWarpsUp = 12, kWarpsDown = 16;

struct Plane27 {
    // of the plane before the centre and of the centre plane: the sums of
    // the rows above and below, and the points themselves; [row][column]
    double em[2][2], e0[2][2], cm[2][2], c0[2][2];

    // A new plane `p` of own rows, with the rows above (`up`) and below
    // (`dn`): the reference's column sums u1 and u2 around the centre plane,
    // then the new plane is the centre.
    __device__ __forceinline__ void step(const double (&p)[2][2], const double (&up)[2], const double (&dn)[2],
                                         double (&s1)[2][2], double (&s2)[2][2])
    {
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const double lo = i ? p[0][k] : up[k], hi = i ? dn[k] : p[1][k];
                s1[i][k] = e0[i][k] + cm[i][k] + p[i][k];
                s2[i][k] = em[i][k] + lo + hi;
                em[i][k] = e0[i][k];
                e0[i][k] = lo + hi;
                cm[i][k] = c0[i][k];
                c0[i][k] = p[i][k];
            }
    }
};

__device__ __forceinline__ int wrap(int f, int n)
{
    f %= n;
    return f < 0 ? f + n : f;
}

// The values left of column 0 and right of column 1 of a lane's pair: the
// left neighbour's column 1 and the right neighbour's column 0.
__device__ __forceinline__ double from_left(double v1) { return __shfl_up_sync(0xffffffffu, v1, 1); }
__device__ __forceinline__ double from_right(double v0) { return __shfl_down_sync(0xffffffffu, v0, 1); }

// r = w - A u at a lane's pair of one row
__device__ __forceinline__ void resid_pair(const double (&ctr)[2], const double (&s1)[2], const double (&s2)[2],
                                           const double (&w)[2], const Coef &cf, double (&r)[2])
{
    const double s1l = from_left(s1[1]), s2l = from_left(s2[1]), s1r = from_right(s1[0]), s2r = from_right(s2[0]);
    r[0] = w[0] - cf.a0 * ctr[0] - cf.a2 * (s2[0] + s1l + s1[1]) - cf.a3 * (s2l + s2[1]);
    r[1] = w[1] - cf.a0 * ctr[1] - cf.a2 * (s2[1] + s1[0] + s1r) - cf.a3 * (s2[0] + s2r);
}

// u + C r at a lane's pair of one row
__device__ __forceinline__ void psinv_pair(const double (&ctr)[2], const double (&s1)[2], const double (&s2)[2],
                                           const double (&u)[2], const Coef &cf, double (&o)[2])
{
    const double s1l = from_left(s1[1]), cl = from_left(ctr[1]), s1r = from_right(s1[0]), cr = from_right(ctr[0]);
    o[0] = u[0] + cf.c0 * ctr[0] + cf.c1 * (cl + ctr[1] + s1[0]) + cf.c2 * (s2[0] + s1l + s1[1]);
    o[1] = u[1] + cf.c0 * ctr[1] + cf.c1 * (ctr[0] + cr + s1[1]) + cf.c2 * (s2[1] + s1[0] + s1r);
}

// A thread's place in a march: warp rows Fy, Fy + 1 and lane columns Fx,
// Fx + 1, the wrapped offset of the first in a plane, and which are its own.
struct March {
    int fx, fy;
    size_t row;  // offset of (Fy, Fx), wrapped, in a plane; the next row is m further
    bool own;
};

template <int W>
__device__ __forceinline__ March march_of(int m)
{
    const int n = m - 2, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    March q;
    q.fx = int(blockIdx.x) * kOwnX - 2 + 2 * lane;
    q.fy = int(blockIdx.y) * (2 * W - 4) - 2 + 2 * w;
    q.row = size_t(wrap(q.fy, n)) * m + wrap(q.fx, n);
    q.own = lane >= 1 && lane <= 30 && w >= 1 && w <= W - 2 && q.fx < n && q.fy < n;
    return q;
}

// The rows v of own points of plane Fz, and their images.
__device__ __forceinline__ void store_rows(double *g, int m, const March &q, int fz, const double (&v)[2][2])
{
    const int n = m - 2;
    const size_t plane = size_t(m) * m;
    for (int z = fz; z < m; z += n) {
        for (int y = q.fy; y < m; y += n) {
            double *p = g + z * plane + size_t(y) * m;
            for (int x = q.fx; x < m; x += n) {
                *reinterpret_cast<double2 *>(p + x) = make_double2(v[0][0], v[0][1]);
                *reinterpret_cast<double2 *>(p + m + x) = make_double2(v[1][0], v[1][1]);
            }
        }
    }
}

__device__ __forceinline__ void load_rows(const double *g, size_t plane_row, int m, double (&v)[2][2])
{
    const double2 a = *reinterpret_cast<const double2 *>(g + plane_row);
    const double2 b = *reinterpret_cast<const double2 *>(g + plane_row + m);
    v[0][0] = a.x;
    v[0][1] = a.y;
    v[1][0] = b.x;
    v[1][1] = b.y;
}

// Rows through shared memory: row index 2 w + i of the CTA's 2 W rows.
__device__ __forceinline__ void put_rows(double2 (*s)[32], const double (&v)[2][2])
{
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    s[2 * w][lane] = make_double2(v[0][0], v[0][1]);
    s[2 * w + 1][lane] = make_double2(v[1][0], v[1][1]);
}
__device__ __forceinline__ void get_row(double2 (*s)[32], int row, int rows, double (&v)[2])
{
    const double2 t = s[min(max(row, 0), rows - 1)][threadIdx.x & 31];
    v[0] = t.x;
    v[1] = t.y;
}

// kAdd: u' = u + P z (the finest level); else u' = 0 + P z.  v: the
// right-hand side (coarse levels: the restricted residual).  u and out are
// different arrays.  zc: own planes a CTA walks (even).
template <int W, bool kAdd>
__global__ void __launch_bounds__(32 * W, 1)
    k_up(const double *z, int mj, const double *u, const double *v, double *out, int m, int zc, Coef cf)
{
    __shared__ double2 su[2 * W][32], sr[2 * W][32];
    wait_for_predecessor();
    const int n = m - 2, w = threadIdx.x >> 5;
    const March q = march_of<W>(m);
    const size_t plane = size_t(m) * m, zplane = size_t(mj) * mj;
    const int z0 = int(blockIdx.z) * zc, z1 = min(n, z0 + zc);
    const size_t zrow = size_t(wrap(q.fy, n) / 2) * mj + wrap(q.fx, n) / 2;
    // the coarse plane i3: z[i2][i1], z[i2][i1+1], z[i2+1][i1], z[i2+1][i1+1]
    auto coarse = [&](int i3, double (&c)[4]) {
        const double *p = z + i3 * zplane + zrow;
        c[0] = p[0];
        c[1] = p[1];
        c[2] = p[mj];
        c[3] = p[mj + 1];
    };
    Plane27 U{}, R{};
    double un[2][2] = {}, vn[2][2] = {}, za[4], zb[4] = {};
    coarse(wrap(z0 - 2, n) / 2, za);
    if (kAdd) load_rows(u, wrap(z0 - 2, n) * plane + q.row, m, un);
    for (int pz = z0 - 2; pz <= z1 + 1; pz++) {
        // u' of plane pz (interp's sums, :836-890)
        double p[2][2];
        {
            const double z1a = za[2] + za[0], z1b = za[3] + za[1];
            double add[2][2];
            if ((pz & 1) == 0) {
                add[0][0] = za[0];
                add[0][1] = 0.5 * (za[1] + za[0]);
                add[1][0] = 0.5 * z1a;
                add[1][1] = 0.25 * (z1a + z1b);
            } else {
                const double z2a = zb[0] + za[0], z2b = zb[1] + za[1];
                const double z3a = zb[2] + zb[0] + z1a, z3b = zb[3] + zb[1] + z1b;
                add[0][0] = 0.5 * z2a;
                add[0][1] = 0.25 * (z2a + z2b);
                add[1][0] = 0.25 * z3a;
                add[1][1] = 0.125 * (z3a + z3b);
            }
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int k = 0; k < 2; k++) p[i][k] = (kAdd ? un[i][k] : 0.0) + add[i][k];
        }
        // loads of the next plane, in flight during this one's work
        double vc[2][2];
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int k = 0; k < 2; k++) vc[i][k] = vn[i][k];
        if (pz <= z1) {
            if (kAdd) load_rows(u, wrap(pz + 1, n) * plane + q.row, m, un);
            load_rows(v, wrap(pz, n) * plane + q.row, m, vn);
            if ((pz & 1) == 0) {
                coarse(wrap(pz, n) / 2 + 1, zb);
            } else {
#pragma unroll
                for (int k = 0; k < 4; k++) za[k] = zb[k];
            }
        }
        double up[2], dn[2], s1[2][2], s2[2][2], uc[2][2], r[2][2], o[2][2];
        put_rows(su, p);
        __syncthreads();
        get_row(su, 2 * w - 1, 2 * W, up);
        get_row(su, 2 * w + 2, 2 * W, dn);
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int k = 0; k < 2; k++) uc[i][k] = U.cm[i][k];  // u' of plane pz - 2
        U.step(p, up, dn, s1, s2);
#pragma unroll
        for (int i = 0; i < 2; i++) resid_pair(U.cm[i], s1[i], s2[i], vc[i], cf, r[i]);  // plane pz - 1
        put_rows(sr, r);
        __syncthreads();
        get_row(sr, 2 * w - 1, 2 * W, up);
        get_row(sr, 2 * w + 2, 2 * W, dn);
        R.step(r, up, dn, s1, s2);
#pragma unroll
        for (int i = 0; i < 2; i++) psinv_pair(R.cm[i], s1[i], s2[i], uc[i], cf, o[i]);  // plane pz - 2
        if (pz - 2 >= z0 && q.own) store_rows(out, m, q, pz - 2, o);
    }
}

// r = v - A u, s (side mj) = its restriction, and r itself when kStore.
template <int W, bool kStore>
__global__ void __launch_bounds__(32 * W, 1)
    k_down(const double *u, const double *v, double *rout, int m, double *s, int mj, int zc, Coef cf)
{
    __shared__ double2 su[2 * W][32], sr[2 * W][32];
    wait_for_predecessor();
    const int n = m - 2, nj = mj - 2, w = threadIdx.x >> 5;
    const March q = march_of<W>(m);
    const size_t plane = size_t(m) * m;
    const int z0 = int(blockIdx.z) * zc, z1 = min(n, z0 + zc);
    Plane27 U{};
    double un[2][2], vn[2][2] = {};
    // of the odd plane before: the rows above, at and below the coarse row;
    // of the even plane: their sum above and below, and the centre
    double mlo[2] = {}, mc[2] = {}, mhi[2] = {}, e0[2] = {}, ec[2] = {};
    load_rows(u, wrap(z0 - 2, n) * plane + q.row, m, un);
    for (int pz = z0 - 2; pz <= z1; pz++) {
        double p[2][2], vc[2][2];
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int k = 0; k < 2; k++) {
                p[i][k] = un[i][k];
                vc[i][k] = vn[i][k];
            }
        if (pz < z1) {
            load_rows(u, wrap(pz + 1, n) * plane + q.row, m, un);
            load_rows(v, wrap(pz, n) * plane + q.row, m, vn);
        }
        double up[2], dn[2], s1[2][2], s2[2][2], r[2][2], lo[2];
        put_rows(su, p);
        __syncthreads();
        get_row(su, 2 * w - 1, 2 * W, up);
        get_row(su, 2 * w + 2, 2 * W, dn);
        U.step(p, up, dn, s1, s2);
#pragma unroll
        for (int i = 0; i < 2; i++) resid_pair(U.cm[i], s1[i], s2[i], vc[i], cf, r[i]);
        const int rz = pz - 1;  // r's plane
        if (kStore && rz >= z0 && q.own) store_rows(rout, m, q, rz, r);
        sr[2 * w + 1][threadIdx.x & 31] = make_double2(r[1][0], r[1][1]);
        __syncthreads();
        get_row(sr, 2 * w - 1, 2 * W, lo);
        if ((rz & 1) == 0) {
#pragma unroll
            for (int k = 0; k < 2; k++) {
                e0[k] = lo[k] + r[1][k];
                ec[k] = r[0][k];
            }
            continue;
        }
        // rprj3's sums (:1724-1790) around plane rz - 1
        double x[2], y[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            x[k] = e0[k] + mc[k] + r[0][k];
            y[k] = mlo[k] + lo[k] + mhi[k] + r[1][k];
            mlo[k] = lo[k];
            mc[k] = r[0][k];
            mhi[k] = r[1][k];
        }
        const double xl = from_left(x[1]), yl = from_left(y[1]), cl = from_left(ec[1]);
        if (rz - 1 >= z0 && q.own) {
            const double val = 0.5 * ec[0] + 0.25 * (cl + ec[1] + x[0]) + 0.125 * (xl + x[1] + y[0]) +
                               0.0625 * (yl + y[1]);
            for (int a = (rz - 1) / 2; a < mj; a += nj)
                for (int b = q.fy / 2; b < mj; b += nj)
                    for (int c = q.fx / 2; c < mj; c += nj) s[at(mj, a, b, c)] = val;
        }
    }
}

// ------------------------------------------------------ the coarse levels
// The V-cycle below a level whose grids are a few hundred KB, as one launch:
// a cluster of kClusterCtas CTAs walks the levels, the operators one after
// another with a cluster barrier between (the grids stay in L2 and the
// barrier costs well under a microsecond, where a launch each took about 4
// us for some 0.1 us of work): 53 us a cycle in place of 20 launches, class S
// (32^3, 4 cycles) 0.68 -> 0.26 ms.  The levels of up to 8^3 points are CTA 0's
// alone.  With `top` the finest level is among them and the launch runs the
// whole benchmark's `cycles` V-cycles, each with the main loop's resid.
constexpr int kClusterCtas = 8;
constexpr int kClusterThreads = 512;
constexpr int kCoarseLevel = 5;     // 32^3
constexpr int kSoloLevel = 3;       // 8^3

struct CoarseArgs {
    double *u[kCoarseLevel + 1], *r[kCoarseLevel + 1];
    const double *v;
    int levels, top, cycles;
    Coef cf;
};

// Points are dealt out as columns: thread t takes x = t % n, y = t / n % n
// and the z run t / n^2, so that a warp reads runs of x.
struct Column {
    int x, y, za, zb;
};
__device__ __forceinline__ Column column_of(int t, int threads, int n)
{
    const int runs = min(n, max(1, threads / (n * n)));
    const int c = t / (n * n), len = (n + runs - 1) / runs;
    Column q;
    q.x = 1 + t % n;
    q.y = 1 + t / n % n;
    q.za = 1 + c * len;
    q.zb = min(n, q.za + len - 1);
    return q;
}

// resid (kPsinv false: out = w - A g) or psinv (out = out + C g) on a column
template <bool kPsinv>
__device__ __forceinline__ void column_stencil(const double *g, const double *w, double *out, int m, const Column &q,
                                               const Coef &cf)
{
    double em[3] = {}, e0[3] = {}, cm[3] = {}, c0[3] = {};
    for (int z = q.za - 1; z <= q.zb + 1; z++) {
        const double *p = g + at(m, z, q.y, q.x);
        double lo[3], c[3], hi[3], s1[3], s2[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            lo[k] = p[k - 1 - m];
            c[k] = p[k - 1];
            hi[k] = p[k - 1 + m];
        }
#pragma unroll
        for (int k = 0; k < 3; k++) {
            s1[k] = e0[k] + cm[k] + c[k];
            s2[k] = em[k] + lo[k] + hi[k];
            em[k] = e0[k];
            e0[k] = lo[k] + hi[k];
            cm[k] = c0[k];
            c0[k] = c[k];
        }
        if (z - 1 < q.za) continue;
        const size_t o = at(m, z - 1, q.y, q.x);
        double val;
        if constexpr (kPsinv)
            val = out[o] + cf.c0 * cm[1] + cf.c1 * (cm[0] + cm[2] + s1[1]) + cf.c2 * (s2[1] + s1[0] + s1[2]);
        else
            val = w[o] - cf.a0 * cm[1] - cf.a2 * (s2[1] + s1[0] + s1[2]) - cf.a3 * (s2[0] + s2[2]);
        store_periodic(out, m, z - 1, q.y, q.x, val);
    }
}

__device__ __forceinline__ void restrict_point(const double *r, int mk, double *s, int mj, int j3, int j2, int j1)
{
    const double *p = r + at(mk, 2 * j3, 2 * j2, 2 * j1);
    const ptrdiff_t row = mk, pl = ptrdiff_t(mk) * mk;
    auto cross = [&](const double *c) { return c[-row] + c[row] + c[-pl] + c[pl]; };
    auto corner = [&](const double *c) { return c[-pl - row] + c[pl - row] + c[-pl + row] + c[pl + row]; };
    const double val = 0.5 * p[0] + 0.25 * (p[-1] + p[1] + cross(p)) + 0.125 * (cross(p - 1) + cross(p + 1) + corner(p)) +
                       0.0625 * (corner(p - 1) + corner(p + 1));
    store_periodic(s, mj, j3, j2, j1, val);
}

// u (side mk) at index (f3, f2, f1), ghosts included: base + P z
__device__ __forceinline__ double interp_point(const double *z, int mj, int f3, int f2, int f1)
{
    const double *p = z + at(mj, f3 >> 1, f2 >> 1, f1 >> 1);
    const ptrdiff_t row = mj, pl = ptrdiff_t(mj) * mj;
    auto line = [&](const double *c) {  // the reference's z1, z2, z3 or the point itself
        if (f3 & 1) return (f2 & 1) ? c[pl + row] + c[pl] + (c[row] + c[0]) : c[pl] + c[0];
        return (f2 & 1) ? c[row] + c[0] : c[0];
    };
    const double scale = ((f3 & 1) ? 0.5 : 1.0) * ((f2 & 1) ? 0.5 : 1.0);
    if ((f1 & 1) == 0) return scale * line(p);
    // odd x adds the two lines; where line is the point itself the reference
    // writes z[i1 + 1] + z[i1]
    if (((f3 | f2) & 1) == 0) return 0.5 * (p[1] + p[0]);
    return 0.5 * scale * (line(p) + line(p + 1));
}

__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    __threadfence();  // plain loads after it see the other CTAs' stores
}

__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kClusterThreads, 1) k_coarse(CoarseArgs A)
{
    wait_for_predecessor();
    const bool solo_cta = blockIdx.x == 0;
    const int gt = int(blockIdx.x) * kClusterThreads + int(threadIdx.x), all = kClusterCtas * kClusterThreads;
    // run an operator of level k by everyone, or by CTA 0 alone below
    auto phase = [&](int k, auto op) {
        if (k > kSoloLevel) {
            op(gt, all);
            cluster_sync();
        } else {
            if (solo_cta) op(int(threadIdx.x), kClusterThreads);
            __syncthreads();
        }
    };
    auto restricted = [&](int k) {  // level k -> k - 1
        phase(k, [&](int t, int threads) {
            const int nj = 1 << (k - 1);
            for (int e = t; e < nj * nj * nj; e += threads)
                restrict_point(A.r[k], 2 * nj + 2, A.r[k - 1], nj + 2, 1 + e / (nj * nj), 1 + e / nj % nj, 1 + e % nj);
        });
    };
    auto stencil = [&](int k, bool psinv, const double *g, const double *w, double *out) {
        phase(k, [&](int t, int threads) {
            const int n = 1 << k;
            const Column q = column_of(t, threads, n);
            if (q.za > n) return;
            if (psinv) column_stencil<true>(g, nullptr, out, n + 2, q, A.cf);
            else column_stencil<false>(g, w, out, n + 2, q, A.cf);
        });
    };
    auto prolonged = [&](int k, bool add) {  // level k - 1 -> k
        phase(k, [&](int t, int threads) {
            const int mk = (1 << k) + 2, mj = (1 << (k - 1)) + 2;
            for (int e = t; e < mk * mk * mk; e += threads) {
                const double p = interp_point(A.u[k - 1], mj, e / (mk * mk), e / mk % mk, e % mk);
                A.u[k][e] = (add ? A.u[k][e] : 0.0) + p;
            }
        });
    };
    const int top_level = A.levels;
    for (int cycle = 0; cycle < A.cycles; cycle++) {
        for (int k = top_level; k >= 2; k--) restricted(k);
        phase(1, [&](int t, int) {  // u = 0 on the coarsest level, then psinv on it
            if (t < 64) A.u[1][t] = 0.0;
        });
        stencil(1, true, A.r[1], nullptr, A.u[1]);
        for (int k = 2; k <= top_level; k++) {
            if (k == kSoloLevel + 1) cluster_sync();  // CTA 0's levels, to everyone
            const bool finest = A.top && k == top_level;
            prolonged(k, finest);
            stencil(k, false, A.u[k], finest ? A.v : A.r[k], A.r[k]);
            stencil(k, true, A.r[k], nullptr, A.u[k]);
            if (finest) stencil(k, false, A.u[k], A.v, A.r[k]);
        }
    }
    cluster_sync();  // no CTA leaves while another's barrier is open
}

// Sum of squares and largest magnitude over the interior: block b takes
// rows (i2, i3) b, b + grid, ... and its threads stride x (at most four
// values of a row each: n <= 1024); the loads of four rows are issued
// before their values are added in the thread's fixed order.  Per-block
// tree, then the last block (ticket) adds the blocks by the same tree.
// out[0] = sum, out[1] = max.
constexpr int kRowsAhead = 4, kMaxPerRow = 4;

__global__ void __launch_bounds__(kNormThreads) k_norm(const double *__restrict__ r, int m, double *part,
                                                       unsigned *ticket, double *out)
{
    __shared__ double ss[kNormThreads], sm[kNormThreads];
    __shared__ bool last;
    wait_for_predecessor();
    const int n = m - 2, rows = n * n, tid = threadIdx.x;
    double s = 0.0, mx = 0.0;
    for (int row0 = blockIdx.x; row0 < rows; row0 += kRowsAhead * gridDim.x) {
        double xv[kRowsAhead][kMaxPerRow];
#pragma unroll
        for (int u = 0; u < kRowsAhead; u++) {
            const int row = row0 + u * int(gridDim.x);
            const double *line = row < rows ? r + at(m, 1 + row / n, 1 + row % n, 0) : nullptr;
#pragma unroll
            for (int j = 0; j < kMaxPerRow; j++) {
                const int i1 = 1 + tid + j * kNormThreads;
                xv[u][j] = (line && i1 <= n) ? line[i1] : 0.0;
            }
        }
#pragma unroll
        for (int u = 0; u < kRowsAhead; u++)
#pragma unroll
            for (int j = 0; j < kMaxPerRow; j++) {
                s = s + xv[u][j] * xv[u][j];
                mx = fmax(mx, fabs(xv[u][j]));
            }
    }
    // thread 0: the block's sum and largest value
    auto block_tree = [&] {
        ss[tid] = s;
        sm[tid] = mx;
        __syncthreads();
        for (int w = kNormThreads / 2; w > 0; w >>= 1) {
            if (tid < w) {
                ss[tid] = ss[tid] + ss[tid + w];
                sm[tid] = fmax(sm[tid], sm[tid + w]);
            }
            __syncthreads();
        }
    };
    block_tree();
    if (tid == 0) {
        part[2 * blockIdx.x] = ss[0];
        part[2 * blockIdx.x + 1] = sm[0];
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    s = mx = 0.0;
    for (int i = tid; i < int(gridDim.x); i += kNormThreads) {
        s = s + __ldcg(part + 2 * i);
        mx = fmax(mx, __ldcg(part + 2 * i + 1));
    }
    block_tree();
    if (tid == 0) {
        out[0] = ss[0];
        out[1] = sm[0];
        *ticket = 0u;
    }
}

__device__ __forceinline__ uint64_t lcg_mul(uint64_t a, uint64_t b) { return (a * b) & kMask46; }

// kSeed * kMult^e mod 2^46 (the low 46 bits of the 64-bit products are exact)
__device__ __forceinline__ uint64_t lcg_jump(uint64_t e)
{
    uint64_t r = kSeed, b = kMult;
    while (e) {
        if (e & 1) r = lcg_mul(r, b);
        b = lcg_mul(b, b);
        e >>= 1;
    }
    return r;
}

// zran3's candidates: draws above hi_t and below lo_t, with their linear
// index L, appended to the lists (counts may pass the capacity: the host
// then retries with tighter thresholds).
__global__ void k_zran3_candidates(long long total, double hi_t, double lo_t, double *hv, long long *hl,
                                   unsigned *hn, double *lv, long long *ll, unsigned *ln)
{
    const long long first = (blockIdx.x * (long long)blockDim.x + threadIdx.x) * kChunk;
    if (first >= total) return;
    const long long end = first + kChunk < total ? first + kChunk : total;
    uint64_t x = lcg_jump(uint64_t(first) + 1);
    for (long long L = first; L < end; L++) {
        const double val = double(x) * 0x1p-46;  // exact
        if (val > hi_t) {
            const unsigned k = atomicAdd(hn, 1u);
            if (k < unsigned(kCandCap)) {
                hv[k] = val;
                hl[k] = L;
            }
        }
        if (val < lo_t) {
            const unsigned k = atomicAdd(ln, 1u);
            if (k < unsigned(kCandCap)) {
                lv[k] = val;
                ll[k] = L;
            }
        }
        x = lcg_mul(x, kMult);
    }
}

// v = -1 at the minus points, then +1 at the plus points, with ghosts
// (v is zero beforehand).  pts: 10 minus then 10 plus (i1, i2, i3).
__global__ void k_set_points(double *v, int m, const int *pts)
{
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    for (int i = 0; i < 20; i++)
        store_periodic(v, m, pts[3 * i + 2], pts[3 * i + 1], pts[3 * i], i < 10 ? -1.0 : 1.0);
}

}  // namespace mg
}  // namespace cgb

using namespace cgb;
using namespace cgb::mg;

struct cgb_mg {
    int device = 0, lt = 0, smoother = 0, sms = 0;
    int m[kMaxLevels + 1] = {};
    double *u[kMaxLevels + 1] = {}, *r[kMaxLevels + 1] = {};
    double *v = nullptr;
    // where the run of `graph_nit` cycles leaves the finest u and r: k_up reads
    // one of u[lt], r[lt] and writes the other (enqueue_region)
    double *u_now = nullptr, *r_now = nullptr;
    double *d_part = nullptr, *d_norm = nullptr;
    unsigned *d_ticket = nullptr;
    int plus[30] = {}, minus[30] = {};
    Coef cf{};
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaGraphExec_t exec = nullptr;
    int graph_nit = -1;
};

namespace {

#define MG_TRY(call)                                                                      \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess)                                                            \
            return set_error(e_ == cudaErrorMemoryAllocation ? CGB_ERR_NOMEM : CGB_ERR_CUDA, \
                             "mg: %s: %s", #call, cudaGetErrorString(e_));                \
    } while (0)

size_t cells(int m) { return size_t(m) * m * m; }

Coef coefficients(int smoother)
{
    // main's coefficients (mg.cu:422-442)
    Coef cf{-8.0 / 3.0, 1.0 / 6.0, 1.0 / 12.0, -3.0 / 8.0, 1.0 / 32.0, -1.0 / 64.0};
    if (smoother) {
        cf.c0 = -3.0 / 17.0;
        cf.c1 = 1.0 / 33.0;
        cf.c2 = -1.0 / 61.0;
    }
    return cf;
}

void mg_release(cgb_mg *g)
{
    if (!g) return;
    cudaSetDevice(g->device);
    if (g->exec) cudaGraphExecDestroy(g->exec);
    for (int k = 0; k <= kMaxLevels; k++) {
        if (g->u[k]) cudaFree(g->u[k]);
        if (g->r[k]) cudaFree(g->r[k]);
    }
    for (void *p : {(void *)g->v, (void *)g->d_part, (void *)g->d_norm, (void *)g->d_ticket})
        if (p) cudaFree(p);
    if (g->ev0) cudaEventDestroy(g->ev0);
    if (g->ev1) cudaEventDestroy(g->ev1);
    if (g->stream) cudaStreamDestroy(g->stream);
    delete g;
}

// x covers [1, m - 1] (the last interior point's right neighbour is a
// column sum), y and z the interior.
dim3 stencil_grid(int m)
{
    return dim3(unsigned((m - 1 + 31) / 32), unsigned((m - 2 + kRows - 1) / kRows), unsigned(m - 2));
}


dim3 interp_grid(int mj)
{
    return dim3(unsigned((mj - 1 + 31) / 32), unsigned((mj - 1 + kRows - 1) / kRows), unsigned(mj - 1));
}

dim3 stencil_rb_grid(int m)
{
    const int n = m - 2;
    return dim3(unsigned((n + 31) / 32), unsigned((n + kRowsRB - 1) / kRowsRB), unsigned((n + kPlanes - 1) / kPlanes));
}

// A launch that may start while its predecessor drains (the kernel begins
// with wait_for_predecessor()).
template <typename... P, typename... A>
void launch(cgb_mg *g, void (*k)(P...), dim3 grid, dim3 block, A... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = g->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k, P(args)...);
}

// The grid of a march over a level, and the own planes a CTA walks: the
// split along z with the fewest planes on the longest SM, counting the four
// (k_up) or two (k_down) extra planes of every walk.
dim3 march_grid(const cgb_mg *g, int m, int warps, int extra, int *zc)
{
    const int n = m - 2, gx = (n + kOwnX - 1) / kOwnX, gy = (n + 2 * warps - 5) / (2 * warps - 4);
    long long best = 0;
    int best_zc = 2;
    for (int c = 2; c <= n; c += 2) {
        const long long chunks = (n + c - 1) / c, waves = (gx * gy * chunks + g->sms - 1) / g->sms;
        const long long cost = waves * (c + extra);
        if (c == 2 || cost <= best) {
            best = cost;
            best_zc = c;
        }
    }
    *zc = best_zc;
    return dim3(unsigned(gx), unsigned(gy), unsigned((n + best_zc - 1) / best_zc));
}

// r (when `store`) and r[lt - 1] from the finest u and v
void launch_down(cgb_mg *g, const double *u, double *r, bool store)
{
    const int lt = g->lt, m = g->m[lt];
    int zc = 0;
    const dim3 grid = march_grid(g, m, kWarpsDown, 2, &zc);
    launch(g, store ? k_down<kWarpsDown, true> : k_down<kWarpsDown, false>, grid, dim3(32 * kWarpsDown), u, g->v,
           r, m, g->r[lt - 1], g->m[lt - 1], zc, g->cf);
}

void launch_up(cgb_mg *g, int k, const double *u, const double *v, double *out)
{
    const int m = g->m[k];
    int zc = 0;
    const dim3 grid = march_grid(g, m, kWarpsUp, 4, &zc);
    launch(g, u ? k_up<kWarpsUp, true> : k_up<kWarpsUp, false>, grid, dim3(32 * kWarpsUp), g->u[k - 1], g->m[k - 1],
           u, v, out, m, zc, g->cf);
}

void launch_coarse(cgb_mg *g, int levels, int top, int cycles)
{
    CoarseArgs A{};
    for (int k = 1; k <= levels; k++) {
        A.u[k] = g->u[k];
        A.r[k] = g->r[k];
    }
    A.v = g->v;
    A.levels = levels;
    A.top = top;
    A.cycles = cycles;
    A.cf = g->cf;
    launch(g, k_coarse, dim3(kClusterCtas), dim3(kClusterThreads), A);
}

void launch_norm(cgb_mg *g, const double *r)
{
    const int n = g->m[g->lt] - 2;
    launch(g, k_norm, dim3(unsigned(std::min(kNormBlocks, (n * n + kRowsAhead - 1) / kRowsAhead))), dim3(kNormThreads),
           r, g->m[g->lt], g->d_part, g->d_ticket, g->d_norm);
}

// The timed region of main (:498-508): resid, norm, nit x (V-cycle (mg3P,
// :1078-1133), resid), norm.  The finest u and r are in *uf and *rf after it:
// above the coarse levels a cycle's k_up reads u and writes the new one over
// r, which nothing reads between the first norm and the last (k_down walks u
// and v, and stores r in the last cycle only), so the two buffers change
// places every cycle.
void enqueue_region(cgb_mg *g, int nit, double **uf, double **rf)
{
    const int lt = g->lt, m = g->m[lt];
    double *u = g->u[lt], *r = g->r[lt];
    if (lt <= kCoarseLevel) {
        k_stencil_rb<false><<<stencil_rb_grid(m), dim3(32, kWarpsRB), 0, g->stream>>>(u, g->v, r, m, g->cf);
        launch_norm(g, r);
        if (nit > 0) launch_coarse(g, lt, 1, nit);
        launch_norm(g, r);
        *uf = u;
        *rf = r;
        return;
    }
    launch_down(g, u, r, true);
    launch_norm(g, r);
    for (int it = 0; it < nit; it++) {
        for (int k = lt - 1; k > kCoarseLevel; k--) {
            const int mj = g->m[k - 1];
            launch(g, k_rprj3, stencil_grid(mj), dim3(32, kRows), g->r[k], g->m[k], g->r[k - 1], mj);
        }
        launch_coarse(g, kCoarseLevel, 0, 1);
        for (int k = kCoarseLevel + 1; k < lt; k++) launch_up(g, k, nullptr, g->r[k], g->u[k]);
        launch_up(g, lt, u, g->v, r);
        std::swap(u, r);
        launch_down(g, u, r, it + 1 == nit);
    }
    launch_norm(g, r);
    *uf = u;
    *rf = r;
}

// zran3 on the device: the candidates, then the host's choice of the ten
// largest and smallest, then v.
int generate_v(cgb_mg *g)
{
    const int m = g->m[g->lt], n = m - 2;
    const long long total = (long long)n * n * n;
    double *hv = nullptr, *lv = nullptr;
    long long *hl = nullptr, *ll = nullptr;
    unsigned *cnt = nullptr;
    int *pts = nullptr;
    auto release = [&] {
        for (void *p : {(void *)hv, (void *)lv, (void *)hl, (void *)ll, (void *)cnt, (void *)pts})
            if (p) cudaFree(p);
    };
    if (cudaMalloc(&hv, sizeof(double) * kCandCap) != cudaSuccess ||
        cudaMalloc(&lv, sizeof(double) * kCandCap) != cudaSuccess ||
        cudaMalloc(&hl, sizeof(long long) * kCandCap) != cudaSuccess ||
        cudaMalloc(&ll, sizeof(long long) * kCandCap) != cudaSuccess ||
        cudaMalloc(&cnt, 2 * sizeof(unsigned)) != cudaSuccess || cudaMalloc(&pts, 60 * sizeof(int)) != cudaSuccess) {
        release();
        return set_error(CGB_ERR_NOMEM, "mg: zran3 buffers");
    }
    double expect = 256.0;
    std::vector<std::pair<double, long long>> hi, lo;
    int st = CGB_OK;
    for (int attempt = 0; attempt < 12; attempt++) {
        const double frac = std::min(0.5, expect / double(total));
        const unsigned threads = 256;
        const long long chunks = (total + kChunk - 1) / kChunk;
        const unsigned blocks = unsigned((chunks + threads - 1) / threads);
        unsigned h_cnt[2] = {0, 0};
        if (cudaMemsetAsync(cnt, 0, 2 * sizeof(unsigned), g->stream) != cudaSuccess) {
            st = set_error(CGB_ERR_CUDA, "mg: zran3 memset");
            break;
        }
        k_zran3_candidates<<<blocks, threads, 0, g->stream>>>(total, 1.0 - frac, frac, hv, hl, cnt, lv, ll,
                                                              cnt + 1);
        if (cudaGetLastError() != cudaSuccess ||
            cudaMemcpyAsync(h_cnt, cnt, sizeof(h_cnt), cudaMemcpyDeviceToHost, g->stream) != cudaSuccess ||
            cudaStreamSynchronize(g->stream) != cudaSuccess) {
            st = set_error(CGB_ERR_CUDA, "mg: zran3 candidates failed");
            break;
        }
        if (h_cnt[0] > unsigned(kCandCap) || h_cnt[1] > unsigned(kCandCap)) {
            expect /= 4.0;
            continue;
        }
        if ((h_cnt[0] < 10 || h_cnt[1] < 10) && frac < 0.5) {
            expect *= 8.0;
            continue;
        }
        std::vector<double> a(h_cnt[0]), b(h_cnt[1]);
        std::vector<long long> ai(h_cnt[0]), bi(h_cnt[1]);
        if (cudaMemcpy(a.data(), hv, sizeof(double) * a.size(), cudaMemcpyDeviceToHost) != cudaSuccess ||
            cudaMemcpy(ai.data(), hl, sizeof(long long) * ai.size(), cudaMemcpyDeviceToHost) != cudaSuccess ||
            cudaMemcpy(b.data(), lv, sizeof(double) * b.size(), cudaMemcpyDeviceToHost) != cudaSuccess ||
            cudaMemcpy(bi.data(), ll, sizeof(long long) * bi.size(), cudaMemcpyDeviceToHost) != cudaSuccess) {
            st = set_error(CGB_ERR_CUDA, "mg: zran3 copy-out failed");
            break;
        }
        for (size_t i = 0; i < a.size(); i++) hi.emplace_back(a[i], ai[i]);
        for (size_t i = 0; i < b.size(); i++) lo.emplace_back(b[i], bi[i]);
        break;
    }
    if (!st && (hi.size() < 10 || lo.size() < 10))
        st = set_error(CGB_ERR_STATE, "mg: zran3 found fewer than ten candidates a side");
    if (!st) {
        // the reference's lists: the ten largest ascending (largest last),
        // the ten smallest descending (smallest last)
        std::sort(hi.begin(), hi.end());
        std::sort(lo.begin(), lo.end(), [](const std::pair<double, long long> &x,
                                           const std::pair<double, long long> &y) { return x.first > y.first; });
        hi.erase(hi.begin(), hi.end() - 10);
        lo.erase(lo.begin(), lo.end() - 10);
        int h_pts[60];
        auto put = [&](int *dst, long long L) {
            dst[0] = 1 + int(L % n);
            dst[1] = 1 + int((L / n) % n);
            dst[2] = 1 + int(L / ((long long)n * n));
        };
        for (int i = 0; i < 10; i++) {
            put(g->minus + 3 * i, lo[i].second);
            put(g->plus + 3 * i, hi[i].second);
            put(h_pts + 3 * i, lo[i].second);
            put(h_pts + 30 + 3 * i, hi[i].second);
        }
        if (cudaMemsetAsync(g->v, 0, sizeof(double) * cells(m), g->stream) != cudaSuccess ||
            cudaMemcpyAsync(pts, h_pts, sizeof(h_pts), cudaMemcpyHostToDevice, g->stream) != cudaSuccess)
            st = set_error(CGB_ERR_CUDA, "mg: v upload failed");
        if (!st) {
            k_set_points<<<1, 32, 0, g->stream>>>(g->v, m, pts);
            if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(g->stream) != cudaSuccess)
                st = set_error(CGB_ERR_CUDA, "mg: v set-up failed");
        }
    }
    release();
    return st;
}

}  // namespace

extern "C" {

int cgb_mg_create(int device, int lt, int smoother, cgb_mg **out)
{
    if (!out) return set_error(CGB_ERR_INVALID, "mg: null output");
    *out = nullptr;
    if (lt < 2 || lt > kMaxLevels - 1) return set_error(CGB_ERR_INVALID, "mg: lt must be in [2, %d]", kMaxLevels - 1);
    if (smoother != 0 && smoother != 1) return set_error(CGB_ERR_INVALID, "mg: smoother must be 0 or 1");
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count)
        return set_error(CGB_ERR_NO_DEVICE, "mg: no CUDA device %d", device);
    int major = 0;
    MG_TRY(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device));
    if (major != 10) return set_error(CGB_ERR_NO_DEVICE, "mg: device %d is not sm_100", device);
    MG_TRY(cudaSetDevice(device));
    cgb_mg *g = new (std::nothrow) cgb_mg;
    if (!g) return set_error(CGB_ERR_NOMEM, "mg: allocation failed");
    g->device = device;
    g->lt = lt;
    g->smoother = smoother;
    g->cf = coefficients(smoother);
    bool ok = cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking) == cudaSuccess &&
              cudaEventCreate(&g->ev0) == cudaSuccess && cudaEventCreate(&g->ev1) == cudaSuccess &&
              cudaMalloc(&g->d_part, sizeof(double) * 2 * kNormBlocks) == cudaSuccess &&
              cudaMalloc(&g->d_norm, sizeof(double) * 2) == cudaSuccess &&
              cudaMalloc(&g->d_ticket, sizeof(unsigned)) == cudaSuccess &&
              cudaMemset(g->d_ticket, 0, sizeof(unsigned)) == cudaSuccess;
    for (int k = 1; k <= lt && ok; k++) {
        g->m[k] = (1 << k) + 2;
        ok = cudaMalloc(&g->u[k], sizeof(double) * cells(g->m[k])) == cudaSuccess &&
             cudaMalloc(&g->r[k], sizeof(double) * cells(g->m[k])) == cudaSuccess &&
             cudaMemset(g->u[k], 0, sizeof(double) * cells(g->m[k])) == cudaSuccess &&
             cudaMemset(g->r[k], 0, sizeof(double) * cells(g->m[k])) == cudaSuccess;
    }
    ok = ok && cudaMalloc(&g->v, sizeof(double) * cells(g->m[lt])) == cudaSuccess &&
         cudaDeviceGetAttribute(&g->sms, cudaDevAttrMultiProcessorCount, device) == cudaSuccess;
    g->u_now = g->u[lt];
    g->r_now = g->r[lt];
    if (!ok) {
        mg_release(g);
        return set_error(CGB_ERR_NOMEM, "mg: device allocation failed (2^%d grid)", lt);
    }
    const int st = generate_v(g);
    if (st) {
        mg_release(g);
        return st;
    }
    *out = g;
    return CGB_OK;
}

int cgb_mg_destroy(cgb_mg *g)
{
    mg_release(g);
    return CGB_OK;
}

int cgb_mg_run(cgb_mg *g, int nit, double *rnm2, double *rnmu, double *device_ms)
{
    if (!g || nit < 0) return set_error(CGB_ERR_INVALID, "mg: null grid or negative nit");
    MG_TRY(cudaSetDevice(g->device));
    const int lt = g->lt, m = g->m[lt];
    if (g->graph_nit != nit) {
        if (g->exec) cudaGraphExecDestroy(g->exec);
        g->exec = nullptr;
        g->graph_nit = -1;
        cudaGraph_t graph = nullptr;
        double *u = nullptr, *r = nullptr;
        MG_TRY(cudaStreamBeginCapture(g->stream, cudaStreamCaptureModeThreadLocal));
        enqueue_region(g, nit, &u, &r);
        const cudaError_t e1 = cudaGetLastError();
        const cudaError_t e2 = cudaStreamEndCapture(g->stream, &graph);
        if (e1 != cudaSuccess || e2 != cudaSuccess) {
            if (graph) cudaGraphDestroy(graph);
            return set_error(CGB_ERR_CUDA, "mg: capture failed: %s",
                             cudaGetErrorString(e1 != cudaSuccess ? e1 : e2));
        }
        const cudaError_t e3 = cudaGraphInstantiate(&g->exec, graph, 0);
        cudaGraphDestroy(graph);
        if (e3 != cudaSuccess) {
            g->exec = nullptr;
            return set_error(CGB_ERR_CUDA, "mg: graph instantiation: %s", cudaGetErrorString(e3));
        }
        g->graph_nit = nit;
        g->u_now = u;
        g->r_now = r;
    }
    // u = 0 on the finest level (main's zero3 before the timed region)
    MG_TRY(cudaMemsetAsync(g->u[lt], 0, sizeof(double) * cells(m), g->stream));
    MG_TRY(cudaEventRecord(g->ev0, g->stream));
    MG_TRY(cudaGraphLaunch(g->exec, g->stream));
    MG_TRY(cudaEventRecord(g->ev1, g->stream));
    double h[2] = {0.0, 0.0};
    MG_TRY(cudaMemcpyAsync(h, g->d_norm, sizeof(h), cudaMemcpyDeviceToHost, g->stream));
    MG_TRY(cudaStreamSynchronize(g->stream));
    float ms = 0.f;
    MG_TRY(cudaEventElapsedTime(&ms, g->ev0, g->ev1));
    const double n = double(m - 2);
    if (rnm2) *rnm2 = std::sqrt(h[0] / (n * n * n));
    if (rnmu) *rnmu = h[1];
    if (device_ms) *device_ms = ms;
    if (!std::isfinite(h[0])) return set_error(CGB_ERR_NUMERIC, "mg: non-finite residual norm");
    return CGB_OK;
}

int cgb_mg_read(cgb_mg *g, int which, double *out, long long count)
{
    if (!g || !out || which < 0 || which > 2) return set_error(CGB_ERR_INVALID, "mg: bad read");
    const size_t need = cells(g->m[g->lt]);
    if (count < (long long)need) return set_error(CGB_ERR_CAPACITY, "mg: %zu doubles needed", need);
    MG_TRY(cudaSetDevice(g->device));
    const double *src = which == 0 ? g->u_now : which == 1 ? g->v : g->r_now;
    MG_TRY(cudaMemcpy(out, src, sizeof(double) * need, cudaMemcpyDeviceToHost));
    return CGB_OK;
}

int cgb_mg_points(cgb_mg *g, int *plus, int *minus)
{
    if (!g) return set_error(CGB_ERR_INVALID, "mg: null grid");
    if (plus) std::memcpy(plus, g->plus, sizeof(g->plus));
    if (minus) std::memcpy(minus, g->minus, sizeof(g->minus));
    return CGB_OK;
}

int cgb_mg_apply(int device, int op, int m, int smoother, const double *in1, const double *in2,
                 double *out)
{
    if (op < 0 || op > 4 || m < 4 || m > (op >= 3 ? 514 : 1026) || (m & 1) || !in1 || !out ||
        (op == 0 && !in2))
        return set_error(CGB_ERR_INVALID, "mg: bad operator call");
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count)
        return set_error(CGB_ERR_NO_DEVICE, "mg: no CUDA device %d", device);
    MG_TRY(cudaSetDevice(device));
    const int mo = op == 2 ? m / 2 + 1 : op >= 3 ? 2 * m - 2 : m;
    const size_t ci = cells(m), co = cells(mo);
    double *a = nullptr, *b = nullptr, *c = nullptr;
    const Coef cf = coefficients(smoother);
    int st = CGB_OK;
    if (cudaMalloc(&a, sizeof(double) * ci) != cudaSuccess || cudaMalloc(&b, sizeof(double) * ci) != cudaSuccess ||
        cudaMalloc(&c, sizeof(double) * co) != cudaSuccess)
        st = set_error(CGB_ERR_NOMEM, "mg: operator buffers");
    if (!st && (cudaMemcpy(a, in1, sizeof(double) * ci, cudaMemcpyHostToDevice) != cudaSuccess ||
                (in2 && cudaMemcpy(b, in2, sizeof(double) * ci, cudaMemcpyHostToDevice) != cudaSuccess) ||
                cudaMemcpy(c, out, sizeof(double) * co, cudaMemcpyHostToDevice) != cudaSuccess))
        st = set_error(CGB_ERR_CUDA, "mg: operator upload");
    if (!st) {
        switch (op) {
        case 0: k_stencil_rb<false><<<stencil_rb_grid(m), dim3(32, kWarpsRB)>>>(a, b, c, m, cf); break;
        case 1: k_stencil_rb<true><<<stencil_rb_grid(m), dim3(32, kWarpsRB)>>>(a, nullptr, c, m, cf); break;
        case 2: k_rprj3<<<stencil_grid(mo), dim3(32, kRows)>>>(a, m, c, mo); break;
        default: k_interp<<<interp_grid(m), dim3(32, kRows)>>>(a, m, c, mo, op == 4); break;
        }
        if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess ||
            cudaMemcpy(out, c, sizeof(double) * co, cudaMemcpyDeviceToHost) != cudaSuccess)
            st = set_error(CGB_ERR_CUDA, "mg: operator failed");
    }
    for (double *p : {a, b, c})
        if (p) cudaFree(p);
    return st;
}

}  // extern "C"

// ft.cu -- the NPB FT benchmark on the GPU: a 3-D complex field evolved in
// Fourier space and transformed back every iteration (GMAP/NPB-GPU
// CUDA/FT/ft.cu: main :335-420, fft :1258-1278, evolve :1245-1256,
// checksum :1124-1153, initial conditions :1188-1227, index map :1166-1186).
//
// Layout: u0, u1 as double2 (real, imaginary), x fastest, as the reference.
// A transform along one axis is one kernel: a CTA stages a tile of L lines
// of that axis in shared memory (rows of L consecutive x values for the y
// and z axes, so every row is one coalesced run; L whole x lines for the x
// axis) and transforms every line by Stockham stages of radix 8 and 16 (4 for
// the rest of 32 points), each stage's butterflies in registers: the first
// stage reads its points from the field, the last writes its outputs to the field, and the
// stages between exchange through shared memory.  So each axis costs one
// read and one write of the field, and where the y and the x axis share a
// kernel (k_fft_yx) the two together do.  The inverse transform's first axis
// (z) also does evolve: it reads the forward transform (kept in u0) and
// multiplies each point by its factor exp(AP t |k|^2) of iteration t, the
// product of three tables of one axis each; only the last iteration writes
// the evolved field back to u0.  The checksum adds its 1024 points in a
// fixed order.
//
// Transform sign: sign +1 is sum x_j exp(+2 pi i jk / n), the reference's
// is = 1 (its forward transform); sign -1 its is = -1.  Results agree with
// the reference's radix-2 Stockham to rounding (the checksums verify at the
// reference's 1e-12; parity tests hold the fields to the oracle).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <new>

#include "cgb_internal.h"

namespace cgb {
namespace ft {

constexpr uint64_t kMask46 = (uint64_t(1) << 46) - 1;
constexpr uint64_t kMult = 1220703125ull;  // A = 5^13 (ft.cu:129)
constexpr uint64_t kSeed = 314159265ull;   // SEED (ft.cu:128)
constexpr double kAlpha = 1.0e-6;          // ALPHA (ft.cu:131)
constexpr double kPi = 3.141592653589793238;
constexpr double kAp = -4.0 * kAlpha * kPi * kPi;  // AP (ft.cu:132), the same order of operations
constexpr int kPoints = 1024;                     // CHECKSUM_TASKS
constexpr int kMaxIter = 64;
constexpr double kRoot2Half = 0.70710678118654752440;

__device__ __forceinline__ uint64_t lcg_mul(uint64_t a, uint64_t b) { return (a * b) & kMask46; }

// kSeed * kMult^e mod 2^46
__device__ __forceinline__ uint64_t jump(uint64_t e)
{
    uint64_t r = kSeed, b = kMult;
    while (e) {
        if (e & 1) r = lcg_mul(r, b);
        b = lcg_mul(b, b);
        e >>= 1;
    }
    return r;
}

// Element e holds draws 2e+1 and 2e+2 after the seed (the planes' seeds of
// ft.cu:1188-1213 and their rows' vranlc runs are one stream in that order).
// A warp fills 32 `per` consecutive elements: lane l takes l, l + 32,
// l + 64, ..., so every store is one coalesced run; it jumps to its first
// element once and steps 32 elements (64 draws) at a time by A^64.
__global__ void k_initial(double2 *u, long long nt, int per)
{
    const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const long long e0 = warp * 32 * per + lane;
    if (e0 >= nt) return;
    uint64_t a64 = kMult;  // A^64
#pragma unroll
    for (int k = 0; k < 6; k++) a64 = lcg_mul(a64, a64);
    uint64_t x = jump(2 * uint64_t(e0) + 1);  // draw 2 e0 + 1
    const long long e1 = min(nt, (warp + 1) * 32 * per);
    for (long long e = e0; e < e1; e += 32) {
        const uint64_t y = lcg_mul(x, kMult);
        u[e] = make_double2(double(x) * 0x1p-46, double(y) * 0x1p-46);
        x = lcg_mul(x, a64);
    }
}

// The index map's integer argument (ft.cu:1166-1186): the squared signed
// frequencies, i'^2 + (j'^2 + k'^2), summed in the reference's order.
__device__ __forceinline__ int k2_of(int i, int j, int k, int nx, int ny, int nz)
{
    const int kk = ((k + nz / 2) % nz) - nz / 2, jj = ((j + ny / 2) % ny) - ny / 2;
    const int ii = ((i + nx / 2) % nx) - nx / 2;
    const int kj2 = jj * jj + kk * kk;
    return ii * ii + kj2;
}

// The twiddle factors by their argument: twk2[k2] = exp(AP k2), for reading
// out (cgb_ft_read).
__global__ void k_twiddle_table(double *twk2, int k2max)
{
    for (int k2 = blockIdx.x * blockDim.x + threadIdx.x; k2 <= k2max; k2 += gridDim.x * blockDim.x)
        twk2[k2] = exp(kAp * (double)k2);
}

// The per-point map itself, for reading out (cgb_ft_read)
__global__ void k_indexmap(double *tw, const double *__restrict__ twk2, int nx, int ny, int nz)
{
    const long long nt = (long long)nx * ny * nz;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nt;
         e += (long long)gridDim.x * blockDim.x) {
        const int i = int(e % nx), j = int((e / nx) % ny), k = int(e / ((long long)nx * ny));
        tw[e] = twk2[k2_of(i, j, k, nx, ny, nz)];
    }
}

// The dependency words of k_fft_yx: the next work item, whether a wait ran
// out, and for each plane how many of its y tiles are written.
struct PlaneSync {
    int *ticket, *failed, *done;
};

// What a run needs beside the field: the roots W[k] = exp(2 pi i k / n),
// k < n; the evolve factors of iteration t = 1 .. niter, one table an axis,
// ev[(t - 1) (nx + ny + nz) + ...] = exp(AP t i'^2) for i' the signed
// frequency (the factor of a point is the product of its three: each is
// within an ulp, where the reference's t-fold product rounds t times); and
// the dependency words, zero.
__global__ void k_tables(double2 *W, int n, double *ev, int nx, int ny, int nz, int niter, PlaneSync s)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k == 0) *s.ticket = *s.failed = 0;
    if (k < nz) s.done[k] = 0;
    if (k < n) {
        double sn, cs;
        sincospi(2.0 * k / n, &sn, &cs);
        W[k] = make_double2(cs, sn);
    }
    const int per = nx + ny + nz;
    if (k < per * niter) {
        int i = k % per, side = nx;
        if (i >= nx) {
            i -= nx;
            side = ny;
            if (i >= ny) {
                i -= ny;
                side = nz;
            }
        }
        const int f = i < side / 2 ? i : i - side;
        ev[k] = exp(kAp * double((k / per + 1) * f * f));
    }
}

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// (i SIGN) z
template <int SIGN>
__device__ __forceinline__ double2 rot90(double2 z)
{
    return SIGN > 0 ? make_double2(-z.y, z.x) : make_double2(z.y, -z.x);
}

// y_k = sum_j x_j w^(jk), w = exp(2 pi i SIGN / 4), in place, natural order
template <int SIGN>
__device__ __forceinline__ void dft4(double2 *x)
{
    const double2 c0 = cadd(x[0], x[2]), c1 = csub(x[0], x[2]);
    const double2 c2 = cadd(x[1], x[3]), c3 = rot90<SIGN>(csub(x[1], x[3]));
    x[0] = cadd(c0, c2);
    x[2] = csub(c0, c2);
    x[1] = cadd(c1, c3);
    x[3] = csub(c1, c3);
}

// the 8-point transform: the sums and the twiddled differences of the two
// halves, each by a 4-point transform, to the even and the odd outputs
template <int SIGN>
__device__ __forceinline__ void dft8(double2 *x)
{
    double2 a[4], b[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        a[k] = cadd(x[k], x[k + 4]);
        b[k] = csub(x[k], x[k + 4]);
    }
    const double c = kRoot2Half, s = SIGN * kRoot2Half;
    b[1] = make_double2(c * b[1].x - s * b[1].y, s * b[1].x + c * b[1].y);
    b[2] = rot90<SIGN>(b[2]);
    b[3] = make_double2(-c * b[3].x - s * b[3].y, s * b[3].x - c * b[3].y);
    dft4<SIGN>(a);
    dft4<SIGN>(b);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        x[2 * k] = a[k];
        x[2 * k + 1] = b[k];
    }
}

// the 16-point transform as 4 x 4: transforms of the points k + 4 j over j,
// their outputs r turned by exp(2 pi i SIGN k r / 16), transforms over k
template <int SIGN>
__device__ __forceinline__ void dft16(double2 *x)
{
    constexpr double c1 = 0.92387953251128675613, s1 = SIGN * 0.38268343236508977173;  // cos, sin of pi/8
    constexpr double h = kRoot2Half;
    double2 a[4][4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
#pragma unroll
        for (int j = 0; j < 4; j++) a[k][j] = x[k + 4 * j];
        dft4<SIGN>(a[k]);
    }
    const double2 w1 = make_double2(c1, s1), w3 = make_double2(SIGN * s1, SIGN * c1);
    auto turn8 = [&](double2 z) { return make_double2(h * (z.x - SIGN * z.y), h * (z.y + SIGN * z.x)); };
    a[1][1] = cmul(a[1][1], w1);
    a[1][2] = turn8(a[1][2]);
    a[1][3] = cmul(a[1][3], w3);
    a[2][1] = turn8(a[2][1]);
    a[2][2] = rot90<SIGN>(a[2][2]);
    a[2][3] = rot90<SIGN>(turn8(a[2][3]));
    a[3][1] = cmul(a[3][1], w3);
    a[3][2] = rot90<SIGN>(turn8(a[3][2]));
    const double2 t = cmul(a[3][3], w1);  // exp(9 pi i / 8) = -exp(pi i / 8)
    a[3][3] = make_double2(-t.x, -t.y);
#pragma unroll
    for (int r = 0; r < 4; r++) {
        double2 b[4] = {a[0][r], a[1][r], a[2][r], a[3][r]};
        dft4<SIGN>(b);
#pragma unroll
        for (int q = 0; q < 4; q++) x[r + 4 * q] = b[q];
    }
}

template <int R, int SIGN>
__device__ __forceinline__ void dft(double2 *x)
{
    static_assert(R == 4 || R == 8 || R == 16, "radix_of");
    if constexpr (R == 16) dft16<SIGN>(x);
    else if constexpr (R == 8) dft8<SIGN>(x);
    else dft4<SIGN>(x);
}

// Radix of the stage that has `rest` points a sub-transform left to do: 16
// where that ends a line in one stage or two, else 8, and 4 for the rest of
// 32.  Lines of 128 .. 2048 points so take 2, 2, 3, 3 and 3 stages (8 and 16
// points) instead of the 3, 3, 3, 4 and 4 of radix 8: a stage less is two
// shared-memory accesses a point and two barriers less.
__host__ __device__ constexpr int radix_of(int rest) { return rest == 4 ? 4 : (rest == 16 || rest == 256 ? 16 : 8); }
template <int N, int NS>
struct StageRadix {
    static constexpr int value = radix_of(N / NS);
};

// Points a thread holds: one butterfly of 16, two of 8 or four of 4 a stage.
constexpr int kPerThread = 16;

// Shared-memory place of point n of line l: rows of P, one spare point after
// every R rows, R the first stage's radix, so that its writes (rows R j + r
// for consecutive j, 16 R P bytes apart without it) fall on different banks.
template <int N, int P>
__device__ __forceinline__ int sidx(int n, int l)
{
    return n * P + l + n / StageRadix<N, 1>::value;
}
template <int N, int P>
constexpr int smem_points()
{
    return N * P + N / StageRadix<N, 1>::value;
}

// Stockham stages over L lines of N points: a stage with sub-transforms of
// NS points and radix R has N/R butterflies a line; butterfly j takes the
// points j + r N/R, twiddles them by W^((j mod NS) r N/(NS R)), transforms
// them and puts them at (j / NS) NS R + (j mod NS) + r NS.  The first stage
// (NS = 1) reads its points straight from the field and the last
// (NS R = N, so its outputs land on j + r NS) writes straight to it: the
// stages between exchange through shared memory, s[sidx(n, l)].

// Butterfly b's line l and index j: in the first and the last stage x
// lines take j fastest (a warp walks a line: coalesced), y and z lines l
// fastest (a warp walks a row of x values).
template <int AXIS, int L, int NB>
__device__ __forceinline__ void bfly(int b, int &l, int &j)
{
    if constexpr (AXIS == 0) {
        j = b % NB;
        l = b / NB;
    } else {
        l = b % L;
        j = b / L;
    }
}

// The twiddles w^r, r < R, of butterfly j: w, w^2, w^4 and w^8 from the roots
// table, the others their products (a few ulps; the transform's rounding is
// of the same order), so a butterfly loads 3 or 4 roots instead of 7 or 15.
template <int N, int NS, int R, int SIGN>
__device__ __forceinline__ void twiddle_dft(double2 *v, int j, const double2 *__restrict__ W, int wscale)
{
    if constexpr (NS > 1) {
        const int step = (j % NS) * (N / (NS * R)) * wscale;
        auto root = [&](int r) {
            double2 w = __ldg(W + step * r);
            if constexpr (SIGN < 0) w.y = -w.y;
            return w;
        };
        if constexpr (R == 16) {
            double2 w[16];
            w[1] = root(1);
            w[2] = root(2);
            w[4] = root(4);
            w[8] = root(8);
#pragma unroll
            for (int r = 3; r < 16; r++) {
                const int top = r >= 8 ? 8 : (r >= 4 ? 4 : 2);
                if (r != 4 && r != 8) w[r] = cmul(w[top], w[r - top]);
            }
#pragma unroll
            for (int r = 1; r < 16; r++) v[r] = cmul(v[r], w[r]);
        } else if constexpr (R == 8) {
            const double2 w1 = root(1), w2 = root(2), w4 = root(4), w3 = cmul(w1, w2);
            v[1] = cmul(v[1], w1);
            v[2] = cmul(v[2], w2);
            v[3] = cmul(v[3], w3);
            v[4] = cmul(v[4], w4);
            v[5] = cmul(v[5], cmul(w1, w4));
            v[6] = cmul(v[6], cmul(w2, w4));
            v[7] = cmul(v[7], cmul(w3, w4));
        } else {
            const double2 w1 = root(1), w2 = root(2);
            v[1] = cmul(v[1], w1);
            v[2] = cmul(v[2], w2);
            v[3] = cmul(v[3], cmul(w1, w2));
        }
    }
    dft<R, SIGN>(v);
}

// A stage between the first and the last: shared to shared, all reads
// before the barrier, all writes after it.  Lines fastest on every axis
// here: the L lanes of a butterfly index share its twiddles (one load for
// them all).
template <int N, int L, int P, int NS, int R, int SIGN>
__device__ __forceinline__ void stage_mid(double2 *s, const double2 *__restrict__ W, int wscale)
{
    constexpr int T = N * L / kPerThread, NB = N / R, PER = NB * L / T;
    double2 v[PER][R];
#pragma unroll
    for (int p = 0; p < PER; p++) {
        int l, j;
        bfly<1, L, NB>(threadIdx.x + p * T, l, j);
#pragma unroll
        for (int r = 0; r < R; r++) v[p][r] = s[sidx<N, P>(j + r * NB, l)];
        twiddle_dft<N, NS, R, SIGN>(v[p], j, W, wscale);
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < PER; p++) {
        int l, j;
        bfly<1, L, NB>(threadIdx.x + p * T, l, j);
        const int d = (j / NS) * NS * R + (j % NS);
#pragma unroll
        for (int r = 0; r < R; r++) s[sidx<N, P>(d + r * NS, l)] = v[p][r];
    }
    __syncthreads();
}

// NS of the last stage
__host__ __device__ constexpr int last_ns(int n)
{
    int ns = 1;
    while (ns * radix_of(n / ns) != n) ns *= radix_of(n / ns);
    return ns;
}

template <int N, int L, int P, int NS, int SIGN>
__device__ __forceinline__ void mid_stages(double2 *s, const double2 *__restrict__ W, int wscale)
{
    if constexpr (NS < last_ns(N)) {
        constexpr int R = StageRadix<N, NS>::value;
        stage_mid<N, L, P, NS, R, SIGN>(s, W, wscale);
        mid_stages<N, L, P, NS * R, SIGN>(s, W, wscale);
    }
}

// Lines a CTA: about TP points a tile, 2 .. 16 lines (x lines); y and z lines
// at least 8 (a row of L consecutive x values is the run each strided row
// read fetches: 128 bytes) and at most 32, and at most 8192 points.  TP is
// 4096 for fields beyond the L2; 2048 for those within it, which have too
// few tiles to fill the SMs evenly: 128^3 points 247 -> 220 us for 6
// iterations, 512 x 256 x 256 11.27 (4096) against 11.39 ms; and 512 for fields
// of up to 2^20 points, whose 2048-point tiles leave SMs without one (8
// iterations, 512 against 2048: 32 x 64 x 32 86.0 and 92.1 us, 128 x 128 x 32 127
// and 131, 128 x 128 x 64 171 and 184; the same at 2^20 and below in every
// other shape or better, at 2^21 between 2 % better and 2 % worse).
constexpr int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }
template <int N, int AXIS, int TP>
struct Tile {
    static constexpr int L = AXIS == 0 ? clampi(TP / N, 2, 16) : clampi(TP / N, 8 < 8192 / N ? 8 : 8192 / N, 32);
    static constexpr int T = N * L / kPerThread;
    static constexpr int CTAS = 8192 / (N * L) < 1 ? 1 : 8192 / (N * L);  // 128 registers a thread
};
constexpr int kLargeTile = 4096, kSmallTile = 2048, kTinyTile = 512;
constexpr long long kTinyPoints = 1 << 20;

// One tile of one axis of the transform, AXIS 0 (x), 1 (y), 2 (z): L lines
// of N points, point n of line l at base + n sn + l sl, by T threads.  in and
// out may be the same array (the CTA reads its whole tile, in the first
// stage, before it writes any of it, in the last).  A point enters as
// `as_read` makes it of what was read (line l, row n), and the outputs go out
// by `put`.  Field loads bypass L1: in k_fft_yx other SMs
// wrote them during the launch.
template <int N, int AXIS, int SIGN, int L, int P, typename Read, typename Put>
__device__ __forceinline__ void axis_tile(const double2 *in, double2 *sbuf, const double2 *__restrict__ W, int wscale,
                                          long long base, long long sn, long long sl, Read as_read,
                                          Put put)
{
    constexpr int T = N * L / kPerThread;
    constexpr int R0 = StageRadix<N, 1>::value;
    static_assert(last_ns(N) >= 8, "a first and a last stage");
    // first stage (NS = 1): butterfly j of line l reads its points, rows
    // j + r N/R0, from the field -- every load before any store (the evolved
    // points go back to u0, which is `in`)
    {
        constexpr int NB = N / R0, PER = NB * L / T;
        double2 v[PER][R0];
#pragma unroll
        for (int p = 0; p < PER; p++) {
            int l, j;
            bfly<AXIS, L, NB>(threadIdx.x + p * T, l, j);
#pragma unroll
            for (int r = 0; r < R0; r++) v[p][r] = __ldcg(in + base + (j + r * NB) * sn + l * sl);
        }
#pragma unroll
        for (int p = 0; p < PER; p++) {
            int l, j;
            bfly<AXIS, L, NB>(threadIdx.x + p * T, l, j);
#pragma unroll
            for (int r = 0; r < R0; r++) v[p][r] = as_read(v[p][r], l, j + r * NB);
            dft<R0, SIGN>(v[p]);
#pragma unroll
            for (int r = 0; r < R0; r++) sbuf[sidx<N, P>(R0 * j + r, l)] = v[p][r];
        }
        __syncthreads();
    }
    mid_stages<N, L, P, R0, SIGN>(sbuf, W, wscale);
    // last stage: its outputs are the rows j + r NS of the field
    {
        constexpr int NS = last_ns(N), R = N / NS, NB = N / R, PER = NB * L / T;
        double2 v[PER][R];
#pragma unroll
        for (int p = 0; p < PER; p++) {
            int l, j;
            bfly<AXIS, L, NB>(threadIdx.x + p * T, l, j);
#pragma unroll
            for (int r = 0; r < R; r++) v[p][r] = sbuf[sidx<N, P>(j + r * NB, l)];
            twiddle_dft<N, NS, R, SIGN>(v[p], j, W, wscale);
        }
#pragma unroll
        for (int p = 0; p < PER; p++) {
            int l, j;
            bfly<AXIS, L, NB>(threadIdx.x + p * T, l, j);
#pragma unroll
            for (int r = 0; r < R; r++) put(base + (j + r * NS) * sn + l * sl, v[p][r]);
        }
    }
}

// One axis over the whole field, a tile a CTA.  EVOLVE: in is u0 as the
// forward transform left it; each point is multiplied by its factor of
// iteration `iter` (the state of ft.cu:1245-1256 after that many), written
// back to u0 when `store` is set (the last iteration), and transformed into
// out.  The factor is ex ey ez from three tables of a few KB: looked up by
// |k|^2 in one table of 1.5 MB (512^3) and applied iter times, this pass ran
// at 3.3 TB/s where the plain z pass ran at 5.2.
template <int N, int AXIS, int SIGN, bool EVOLVE, int TP>
__global__ void __launch_bounds__(Tile<N, AXIS, TP>::T, Tile<N, AXIS, TP>::CTAS)
    k_fft(const double2 *in, double2 *out, double2 *u0, const double *__restrict__ ev,
          const double2 *__restrict__ W, int wscale, int nx, int ny, int nz, int iter, int store)
{
    static_assert(!EVOLVE || AXIS == 2, "evolve rides on the z lines");
    constexpr int L = Tile<N, AXIS, TP>::L, P = AXIS == 0 ? L + 1 : L;
    extern __shared__ double2 sbuf[];
    long long base, sn, sl;
    int x0 = 0, q = 0;  // y and z lines: the tile's first x and its z (y lines) or y (z lines)
    if constexpr (AXIS == 0) {
        base = (long long)blockIdx.x * L * nx;
        sn = 1;
        sl = nx;
    } else {
        const int tiles_x = nx / L;
        x0 = (blockIdx.x % tiles_x) * L;
        q = blockIdx.x / tiles_x;
        base = AXIS == 1 ? (long long)q * nx * ny + x0 : (long long)q * nx + x0;
        sn = AXIS == 1 ? (long long)nx : (long long)nx * ny;
        sl = 1;
    }
    const double *e = ev + (long long)(iter - 1) * (nx + ny + nz);
    const double ey = EVOLVE ? __ldg(e + nx + q) : 1.0;
    axis_tile<N, AXIS, SIGN, L, P>(
        in, sbuf, W, wscale, base, sn, sl,
        [&](double2 v, int l, int n) {
            if constexpr (EVOLVE) {
                const double t = __ldg(e + x0 + l) * ey * __ldg(e + nx + ny + n);
                v = make_double2(v.x * t, v.y * t);
                if (store) u0[base + n * sn + l] = v;
            }
            return v;
        },
        [&](long long e, double2 v) { out[e] = v; });
}

// The y and then the x axis in one kernel, in place, for fields beyond the
// L2: a plane's y tiles are written and its x tiles read a few planes later,
// while the plane is still in L2, so the two axes together read and write
// HBM once.  Work items (tiles of 4096 points, 256 threads, two CTAs an SM)
// are handed out by a ticket in this order: the y tiles of planes 0 .. lag-1,
// then those of plane lag + i and the x tiles of plane i in turn, then the
// last planes' x tiles.  An x tile waits until its plane's y tiles are
// counted; it only ever waits for items handed out before it, and y items
// wait for none, so the items always finish whatever CTAs are resident.
// The wait is bounded all the same.
//
// Large fields: those that do not stay in L2 from one pass to the next.  At
// 256 x 256 x 64 (67 MB) the separate passes take 433 us for 6 iterations and
// this one 469; at 256 x 256 x 128 (134 MB) 978 and 942; at 512 x 256 x 256
// and 20 iterations 11.27 and 11.04 ms, at 512^3 52.2 and 49.6.
constexpr long long kLargeBytes = 100LL << 20;
constexpr int kTilePoints = kLargeTile;
constexpr int kTileThreads = kTilePoints / kPerThread;
constexpr long long kWaitNs = 2000000000LL;

__device__ __forceinline__ bool wait_count(const int *count, int want, const int *failed, long long limit_ns)
{
    unsigned long long t0 = 0;
    for (unsigned spins = 0;; spins++) {
        int v;
        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
        if (v >= want) return true;
        if ((spins & 63u) == 63u) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (t0 == 0) t0 = t;
            if ((long long)(t - t0) > limit_ns || *(volatile const int *)failed) return false;
        }
    }
}

template <int NX, int NY, int SIGN>
__global__ void __launch_bounds__(kTileThreads, 2)
    k_fft_yx(double2 *u, const double2 *__restrict__ W, int wscale_x, int wscale_y, int nz, int lag, PlaneSync s,
             long long limit_ns)
{
    constexpr int LX = kTilePoints / NX, LY = kTilePoints / NY, TP = NX * NY / kTilePoints;
    extern __shared__ double2 sbuf[];
    __shared__ int next, stop;
    if (threadIdx.x == 0) {
        next = atomicAdd(s.ticket, 1);
        stop = 0;
    }
    for (;;) {
        __syncthreads();  // the item is known, and the last one's shared reads are over
        const int item = next;
        if (item >= 2 * nz * TP) return;
        const int g = item / TP, tile = item % TP;
        int plane, x_axis;
        if (g < lag) {
            plane = g;
            x_axis = 0;
        } else if (g < 2 * nz - lag) {
            x_axis = (g - lag) & 1;
            plane = (g - lag) / 2 + (x_axis ? 0 : lag);
        } else {
            plane = g - nz;
            x_axis = 1;
        }
        if (threadIdx.x == 0 && x_axis && !wait_count(s.done + plane, TP, s.failed, limit_ns)) {
            atomicExch(s.failed, 1);
            stop = 1;
        }
        __syncthreads();
        if (stop) return;
        int ahead = 0;
        if (threadIdx.x == 0) ahead = atomicAdd(s.ticket, 1);
        const long long corner = (long long)plane * NX * NY;
        const auto as_read = [](double2 v, int, int) { return v; };
        if (x_axis) {  // the outputs are next read an iteration later: out of L2 first
            axis_tile<NX, 0, SIGN, LX, LX + 1>(u, sbuf, W, wscale_x, corner + (long long)tile * LX * NX, 1, NX, as_read,
                                               [&](long long e, double2 v) { __stcs(u + e, v); });
        } else {
            axis_tile<NY, 1, SIGN, LY, LY>(u, sbuf, W, wscale_y, corner + tile * LY, NX, 1, as_read,
                                           [&](long long e, double2 v) { u[e] = v; });
            __syncthreads();
            if (threadIdx.x == 0) {
                __threadfence();
                asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(s.done + plane) : "memory");
            }
        }
        if (threadIdx.x == 0) next = ahead;
    }
}

// sums[it] = the sum of u1 at the 1024 points, over nt (warp by warp, then
// the warps, in a fixed order); and the dependency words back to zero for
// the next iteration's k_fft_yx.
__global__ void __launch_bounds__(kPoints) k_checksum(const double2 *u1, int nx, int ny, int nz, int it,
                                                      double2 *sums, PlaneSync s)
{
    __shared__ double2 sh[kPoints / 32];
    const int j = threadIdx.x + 1;
    const long long e = (long long)(j % nx) + (long long)(3 * j % ny) * nx + (long long)(5 * j % nz) * nx * ny;
    double2 v = u1[e];
    for (int k = threadIdx.x; k < nz; k += kPoints) s.done[k] = 0;
    if (threadIdx.x == 0) *s.ticket = 0;
    auto warp_sum = [&] {
#pragma unroll
        for (int w = 16; w > 0; w >>= 1) {
            v.x += __shfl_down_sync(0xffffffffu, v.x, w);
            v.y += __shfl_down_sync(0xffffffffu, v.y, w);
        }
    };
    warp_sum();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        v = sh[threadIdx.x];
        warp_sum();
        const double nt = (double)nx * ny * nz;
        if (threadIdx.x == 0) sums[it] = make_double2(v.x / nt, v.y / nt);
    }
}

using FftKernel = void (*)(const double2 *, double2 *, double2 *, const double *, const double2 *, int, int, int,
                           int, int, int);
using FusedKernel = void (*)(double2 *, const double2 *, int, int, int, int, PlaneSync, long long);

struct Launch {
    FftKernel k = nullptr;
    int threads = 0, lines = 0;
    size_t smem = 0;
};

struct FusedLaunch {
    FusedKernel k = nullptr;
    size_t smem = 0;
    int lag = 0, grid = 0;
};

template <int NX, int NY>
FusedLaunch make_fused()
{
    constexpr int LX = kTilePoints / NX, LY = kTilePoints / NY;
    constexpr int px = smem_points<NX, LX + 1>(), py = smem_points<NY, LY>();
    FusedLaunch a;
    a.k = k_fft_yx<NX, NY, -1>;
    a.smem = sizeof(double2) * (px > py ? px : py);
    return a;
}

template <int NX>
FusedLaunch pick_fused_y(int ny)
{
    switch (ny) {
    case 128: return make_fused<NX, 128>();
    case 256: return make_fused<NX, 256>();
    case 512: return make_fused<NX, 512>();
    case 1024: return make_fused<NX, 1024>();
    default: return FusedLaunch{};
    }
}

FusedLaunch pick_fused(int nx, int ny)
{
    switch (nx) {
    case 128: return pick_fused_y<128>(ny);
    case 256: return pick_fused_y<256>(ny);
    case 512: return pick_fused_y<512>(ny);
    case 1024: return pick_fused_y<1024>(ny);
    default: return FusedLaunch{};
    }
}

template <int N, int AXIS, int SIGN, bool EVOLVE, int TP>
Launch make_launch()
{
    constexpr int L = Tile<N, AXIS, TP>::L, P = AXIS == 0 ? L + 1 : L;
    Launch a;
    a.k = k_fft<N, AXIS, SIGN, EVOLVE, TP>;
    a.threads = Tile<N, AXIS, TP>::T;
    a.lines = L;
    a.smem = sizeof(double2) * smem_points<N, P>();
    return a;
}

template <int AXIS, int SIGN, bool EVOLVE, int TP>
Launch pick_tile(int n)
{
    switch (n) {
    case 32: return make_launch<32, AXIS, SIGN, EVOLVE, TP>();
    case 64: return make_launch<64, AXIS, SIGN, EVOLVE, TP>();
    case 128: return make_launch<128, AXIS, SIGN, EVOLVE, TP>();
    case 256: return make_launch<256, AXIS, SIGN, EVOLVE, TP>();
    case 512: return make_launch<512, AXIS, SIGN, EVOLVE, TP>();
    case 1024: return make_launch<1024, AXIS, SIGN, EVOLVE, TP>();
    case 2048:  // with sides of 32 at least, such a field is never a tiny one
        if constexpr (TP != kTinyTile) return make_launch<2048, AXIS, SIGN, EVOLVE, TP>();
        return Launch{};
    default: return Launch{};
    }
}

template <int AXIS, int SIGN, bool EVOLVE>
Launch pick(int n, long long points)
{
    if (points <= kTinyPoints) return pick_tile<AXIS, SIGN, EVOLVE, kTinyTile>(n);
    if (points * (long long)sizeof(double2) < kLargeBytes) return pick_tile<AXIS, SIGN, EVOLVE, kSmallTile>(n);
    return pick_tile<AXIS, SIGN, EVOLVE, kLargeTile>(n);
}

}  // namespace ft
}  // namespace cgb

using namespace cgb;
using namespace cgb::ft;

struct cgb_ft {
    int device = 0, nx = 0, ny = 0, nz = 0, maxdim = 0;
    long long nt = 0;
    double2 *u0 = nullptr, *u1 = nullptr;
    // one allocation: the roots, the checksums, the evolve factors (kMaxIter
    // (nx + ny + nz)) and PlaneSync's words (ticket, failed, nz counts)
    double2 *W = nullptr, *sums = nullptr;
    double *ev = nullptr;
    int *sync = nullptr;
    int k2max = 0;
    Launch fwd[3], inv[3];  // x, y, z passes; inv[2] evolves
    FusedLaunch inv_yx;     // y and x in one kernel (k null: the separate passes)
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaGraphExec_t exec = nullptr;
    int exec_niter = -1;
};

namespace {

#define FT_TRY(call)                                                                      \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess)                                                            \
            return set_error(e_ == cudaErrorMemoryAllocation ? CGB_ERR_NOMEM : CGB_ERR_CUDA, \
                             "ft: %s: %s", #call, cudaGetErrorString(e_));                \
    } while (0)

void ft_release(cgb_ft *f)
{
    if (!f) return;
    cudaSetDevice(f->device);
    if (f->exec) cudaGraphExecDestroy(f->exec);
    for (void *p : {(void *)f->u0, (void *)f->u1, (void *)f->W})
        if (p) cudaFree(p);
    if (f->ev0) cudaEventDestroy(f->ev0);
    if (f->ev1) cudaEventDestroy(f->ev1);
    if (f->stream) cudaStreamDestroy(f->stream);
    delete f;
}

bool pow2_in(int v, int lo, int hi) { return v >= lo && v <= hi && (v & (v - 1)) == 0; }

PlaneSync plane_sync(cgb_ft *f) { return PlaneSync{f->sync, f->sync + 1, f->sync + 2}; }

void run_pass(cgb_ft *f, const Launch &a, int axis, const double2 *in, double2 *out, int iter = 0, int store = 0)
{
    const int dims[3] = {f->nx, f->ny, f->nz};
    const unsigned tiles = unsigned(f->nt / ((long long)dims[axis] * a.lines));
    a.k<<<tiles, a.threads, a.smem, f->stream>>>(in, out, f->u0, f->ev, f->W, f->maxdim / dims[axis], f->nx, f->ny,
                                                  f->nz, iter, store);
}

bool is_large(const cgb_ft *f) { return f->nt * (long long)sizeof(double2) >= kLargeBytes; }

// The fused y and x pass, where it is compiled (sides 128 .. 1024) and pays.
bool plan_fused(cgb_ft *f)
{
    FusedLaunch a = pick_fused(f->nx, f->ny);
    if (!a.k || !is_large(f)) return true;
    int sms = 0, ctas = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, f->device) != cudaSuccess ||
        cudaFuncSetAttribute(a.k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(a.smem)) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, a.k, kTileThreads, a.smem) != cudaSuccess || ctas < 1)
        return false;
    const int per_plane = f->nx * f->ny / kTilePoints;
    a.grid = std::min(sms * ctas, 2 * f->nz * per_plane);
    // planes between a plane's y and x tiles: two rounds of tiles, so that an
    // x tile seldom waits (38 MB of planes at 296 CTAs, well inside the L2)
    a.lag = std::min(f->nz, (2 * a.grid + per_plane - 1) / per_plane);
    f->inv_yx = a;
    return true;
}

// main's timed region (ft.cu:391-408): index map (as one table an axis and
// iteration), initial conditions, the roots, the forward transform u1 -> u0,
// then niter x (evolve, inverse transform, checksum).
void enqueue_benchmark(cgb_ft *f, int niter)
{
    const PlaneSync sync = plane_sync(f);
    const int tables = std::max(f->maxdim, (f->nx + f->ny + f->nz) * niter);
    k_tables<<<(tables + 255) / 256, 256, 0, f->stream>>>(f->W, f->maxdim, f->ev, f->nx, f->ny, f->nz, niter, sync);
    // elements a lane: 64 on large fields (a jump costs about 40 steps), fewer
    // where that would leave SMs idle
    const int per = int(std::min<long long>(64, std::max<long long>(4, f->nt / (148 * 1024))));
    const long long warps = (f->nt + 32LL * per - 1) / (32LL * per);
    k_initial<<<unsigned((warps + 7) / 8), 256, 0, f->stream>>>(f->u1, f->nt, per);
    run_pass(f, f->fwd[0], 0, f->u1, f->u1);
    run_pass(f, f->fwd[1], 1, f->u1, f->u1);
    run_pass(f, f->fwd[2], 2, f->u1, f->u0);
    for (int it = 1; it <= niter; it++) {
        run_pass(f, f->inv[2], 2, f->u0, f->u1, it, it == niter);
        if (f->inv_yx.k) {
            f->inv_yx.k<<<f->inv_yx.grid, kTileThreads, f->inv_yx.smem, f->stream>>>(
                f->u1, f->W, f->maxdim / f->nx, f->maxdim / f->ny, f->nz, f->inv_yx.lag, sync, kWaitNs);
        } else {
            run_pass(f, f->inv[1], 1, f->u1, f->u1);
            run_pass(f, f->inv[0], 0, f->u1, f->u1);
        }
        k_checksum<<<1, kPoints, 0, f->stream>>>(f->u1, f->nx, f->ny, f->nz, it, f->sums, sync);
    }
}

}  // namespace

extern "C" {

int cgb_ft_create(int device, int nx, int ny, int nz, cgb_ft **out)
{
    if (!out) return set_error(CGB_ERR_INVALID, "ft: null output");
    *out = nullptr;
    if (!pow2_in(nx, 32, 2048) || !pow2_in(ny, 32, 2048) || !pow2_in(nz, 32, 2048))
        return set_error(CGB_ERR_INVALID, "ft: each dimension a power of two in [32, 2048]");
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count)
        return set_error(CGB_ERR_NO_DEVICE, "ft: no CUDA device %d", device);
    int major = 0;
    FT_TRY(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device));
    if (major != 10) return set_error(CGB_ERR_NO_DEVICE, "ft: device %d is not sm_100", device);
    FT_TRY(cudaSetDevice(device));
    cgb_ft *f = new (std::nothrow) cgb_ft;
    if (!f) return set_error(CGB_ERR_NOMEM, "ft: allocation failed");
    f->device = device;
    f->nx = nx;
    f->ny = ny;
    f->nz = nz;
    f->maxdim = std::max(nx, std::max(ny, nz));
    f->nt = (long long)nx * ny * nz;
    f->k2max = (nx / 2) * (nx / 2) + (ny / 2) * (ny / 2) + (nz / 2) * (nz / 2);
    f->fwd[0] = pick<0, 1, false>(nx, f->nt);
    f->fwd[1] = pick<1, 1, false>(ny, f->nt);
    f->fwd[2] = pick<2, 1, false>(nz, f->nt);
    f->inv[0] = pick<0, -1, false>(nx, f->nt);
    f->inv[1] = pick<1, -1, false>(ny, f->nt);
    f->inv[2] = pick<2, -1, true>(nz, f->nt);
    bool ok = true;
    for (const Launch *a : {&f->fwd[0], &f->fwd[1], &f->fwd[2], &f->inv[0], &f->inv[1], &f->inv[2]})
        ok = ok && a->k &&
             cudaFuncSetAttribute(a->k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(a->smem)) == cudaSuccess;
    ok = ok && plan_fused(f);
    ok = ok && cudaStreamCreateWithFlags(&f->stream, cudaStreamNonBlocking) == cudaSuccess &&
         cudaEventCreate(&f->ev0) == cudaSuccess && cudaEventCreate(&f->ev1) == cudaSuccess;
    if (!ok) {
        ft_release(f);
        return set_error(CGB_ERR_CUDA, "ft: kernel set-up failed");
    }
    const size_t points = size_t(f->maxdim) + kMaxIter + 1, factors = size_t(nx + ny + nz) * kMaxIter;
    ok = cudaMalloc(&f->u0, sizeof(double2) * size_t(f->nt)) == cudaSuccess &&
         cudaMalloc(&f->u1, sizeof(double2) * size_t(f->nt)) == cudaSuccess &&
         cudaMalloc(&f->W, sizeof(double2) * points + sizeof(double) * factors + sizeof(int) * size_t(nz + 2)) ==
             cudaSuccess;
    if (ok) {
        f->sums = f->W + f->maxdim;
        f->ev = reinterpret_cast<double *>(f->W + points);
        f->sync = reinterpret_cast<int *>(f->ev + factors);
    }
    if (!ok) {
        ft_release(f);
        return set_error(CGB_ERR_NOMEM, "ft: device allocation failed (%d x %d x %d)", nx, ny, nz);
    }
    *out = f;
    return CGB_OK;
}

int cgb_ft_destroy(cgb_ft *f)
{
    ft_release(f);
    return CGB_OK;
}

int cgb_ft_run(cgb_ft *f, int niter, double *sums, double *device_ms)
{
    if (!f) return set_error(CGB_ERR_INVALID, "ft: null instance");
    if (niter < 1 || niter > kMaxIter) return set_error(CGB_ERR_INVALID, "ft: niter must be in [1, %d]", kMaxIter);
    FT_TRY(cudaSetDevice(f->device));
    const cudaStream_t st = f->stream;
    if (!f->exec || f->exec_niter != niter) {
        if (f->exec) cudaGraphExecDestroy(f->exec);
        f->exec = nullptr;
        cudaGraph_t graph = nullptr;
        FT_TRY(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        enqueue_benchmark(f, niter);
        const cudaError_t e1 = cudaGetLastError();
        const cudaError_t e2 = cudaStreamEndCapture(st, &graph);
        if (e1 != cudaSuccess || e2 != cudaSuccess) {
            if (graph) cudaGraphDestroy(graph);
            return set_error(CGB_ERR_CUDA, "ft: capture failed: %s", cudaGetErrorString(e1 != cudaSuccess ? e1 : e2));
        }
        const cudaError_t e3 = cudaGraphInstantiate(&f->exec, graph, 0);
        cudaGraphDestroy(graph);
        if (e3 != cudaSuccess) {
            f->exec = nullptr;
            return set_error(CGB_ERR_CUDA, "ft: graph instantiation failed");
        }
        f->exec_niter = niter;
    }
    FT_TRY(cudaEventRecord(f->ev0, st));
    FT_TRY(cudaGraphLaunch(f->exec, st));
    FT_TRY(cudaEventRecord(f->ev1, st));
    double2 h[kMaxIter + 1];
    int failed = 0;
    FT_TRY(cudaMemcpyAsync(h, f->sums, sizeof(double2) * (niter + 1), cudaMemcpyDeviceToHost, st));
    if (f->inv_yx.k) FT_TRY(cudaMemcpyAsync(&failed, f->sync + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
    FT_TRY(cudaStreamSynchronize(st));
    if (failed) return set_error(CGB_ERR_TIMEOUT, "ft: a plane's y tiles were not done within the wait limit");
    float ms = 0.f;
    FT_TRY(cudaEventElapsedTime(&ms, f->ev0, f->ev1));
    if (sums)
        for (int it = 1; it <= niter; it++) {
            sums[2 * (it - 1)] = h[it].x;
            sums[2 * (it - 1) + 1] = h[it].y;
        }
    if (device_ms) *device_ms = ms;
    return CGB_OK;
}

int cgb_ft_selftest_wait(cgb_ft *f, long long limit_ns)
{
    if (!f || limit_ns <= 0 || limit_ns > 10000000000LL)
        return set_error(CGB_ERR_INVALID, "ft: limit_ns must be in (0, 1e10]");
    if (!f->inv_yx.k) return set_error(CGB_ERR_STATE, "ft: this field takes the y and x axes apart");
    FT_TRY(cudaSetDevice(f->device));
    const cudaStream_t st = f->stream;
    const PlaneSync sync = plane_sync(f);
    // only the last item is left to hand out, an x tile; no plane has a y tile
    const int last = 2 * f->nz * (f->nx * f->ny / kTilePoints) - 1;
    FT_TRY(cudaMemsetAsync(f->sync, 0, sizeof(int) * size_t(f->nz + 2), st));
    FT_TRY(cudaMemcpyAsync(sync.ticket, &last, sizeof(int), cudaMemcpyHostToDevice, st));
    f->inv_yx.k<<<f->inv_yx.grid, kTileThreads, f->inv_yx.smem, st>>>(
        f->u1, f->W, f->maxdim / f->nx, f->maxdim / f->ny, f->nz, f->inv_yx.lag, sync, limit_ns);
    FT_TRY(cudaGetLastError());
    int failed = 0;
    FT_TRY(cudaMemcpyAsync(&failed, sync.failed, sizeof(int), cudaMemcpyDeviceToHost, st));
    FT_TRY(cudaStreamSynchronize(st));
    if (failed) return set_error(CGB_ERR_TIMEOUT, "ft: a plane's y tiles were not done within the wait limit");
    return CGB_OK;
}

int cgb_ft_read(cgb_ft *f, int which, double *out, long long count)
{
    if (!f || !out || which < 0 || which > 2) return set_error(CGB_ERR_INVALID, "ft: bad read");
    const long long need = which == 2 ? f->nt : 2 * f->nt;
    if (count < need) return set_error(CGB_ERR_CAPACITY, "ft: %lld doubles needed", need);
    FT_TRY(cudaSetDevice(f->device));
    if (which == 2) {  // the per-point map, expanded from the table into a scratch array
        double *tw = nullptr, *twk2 = nullptr;
        FT_TRY(cudaMalloc(&tw, sizeof(double) * size_t(f->nt)));
        if (cudaMalloc(&twk2, sizeof(double) * size_t(f->k2max + 1)) != cudaSuccess) {
            cudaFree(tw);
            return set_error(CGB_ERR_NOMEM, "ft: no memory for the twiddle table");
        }
        k_twiddle_table<<<(f->k2max + 256) / 256, 256, 0, f->stream>>>(twk2, f->k2max);
        k_indexmap<<<8 * 148, 256, 0, f->stream>>>(tw, twk2, f->nx, f->ny, f->nz);
        const cudaError_t e1 = cudaGetLastError(), e2 = cudaStreamSynchronize(f->stream);
        const cudaError_t e3 = cudaMemcpy(out, tw, sizeof(double) * size_t(need), cudaMemcpyDeviceToHost);
        cudaFree(tw);
        cudaFree(twk2);
        if (e1 != cudaSuccess || e2 != cudaSuccess || e3 != cudaSuccess)
            return set_error(CGB_ERR_CUDA, "ft: reading the twiddle factors failed");
        return CGB_OK;
    }
    const void *src = which == 0 ? (const void *)f->u0 : (const void *)f->u1;
    FT_TRY(cudaMemcpy(out, src, sizeof(double) * size_t(need), cudaMemcpyDeviceToHost));
    return CGB_OK;
}

}  // extern "C"

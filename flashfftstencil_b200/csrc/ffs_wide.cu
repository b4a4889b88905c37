// FP64 butterfly form on wide tiles: one fused pass as three kernels over a workspace.
//
// Why: the halo is r tau per side, so the tile edge bounds the fused step count and the
// share of points that are kept.  A 128 x 128 tile (the largest in one SM's shared memory)
// keeps (96 / 128)^2 = 0.56 of its points at r tau = 16, and T = 32 needs two such passes; a
// 512 x 512 tile keeps 0.77 at r tau = 32 in one pass, a 2048 x 2048 one 0.77 at r tau = 128.
// The price is that the transform leaves the SM between its x and y parts.
//
// One tile is Nx x Ny real points, held as Ny / 2 packed complex rows (row y + i row y + Ny/2):
//   rows_fwd   packed row from the grid, FFT-Nx, stored half by half: Z[j] at slot j and
//              Z[Nx - j] at slot Hoff + j (j = 0 .. Nx/2, Hoff = Nx/2 + kPad), so that the two
//              values a column needs lie at the same offset of two aligned segments;
//   columns    for each kx = j: the true rows' half spectra (Z[j] +- conj Z[Nx-j]) for y and
//              y + Ny/2, which one thread holds (y = t + L a), FFT-Ny, times S^tau, inverse
//              FFT-Ny, stored in place: row y's value at slot j (y < Ny/2) or Hoff + j;
//   rows_inv   two useful rows packed again, inverse FFT-Nx, cropped stores.
// Every global access of a line's threads is to consecutive addresses, every exchange is
// conflict-free (ffs_wide.cuh).
// Bound: rows by HBM (rows_fwd 0.87 of the copy rate, rows_inv 0.72 to 0.78: Box2D9P 4096^2, periodic, T = 32
// in 100 tiles of 512 x 512 73 and 68 us); the columns (127 us, 0.48) by the sum of their loads, four exchanges
// and stores, with 16 warps on an SM at 128 registers (of 9.5 cycles between two issues of a warp 3.8 wait for
// global loads, 2.0 for shared memory; FP64 pipe 39 %).  8 points a thread and twice the warps spill (49 us
// against 44 a launch of fewer tiles).  Against the 128 x 128 tiles: that grid with a fixed boundary (81 tiles)
// 505 -> 296 us, Box2D25P 8192^2, periodic, T = 128 12878 -> 1720.  Replaces rfft_2d (src/2D/rfft_2d/2d_rfft_1_async.cu:17-364)
// like the one-SM tiles do.
#include "ffs_wide.cuh"

#include <algorithm>

#include "ffs_band.cuh"
#include "ffs_chain.cuh"
#include "ffs_kernels.h"

namespace ffst {
namespace wide {

constexpr int kRowThreads = 128;

// Points per thread of a row and of a column line, and the threads of a column block.
constexpr int row_points(int n) { return n <= 512 ? 8 : 16; }
constexpr int col_points(int n) { return n <= 256 ? 8 : 16; }
constexpr int col_threads(int n) { return n <= 1024 ? 256 : 512; }
constexpr int col_blocks_per_sm(int n) { return n <= 256 ? 3 : (n <= 1024 ? 2 : 1); }
template <int N>
using RowShape = Shape<N, row_points(N)>;
template <int N>
using ColShape = Shape<N, col_points(N)>;
template <int N>
constexpr int col_count() { return col_threads(N) / ColShape<N>::L; } // columns side by side in a block
// row blocks per SM: 64 registers a thread with 8 points, 128 with 16
constexpr int row_blocks_per_sm(int n) { return 65536 / (row_points(n) == 8 ? 64 : 128) / kRowThreads; }

struct BlockSync {
    __device__ __forceinline__ void operator()() const { __syncthreads(); }
};
template <int N>
struct RowSync {
    __device__ __forceinline__ void operator()() const
    {
        if constexpr (RowShape<N>::L <= 32)
            __syncwarp();
        else
            __syncthreads();
    }
};

__device__ __forceinline__ int64_t wrap(int64_t x, int64_t n)
{
    const int64_t m = x % n;
    return m < 0 ? m + n : m;
}

template <int N>
__global__ void __launch_bounds__(kRowThreads, row_blocks_per_sm(N)) rows_fwd_kernel(const __grid_constant__ WideWork p)
{
    using S = RowShape<N>;
    extern __shared__ __align__(16) double2 smem[];
    chain_wait();
    const int l = threadIdx.x / S::L, t = threadIdx.x % S::L;
    constexpr int LPB = kRowThreads / S::L;
    const int half = p.tile[1] >> 1;
    const int line = blockIdx.x * LPB + l; // Ny / 2 is a multiple of LPB
    const int tl = line / half, r = line - tl * half;
    const int64_t tile = p.tile0 + tl;
    const int64_t ty = tile / p.nt[0], tx = tile - ty * p.nt[0];
    const int64_t x0 = p.org[0] + tx * p.useful[0] + t, y0 = p.org[1] + ty * p.useful[1] + r;
    double xr[S::P], xi[S::P];
    if (p.periodic) {
        const double *ra = p.in + wrap(y0, p.n[1]) * p.n[0], *rb = p.in + wrap(y0 + half, p.n[1]) * p.n[0];
        const int nx = (int)p.n[0];
        int x = (int)wrap(x0, p.n[0]);
#pragma unroll
        for (int a = 0; a < S::P; ++a) {
            xr[a] = __ldg(ra + x);
            xi[a] = __ldg(rb + x);
            x += S::L; // L <= 128 <= nx (the plan builder's bound for wide tiles)
            x -= x >= nx ? nx : 0;
        }
    } else {
        const bool ina = y0 >= 0 && y0 < p.n[1], inb = y0 + half >= 0 && y0 + half < p.n[1];
        const double *ra = p.in + y0 * p.n[0], *rb = p.in + (y0 + half) * p.n[0];
#pragma unroll
        for (int a = 0; a < S::P; ++a) {
            const int64_t x = x0 + S::L * a;
            const bool in = x >= 0 && x < p.n[0];
            xr[a] = in && ina ? __ldg(ra + x) : 0.0;
            xi[a] = in && inb ? __ldg(rb + x) : 0.0;
        }
    }
    line_fft<N, false, 1, S::P>(xr, xi, t, smem + l * S::SLOTS, p.tw[0], RowSync<N>());
    constexpr int H = N / 2 + kPad;
    double2 *w = p.work + (size_t)line * (2 * H);
#pragma unroll
    for (int a = 0; a < S::P; ++a) {
        const int f = t + S::L * a;
        const double2 v = make_double2(xr[a], xi[a]);
        if (a < S::P / 2) {
            w[f] = v;
            if (a == 0 && t == 0)
                w[H] = v; // the partner of 0 is 0
        } else {
            w[H + N - f] = v;
            if (a == S::P / 2 && t == 0)
                w[N / 2] = v; // the partner of N / 2 is N / 2
        }
    }
}

// Columns of a 2D tile: forward, spectrum, inverse.
template <int N>
__global__ void __launch_bounds__(col_threads(N), col_blocks_per_sm(N)) cols_kernel(const __grid_constant__ WideWork p)
{
    using S = ColShape<N>;
    constexpr int C = col_count<N>();
    extern __shared__ __align__(16) double2 smem[];
    chain_wait();
    const int c = threadIdx.x % C, t = threadIdx.x / C;
    const int hx = p.tile[0] >> 1;
    const int groups = hx / C + 1;
    // The tiles' blocks of one group of columns one after the other: they share its part of the spectrum,
    // which, from 16 MB on (2^20 points), the workspace streaming by takes out of L2 before the next tile
    // needs it (2048 x 2048 tiles, Box2D25P 8192^2 at T = 128 1813 -> 1720 us; 1024 x 2048 2200 -> 2125).
    // Below, tile by tile: adjacent segments then lie close in time (1024 x 512 and smaller 2 % faster).
    const bool by_group = N * hx >= 1 << 20;
    const int outer = by_group ? p.ntiles : groups, hi_index = blockIdx.x / outer, lo_index = blockIdx.x - hi_index * outer;
    const int tl = by_group ? lo_index : hi_index, j = (by_group ? hi_index : lo_index) * C + c;
    const bool live = j <= hx;
    const int H = hx + kPad, P = 2 * H;
    double2 *w = p.work + (size_t)tl * (N / 2) * P + j;
    double xr[S::P], xi[S::P];
    // twice the half spectra of rows y and y + Ny / 2 (the spectrum carries the factor 1/2)
#pragma unroll
    for (int a = 0; a < S::P / 2; ++a) {
        double2 zk = make_double2(0.0, 0.0), zm = zk;
        if (live) {
            const double2 *row = w + (t + S::L * a) * P;
            zk = row[0];
            zm = row[H];
        }
        xr[a] = zk.x + zm.x;
        xi[a] = zk.y - zm.y;
        xr[a + S::P / 2] = zk.y + zm.y;
        xi[a + S::P / 2] = zm.x - zk.x;
    }
    line_fft<N, false, C, S::P>(xr, xi, t, smem + c, p.tw[1], BlockSync());
    const double2 *sp = p.spec + j;
#pragma unroll
    for (int a = 0; a < S::P; ++a) {
        const double2 s = live ? __ldg(sp + (t + S::L * a) * H) : make_double2(0.0, 0.0);
        f128::cmul(xr[a], xi[a], s.x, s.y);
    }
    __syncthreads(); // the forward transform's last gets before the inverse's first puts
    line_fft<N, true, C, S::P>(xr, xi, t, smem + c, p.tw[1], BlockSync());
    const int lo = p.halo[1], hi = p.halo[1] + (int)p.useful[1];
    if (!live)
        return;
#pragma unroll
    for (int a = 0; a < S::P; ++a) {
        const int y = t + S::L * a;
        if (y >= lo && y < hi)
            w[(t + S::L * (a % (S::P / 2))) * P + (a < S::P / 2 ? 0 : H)] = make_double2(xr[a], xi[a]);
    }
}

template <int N>
__global__ void __launch_bounds__(kRowThreads, row_blocks_per_sm(N)) rows_inv_kernel(const __grid_constant__ WideWork p)
{
    using S = RowShape<N>;
    extern __shared__ __align__(16) double2 smem[];
    chain_wait();
    const int l = threadIdx.x / S::L, t = threadIdx.x % S::L;
    constexpr int LPB = kRowThreads / S::L;
    const int half = p.tile[1] >> 1;
    const int pairs = ((int)p.useful[1] + 1) >> 1;
    const int ppb = (pairs + LPB - 1) / LPB * LPB; // pairs per tile, rounded to whole blocks
    const int line = blockIdx.x * LPB + l;
    const int tl = line / ppb, q = line - tl * ppb;
    const int64_t tile = p.tile0 + tl;
    const int64_t ty = tile / p.nt[0], tx = tile - ty * p.nt[0];
    const int64_t x0 = p.org[0] + tx * p.useful[0] + t, yt = p.org[1] + ty * p.useful[1];
    const int ya = p.halo[1] + q, yb = ya + pairs;
    const bool ona = q < pairs && yt + ya < p.vhi[1];
    const bool onb = ona && yb < p.halo[1] + (int)p.useful[1] && yt + yb < p.vhi[1];
    if constexpr (S::L <= 32) { // a warp holds whole lines and waits for no other
        if (__all_sync(0xffffffffu, !ona)) // every lane votes
            return;
    }
    constexpr int H = N / 2 + kPad;
    const double2 *wt = p.work + (size_t)tl * half * (2 * H);
    const double2 *wa = wt + (size_t)(ya < half ? ya : ya - half) * (2 * H) + (ya < half ? 0 : H);
    const double2 *wb = wt + (size_t)(yb < half ? yb : yb - half) * (2 * H) + (yb < half ? 0 : H);
    double xr[S::P], xi[S::P];
    const double2 zero = make_double2(0.0, 0.0);
#pragma unroll
    for (int a = 0; a < S::P; ++a) {
        const int f = t + S::L * a;
        const int j = a < S::P / 2 ? f : N - f;
        const double2 u = ona ? wa[j] : zero, v = onb ? wb[j] : zero;
        if (a < S::P / 2) { // A + i B
            xr[a] = u.x - v.y;
            xi[a] = u.y + v.x;
        } else { // conj A + i conj B
            xr[a] = u.x + v.y;
            xi[a] = v.x - u.y;
        }
    }
    line_fft<N, true, 1, S::P>(xr, xi, t, smem + l * S::SLOTS, p.tw[0], RowSync<N>());
    const int lo = p.halo[0], hi = p.halo[0] + (int)p.useful[0];
    double *oa = p.out + (yt + ya) * p.n[0], *ob = p.out + (yt + yb) * p.n[0];
#pragma unroll
    for (int a = 0; a < S::P; ++a) {
        const int x = t + S::L * a;
        const int64_t gx = x0 + S::L * a;
        if (x >= lo && x < hi && gx < p.vhi[0]) {
            if (ona)
                oa[gx] = xr[a];
            if (onb)
                ob[gx] = xi[a];
        }
    }
}

// ---- 1-D: a pair of tiles per line ----
//
// Two tiles of N cells are one complex line (re = tile 2q, im = tile 2q + 1) that stays in its
// threads' registers: forward, spectrum, inverse, cropped stores, four exchanges and no other
// shared-memory traffic.  The one-SM tile (ffs_fft1d.cu) stages 4096-cell pairs through shared
// memory, one per SM, 10.5 us a wave; here an SM holds 8192 points in lines of 1024 to 4096, so short
// grids spread over more SMs.  The fixed boundary's boxes are blocks of the same launch.

constexpr int kLineThreads = 256;
template <int N>
using LineShape = Shape<N, 16>;

// (not inlined: inside the kernel its registers made the lines' code spill)
template <int WARPS>
__device__ __noinline__ void band_block(const BandWork &band, int box, unsigned char *smem)
{
    band::process_box<1, 0, false, WARPS>(band, box, smem, kLineThreads);
}

template <int N>
__global__ void __launch_bounds__(kLineThreads, 2) line_tiles_kernel(const __grid_constant__ WideWork p,
                                                                     const __grid_constant__ BandWork band, int tile_blocks)
{
    using S = LineShape<N>;
    constexpr int LPB = kLineThreads / S::L;
    extern __shared__ __align__(16) double2 smem[];
    chain_wait();
    if ((int)blockIdx.x >= tile_blocks) {
        const int box = (int)blockIdx.x - tile_blocks;
        if (band::warp_multiple(band) == 2)
            band_block<2>(band, box, reinterpret_cast<unsigned char *>(smem));
        else
            band_block<1>(band, box, reinterpret_cast<unsigned char *>(smem));
        return;
    }
    const int l = threadIdx.x / S::L, t = threadIdx.x % S::L;
    const int64_t q = (int64_t)blockIdx.x * LPB + l;
    const bool ona = 2 * q < p.nt[0], onb = 2 * q + 1 < p.nt[0];
    const int64_t n = p.n[0], oa = p.org[0] + 2 * q * p.useful[0], ob = oa + p.useful[0]; // the tiles' first cells
    double xr[S::P], xi[S::P];
    if (oa >= 0 && ob + N <= n && onb) { // both tiles inside the grid
        const double *a0 = p.in + oa + t, *b0 = p.in + ob + t;
#pragma unroll
        for (int a = 0; a < S::P; ++a) {
            xr[a] = __ldg(a0 + S::L * a);
            xi[a] = __ldg(b0 + S::L * a);
        }
    } else {
#pragma unroll
        for (int a = 0; a < S::P; ++a) {
            int64_t x = oa + t + S::L * a, y = x + p.useful[0];
            if (p.periodic) { // (N <= n: at most one period off)
                x += x < 0 ? n : x >= n ? -n : 0;
                y += y < 0 ? n : y >= n ? -n : 0;
            }
            xr[a] = ona && x >= 0 && x < n ? __ldg(p.in + x) : 0.0;
            xi[a] = onb && y >= 0 && y < n ? __ldg(p.in + y) : 0.0;
        }
    }
    double2 *sm = smem + l * S::SLOTS;
    line_fft<N, false, 1, S::P>(xr, xi, t, sm, p.tw[0], BlockSync());
#pragma unroll
    for (int a = 0; a < S::P; ++a) {
        const int f = t + S::L * a; // real weights: S(-f) = conj S(f)
        const double2 s = p.spec[a < S::P / 2 ? f : N - f];
        f128::cmul(xr[a], xi[a], s.x, a < S::P / 2 ? s.y : -s.y);
        if (a % 4 == 3)
            f128::hoist_fence();
    }
    __syncthreads(); // the forward transform's last gets before the inverse's first puts
    int ti = t;
    asm volatile("" : "+r"(ti)); // hides that the inverse reads the same twiddles: kept over, they spill
    line_fft<N, true, 1, S::P>(xr, xi, ti, sm, p.tw[0], BlockSync());
    // useful cells below vhi
    const int lo = p.halo[0];
    const int64_t end = lo + p.useful[0];
    const int ha = ona ? (int)min(end, p.vhi[0] - oa) : 0, hb = onb ? (int)min(end, p.vhi[0] - ob) : 0;
    double *a1 = p.out + oa + t, *b1 = p.out + ob + t;
#pragma unroll
    for (int a = 0; a < S::P; ++a) {
        const int c = t + S::L * a;
        if (c >= lo && c < ha)
            a1[S::L * a] = xr[a];
        if (c >= lo && c < hb)
            b1[S::L * a] = xi[a];
    }
}

template <int N>
cudaError_t line_tiles(const WideWork &w, const BandWork &band, size_t band_smem, cudaStream_t s)
{
    using S = LineShape<N>;
    constexpr int LPB = kLineThreads / S::L;
    const size_t smem = std::max(sizeof(double2) * S::SLOTS * LPB, band_smem);
    const int64_t blocks = ((w.nt[0] + 1) / 2 + LPB - 1) / LPB;
    return launch_chained(line_tiles_kernel<N>, (unsigned)(blocks + band.nboxes), kLineThreads, smem, s, w, band, (int)blocks);
}

// ---- the spectrum S^tau, in double-double arithmetic ----
//
// S(k)^tau by repeated squaring multiplies the relative error of S by tau, so plain FP64
// would lose log2(tau) bits where |S| is close to 1.  A double-double pair carries 106
// bits (sums by Knuth's and Dekker's error-free additions, products by a fused
// multiply-add's exact remainder); the roots come from the host in extended precision.

struct DD {
    double hi, lo;
};
__device__ __forceinline__ DD quick_two_sum(double a, double b)
{
    const double s = a + b;
    return {s, b - (s - a)};
}
__device__ __forceinline__ DD dd_add(DD a, DD b)
{
    const double s = a.hi + b.hi, v = s - a.hi;
    const double e = (a.hi - (s - v)) + (b.hi - v);
    return quick_two_sum(s, e + (a.lo + b.lo));
}
__device__ __forceinline__ DD dd_neg(DD a) { return {-a.hi, -a.lo}; }
__device__ __forceinline__ DD dd_mul(DD a, DD b)
{
    const double p = a.hi * b.hi;
    const double e = fma(a.hi, b.hi, -p) + (a.hi * b.lo + a.lo * b.hi);
    return quick_two_sum(p, e);
}
struct CDD {
    DD re, im;
};
__device__ __forceinline__ CDD cdd_mul(CDD a, CDD b)
{
    return {dd_add(dd_mul(a.re, b.re), dd_neg(dd_mul(a.im, b.im))), dd_add(dd_mul(a.re, b.im), dd_mul(a.im, b.re))};
}
__device__ __forceinline__ CDD cdd_add(CDD a, CDD b) { return {dd_add(a.re, b.re), dd_add(a.im, b.im)}; }

// roots[m] = exp(+2 pi i m / n) as {re.hi, re.lo}, {im.hi, im.lo}
__device__ __forceinline__ CDD root_of(const double2 *roots, int n, int d, int k)
{
    int m = (int)(((int64_t)d * k) % n);
    m += m < 0 ? n : 0;
    const double2 a = __ldg(roots + 2 * m), b = __ldg(roots + 2 * m + 1);
    return {{a.x, a.y}, {b.x, b.y}};
}

__global__ void __launch_bounds__(256) spectrum_kernel(const WideSpectrum p)
{
    const int H = p.tile[0] / 2 + kPad;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t line = i / H;
    const int kx = (int)(i - line * H);
    if (line >= p.tile[1])
        return;
    if (kx > p.tile[0] / 2) {
        p.out[i] = make_double2(0.0, 0.0);
        return;
    }
    const int ky = (int)line, r = p.r, ry = p.dim == 2 ? r : 0, K = 2 * r + 1;
    const DD z0 = {0.0, 0.0};
    CDD s = {z0, z0};
    for (int dy = -ry; dy <= ry; ++dy) {
        CDD row = {z0, z0};
        for (int dx = -r; dx <= r; ++dx) {
            const double w = __ldg(p.weights + (dy + ry) * K + (dx + r));
            if (w != 0.0) {
                const CDD e = root_of(p.roots[0], p.tile[0], dx, kx);
                const DD wd = {w, 0.0};
                row = cdd_add(row, {dd_mul(e.re, wd), dd_mul(e.im, wd)});
            }
        }
        s = cdd_add(s, p.dim == 2 ? cdd_mul(row, root_of(p.roots[1], p.tile[1], dy, ky)) : row);
    }
    CDD v = {{1.0, 0.0}, z0};
    for (int e = p.tau; e > 0; e >>= 1) {
        if (e & 1)
            v = cdd_mul(v, s);
        s = cdd_mul(s, s);
    }
    p.out[i] = make_double2(v.re.hi * p.scale, v.im.hi * p.scale); // scale: a power of two
}

template <int N>
cudaError_t prepare_one()
{
    const int rows = (int)sizeof(double2) * RowShape<N>::SLOTS * (kRowThreads / RowShape<N>::L);
    const int cols = (int)sizeof(double2) * ColShape<N>::SLOTS * col_count<N>();
    cudaError_t e = cudaFuncSetAttribute(rows_fwd_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, rows);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(rows_inv_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, rows);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(cols_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, cols);
    return e;
}

template <int N>
cudaError_t rows(const WideWork &w, bool inverse, cudaStream_t s)
{
    constexpr int LPB = kRowThreads / RowShape<N>::L;
    const size_t smem = sizeof(double2) * RowShape<N>::SLOTS * LPB;
    if (!inverse) {
        return launch_chained(rows_fwd_kernel<N>, (unsigned)((int64_t)w.ntiles * (w.tile[1] / 2) / LPB), kRowThreads, smem,
                              s, w);
    }
    const int pairs = ((int)w.useful[1] + 1) / 2;
    const int64_t blocks = (int64_t)w.ntiles * ((pairs + LPB - 1) / LPB);
    return launch_chained(rows_inv_kernel<N>, (unsigned)blocks, kRowThreads, smem, s, w);
}

template <int N>
cudaError_t cols(const WideWork &w, cudaStream_t s)
{
    constexpr int C = col_count<N>();
    const size_t smem = sizeof(double2) * ColShape<N>::SLOTS * C;
    return launch_chained(cols_kernel<N>, (unsigned)(w.ntiles * (w.tile[0] / 2 / C + 1)), col_threads(N), smem, s, w);
}

#define FFS_WIDE_BY_EDGE(edge, call)                                                                                \
    switch (edge) {                                                                                                 \
    case 256: { constexpr int N = 256; return call; }                                                               \
    case 512: { constexpr int N = 512; return call; }                                                               \
    case 1024: { constexpr int N = 1024; return call; }                                                             \
    case 2048: { constexpr int N = 2048; return call; }                                                             \
    default: return cudaErrorInvalidValue;                                                                          \
    }

cudaError_t rows_any(const WideWork &w, bool inverse, cudaStream_t s)
{
    FFS_WIDE_BY_EDGE(w.tile[0], (rows<N>(w, inverse, s)))
}
cudaError_t cols_any(const WideWork &w, cudaStream_t s)
{
    FFS_WIDE_BY_EDGE(w.tile[1], (cols<N>(w, s)))
}

constexpr size_t kLineSmemLimit = 200 * 1024; // (a band box may need more than the lines)

template <int N>
cudaError_t prepare_line()
{
    return cudaFuncSetAttribute(line_tiles_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLineSmemLimit);
}

} // namespace wide

cudaError_t launch_wide1(const WideWork &w, const BandWork &band, size_t band_smem, cudaStream_t s)
{
    switch (w.tile[0]) {
    case 1024: return wide::line_tiles<1024>(w, band, band_smem, s);
    case 2048: return wide::line_tiles<2048>(w, band, band_smem, s);
    case 4096: return wide::line_tiles<4096>(w, band, band_smem, s);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t prepare_wide()
{
    cudaError_t e = wide::prepare_line<1024>();
    if (e == cudaSuccess)
        e = wide::prepare_line<2048>();
    if (e == cudaSuccess)
        e = wide::prepare_line<4096>();
    if (e == cudaSuccess)
        e = wide::prepare_one<256>();
    if (e == cudaSuccess)
        e = wide::prepare_one<512>();
    if (e == cudaSuccess)
        e = wide::prepare_one<1024>();
    if (e == cudaSuccess)
        e = wide::prepare_one<2048>();
    return e;
}

cudaError_t launch_wide(const WideWork &w, int64_t tiles, int chunk, cudaStream_t s)
{
    for (int64_t t = 0; t < tiles; t += chunk) {
        WideWork c = w;
        c.tile0 = t;
        c.ntiles = (int)(tiles - t < chunk ? tiles - t : chunk);
        cudaError_t e = wide::rows_any(c, false, s);
        if (e == cudaSuccess)
            e = wide::cols_any(c, s);
        if (e == cudaSuccess)
            e = wide::rows_any(c, true, s);
        if (e != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}

int wide_points(int n, int axis) { return axis == 0 ? wide::row_points(n) : wide::col_points(n); }

size_t wide_tile_bytes(const int tile[2]) // workspace of one tile
{
    return sizeof(double2) * (size_t)(tile[0] + 2 * wide::kPad) * (tile[1] / 2);
}

size_t wide_spectrum_count(const int tile[2])
{
    return (size_t)(tile[0] / 2 + wide::kPad) * tile[1];
}

cudaError_t launch_wide_spectrum(const WideSpectrum &p, cudaStream_t s)
{
    const int64_t count = (int64_t)wide_spectrum_count(p.tile);
    wide::spectrum_kernel<<<(unsigned)((count + 255) / 256), 256, 0, s>>>(p);
    return cudaGetLastError();
}

} // namespace ffst

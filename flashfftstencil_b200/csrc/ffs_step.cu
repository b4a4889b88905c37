// Direct FP64 time stepping of 2-D regions by blocks that hold their tile in registers: many
// steps of a few cells.
//
// Where: the fixed boundary's frame of the wide tiles, deep bands of the one-SM tiles, and small grids
// stepped directly (300 x 260, T = 12: 14.4 -> 12.3 us), where a launch is bound by the length of its
// units.  The marching kernel (ffs_march.cu) has more useful cells per multiply-add on large grids, but
// its warps walk 2 r tau rows before their first output and leave most of the GPU idle on a strip: 8
// launches of 4 steps on the frame of 2048^2 took 170 us (a whole solve with this kernel 113).
//
// A block of kWarps warps holds a tile of 32 K columns x M kWarps rows: a lane K consecutive columns
// of the warp's M rows.  Per step a warp leaves its first and last r rows in shared memory (two
// buffers, one block barrier a step), reads its neighbours' r rows on either side, and goes down its
// rows once: each source row (with the lane's neighbour cells by shuffles) adds its taps to the up to
// 2r + 1 output rows it feeds, and a finished row replaces its source, which is no longer read.
// Tiles overlap by r steps per side (none at a fixed face: the ring holds there), warps whose rows
// no longer matter skip the arithmetic.  A cell's taps are summed in the tap list's order (dy, then
// dx).  The ring's cells keep their value by a select.
// Bound: the FP64 pipe within a step, the barrier and the shuffles' latency between steps.
#include <algorithm>

#include "ffs_chain.cuh"
#include "ffs_kernels.h"

namespace ffst {
namespace step {

constexpr int kWarps = 16;
constexpr int K = 2; // columns per lane: with 4 (128 x 64 tiles) a step of the frame took 1.4 times as long
constexpr int M = 4; // rows per warp
constexpr int W = 32 * K, kRows = M * kWarps;

// Tile i of n along one axis of a region: output cells [a, b), first cell of the tile.
struct Span {
    int a, b, org;
};
__device__ __forceinline__ Span span(int lo, int hi, bool wall_lo, int i, int n, int U, int H)
{
    const int first = wall_lo ? H : 0; // the first tile's extra cells at a fixed face
    Span s;
    s.a = i == 0 ? lo : lo + first + i * U;
    s.b = i == n - 1 ? hi : lo + first + (i + 1) * U;
    s.org = i == 0 && wall_lo ? lo : s.a - H;
    return s;
}

template <int R, bool STAR>
__global__ void __launch_bounds__(32 * kWarps, 1) step2d_kernel(const __grid_constant__ MarchWork p, int steps)
{
    constexpr int D = 2 * R + 1;
    extern __shared__ __align__(16) double edges[];
    auto edge = reinterpret_cast<double (*)[kWarps][2 * R][W]>(edges); // [step & 1][warp][first, last r rows]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    chain_wait();
    int u = blockIdx.x, k = 0;
    for (int i = 1; i < p.nregions; ++i)
        if (u >= p.reg[i].first_unit)
            k = i;
    const MarchRegion &g = p.reg[k];
    u -= g.first_unit;
    const int H = R * steps;
    const bool fixed = !p.periodic;
    const int ty = u / g.strips, tx = u - ty * g.strips;
    const Span sx = span(g.ox0, g.ox1, fixed && g.ox0 < p.rx0, tx, g.strips, W - 2 * H, H);
    const Span sy = span(g.oy0, g.oy1, fixed && g.oy0 < p.ry0, ty, g.chunk, kRows - 2 * H, H);
    const int x0 = sx.org + lane * K, y0 = sy.org + warp * M;

    double v[M][K];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        int y = y0 + m;
        bool in = true;
        if (fixed) {
            in = y >= g.sy0 && y < g.sy1;
        } else {
            y %= p.ny;
            y += y < 0 ? p.ny : 0;
        }
        const double *src = g.src + (int64_t)y * g.spitch;
#pragma unroll
        for (int i = 0; i < K; ++i) {
            int x = x0 + i;
            bool on = in;
            if (fixed) {
                on = in && x >= g.sx0 && x < g.sx1;
            } else {
                x %= p.nx;
                x += x < 0 ? p.nx : 0;
            }
            v[m][i] = on ? __ldg(src + x) : 0.0;
        }
    }
    double w[D * D];
#pragma unroll
    for (int i = 0; i < D * D; ++i)
        if (!STAR || i / D == R || i % D == R) {
            w[i] = p.w[i];
            if (R == 1 || STAR)
                asm volatile("" : "+d"(w[i])); // in registers, not fetched again at each use
        }
    bool ring_col[K], ring_row[M];
    bool any = false;
#pragma unroll
    for (int i = 0; i < K; ++i)
        any |= ring_col[i] = x0 + i < p.rx0 || x0 + i >= p.rx1;
#pragma unroll
    for (int m = 0; m < M; ++m)
        any |= ring_row[m] = y0 + m < p.ry0 || y0 + m >= p.ry1;
    const bool ring = fixed && __any_sync(0xffffffffu, any);

    for (int s = 0; s < steps; ++s) {
        double (*mine)[W] = edge[s & 1][warp];
#pragma unroll
        for (int j = 0; j < R; ++j)
#pragma unroll
            for (int i = 0; i < K; i += 2) {
                const int c = lane * K + i;
                *reinterpret_cast<double2 *>(&mine[j][c]) = make_double2(v[j][i], v[j][i + 1]);
                *reinterpret_cast<double2 *>(&mine[R + j][c]) = make_double2(v[M - R + j][i], v[M - R + j][i + 1]);
            }
        __syncthreads();
        // rows that still matter: within r (steps - 1 - s) of the tile's output
        const int reach = R * (steps - 1 - s);
        if (y0 + M <= sy.a - reach || y0 >= sy.b + reach)
            continue; // (the same for the whole warp; the barrier is above)
        // the tile's outermost warps have no neighbour on one side: any finite rows do there
        double (*above)[W] = edge[s & 1][warp > 0 ? warp - 1 : 0], (*below)[W] = edge[s & 1][warp < kWarps - 1 ? warp + 1 : warp];
        double acc[M][K];
#pragma unroll
        for (int j = -R; j < M + R; ++j) { // source row y0 + j
            double e[K + 2 * R];
#pragma unroll
            for (int i = 0; i < K; i += 2) {
                if (j >= 0 && j < M) {
                    e[R + i] = v[j < 0 || j >= M ? 0 : j][i];
                    e[R + i + 1] = v[j < 0 || j >= M ? 0 : j][i + 1];
                } else {
                    const double *row = j < 0 ? above[2 * R + j] : below[j - M];
                    const double2 d = *reinterpret_cast<const double2 *>(row + lane * K + i);
                    e[R + i] = d.x;
                    e[R + i + 1] = d.y;
                }
            }
            // a star's rows off the output row feed only the column itself, but every row of the
            // tile is some output's own row
            if (!STAR || (j >= 0 && j < M)) {
#pragma unroll
                for (int q = 0; q < R; ++q) {
                    e[q] = __shfl_up_sync(0xffffffffu, e[K + q], 1);
                    e[K + R + q] = __shfl_down_sync(0xffffffffu, e[R + q], 1);
                }
            }
#pragma unroll
            for (int dx = -R; dx <= R; ++dx)
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const int dy = j - m;
                    if (dy < -R || dy > R || (STAR && dx != 0 && dy != 0))
                        continue;
#pragma unroll
                    for (int i = 0; i < K; ++i) {
                        const double wt = w[(dy + R) * D + dx + R];
                        if (dy == -R && dx == (STAR ? 0 : -R))
                            acc[m][i] = wt * e[R + i + dx];
                        else
                            acc[m][i] = fma(wt, e[R + i + dx], acc[m][i]);
                    }
                }
            if (j - R >= 0) { // row j - R is finished; its source is not read again
                const int m = j - R;
#pragma unroll
                for (int i = 0; i < K; ++i)
                    v[m][i] = ring && (ring_row[m] || ring_col[i]) ? v[m][i] : acc[m][i];
            }
        }
    }
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const int y = y0 + m;
        if (y < sy.a || y >= sy.b)
            continue;
        double *dst = g.dst + (int64_t)y * g.dpitch;
#pragma unroll
        for (int i = 0; i < K; ++i)
            if (x0 + i >= sx.a && x0 + i < sx.b)
                dst[x0 + i] = v[m][i];
    }
}

template <int R, bool STAR>
cudaError_t launch(const MarchWork &w, int steps, cudaStream_t s)
{
    constexpr size_t smem = (size_t)2 * kWarps * 2 * R * W * sizeof(double);
    if (w.units <= 0) // set-up call
        return cudaFuncSetAttribute(step2d_kernel<R, STAR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return launch_chained(step2d_kernel<R, STAR>, (unsigned)w.units, 32 * kWarps, smem, s, w, steps);
}

cudaError_t dispatch(const MarchWork &w, int r, bool star, int steps, cudaStream_t s)
{
    if (r == 1)
        return star ? launch<1, true>(w, steps, s) : launch<1, false>(w, steps, s);
    if (r == 2)
        return star ? launch<2, true>(w, steps, s) : launch<2, false>(w, steps, s);
    return cudaErrorInvalidValue;
}

} // namespace step

cudaError_t prepare_step()
{
    const MarchWork none{};
    cudaError_t e = cudaSuccess;
    for (int r : {1, 2})
        for (bool star : {true, false})
            if (e == cudaSuccess)
                e = step::dispatch(none, r, star, 1, nullptr);
    return e;
}

int step_max_steps(int r) { return r == 1 ? 16 : r == 2 ? 8 : 0; } // half the tile's 64 cells are margin
int step_width(int r, int steps) { return step::W - 2 * r * steps; }

// Tiles of each region.
void step_tiles(MarchWork *w, int r, int steps)
{
    const int H = r * steps;
    auto count = [&](int lo, int hi, int stepped_lo, int stepped_hi, int edge) {
        const int walls = w->periodic ? 0 : (lo < stepped_lo) + (hi > stepped_hi);
        const int U = edge - 2 * H;
        return std::max(1, (hi - lo - walls * H + U - 1) / U);
    };
    w->units = 0;
    for (int i = 0; i < w->nregions; ++i) {
        MarchRegion &g = w->reg[i];
        g.strips = count(g.ox0, g.ox1, w->rx0, w->rx1, step::W);
        g.chunk = count(g.oy0, g.oy1, w->ry0, w->ry1, step::kRows);
        g.first_unit = w->units;
        w->units += g.strips * g.chunk;
    }
}

cudaError_t launch_step2d(const MarchWork &w, int r, bool star, int steps, cudaStream_t s)
{
    return w.units > 0 ? step::dispatch(w, r, star, steps, s) : cudaSuccess;
}

} // namespace ffst

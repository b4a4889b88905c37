// Direct FP64 time stepping of 2-D regions in registers: tau fused steps while a warp marches
// down the rows.
//
// Where: short runs (few steps between two uses of a grid), where tau (2r+1)^2 multiply-adds
// per cell cost less than two transforms (Star2D9P 1999 x 2047, T = 4: 64 x 64 tiles 82 us, this 34).
//
// A warp owns a strip of 32 K columns, K consecutive ones per lane, and reads the region's rows
// in order.  Level s (0-based) turns row y of step s into row y - r of step s + 1: row y adds its
// taps to the 2r pending output rows that a lane keeps in registers, completes the oldest and
// opens a new one, and the completed row goes straight to level s + 1.  So a row is read once
// and written once for tau steps, with no block barrier: per level the only traffic is the 2r
// neighbour cells of a lane's chunk, by shuffles.  A cell's taps are summed in the tap list's
// order (dy, then dx).
// Cells within r tau of a strip's side or of a chunk's first and last row are recomputed by the
// neighbours: U = 32 K - 2 r tau columns and all rows of the chunk are written.
// Registers bound tau: 2 r K accumulators per level, 64 doubles in all (tau 8 at r = 1, 4 at r = 2;
// 2 for the 25 taps of a dense r = 2, which are registers too).
// Rows come by cp.async into a per-warp ring of kRing rows in shared memory, kAhead rows early,
// and leave through one more row of it, so that global accesses are to consecutive cells while a
// lane holds K of them (loading and storing a lane's own K cells directly wrote quarter sectors).
// The ring also holds the fixed ring's values: its cells keep their initial value, and row
// y - r (s + 1) was read at most r tau rows ago.
// Bound: the FP64 pipe ((2r+1)^2 FMA per cell-step; 4 shuffles per K cells beside them).
// No counterpart in the reference, whose tile kernel is its only stepper.
#include <algorithm>
#include <type_traits>

#include "ffs_chain.cuh"
#include "ffs_kernels.h"

namespace ffst {
namespace march {

constexpr int kWarps = 4; // per block
constexpr int K = 4;      // columns per lane
constexpr int W = 32 * K; // columns of a strip
constexpr int kRing = 16; // rows kept: r tau (at most 8) behind, kAhead before the current one
constexpr int kAhead = 4;
constexpr int kRowBytes = W * (int)sizeof(double);

// Position of cell c in a staged row: 16-byte pairs of cells, their index XORed so that the 8
// lanes of a quarter warp, 2 pairs apart, hit distinct bank groups.
__device__ __forceinline__ int staged(int c)
{
    const int q = c >> 1;
    return ((q ^ ((q >> 3) & 1)) << 1) | (c & 1);
}

// n = 8: copies one cell; 0: fills with zero
__device__ __forceinline__ void copy8_async(uint32_t dst, const double *src, int n)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

// Blocks per SM: 3 where the kernel fits 168 registers a thread without spilling (spilling a
// few of them to do so cost 1.6 times the time of tau = 4 with a fixed boundary).
constexpr int blocks_per_sm(int r, bool star, bool fixed, int tau)
{
    return r == 1 ? (tau <= (fixed ? 3 : 4) ? 3 : 2) : (tau <= (fixed || !star ? 1 : 2) && (star || !fixed) ? 3 : 2);
}

template <int R, bool STAR, bool FIXED, int TAU>
__global__ void __launch_bounds__(32 * kWarps, blocks_per_sm(R, STAR, FIXED, TAU)) march2d_kernel(const __grid_constant__ MarchWork p)
{
    extern __shared__ __align__(16) double stage[];
    chain_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int u = blockIdx.x * kWarps + warp;
    if (u >= p.units)
        return;
    int k = 0;
#pragma unroll
    for (int i = 1; i < kMarchRegions; ++i)
        if (i < p.nregions && u >= p.reg[i].first_unit)
            k = i;
    const MarchRegion &g = p.reg[k];
    u -= g.first_unit;
    const int chunk = u / g.strips, strip = u - chunk * g.strips;
    constexpr int H = R * TAU, U = W - 2 * H;
    const int xw = g.ox0 + strip * U - H; // the strip's first staged column
    const int ya = g.oy0 + chunk * g.chunk, yb = min(ya + g.chunk, g.oy1);
    double *ring = stage + warp * (kRing + 1) * W, *outrow = ring + kRing * W;
    const uint32_t ring_s = (uint32_t)__cvta_generic_to_shared(ring);
    const int xs = xw + lane * K; // this lane's first column in registers
    // staging: the lane copies columns xw + lane + 32 i, from offset off in a row of src, `bytes`
    // each (0: outside src, reads as zero)
    int off[K], bytes[K];
    uint32_t put[K];
    bool keep[K]; // columns to write
#pragma unroll
    for (int i = 0; i < K; ++i) {
        const int c = lane + 32 * i, x = xw + c;
        put[i] = ring_s + (uint32_t)(staged(c) * sizeof(double));
        keep[i] = c >= H && c < H + U && x < g.ox1;
        if constexpr (FIXED) {
            bytes[i] = x >= g.sx0 && x < g.sx1 ? 8 : 0;
            off[i] = max(g.sx0, min(x, g.sx1 - 1));
        } else {
            const int m = x % p.nx;
            bytes[i] = 8;
            off[i] = m < 0 ? m + p.nx : m;
        }
    }
    bool ring_col[K];
#pragma unroll
    for (int i = 0; i < K; ++i)
        ring_col[i] = xs + i < p.rx0 || xs + i >= p.rx1;

    // the taps stay in registers: as kernel parameters each use fetched them again
    constexpr int D = 2 * R + 1;
    double w[D * D];
#pragma unroll
    for (int i = 0; i < D * D; ++i)
        if (!STAR || i / D == R || i % D == R) {
            w[i] = p.w[i];
            asm volatile("" : "+d"(w[i]));
        }

    // Level s keeps D rows of K cells: 2r pending output rows and the row it completes.  At row
    // y0 + ph (mod D) the pending row y - R + j is in slot (ph + j) % D: the row loop is unrolled
    // D times, so that rows change roles without register moves (those, 2 per double, were a
    // quarter of the instructions).
    double acc[TAU][D][K];
#pragma unroll
    for (int s = 0; s < TAU; ++s)
#pragma unroll
        for (int j = 0; j < D; ++j)
#pragma unroll
            for (int i = 0; i < K; ++i)
                acc[s][j][i] = 0.0;

    const int y0 = FIXED ? max(ya - H, g.sy0) : ya - H;
    int row = y0; // the row of src that fetch() copies next
    if constexpr (!FIXED) {
        row %= p.ny;
        row += row < 0 ? p.ny : 0;
    }
    auto fetch = [&](int y) { // y: the row in the region's coordinates
        const double *src = g.src + (int64_t)row * g.spitch;
        const uint32_t slot = (uint32_t)((y & (kRing - 1)) * kRowBytes);
        const bool in = !FIXED || y < g.sy1;
#pragma unroll
        for (int i = 0; i < K; ++i)
            copy8_async(put[i] + slot, src + off[i], in ? bytes[i] : 0);
        asm volatile("cp.async.commit_group;" ::: "memory");
        if constexpr (FIXED) {
            row = min(row + 1, g.sy1 - 1); // rows below src read as zero
        } else {
            row = row + 1 == p.ny ? 0 : row + 1;
        }
    };
    auto held = [&](int y, double (&v)[K]) { // the lane's cells of staged row y
        const double *r = ring + (y & (kRing - 1)) * W;
#pragma unroll
        for (int i = 0; i < K; i += 2) {
            const double2 d = *reinterpret_cast<const double2 *>(r + staged(lane * K + i));
            v[i] = d.x;
            v[i + 1] = d.y;
        }
    };
    const int end = yb + H;
    auto step_row = [&](int y, auto phase, auto at_ring) {
        constexpr int PH = decltype(phase)::value;
        constexpr bool RING = decltype(at_ring)::value;
        asm volatile("cp.async.wait_group %0;" ::"n"(kAhead - 1) : "memory");
        __syncwarp(); // row y is staged; row y + kAhead - kRing is no longer read
        fetch(y + kAhead);
        double v[K];
        held(y, v);
#pragma unroll
        for (int s = 0; s < TAU; ++s) {
            // the row with R neighbours on either side
            double e[K + 2 * R];
#pragma unroll
            for (int j = 0; j < R; ++j) {
                e[j] = __shfl_up_sync(0xffffffffu, v[K - R + j], 1);
                e[K + R + j] = __shfl_down_sync(0xffffffffu, v[j], 1);
            }
#pragma unroll
            for (int i = 0; i < K; ++i)
                e[R + i] = v[i];
            // the pending rows y - r .. y + r - 1 and the new row y + r take the row's taps dy = r ..
            // -r; tap by tap over all of them, so that consecutive multiply-adds are independent
#pragma unroll
            for (int dx = -R; dx <= R; ++dx)
#pragma unroll
                for (int j = 0; j < D; ++j)
                    if (!STAR || dx == 0 || j == R)
#pragma unroll
                        for (int i = 0; i < K; ++i) {
                            double &t = acc[s][(PH + j) % D][i];
                            const double wt = w[(2 * R - j) * D + dx + R];
                            if (j == 2 * R && dx == (STAR ? 0 : -R))
                                t = wt * e[R + i + dx];
                            else
                                t = fma(wt, e[R + i + dx], t);
                        }
            double (&done)[K] = acc[s][PH % D];
            if constexpr (RING) {
                const int yo = y - R * (s + 1); // the completed row
                const bool ring_row = yo < p.ry0 || yo >= p.ry1;
                double o[K];
                held(yo, o); // (before y0: a row that nothing written depends on)
#pragma unroll
                for (int i = 0; i < K; ++i)
                    done[i] = ring_row || ring_col[i] ? o[i] : done[i];
            }
#pragma unroll
            for (int i = 0; i < K; ++i)
                v[i] = done[i];
        }
        const int yo = y - H;
        if (yo >= ya && yo < yb) {
#pragma unroll
            for (int i = 0; i < K; i += 2)
                *reinterpret_cast<double2 *>(outrow + staged(lane * K + i)) = make_double2(v[i], v[i + 1]);
            __syncwarp();
            double *dst = g.dst + (int64_t)yo * g.dpitch + xw + lane;
#pragma unroll
            for (int i = 0; i < K; ++i)
                if (keep[i])
                    dst[32 * i] = outrow[staged(lane + 32 * i)];
        } // (the next row's __syncwarp comes before outrow is written again)
    };

#pragma unroll
    for (int i = 0; i < kAhead; ++i)
        fetch(y0 + i);
    auto step_rows = [&](int y, auto at_ring) {
        step_row(y, std::integral_constant<int, 0>(), at_ring);
        step_row(y + 1, std::integral_constant<int, 1>(), at_ring);
        step_row(y + 2, std::integral_constant<int, 2>(), at_ring);
        if constexpr (D > 3) {
            step_row(y + 3, std::integral_constant<int, 3>(), at_ring);
            step_row(y + 4, std::integral_constant<int, 4>(), at_ring);
        }
    };
    // the ring's cells cost every level, so rows and strips away from it run without (the same
    // for the whole warp)
    const bool ring_cols = xw < p.rx0 || xw + W > p.rx1;
    for (int y = y0; y < end; y += D) { // up to D - 1 rows past the end, which write nothing
        if (FIXED && (ring_cols || y - H < p.ry0 || y + D - 1 - R >= p.ry1))
            step_rows(y, std::true_type());
        else
            step_rows(y, std::false_type());
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

constexpr size_t kSmemBytes = (size_t)kWarps * (kRing + 1) * kRowBytes;

template <int R, bool STAR, int TAU>
cudaError_t launch(const MarchWork &w, cudaStream_t s)
{
    const int blocks = (w.units + kWarps - 1) / kWarps;
    return w.periodic ? launch_chained(march2d_kernel<R, STAR, false, TAU>, blocks, 32 * kWarps, kSmemBytes, s, w)
                      : launch_chained(march2d_kernel<R, STAR, true, TAU>, blocks, 32 * kWarps, kSmemBytes, s, w);
}

// Most steps of one launch: 2 r K accumulators per level beside the taps.
template <int R, bool STAR>
constexpr int max_tau() { return R == 1 ? 8 : (STAR ? 4 : 2); }

template <int R, bool STAR, int TAU = max_tau<R, STAR>()>
cudaError_t by_tau(const MarchWork &w, int tau, cudaStream_t s)
{
    if (tau == TAU)
        return launch<R, STAR, TAU>(w, s);
    if constexpr (TAU > 1)
        return by_tau<R, STAR, TAU - 1>(w, tau, s);
    return cudaErrorInvalidValue;
}

template <int R, bool STAR, int TAU = max_tau<R, STAR>()>
cudaError_t prepare_up_to()
{
    cudaError_t e = cudaFuncSetAttribute(march2d_kernel<R, STAR, false, TAU>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(march2d_kernel<R, STAR, true, TAU>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kSmemBytes);
    if constexpr (TAU > 1)
        if (e == cudaSuccess)
            e = prepare_up_to<R, STAR, TAU - 1>();
    return e;
}

} // namespace march

cudaError_t prepare_march()
{
    cudaError_t e = march::prepare_up_to<1, true>();
    if (e == cudaSuccess)
        e = march::prepare_up_to<1, false>();
    if (e == cudaSuccess)
        e = march::prepare_up_to<2, true>();
    if (e == cudaSuccess)
        e = march::prepare_up_to<2, false>();
    return e;
}

int march_max_tau(int r, bool star)
{
    return r == 1 ? march::max_tau<1, true>() : r == 2 ? (star ? march::max_tau<2, true>() : march::max_tau<2, false>()) : 0;
}
int march_warps(int r, bool star, bool fixed, int tau) { return march::kWarps * march::blocks_per_sm(r, star, fixed, tau); }
int march_width(int r, int tau) { return march::W - 2 * r * tau; }

// Splits a region's output (one region: with a fixed boundary it becomes up to three) into strips and row
// chunks, one unit for every resident warp (each unit re-reads 2 r tau rows of its neighbours, so chunks are as long as that allows).  With a
// fixed boundary the strips at the ring are regions of their own with shorter chunks: their
// rows take about 1.5 times as long, and the launch ends with its longest unit.
void march_units(MarchWork *w, int r, bool star, int tau, int num_sms)
{
    const int U = march_width(r, tau);
    MarchRegion all[kMarchRegions];
    int n = 0;
    for (int i = 0; i < w->nregions; ++i) {
        const MarchRegion g = w->reg[i];
        const int strips = (g.ox1 - g.ox0 + U - 1) / U;
        if (w->periodic || strips < 3) {
            all[n++] = g;
            continue;
        }
        const int cut[4] = {g.ox0, g.ox0 + U, g.ox0 + (strips - 1) * U, g.ox1};
        for (int k = 0; k < 3; ++k) {
            all[n] = g;
            all[n].ox0 = cut[k];
            all[n++].ox1 = cut[k + 1];
        }
    }
    double area = 0; // rows of strips, weighted
    for (int i = 0; i < n; ++i) {
        all[i].strips = (all[i].ox1 - all[i].ox0 + U - 1) / U;
        const bool ring = !w->periodic && (all[i].ox0 - r * tau < w->rx0 || all[i].ox1 + U > w->rx1);
        all[i].first_unit = ring;
        area += (double)all[i].strips * (all[i].oy1 - all[i].oy0) * (ring ? 1.5 : 1.0);
    }
    // rows per unit for the resident warps: as few as leave no unit for a second wave (22 strips of 61 rows are 1188
    // units of 3279 rows for 1184 warps: Heat-2D 2394 x 3279, periodic, tau 8 73 us a pass)
    constexpr int kLeastRows = 8; // (a launch of few rows is bound by its units' length: on the
                                  // frame of 1500 x 1300 at tau 4, 8 / 16 rows took 80 / 148 us in all)
    const int slots = num_sms * march_warps(r, star, !w->periodic, tau);
    w->nregions = n;
    auto split = [&](double rows) { // fills the regions, returns the units
        int units = 0;
        for (int i = 0; i < n; ++i) {
            MarchRegion &g = w->reg[i] = all[i];
            const int total = g.oy1 - g.oy0;
            const int chunk = std::max((int)(all[i].first_unit ? rows / 1.5 : rows) + 1, kLeastRows);
            const int parts = (total + chunk - 1) / chunk;
            g.chunk = (total + parts - 1) / parts;
            g.first_unit = units;
            units += g.strips * ((total + g.chunk - 1) / g.chunk);
        }
        return units;
    };
    double rows = area / (double)slots;
    w->units = split(rows);
    for (int k = 0; k < 8 && w->units > slots && rows >= kLeastRows; ++k)
        w->units = split(rows *= 1.01);
}

cudaError_t launch_march2d(const MarchWork &w, int r, bool star, int tau, cudaStream_t s)
{
    if (w.units <= 0)
        return cudaSuccess;
    if (r == 1)
        return star ? march::by_tau<1, true>(w, tau, s) : march::by_tau<1, false>(w, tau, s);
    if (r == 2)
        return star ? march::by_tau<2, true>(w, tau, s) : march::by_tau<2, false>(w, tau, s);
    return cudaErrorInvalidValue;
}

} // namespace ffst

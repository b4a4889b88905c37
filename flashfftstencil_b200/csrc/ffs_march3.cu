// Direct FP64 time stepping of 3-D grids (radius 1), one step per launch: a block marches through the
// z planes.
//
// Where: most 3-D runs.  The 16^3 tile's transforms keep (12 / 16)^3 = 0.42 of their points at two
// fused steps: Box3D27P 512^3 takes 768 us a step that way, Heat-3D 740; one direct step 460 to 510 (the
// more solves in a row, the longer) and 396 to 420 (HBM alone: 323).
//
// A block of 256 threads owns a 64 x 32 tile of a plane, a thread one column of kRows rows.  Planes (the
// tile and one cell around it) come by cp.async into a ring in shared memory, kAhead planes early.  A
// source plane is read once per thread, 3 (kRows + 2) values, and each feeds the up to nine outputs it
// belongs to in the three pending planes that the thread keeps in registers; the oldest is finished and
// written out.  Pending planes change roles by unrolling the plane loop three times.  A cell's taps are
// summed in the tap list's order (dz, dy, dx).
// The fixed ring's cells keep their value by a select from the source plane's centre.
// Bound: HBM (16 bytes a cell) with few taps; with 27 the FP64 pipe and issue (counters at 256^3: pipe 48 %,
// issue 58 %, HBM 56 % of the copy rate, no dominant stall).  Two steps a launch, the second level's source through shared memory,
// took as long per step (Heat-3D 401, Box3D27P 570 us at 512^3): HBM traffic halves, but the margins, a
// second barrier per plane and spills at 128 registers take it back.
#include <cmath>
#include <type_traits>

#include "ffs_chain.cuh"
#include "ffs_kernels.h"

namespace ffst {
namespace march3 {

constexpr int NT = 256;
constexpr int kAhead = 3;
constexpr int kSlots = kAhead + 2; // and the plane being read, and the one before it (the ring's values)

// A block's tile of a plane: X cells wide, ROWS rows per thread.
template <int X, int ROWS>
struct Tile {
    static constexpr int TX = X, TY = ROWS * (NT / X), kRows = ROWS;
    static constexpr int PX = TX + 2, PY = TY + 2, kPlane = PX * PY; // a staged plane
    static constexpr size_t kSmemBytes = sizeof(double) * kPlane * kSlots;
};
using Large = Tile<64, 8>; // 64 x 32
using Small = Tile<32, 4>; // 32 x 32
static_assert(2 * Large::kSmemBytes <= 226 * 1024, "two blocks per SM");

__device__ __forceinline__ void copy8_async(uint32_t dst, const double *src, int n)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

__device__ __forceinline__ int wrap(int x, int n)
{
    x %= n;
    return x < 0 ? x + n : x;
}

// Adds source plane z (at `plane`, the thread's first cell) to the pending planes z - 1, z and z + 1 in
// slots PH, PH + 1 and PH + 2 (mod 3).
template <bool STAR, int PH, int PX, int kRows>
__device__ __forceinline__ void add_plane(const double *plane, const double (&w)[27], double (&acc)[3][kRows])
{
#pragma unroll
    for (int j = -1; j <= kRows; ++j) {
        double e[3];
        const double *row = plane + j * PX;
        e[1] = row[0];
        if (!STAR || (j >= 0 && j < kRows)) {
            e[0] = row[-1];
            e[2] = row[1];
        }
#pragma unroll
        for (int m = 0; m < kRows; ++m) {
            const int dy = j - m;
            if (dy < -1 || dy > 1)
                continue;
#pragma unroll
            for (int p = 0; p < 3; ++p) { // pending plane z - 1 + p: dz = 1 - p
                const int dz = 1 - p;
                double &a = acc[(PH + p) % 3][m];
#pragma unroll
                for (int dx = -1; dx <= 1; ++dx) {
                    if (STAR && (dx != 0) + (dy != 0) + (dz != 0) > 1)
                        continue;
                    const double wt = w[(dz + 1) * 9 + (dy + 1) * 3 + dx + 1];
                    // the first tap of the plane that opens
                    if (p == 2 && (STAR || (dy == -1 && dx == -1)))
                        a = wt * e[dx + 1];
                    else
                        a = fma(wt, e[dx + 1], a);
                }
            }
        }
    }
}

template <class T, bool STAR, bool FIXED>
__global__ void __launch_bounds__(NT, 2) march3d_kernel(const __grid_constant__ March3Work p)
{
    constexpr int TX = T::TX, TY = T::TY, kRows = T::kRows, PX = T::PX, PY = T::PY, kPlane = T::kPlane;
    extern __shared__ __align__(16) double smem[];
    chain_wait();
    int u = blockIdx.x;
    const int chunk = u / (p.tiles[0] * p.tiles[1]);
    u -= chunk * p.tiles[0] * p.tiles[1];
    const int ty = u / p.tiles[0], tx = u - ty * p.tiles[0];
    const int x0 = tx * TX, y0 = ty * TY;                                       // the tile's first cell
    const int za = chunk * p.chunk, zb = min(za + p.chunk, p.n[2]);             // planes to write
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cx = threadIdx.x & (TX - 1), cy = (threadIdx.x / TX) * kRows; // the thread's cells in the tile
    const int nx = p.n[0];
    const int64_t plane_cells = (int64_t)nx * p.n[1];

    // staging: rows warp, warp + 8 .. of the plane, columns lane, lane + 32, lane + 64 (< PX): their
    // offsets in a plane (the same for every plane; computing them per plane was a third of the
    // instructions; one offset per cell instead of a row's and a column's spilled) and which of
    // them are inside the grid (the others read as zero)
    constexpr int RP = (PY + NT / 32 - 1) / (NT / 32); // rows per warp
    int row_off[RP], col_off[3];
    unsigned live = 0; // bit j: row j, bit 8 + i: column i
#pragma unroll
    for (int j = 0; j < RP; ++j) {
        const int y = y0 - 1 + warp + NT / 32 * j;
        row_off[j] = (FIXED ? max(0, min(y, p.n[1] - 1)) : wrap(y, p.n[1])) * nx;
        live |= (y >= 0 && y < p.n[1] ? 1u : 0u) << j;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int x = x0 - 1 + lane + 32 * i;
        col_off[i] = FIXED ? max(0, min(x, nx - 1)) : wrap(x, nx);
        live |= (x >= 0 && x < nx ? 1u : 0u) << (8 + i);
    }
    const uint32_t smem_s = (uint32_t)__cvta_generic_to_shared(smem + warp * PX + lane);
    // fetch() copies plane fz next, into slot fslot
    int fz = FIXED ? za - 1 : wrap(za - 1, p.n[2]), fslot = 0;
    const double *src = p.in + max(0, fz) * plane_cells;
    auto fetch = [&]() {
        const unsigned on = !FIXED || (fz >= 0 && fz < p.n[2]) ? live : 0;
        const uint32_t dst = smem_s + (uint32_t)(fslot * kPlane * sizeof(double));
#pragma unroll
        for (int j = 0; j < RP; ++j) {
            if (warp + NT / 32 * j >= PY)
                continue;
#pragma unroll
            for (int i = 0; i < 3; ++i)
                if (lane + 32 * i < PX)
                    copy8_async(dst + (uint32_t)((NT / 32 * j * PX + 32 * i) * sizeof(double)), src + (row_off[j] + col_off[i]),
                                !FIXED || (on >> j & on >> (8 + i) & 1) ? 8 : 0);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        ++fz;
        if (!FIXED && fz == p.n[2]) {
            fz = 0;
            src = p.in;
        } else if (fz > 0 && (!FIXED || fz < p.n[2])) { // (planes outside read as zero, from any address)
            src += plane_cells;
        }
        fslot = fslot + 1 == kSlots ? 0 : fslot + 1;
    };

    double w[27];
#pragma unroll
    for (int i = 0; i < 27; ++i)
        if (!STAR || (i / 9 != 1) + (i / 3 % 3 != 1) + (i % 3 != 1) <= 1) {
            w[i] = p.w[i];
            asm volatile("" : "+d"(w[i])); // in registers, not fetched again at each use
        }
    double acc[3][kRows];
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int m = 0; m < kRows; ++m)
            acc[j][m] = 0.0;
    const int gx = x0 + cx, gy = y0 + cy;
    // rows of the thread's column: held by the ring in every plane, and to write
    unsigned held = 0, keep = 0;
#pragma unroll
    for (int m = 0; m < kRows; ++m) {
        if (gx < p.slo[0] || gx >= p.shi[0] || gy + m < p.slo[1] || gy + m >= p.shi[1])
            held |= 1u << m;
        if (gx < nx && gy + m < p.n[1])
            keep |= 1u << m;
    }
    const bool ring_tile = x0 < p.slo[0] || x0 + TX > p.shi[0] || y0 < p.slo[1] || y0 + TY > p.shi[1];
    const int at = (cy + 1) * PX + cx + 1; // the thread's first cell in a staged plane
    double *dst = p.out + za * plane_cells + (int64_t)gy * nx + gx;
    int slot = 0; // of source plane z

    auto step_plane = [&](int z, auto phase) {
        constexpr int PH = decltype(phase)::value;
        asm volatile("cp.async.wait_group %0;" ::"n"(kAhead - 1) : "memory");
        __syncthreads(); // plane z is staged; plane z - 2 is no longer read
        fetch();
        add_plane<STAR, PH, PX>(smem + slot * kPlane + at, w, acc);
        double (&done)[kRows] = acc[PH % 3]; // plane z - 1
        const int zo = z - 1;
        if (zo >= za && zo < zb) {
            if (FIXED && (ring_tile || zo < p.slo[2] || zo >= p.shi[2])) {
                const double *before = smem + (slot == 0 ? kSlots - 1 : slot - 1) * kPlane + at; // plane zo
                const unsigned hold = zo < p.slo[2] || zo >= p.shi[2] ? ~0u : held;
#pragma unroll
                for (int m = 0; m < kRows; ++m)
                    if (keep >> m & 1)
                        dst[m * nx] = hold >> m & 1 ? before[m * PX] : done[m];
            } else {
#pragma unroll
                for (int m = 0; m < kRows; ++m)
                    if (keep >> m & 1)
                        dst[m * nx] = done[m];
            }
            dst += plane_cells;
        }
        slot = slot + 1 == kSlots ? 0 : slot + 1;
    };
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
        fetch();
    for (int z = za - 1; z <= zb; z += 3) { // up to two planes past the end, which write nothing
        step_plane(z, std::integral_constant<int, 0>());
        step_plane(z + 1, std::integral_constant<int, 1>());
        step_plane(z + 2, std::integral_constant<int, 2>());
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

template <class T, bool STAR, bool FIXED>
cudaError_t launch(const March3Work &w, cudaStream_t s)
{
    if (w.units <= 0) // set-up call
        return cudaFuncSetAttribute(march3d_kernel<T, STAR, FIXED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)T::kSmemBytes);
    return launch_chained(march3d_kernel<T, STAR, FIXED>, (unsigned)w.units, NT, T::kSmemBytes, s, w);
}

template <class T>
cudaError_t by_boundary(const March3Work &w, bool star, cudaStream_t s)
{
    if (w.periodic)
        return star ? launch<T, true, false>(w, s) : launch<T, false, false>(w, s);
    return star ? launch<T, true, true>(w, s) : launch<T, false, true>(w, s);
}

cudaError_t dispatch(const March3Work &w, bool star, cudaStream_t s)
{
    return w.small ? by_boundary<Small>(w, star, s) : by_boundary<Large>(w, star, s);
}

// A plane of an SM's two blocks, and per tap (one block per SM takes about half: Heat-3D 100 x 90 x 70 in
// 144 units of 6 planes 5.8 us a step, in 288 of 3 planes 7.8; but Box3D27P 512^3 in 128 units 667, in 1152
// 453).  Measured, us a step,
// Large / Small: Heat-3D 65 x 33 x 9 4.8 / 3.4, 100 x 90 x 70 6.2 / 5.8, 236 x 144 x 99 15.0 / 15.6, 256^3 57 / 60;
// Box3D27P 100 x 90 x 70 7.5 / 7.1, 256^3 60 / 64; Large at 512^3, fixed, 413 and 453 (a first solve; up to 420 and 510 in a row).
constexpr double kMarch3PlaneSeconds = 1.5e-6, kMarch3TapSeconds = 0.012e-6;
constexpr double kMarch3SmallPlaneSeconds = 0.85e-6, kMarch3SmallTapSeconds = 0.007e-6;
constexpr double kMarch3LaunchSeconds = 2e-6;

} // namespace march3


cudaError_t prepare_march3()
{
    March3Work w{};
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < 8; ++k) {
        w.periodic = k & 1;
        w.small = k >> 1 & 1;
        if (e == cudaSuccess)
            e = march3::dispatch(w, k & 4, nullptr);
    }
    return e;
}

// Tile, and z chunks: the choice whose waves (two blocks per SM) take least; a chunk steps two planes
// beside its own and starts up in about the time of two more.  Returns the modelled seconds.
double march3_units(March3Work *w, int taps, int num_sms)
{
    double best = 1e300;
    const March3Work in = *w;
    for (bool small : {false, true}) {
        const int tx = small ? march3::Small::TX : march3::Large::TX, ty = small ? march3::Small::TY : march3::Large::TY;
        const int x = (in.n[0] + tx - 1) / tx, y = (in.n[1] + ty - 1) / ty;
        using namespace march3;
        // a plane of an SM's two blocks, and of one block alone
        const double fixed = in.periodic ? 1.0 : 1.15, base = small ? kMarch3SmallPlaneSeconds : kMarch3PlaneSeconds,
                     tap = (small ? kMarch3SmallTapSeconds : kMarch3TapSeconds) * taps;
        const double two = fixed * (base + tap),
                     one = (in.periodic ? 0.8 : 1.1) * (0.5 * base + 1.2 * tap);
        for (int n = 1; n <= in.n[2] && n <= 4096; ++n) {
            const int len = (in.n[2] + n - 1) / n;
            if ((in.n[2] + len - 1) / len != n)
                continue;
            const int64_t units = (int64_t)x * y * n;
            const double cost = std::ceil((double)units / (2.0 * num_sms)) * (len + 4) * (units <= num_sms ? one : two);
            if (units < INT32_MAX && cost < best) {
                best = cost;
                w->small = small;
                w->tiles[0] = x;
                w->tiles[1] = y;
                w->chunk = len;
                w->units = (int)units;
            }
        }
    }
    return best + march3::kMarch3LaunchSeconds;
}

cudaError_t launch_march3d(const March3Work &w, bool star, cudaStream_t s)
{
    return w.units > 0 ? march3::dispatch(w, star, s) : cudaSuccess;
}

} // namespace ffst

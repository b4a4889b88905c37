// Direct FP64 time stepping of 1-D grids: a warp holds a piece of the line in registers and steps it
// many times.
//
// Where: short runs, and lines of up to some 10^5 cells.  A tile's launch takes 14 us (4096 cells in
// shared memory) or 10.6 (ffs_wide.cu) however few cells there are; a step here is one exchange between
// neighbouring lanes and (2r+1) multiply-adds per cell: 10000 cells, radius 2, T = 16 14.4 -> 7.8 us,
// 2.5 M cells, T = 3 37.3 -> 12.7.
//
// A warp owns 32 K consecutive cells, K per lane, of which the outer r steps on either side are margin
// (none at a fixed face, where the ring holds).  Per step a lane gets the r cells beyond each end of its
// chunk by shuffles.  Cells come and go through shared memory, so that global accesses are to
// consecutive cells; position c + c / K there puts a half warp's lanes, K cells apart, on distinct
// banks.  A cell's taps are summed in the tap list's order.
// Bound: HBM for few steps, the FP64 pipe for many, the chain of a step's shuffles and multiply-adds on
// short lines.  K = 8 has twice the warps, K = 16 half the margin: long runs take 16.
#include <type_traits>

#include "ffs_chain.cuh"
#include "ffs_kernels.h"

namespace ffst {
namespace line {

constexpr int kWarps = 4; // per block

template <int R, int K>
__global__ void __launch_bounds__(32 * kWarps) line_kernel(const __grid_constant__ LineWork p)
{
    constexpr int W = 32 * K, PITCH = W + 32;
    __shared__ double stage[kWarps][PITCH];
    chain_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t u = (int64_t)blockIdx.x * kWarps + warp;
    if (u >= p.units)
        return;
    const int H = R * p.steps, U = W - 2 * H;
    const int64_t a = u * U, org = a - H; // cells [a, a + U) are written
    double *s = stage[warp];
#pragma unroll
    for (int i = 0; i < K; ++i) {
        const int c = lane + 32 * i;
        int64_t x = org + c;
        bool in = true;
        if (p.periodic) {
            if (x < 0 || x >= p.n) {
                x %= p.n;
                x += x < 0 ? p.n : 0;
            }
        } else {
            in = x >= 0 && x < p.n;
        }
        s[c + c / K] = in ? __ldg(p.in + x) : 0.0;
    }
    __syncwarp();
    double v[K], w[2 * R + 1];
#pragma unroll
    for (int i = 0; i < K; ++i)
        v[i] = s[lane * (K + 1) + i];
#pragma unroll
    for (int i = 0; i < 2 * R + 1; ++i)
        w[i] = p.w[i];
    const int64_t x0 = org + lane * K;
    unsigned hold = 0; // cells of the fixed ring
#pragma unroll
    for (int i = 0; i < K; ++i)
        if (x0 + i < p.slo || x0 + i >= p.shi)
            hold |= 1u << i;
    const bool ring = !p.periodic && __any_sync(0xffffffffu, hold != 0);
    auto steps = [&](auto at_ring) {
        constexpr bool RING = decltype(at_ring)::value;
        for (int t = 0; t < p.steps; ++t) {
            double e[K + 2 * R], nv[K];
#pragma unroll
            for (int j = 0; j < R; ++j) {
                e[j] = __shfl_up_sync(0xffffffffu, v[K - R + j], 1);
                e[K + R + j] = __shfl_down_sync(0xffffffffu, v[j], 1);
            }
#pragma unroll
            for (int i = 0; i < K; ++i)
                e[R + i] = v[i];
#pragma unroll
            for (int d = 0; d < 2 * R + 1; ++d)
#pragma unroll
                for (int i = 0; i < K; ++i)
                    nv[i] = d == 0 ? w[0] * e[i] : fma(w[d], e[i + d], nv[i]);
#pragma unroll
            for (int i = 0; i < K; ++i)
                v[i] = RING && (hold >> i & 1) ? v[i] : nv[i];
        }
    };
    if (ring)
        steps(std::true_type());
    else
        steps(std::false_type());
    __syncwarp();
#pragma unroll
    for (int i = 0; i < K; ++i)
        s[lane * (K + 1) + i] = v[i];
    __syncwarp();
#pragma unroll
    for (int i = 0; i < K; ++i) {
        const int c = lane + 32 * i;
        if (c >= H && c < H + U && org + c < p.n)
            p.out[org + c] = s[c + c / K];
    }
}

// Loads the kernels: otherwise their first launch does.
template <int R>
cudaError_t load()
{
    cudaFuncAttributes a;
    const cudaError_t e = cudaFuncGetAttributes(&a, line_kernel<R, 8>);
    return e != cudaSuccess ? e : cudaFuncGetAttributes(&a, line_kernel<R, 16>);
}

template <int R>
cudaError_t launch(const LineWork &w, int k, cudaStream_t s)
{
    const unsigned blocks = (unsigned)((w.units + kWarps - 1) / kWarps);
    return k == 8 ? launch_chained(line_kernel<R, 8>, blocks, 32 * kWarps, 0, s, w)
                  : launch_chained(line_kernel<R, 16>, blocks, 32 * kWarps, 0, s, w);
}

} // namespace line

// The first line of a process took 490 to 710 us with the kernels loaded in it, 100 with this.
cudaError_t prepare_line()
{
    for (cudaError_t e : {line::load<1>(), line::load<2>(), line::load<3>(), line::load<4>()})
        if (e != cudaSuccess)
            return e;
    return cudaSuccess;
}

int line_max_steps(int r, int k) { return r >= 1 && r <= 4 ? (32 * k - 64) / 2 / r : 0; } // 64 cells written at least

cudaError_t launch_line(LineWork w, int r, int k, cudaStream_t s)
{
    const int U = 32 * k - 2 * r * w.steps;
    w.units = (w.n + U - 1) / U;
    switch (r) {
    case 1: return line::launch<1>(w, k, s);
    case 2: return line::launch<2>(w, k, s);
    case 3: return line::launch<3>(w, k, s);
    case 4: return line::launch<4>(w, k, s);
    default: return cudaErrorInvalidValue;
    }
}

} // namespace ffst

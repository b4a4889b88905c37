// Host-side launch interface of the sm_100a kernels (internal to libffs.so).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace ffst {

// Codes a kernel writes into the plan's device status word.
enum DeviceError : int {
    kDevOk = 0,
    kDevTimeoutTma = 1,
    kDevTimeoutMma = 2,
    kDevBadConfig = 3,
    kDevTimeoutDep = 4,
};

// Tile-pair work description shared by the fused DFT-tile kernels.  Tiles of
// edge n overlap by `halo` cells per side; each produces a u = n - 2*halo edge of
// outputs.  Two tiles adjacent along x are packed as the real and imaginary
// parts of one complex tile (the reference's "two real tiles per complex tile",
// src/2D/rfft_2d/2d_rfft_1_async.cu:73-92).
struct TileWork {
    const double *in;
    double *out;
    const double2 *spec;   // spectrum^tau / n^d, in the kernel's frequency-position order
    const double2 *tables; // DFT-8 roots (8) then n-th roots of unity (n or n^2 for 1D)
    int *status;           // device error word (0 = ok)
    int64_t nx, ny, nz;
    int halo, useful;
    int64_t t0[3];   // first tile index per dim (x, y, z)
    int64_t nt[3];   // tiles per dim in the range (x, y, z)
    int64_t npx;     // tile pairs along x = ceil(nt[0] / 2)
    int64_t nitems;  // npx * nt[1] * nt[2]
    int64_t vlo[3], vhi[3]; // store window per dim (spectrally exact cells)
    int periodic;
    int use_tma;
};

cudaError_t prepare_dmma2d(); // sets the shared-memory attribute on the current device
cudaError_t launch_dmma2d(const CUtensorMap *tmap, const TileWork &w, int grid, cudaStream_t s);
size_t dmma2d_smem_bytes();
int dmma2d_tile();

// 2D FP64 radix-8 butterfly form (same tile geometry and spectrum layout as tc2d).
cudaError_t prepare_fft2d();
cudaError_t launch_fft2d(const CUtensorMap *tmap, const TileWork &w, int grid, cudaStream_t s);
size_t fft2d_smem_bytes();

// 3D FP64 butterfly form (two CTAs per SM; `grid` is the SM count bound).
cudaError_t prepare_fft3d();
cudaError_t launch_fft3d(const TileWork &w, int grid, cudaStream_t s);
int64_t fft3d_grid(int64_t nitems, int num_sms); // the CTA count launch_fft3d uses
size_t fft3d_smem_bytes();
// 2D FP64 butterfly form on one 128 x 128 real tile per CTA (single tiles, not pairs).
cudaError_t prepare_fft2d128();
cudaError_t launch_fft2d128(const TileWork &w, int grid, cudaStream_t s);
size_t fft2d128_smem_bytes();
// 3D FP64 butterfly form on a 32^3 tile held by a cluster of four CTAs (one per SM).
cudaError_t prepare_fft3d32();
cudaError_t launch_fft3d32(const TileWork &w, int num_sms, cudaStream_t s);
size_t fft3d32_smem_bytes();

// FP64 butterfly form on wide tiles (256 .. 2048 cells per axis): three kernels per chunk of
// tiles over a workspace (ffs_wide.cu).  Tile i covers grid cells from org + (i per axis) *
// useful; its useful cells start `halo` cells in and are stored below vhi.
struct WideWork {
    const double *in;
    double *out;
    double2 *work;        // `chunk` tiles of packed rows
    const double2 *spec;  // S^tau / (2 Nx Ny), [ky][kx], kx padded to Nx / 2 + 16 (1-D: S^tau / N)
    const double2 *tw[2]; // per axis, P points a thread: w_N^(m k1), then w_(N/P)^(m2 k2)
    int64_t n[2], org[2], useful[2], vhi[2], nt[2];
    int64_t tile0;        // first tile of the chunk
    int ntiles;           // tiles of the chunk
    int tile[2], halo[2];
    int periodic;
};
struct WideSpectrum {
    double2 *out;
    const double *weights;
    const double2 *roots[2]; // exp(+2 pi i m / n) per axis, {re hi, re lo}, {im hi, im lo}
    int dim, r, tau;
    int tile[2];
    double scale;
};
int wide_points(int n, int axis); // points per thread of a line of n (axis 0: rows, else columns)
cudaError_t prepare_wide();
cudaError_t launch_wide(const WideWork &w, int64_t tiles, int chunk, cudaStream_t s);
size_t wide_tile_bytes(const int tile[2]);
size_t wide_spectrum_count(const int tile[2]);
cudaError_t launch_wide_spectrum(const WideSpectrum &p, cudaStream_t s);

// 1D FP64 butterfly form (four-step DFT-4096 of radix-8 lines).
cudaError_t prepare_fft1d();
cudaError_t launch_fft1d(const TileWork &w, int grid, cudaStream_t s);
size_t fft1d_smem_bytes();

cudaError_t prepare_dmma1d();
cudaError_t launch_dmma1d(const TileWork &w, int grid, cudaStream_t s);
size_t dmma1d_smem_bytes();
int dmma1d_tile();

cudaError_t prepare_dmma3d();
cudaError_t launch_dmma3d(const CUtensorMap *tmap, const TileWork &w, int grid, cudaStream_t s);
size_t dmma3d_smem_bytes();
int dmma3d_tile();

// tcgen05 2D and 3D forms (Ozaki INT8 slices / 3-way BF16 split).
constexpr int kFormOzaki = 2;
constexpr int kFormBf16 = 3;
cudaError_t prepare_tc2d();
cudaError_t launch_tc2d(int form, int slices, const TileWork &w, const unsigned char *a_slices, int grid,
                        cudaStream_t s);
size_t tc2d_smem_bytes(int form, int slices);
cudaError_t prepare_tc3d();
cudaError_t launch_tc3d(int form, int slices, const TileWork &w, const unsigned char *f_slices, int grid,
                        cudaStream_t s);
size_t tc3d_smem_bytes(int form, int slices);

// Direct FP64 time stepping of boxes near a fixed boundary.
struct BandBox {
    int64_t lo[3]; // box origin (x, y, z)
    int32_t ext[3]; // box extents
};
struct BandWork {
    const double *in;
    double *out;
    const double *weights; // dense (2r+1)^dim, device
    const BandBox *boxes;
    int nboxes;
    int dim, r, tau;
    int64_t n[3];
    int64_t max_vol;       // largest staged region (box + halo) over all boxes, in cells
    const int4 *taps;      // non-zero taps: {dx, dy, dz, index into weights}
    int ntaps;
    int *status;
    int warp_rows;         // 2-D 3 x 3 box: most staged widths are multiples of 32, step by warp rows
};
// 1-D wide tiles (pairs of 1024 .. 4096 cells) and the fixed boundary's boxes in one launch.
cudaError_t launch_wide1(const WideWork &w, const BandWork &band, size_t band_smem, cudaStream_t s);
cudaError_t prepare_band(size_t max_smem);

// Direct stepping of 2-D regions in registers (ffs_march.cu).  Coordinates are the grid's:
// src and dst are offset so that src[y * spitch + x] is cell (x, y).
struct MarchRegion {
    const double *src;
    double *dst;
    int64_t spitch, dpitch;
    int sx0, sx1, sy0, sy1; // readable cells of src (fixed boundary)
    int ox0, ox1, oy0, oy1; // cells to write
    int strips, chunk, first_unit; // set by march_units
};
constexpr int kMarchRegions = 4;
struct MarchWork {
    MarchRegion reg[kMarchRegions];
    double w[25]; // dense (2r+1)^2 taps
    int nregions, units;
    int nx, ny, periodic;
    int rx0, rx1, ry0, ry1; // cells that are stepped (fixed boundary); the others keep their value
};
cudaError_t prepare_march();
int march_max_tau(int r, bool star); // most steps of one launch, 0: radius not supported
int march_warps(int r, bool star, bool fixed, int tau); // resident warps per SM
int march_width(int r, int tau);     // columns a warp writes
void march_units(MarchWork *w, int r, bool star, int tau, int num_sms);
cudaError_t launch_march2d(const MarchWork &w, int r, bool star, int tau, cudaStream_t s);

// The same regions stepped by blocks that hold a 64 x 64 tile in registers (ffs_step.cu): for
// regions that do not fill the GPU.
cudaError_t prepare_step();
int step_max_steps(int r);          // most steps of one launch, 0: radius not supported
int step_width(int r, int steps);   // cells of a tile's edge that it writes
void step_tiles(MarchWork *w, int r, int steps);
cudaError_t launch_step2d(const MarchWork &w, int r, bool star, int steps, cudaStream_t s);

// One direct step of a 3-D grid, radius 1 (ffs_march3.cu).
struct March3Work {
    const double *in;
    double *out;
    double w[27];
    int n[3], periodic;
    int slo[3], shi[3];         // cells that are stepped (fixed boundary); the others keep their value
    int small, tiles[2], chunk, units; // set by march3_units
};
cudaError_t prepare_march3();
double march3_units(March3Work *w, int taps, int num_sms); // the modelled seconds
cudaError_t launch_march3d(const March3Work &w, bool star, cudaStream_t s);

// `steps` direct steps of a 1-D grid, radius 1 .. 4 (ffs_line.cu), k = 8 or 16 cells per lane.
struct LineWork {
    const double *in;
    double *out;
    double w[9];
    int64_t n, units; // units: set by launch_line
    int64_t slo, shi; // cells that are stepped (fixed boundary); the others keep their value
    int steps, periodic;
};
cudaError_t prepare_line();
int line_max_steps(int r, int k);
cudaError_t launch_line(LineWork w, int r, int k, cudaStream_t s);

// Autotuner utilities: a seeded uniform [0, 1) fill, and out[0] = max |y - r|,
// out[1] = max |r| as ordered bit patterns (out zeroed by the caller).
cudaError_t launch_fill_uniform(double *d, size_t n, uint64_t seed, cudaStream_t s);
cudaError_t launch_max_diff(const double *y, const double *r, size_t n, unsigned long long *out, cudaStream_t s);
cudaError_t launch_band(const BandWork &w, size_t smem_bytes, cudaStream_t s);
size_t band_smem_bytes(int64_t max_vol, int ntaps);

// One (problem, pass) of a batch: its tile work and band boxes, plus the stage
// of the same problem's previous pass that must finish first.
struct BatchStage {
    TileWork tw;
    BandWork bw;
    int dim;
    int dep;           // index of the previous pass's stage, -1 for the first pass
    int64_t dep_count; // items of that stage
};
size_t batch_tile_smem_bytes();
cudaError_t prepare_batch(size_t max_smem);
// Polls (128 ns apart) a batch item waits for its problem's previous pass before it
// records kDevTimeoutDep and goes on: seconds, far above any real wait.
constexpr uint32_t kDepSpinLimit = 1u << 24;
cudaError_t launch_batch(const BatchStage *stages, const int64_t *start, int nstages, int64_t total, int *done,
                         unsigned long long *head, int *status, uint32_t dep_limit, size_t smem, int grid,
                         cudaStream_t s);

} // namespace ffst

// Host-only plan builder.  Replaces the reference's CreatePlan
// (src/1D/create_fft_pfa_plan.cu:19-228, src/2D/create_fft_pfa_plan.cu:17-147,
// src/3D/create_fft_pfa_plan.cu:17-139), which builds DFT-8 matrices with
// cos/sin and the kernel spectrum with cuFFT and uploads both to __constant__.
// Here everything is FP64 host arithmetic: the spectrum is a direct DFT of the
// (2r+1)^d taps (no cuFFT), raised to the fused step count by repeated
// squaring in extended precision, divided by n^d, and permuted into the order in
// which the tile kernel holds its frequencies.
#include "ffs_plan.h"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

namespace ffst {

namespace {

const ShapeDef kShapes[] = {
    {"Heat-1D", FFS_SHAPE_HEAT_1D, 1, 1, "1d1r"},       {"1D5P", FFS_SHAPE_1D5P, 1, 2, "1d2r"},
    {"1D7P", FFS_SHAPE_1D7P, 1, 3, "1d3r"},             {"Heat-2D", FFS_SHAPE_HEAT_2D, 2, 1, "star_2d1r"},
    {"Box2D9P", FFS_SHAPE_BOX2D9P, 2, 1, "box_2d1r"},   {"Star2D9P", FFS_SHAPE_STAR2D9P, 2, 2, "star_2d2r"},
    {"Box2D25P", FFS_SHAPE_BOX2D25P, 2, 2, "box_2d2r"}, {"Heat-3D", FFS_SHAPE_HEAT_3D, 3, 1, "star_3d1r"},
    {"Box3D27P", FFS_SHAPE_BOX3D27P, 3, 1, "box_3d1r"},
};

bool iequals(const char *a, const char *b)
{
    for (; *a && *b; ++a, ++b)
        if (tolower((unsigned char)*a) != tolower((unsigned char)*b))
            return false;
    return *a == *b;
}

struct CLD { // extended-precision complex for spectrum powers
    long double re, im;
};
inline CLD mul(CLD a, CLD b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
CLD cpow(CLD z, int e)
{
    CLD r{1.0L, 0.0L};
    while (e > 0) {
        if (e & 1)
            r = mul(r, z);
        z = mul(z, z);
        e >>= 1;
    }
    return r;
}

// exp(-2 pi i m / n) for m in [0, n), computed in long double.
std::vector<CLD> roots(int n)
{
    std::vector<CLD> r(n);
    const long double two_pi = 6.283185307179586476925286766559L;
    for (int m = 0; m < n; ++m) {
        long double a = two_pi * (long double)m / (long double)n;
        r[m] = {cosl(a), -sinl(a)};
    }
    return r;
}

int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Symbol of the correlation stencil at integer frequency k (per dim) on an n^d
// grid: S(k) = sum_d w[d] exp(+2 pi i d.k / n).
CLD symbol(const PlanSpec &sp, const std::vector<CLD> &rt, int n, const int k[3])
{
    const int r = sp.radius, K = 2 * r + 1;
    const int ry = sp.dim >= 2 ? r : 0, rz = sp.dim >= 3 ? r : 0, Ky = 2 * ry + 1;
    CLD s{0.0L, 0.0L};
    for (int dz = -rz; dz <= rz; ++dz)
        for (int dy = -ry; dy <= ry; ++dy)
            for (int dx = -r; dx <= r; ++dx) {
                const double w = sp.weights[((dz + rz) * Ky + (dy + ry)) * K + (dx + r)];
                if (w == 0.0)
                    continue;
                // exp(+2 pi i m / n) = conj(root[m]) = root[(-m) mod n]
                int64_t m = (int64_t)dx * k[0] + (int64_t)dy * k[1] + (int64_t)dz * k[2];
                m = ((-m) % n + n) % n;
                s.re += (long double)w * rt[m].re;
                s.im += (long double)w * rt[m].im;
            }
    return s;
}

// ---- per-form tile geometry ----
int tile_edge(int dim, ffs_form form)
{
    (void)form;
    switch (dim) {
    case 1:
        return 4096;
    case 2:
        return 64;
    default:
        return 16;
    }
}

// Second tile edge of the FP64 butterfly form: 128 x 128 (one real tile per CTA) in 2D,
// 32^3 (a four-CTA cluster per pair) in 3D; 0 for the forms with one edge.
int alt_tile_edge(int dim, ffs_form form)
{
    if (form != FFS_FORM_FP64_FFT)
        return 0;
    return dim == 2 ? 128 : (dim == 3 ? 32 : 0);
}

int round_even(int v) { return (v + 1) & ~1; }

// Geometry of one pass kind with fusion depth tau.
void geometry(const PlanSpec &sp, int tau, PassSpec *ps)
{
    const int n = sp.tile;
    ps->tau = tau;
    ps->halo = round_even(sp.radius * tau);
    ps->useful = n - 2 * ps->halo;
    const int64_t rt = (int64_t)sp.radius * tau;
    for (int d = 0; d < 3; ++d) {
        if (d >= sp.dim) {
            ps->vlo[d] = 0;
            ps->vhi[d] = 1;
            ps->t0[d] = 0;
            ps->nt[d] = 1;
            continue;
        }
        if (sp.boundary == FFS_BOUNDARY_PERIODIC) {
            ps->vlo[d] = 0;
            ps->vhi[d] = sp.n[d];
        } else { // cells within r*tau of a fixed face go to the band; an open face has none
            ps->vlo[d] = (sp.open_faces >> (2 * d) & 1) ? 0 : std::min<int64_t>(rt, sp.n[d]);
            ps->vhi[d] = (sp.open_faces >> (2 * d + 1) & 1) ? sp.n[d]
                                                             : std::max<int64_t>(sp.n[d] - rt, ps->vlo[d]);
        }
        ps->t0[d] = ps->vlo[d] / ps->useful;
        const int64_t t1 = ceil_div(ps->vhi[d], ps->useful);
        ps->nt[d] = std::max<int64_t>(0, t1 - ps->t0[d]);
    }
    bool empty = false;
    for (int d = 0; d < sp.dim; ++d)
        empty |= ps->vhi[d] <= ps->vlo[d];
    if (empty) {
        ps->npx = 0;
        ps->nitems = 0;
    } else {
        // tile pairs along x (re / im of one complex tile), except the 2D 128 x 128 kernel,
        // which packs row pairs of one real tile instead
        ps->npx = (sp.dim == 2 && sp.tile == 128) ? ps->nt[0] : ceil_div(ps->nt[0], 2);
        ps->nitems = ps->npx * ps->nt[1] * ps->nt[2];
    }
}

// Fixed-boundary band: every cell outside the exact window, partitioned into
// slabs (cell goes to the highest dim in which it is in the band) and boxes
// small enough that box + r*tau halo fits the band kernel's shared memory.
struct BandSlab {
    int64_t lo[3], hi[3], chunk[3];
};
std::vector<BandSlab> band_slabs(const PlanSpec &sp, const PassSpec &ps)
{
    std::vector<BandSlab> slabs;
    if (sp.boundary != FFS_BOUNDARY_FIXED || ps.tau == 0)
        return slabs;
    const int64_t rt = (int64_t)sp.radius * ps.tau;
    const size_t tap_bytes = sp.taps.size() * (sizeof(int4) + sizeof(double)) + 64;
    const int64_t vol_limit = (int64_t)((kBandSmemLimit - tap_bytes) / (2 * sizeof(double)));
    for (int d = sp.dim - 1; d >= 0; --d) {
        for (int side = 0; side < 2; ++side) {
            int64_t lo[3], hi[3];
            for (int e = 0; e < 3; ++e) {
                if (e >= sp.dim) {
                    lo[e] = 0;
                    hi[e] = 1;
                } else if (e > d) {
                    lo[e] = ps.vlo[e];
                    hi[e] = ps.vhi[e];
                } else if (e < d) {
                    lo[e] = 0;
                    hi[e] = sp.n[e];
                } else if (side == 0) {
                    lo[e] = 0;
                    hi[e] = ps.vlo[e];
                } else {
                    lo[e] = ps.vhi[e];
                    hi[e] = sp.n[e];
                }
            }
            bool empty = false;
            for (int e = 0; e < 3; ++e)
                empty |= hi[e] <= lo[e];
            if (empty)
                continue;
            int64_t chunk[3];
            for (int e = 0; e < 3; ++e)
                chunk[e] = hi[e] - lo[e];
            auto staged_bound = [&]() {
                int64_t v = 1;
                for (int e = 0; e < sp.dim; ++e)
                    v *= std::min<int64_t>(chunk[e] + 2 * rt, sp.n[e]);
                return v;
            };
            // cap the long dims of a box: the band kernel runs beside the tile kernel, and its
            // CTAs hold SMs the tile CTAs then start late on.  2D: 32 (Box2D9P 4096^2, caps
            // 16 / 32 / 64 / 256 -> 826 / 849 / 831 / 657 GStencil/s; with the band launched
            // after the 128 x 128 tile kernel, caps 24 / 32 / 48 / 64 -> 955 / 990 / 918 / 918,
            // and Box2D9P 8192^2 1117 / 1124 / 1110 / 1110; on grids below 2^24 cells
            // the 512-problem mixed batch took 204.0 / 210.9 / 207.1 at 16 / 32 / 64 with the 3D
            // cap at 16).  3D: 64 on grids of 2^24 cells and more (Box3D27P 512^3, caps 16 / 64
            // -> 149.5 / 151.9), 32 below (the batch: 217.0 against 210.9 at 16, 2D cap 32).
            const bool big = sp.cells >= (size_t)1 << 24;
            const int64_t long_cap = sp.dim == 1 ? (int64_t)1 << 30 : (sp.dim == 2 ? 32 : (big ? 64 : 32));
            for (int e = 0; e < sp.dim; ++e)
                if (e != d)
                    chunk[e] = std::min(chunk[e], long_cap);
            while (staged_bound() > vol_limit) {
                int big = -1;
                for (int e = 0; e < sp.dim; ++e)
                    if (chunk[e] > 1 && (big < 0 || chunk[e] > chunk[big]))
                        big = e;
                if (big < 0)
                    break;
                chunk[big] = (chunk[big] + 1) / 2;
            }
            BandSlab b;
            for (int e = 0; e < 3; ++e) {
                b.lo[e] = lo[e];
                b.hi[e] = hi[e];
                b.chunk[e] = chunk[e];
            }
            slabs.push_back(b);
        }
    }
    return slabs;
}

// Largest staged region of the band's boxes: per slab the product of each axis' longest staged run
// (the boxes are all combinations of the axes' segments).
int64_t band_max_volume(const PlanSpec &sp, const PassSpec &ps, const std::vector<BandSlab> &slabs)
{
    const int64_t rt = (int64_t)sp.radius * ps.tau;
    int64_t most = 0;
    for (const BandSlab &b : slabs) {
        int64_t vol = 1;
        for (int e = 0; e < sp.dim; ++e) {
            int64_t run = 0;
            for (int64_t o = b.lo[e]; o < b.hi[e]; o += b.chunk[e]) {
                const int64_t end = std::min(o + b.chunk[e], b.hi[e]);
                run = std::max(run, std::min<int64_t>(end + rt, sp.n[e]) - std::max<int64_t>(o - rt, 0));
            }
            vol *= run;
        }
        most = std::max(most, vol);
    }
    return most;
}

void band_boxes(const PlanSpec &sp, PassSpec *ps)
{
    ps->boxes.clear();
    const std::vector<BandSlab> slabs = band_slabs(sp, *ps);
    ps->band_max_vol = band_max_volume(sp, *ps, slabs);
    for (const BandSlab &b : slabs)
        for (int64_t z = b.lo[2]; z < b.hi[2]; z += b.chunk[2])
            for (int64_t y = b.lo[1]; y < b.hi[1]; y += b.chunk[1])
                for (int64_t x = b.lo[0]; x < b.hi[0]; x += b.chunk[0]) {
                    BandBox box;
                    const int64_t o[3] = {x, y, z};
                    for (int e = 0; e < 3; ++e) {
                        box.lo[e] = o[e];
                        box.ext[e] = (int32_t)std::min<int64_t>(b.chunk[e], b.hi[e] - o[e]);
                    }
                    ps->boxes.push_back(box);
                }
}

// One 32^3 complex tile pair on a four-SM cluster (FP64 butterflies), measured: 27-33 us
// per pair on Box3D27P 512^3 (2.97 ms for 3610 pairs at tau 2, 5.25 ms for 5324 at tau 4),
// with 33 clusters resident on 148 SMs.  The pair holds ten times the butterfly work of a
// 16^3 pair, but a CTA of 32-point lines runs 8 warps per SM against 24.
constexpr double kTile32PairSeconds = 30e-6;
constexpr double kTile32ClustersPerSm = 33.0 / 148.0;

// One 128 x 128 real tile on one SM (FP64 butterflies), measured: 20 us (Box2D9P 4096^2,
// tau 16: 0.251-0.257 ms for 1849 tiles, 12.5 per SM), against 5.8 us for a 64 x 64 pair.
constexpr double kTile128Seconds = 20e-6;

// Modelled seconds of a pass's band.  Boxes run concurrently, several per SM; a box costs its
// direct stepping work plus a per-step barrier latency.  Along an axis a slab's boxes have at most
// two extents (the chunk and a remainder), so the sum needs no list of boxes: a 512^3 shell at
// large tau has millions, and the models of all step counts took seconds.
double band_cost(const PlanSpec &sp, const PassSpec &ps, int num_sms)
{
    double box_max = 0.0, box_sum = 0.0;
    for (const BandSlab &b : band_slabs(sp, ps)) {
        double count[3][2] = {{1, 0}, {1, 0}, {1, 0}}, size[3][2] = {{1, 1}, {1, 1}, {1, 1}};
        for (int e = 0; e < sp.dim; ++e) {
            const int64_t len = b.hi[e] - b.lo[e], rem = len % b.chunk[e];
            count[e][0] = (double)(len / b.chunk[e]);
            count[e][1] = rem ? 1.0 : 0.0;
            size[e][0] = std::min<double>((double)b.chunk[e] + 2.0 * sp.radius * ps.tau, (double)sp.n[e]);
            size[e][1] = std::min<double>((double)rem + 2.0 * sp.radius * ps.tau, (double)sp.n[e]);
        }
        for (int k = 0; k < 8; ++k) {
            const int i = k & 1, j = k >> 1 & 1, l = k >> 2;
            const double boxes = count[0][i] * count[1][j] * count[2][l];
            if (boxes == 0.0)
                continue;
            const double v = size[0][i] * size[1][j] * size[2][l];
            const double bt = v * ps.tau * (double)sp.taps.size() / 60e9 + ps.tau * 0.3e-6;
            box_max = std::max(box_max, bt);
            box_sum += boxes * bt;
        }
    }
    return box_sum == 0.0 ? 0.0 : std::max(box_max, box_sum / (num_sms * 4.0)) + 3e-6;
}

// Model of one pass in seconds (used to pick tau).  Rough per-form constants;
// the tile cost is the measured order of one tile pair per SM.
double pass_cost(const PlanSpec &sp, const PassSpec &ps, int num_sms)
{
    double tile_pair_s = 12e-6; // one 64x64 (2D) or 4096 (1D) complex tile pair on one SM (FP64 DMMA)
    if (sp.dim == 3)
        tile_pair_s = 10e-6;
    if (sp.form == FFS_FORM_OZAKI_I8)
        tile_pair_s = 4e-6 * sp.slices;
    else if (sp.form == FFS_FORM_FP64_FFT)
        tile_pair_s = sp.dim == 3 ? 3e-6 : (sp.dim == 2 ? 5.7e-6 : 6e-6); // 2D: 0.142 ms for 3698 pairs, 25 per SM
    else if (sp.form == FFS_FORM_BF16X3)
        tile_pair_s = 6e-6;
    // the 32^3 tile: one pair per four-SM cluster at a time
    const bool cluster = sp.dim == 3 && sp.tile == 32;
    if (cluster)
        tile_pair_s = kTile32PairSeconds;
    if (sp.dim == 2 && sp.tile == 128)
        tile_pair_s = kTile128Seconds;
    const double waves = std::ceil((double)ps.nitems / (cluster ? std::floor(kTile32ClustersPerSm * num_sms) : num_sms));
    return waves * tile_pair_s + band_cost(sp, ps, num_sms) + 4e-6;
}

int max_tau(const PlanSpec &sp)
{
    const int n = sp.tile;
    const int r = sp.radius;
    int tau_max = sp.T;
    if (r > 0)
        tau_max = std::min(tau_max, (n - 8) / 2 / r); // keep u >= 8
    tau_max = std::max(tau_max, 1);
    if (r > 0) // halo is rounded up to even: make sure u stays >= 8
        while (tau_max > 1 && n - 2 * round_even(r * tau_max) < 8)
            --tau_max;
    return tau_max;
}

// Whether the tile has cells left between the halos of tau steps (a 16^3 tile has none at radius 7
// and 8; the geometry divides by their number).
bool tile_holds(const PlanSpec &sp, int tau) { return sp.tile > 2 * round_even(sp.radius * tau); }

double model_cost(const PlanSpec &sp, int tau)
{
    if (!tile_holds(sp, tau))
        return INFINITY;
    PassSpec ps;
    geometry(sp, tau, &ps);
    const int passes = (sp.T + tau - 1) / tau;
    return passes * pass_cost(sp, ps, 148);
}

void pick_tau(PlanSpec *sp, int tau_override)
{
    const int n = sp->tile;
    const int r = sp->radius;
    int tau_max = sp->T;
    if (r > 0)
        tau_max = std::min(tau_max, (n - 8) / 2 / r); // keep u >= 8
    tau_max = std::max(tau_max, 1);
    if (r > 0) // halo is rounded up to even: make sure u stays >= 8
        while (tau_max > 1 && n - 2 * round_even(r * tau_max) < 8)
            --tau_max;
    int best = tau_override > 0 ? std::min(tau_override, tau_max) : 0;
    if (!best) { // a measured choice for this problem class wins over the model
        const int tuned = tune_lookup(tune_key(*sp));
        if (tuned > 0 && tuned <= tau_max)
            best = tuned;
    }
    if (!best) {
        double best_cost = 1e300;
        best = 1; // (of an edge too small for the radius, which the caller refuses)
        for (int tau = 1; tau <= tau_max; ++tau) {
            const double c = model_cost(*sp, tau);
            if (c < best_cost * (1 - 1e-9)) {
                best_cost = c;
                best = tau;
            }
        }
    }
    sp->tau = best;
    sp->passes = (sp->T + best - 1) / best;
    sp->tau_last = sp->T - (sp->passes - 1) * best;
}

// Tile edge of the 3D butterfly form: the autotuner's measured choice for the problem
// class when it has one, else the edge whose best modelled solve is shorter.
int pick_tile(const PlanSpec &sp, int tau_override)
{
    const int tuned = tune_lookup(tile_key(sp));
    const int edges[2] = {tile_edge(sp.dim, sp.form), alt_tile_edge(sp.dim, sp.form)};
    const int tuned_ok = tuned == edges[0] || tuned == edges[1];
    if (tuned_ok)
        return tuned;
    int best = edges[0];
    double best_cost = 1e300;
    for (int tile : edges) {
        PlanSpec t = sp;
        t.tile = tile;
        pick_tau(&t, tau_override);
        const double c = model_cost(t, t.tau);
        if (c < best_cost * (1 - 1e-9)) {
            best_cost = c;
            best = tile;
        }
    }
    return best;
}

// ---- direct stepping ----

constexpr double kMarchLaunchSeconds = 5e-6; // launch, first rows
constexpr double kMarchBytesPerSecond = 5e12, kMarchCachedBytesPerSecond = 7e12;
// 1-D: launch and copies; a step of a warp alone; multiply-adds with every SM busy
constexpr double kLineLaunchSeconds = 6e-6, kLineStepSeconds = 0.04e-6, kLineCellSeconds = 1.5e-9;
constexpr double kLineChainSeconds = 1.5e-6; // what a pass behind another does not wait for
constexpr double kLineFmaPerSecond = 9e12;

// The marching kernel by radius, taps and boundary: seconds of a cell's step with every SM busy, margins counted, and of
// one level of one row for a warp alone (300 x 260).  The first from 1500 x 1300 and 4130 x 5900, us, measured / model:
// Heat-2D, periodic, tau 6 19.3 / 19.4 and 108 / 106, fixed, tau 4 17.5 / 16.9 and 108 / 103; Box2D9P, fixed, tau 4 21.7 /
// 21.5 and 140 / 140; Star2D9P, fixed, tau 3 24.3 / 24.1 and 129 / 139; 25 taps, fixed, tau 2 25.8 / 25.2 and 158 / 167.
struct MarchRate {
    double cell, row;
};
MarchRate march_rate(int r, bool star, bool fixed, int tau)
{
    if (r == 1)
        return star ? (fixed ? MarchRate{0.88e-12, 0.09e-6} : MarchRate{0.6e-12, 0.05e-6})
                    : (fixed ? MarchRate{1.22e-12, 0.115e-6} : MarchRate{0.9e-12, 0.07e-6});
    if (star)
        return fixed ? MarchRate{tau == 4 ? 1.95e-12 : 1.6e-12, 0.195e-6} : MarchRate{1.15e-12, 0.13e-6};
    return fixed ? MarchRate{tau == 1 ? 3.7e-12 : 3e-12, 0.33e-6} : MarchRate{2.5e-12, 0.21e-6};
}

// Modelled seconds of `tau` fused steps of one nx x ny region.
double march_cost(const PlanSpec &sp, double nx, double ny, int tau)
{
    const int r = sp.radius;
    const bool fixed = sp.boundary == FFS_BOUNDARY_FIXED;
    const int warps = march_warps(r, sp.star, fixed, tau);
    const MarchRate rate = march_rate(r, sp.star, fixed, tau);
    const double U = march_width(r, tau), h = 2.0 * r * tau;
    const double strips = std::ceil(nx / U);
    const double rows = std::min(std::max(strips * ny / (148.0 * warps), 8.0), ny); // march_units
    const double cells = strips * 128 * ny * (rows + h) / rows;
    const double steps = cells * tau * rate.cell, latency = (rows + h) * tau * rate.row;
    // grids of up to 100 MB, both counted, stay in L2 between passes, and part of them up to 300
    const double moved = 16.0 * nx * ny, far = std::min(std::max((moved - 100e6) / 200e6, 0.0), 1.0);
    const double bytes = moved / (kMarchCachedBytesPerSecond + far * (kMarchBytesPerSecond - kMarchCachedBytesPerSecond));
    return std::max(std::max(steps, latency), bytes) + kMarchLaunchSeconds;
}

// The block kernel's steps of its tiles, one per SM at a time (5 taps 0.85 us, 9 taps 1.05, 25 taps 1.8,
// measured on 300 x 260).
double step_seconds(const PlanSpec &sp, double tiles, int steps)
{
    return steps * (0.6e-6 + 0.05e-6 * (double)sp.taps.size()) * std::ceil(tiles / 148.0);
}

// Its tiles of a grid (step_tiles: a tile at a fixed face has no margin there).
double step_grid_tiles(const PlanSpec &sp, int steps)
{
    const double U = step_width(sp.radius, steps), H = sp.radius * steps;
    double tiles = 1.0;
    for (int d = 0; d < 2; ++d) {
        const int walls = sp.boundary != FFS_BOUNDARY_FIXED ? 0
                                                             : !(sp.open_faces >> 2 * d & 1) + !(sp.open_faces >> (2 * d + 1) & 1);
        tiles *= std::max(std::ceil(((double)sp.n[d] - walls * H) / U), 1.0);
    }
    return tiles;
}

// One launch of it over a grid.  A tile is loaded and stored with nothing else on its SM: after the first, which
// overlaps the launch, 2.7 us (4130 x 5900, one step of 44 to 47 tiles per SM, 5, 9 and 25 taps 162, 169 and 218 us).
constexpr double kStepTileSeconds = 2.7e-6;
double step_cost(const PlanSpec &sp, int steps)
{
    const double tiles = step_grid_tiles(sp, steps);
    return kMarchLaunchSeconds + step_seconds(sp, tiles, steps) + kStepTileSeconds * (std::ceil(tiles / 148.0) - 1);
}

// FFS_DIRECT: "0" keeps direct stepping off, "march" or "blocks" takes that kernel wherever it
// can run.
std::string direct_override()
{
    const char *env = getenv("FFS_DIRECT");
    return env ? env : "";
}

// Modelled seconds of one direct step of a 3-D grid.
double march3_cost(const PlanSpec &sp)
{
    March3Work w{};
    for (int d = 0; d < 3; ++d)
        w.n[d] = (int)sp.n[d];
    w.periodic = sp.boundary == FFS_BOUNDARY_PERIODIC;
    return std::max(march3_units(&w, (int)sp.taps.size(), 148), 16.0 * (double)sp.cells / kMarchBytesPerSecond);
}

// 1-D: seconds of a step of the box at a fixed face, 2 r tau staged cells (measured on 7001 to 20000 cells, radius 1
// to 8).  Up to radius 4 and 512 cells one warp steps it, 8 or 16 cells a lane.  Else a block does with a barrier per
// step, 1024 cells at a time: radius 7, us a step, 0.85 in a launch of its own, as a block among line tiles 0.95
// up to 1024 cells, 1.65 to 2048, 2.4 to 3072 and 3.2 above; radius 1, 2, 5 and 8 there 0.41, 0.51, 0.75 and 1.05.
double box1_step(const PlanSpec &sp, int tau, bool among_lines)
{
    const int64_t staged = std::min<int64_t>(2ll * sp.radius * tau, sp.n[0]);
    if (sp.boundary != FFS_BOUNDARY_FIXED || staged == 0 || (sp.open_faces & 3) == 3)
        return 0.0;
    if (sp.radius <= 4 && staged <= 512)
        return staged <= 256 ? 0.03e-6 + 0.04e-6 * sp.radius : 0.06e-6 + 0.055e-6 * sp.radius;
    const double chunk = (among_lines ? 0.046e-6 : 0.038e-6) * (double)sp.taps.size();
    return (among_lines ? 0.27e-6 : 0.28e-6) + chunk * std::ceil((double)staged / 1024);
}

bool strips_win(const PlanSpec &sp);

// The modelled solve on the form's one-SM tiles, to compare with the other routes.  Corrections to the
// model that ranks the tiles' own step counts:
// - 3-D: it counts 3 us per pair of 16^3 tiles (its band and launch terms were fitted with that), but a
//   pair takes 6 us: 100 x 90 x 70, periodic, T = 10 81 us, 256^3 at T = 4 443 us;
// - 2-D, 64 x 64: the tiles at a periodic face wrap with plain loads, and an odd row length rules TMA out for all (us,
//   measured at 1, 2, 6, 14 and 34 waves: periodic 14.6, 27, 54, 98 to 103, 229, odd rows 16.5, -, 68, 168, 421;
//   fixed 10.5, 21, 43, 89, -, odd rows 12.5, 21, -, 120, -).  A fixed boundary's boxes run beside the tiles: up to a
//   depth of 8 cells 5.5 us of their modelled time do not show, to 14 3, then 2 (a band that is stepped on the frame
//   shows as modelled), and 10 beside the longer 128 x 128 tiles.  One wave that leaves them few SMs may become two
//   (25 taps, 752 x 885, T = 3, 136 tiles 16.9 or 24.7 us, 99 of them 10.6);
// - 1-D: a wave takes 10.5 us, not 6 (16.7 M cells 150 us, 44.3 M 404 us, a few thousand 14.8), and the boxes are
//   stepped beside the tiles (radius 7, 8 and 5, one pass of 18, 32 and 80 steps 18.4, 31.9 and 59.0 us).  The
//   tiles that share their SMs are late: 4.8 M cells, radius 3, 140 steps 91 us (tiles 57, boxes 76), 9.8 M, radius
//   5, 154 steps 274 us (140, 171), 2.1 M, radius 6, 65 steps 52 us (36, 51).
double tile_route_cost(const PlanSpec &sp)
{
    double c = model_cost(sp, sp.tau);
    if (sp.form != FFS_FORM_FP64_FFT || !tile_holds(sp, sp.tau))
        return c;
    PassSpec ps;
    geometry(sp, sp.tau, &ps);
    const double waves = std::ceil((double)ps.nitems / 148);
    if (sp.dim == 1) {
        const double tiles = waves * 10.5e-6 + 4e-6, boxes = sp.tau * box1_step(sp, sp.tau, false);
        return sp.passes * std::max(tiles, boxes + 3e-6 + 0.8 * std::max(tiles - 25e-6, 0.0));
    }
    if (sp.dim == 2 && ps.nitems > 0) {
        const bool periodic = sp.boundary == FFS_BOUNDARY_PERIODIC, odd = sp.n[0] & 1;
        const double items = (double)ps.nitems;
        const double w = !periodic && items > 118 ? std::max(waves, 1.5) : waves;
        double tiles;
        if (sp.tile == 128)
            tiles = 4e-6 + waves * kTile128Seconds;
        else if (periodic)
            tiles = odd ? 5e-6 + w * 11.9e-6 : std::min(w * 14.6e-6, 20e-6 + w * 5.75e-6);
        else
            tiles = odd ? 4.5e-6 + w * 8.2e-6 : w == 1 ? 10.5e-6 : 8e-6 + w * 5.75e-6;
        const int depth = sp.radius * sp.tau;
        double hidden = depth <= 8 ? 5.5e-6 : depth <= 14 ? 3e-6 : 2e-6;
        if (sp.tile == 128)
            hidden = waves > 1 || items <= 104 ? 10e-6 : 0.0;
        else if (strips_win(sp))
            hidden = 0.0;
        return sp.passes * (tiles + std::max(band_cost(sp, ps, 148) - hidden, 0.0));
    }
    if (sp.dim == 3 && sp.tile == 16)
        c += sp.passes * waves * 3e-6;
    return c;
}

double pick_direct3(PlanSpec *sp, bool forced)
{
    // (an open face's stepped cells end at +-2^30; offsets in a plane are 32-bit)
    if (sp->radius != 1 || sp->n[0] >= 1 << 30 || sp->n[1] >= 1 << 30 || sp->n[2] >= 1 << 30 ||
        sp->n[0] * sp->n[1] >= 1ll << 31)
        return INFINITY;
    sp->tau = sp->tau_last = 1;
    sp->passes = sp->T;
    return forced ? 0.0 : sp->T * march3_cost(*sp);
}

// Modelled seconds of `steps` direct steps of a line, k cells per lane.
double line_cost(const PlanSpec &sp, int k, int steps)
{
    const double taps = 2.0 * sp.radius + 1, n = (double)sp.n[0];
    const double units = std::ceil(n / (32.0 * k - 2.0 * sp.radius * steps));
    // a warp loads, steps and stores in turn, so bytes and multiply-adds add up (fewer warps per SM
    // with 16 cells a lane)
    const double busy = 16.0 * n / (k == 8 ? 5e12 : 4e12) + units * 32 * k * steps * taps / kLineFmaPerSecond + 2.5e-6;
    return std::max(busy, steps * (kLineStepSeconds + kLineCellSeconds * taps * k) + kLineLaunchSeconds);
}

// Calls use(tau, passes) for the step counts, most at a time, that split T evenly into up to `times` the
// fewest passes: each count once with its fewest passes, so a plan for 10^9 steps looks at no more of them
// than one for 1000.
template <class Use>
void even_steps(int T, int most, int times, Use use)
{
    const int64_t limit = times * ceil_div(T, most);
    for (int tau = std::min(most, T); tau >= 1 && ceil_div(T, tau) <= limit; --tau)
        if (ceil_div(T, ceil_div(T, tau)) == tau)
            use(tau, (int)ceil_div(T, tau));
}

double pick_direct1(PlanSpec *sp, bool forced)
{
    double best = INFINITY;
    for (int k : {8, 16}) {
        const int most = line_max_steps(sp->radius, k);
        if (most == 0)
            continue;
        even_steps(sp->T, most, 3, [&](int tau, int passes) {
            // (a pass starts up while the one before it ends: radius 3, 17121 cells, three passes of 32 steps take
            // 20.9 us, radius 2, 116920 cells, eight of 41 86.3)
            const double c = passes * line_cost(*sp, k, tau) - (passes - 1) * kLineChainSeconds;
            if (c < best) {
                best = c;
                sp->line_k = k;
                sp->tau = tau;
                sp->passes = passes;
                sp->tau_last = sp->T - (passes - 1) * tau;
            }
        });
    }
    return forced && best < INFINITY ? 0.0 : best;
}

// The whole solve stepped directly: fills tau, passes and the kernel, returns seconds.
double pick_direct(PlanSpec *sp)
{
    const int r = sp->radius;
    const std::string only = direct_override();
    if (sp->dim == 1)
        return only == "blocks" ? INFINITY : pick_direct1(sp, only == "march");
    if (sp->dim == 3)
        return only == "blocks" ? INFINITY : pick_direct3(sp, only == "march");
    if (sp->dim != 2 || march_max_tau(r, sp->star) == 0 || sp->n[0] >= 1 << 30 || sp->n[1] >= 1 << 30)
        return INFINITY;
    double best = INFINITY;
    for (bool blocks : {false, true}) {
        if (only == (blocks ? "march" : "blocks"))
            continue;
        const int most = blocks ? step_max_steps(r) : march_max_tau(r, sp->star);
        even_steps(sp->T, most, 2, [&](int tau, int passes) {
            auto pass = [&](int steps) {
                return blocks ? step_cost(*sp, steps) : march_cost(*sp, (double)sp->n[0], (double)sp->n[1], steps);
            };
            const double c = (passes - 1) * pass(tau) + pass(sp->T - (passes - 1) * tau);
            if (c < best) {
                best = c;
                sp->blocks = blocks;
                sp->tau = tau;
                sp->passes = passes;
                sp->tau_last = sp->T - (passes - 1) * tau;
            }
        });
    }
    return only == "march" || only == "blocks" ? 0.0 : best;
}

// Modelled seconds of one direct pass.
double direct_cost(const PlanSpec &sp, int tau)
{
    if (sp.dim == 1)
        return line_cost(sp, sp.line_k, tau);
    if (sp.dim == 3)
        return march3_cost(sp);
    return sp.blocks ? step_cost(sp, tau) : march_cost(sp, (double)sp.n[0], (double)sp.n[1], tau);
}

// The band of one wide pass, stepped on the frame: its seconds alone, and the share of them in
// which the whole GPU is busy with it (what the tiles beside it lose).
double frame_cost(const PlanSpec &sp, int tau, double *busy)
{
    *busy = 0.0;
    if (sp.boundary != FFS_BOUNDARY_FIXED)
        return 0.0;
    const int most = frame_steps(sp), n = (tau + most - 1) / most, steps = (tau + n - 1) / n;
    const double U = step_width(sp.radius, steps), b = sp.radius * tau;
    const double tiles = 2.0 * ((double)sp.n[0] + (double)sp.n[1]) / U * std::ceil((1.5 * b - sp.radius * steps) / U);
    const double launch = step_seconds(sp, tiles, steps);
    *busy = n * launch * std::min(1.0, tiles / 148.0);
    return n * (launch + kMarchLaunchSeconds);
}

// Whether the one-SM tiles' band is stepped on the frame too (the same sums in the same order), rather
// than by a block per box: the boxes' halos are r tau wide on both sides, so past a depth of 16 cells
// they step little else, and from 8 on a long frame has more of them than SMs (us a solve, boxes / frame:
// 1536 x 1024, Box2D9P, T = 12 58.8 / 51.5, Box2D25P, T = 4 43.3 / 41.1, T = 12 123.6 / 103.7 in FP64;
// 4096 x 2048, Box2D25P, T = 12 in 128 x 128 tiles 288 / 197; 200 x 150, Box2D9P, T = 20 37.1 / 24.8).
// A short or shallow frame costs a second launch or as much as the boxes: 200 x 150, T = 12 16.4 / 18.7;
// 1536 x 1024, T = 4 27.1 / 29.0.
bool strips_win(const PlanSpec &sp)
{
    if (march_max_tau(sp.radius, sp.star) == 0 || sp.n[0] >= 1 << 30 || sp.n[1] >= 1 << 30)
        return false;
    PassSpec ps;
    geometry(sp, sp.tau, &ps);
    const int depth = sp.radius * sp.tau;
    return ps.nitems > 0 && (depth >= 16 || (depth >= 8 && sp.n[0] + sp.n[1] >= 1024));
}

// ---- wide tiles ----

constexpr int kWideEdges[] = {256, 512, 1024, 2048};
// Workspace of one chunk of tiles.  Fewer, larger launches win over a workspace that stays in
// the 126 MB L2: Box2D25P 8192^2, T = 128, took 2297 / 2213 / 2018 / 1821 us with chunks of
// 32 / 80 / 160 / 1000 MB (1720 since its columns go group by group), Box2D9P 4096^2 at T = 32 321 / 293 / 280 / 267 us.
constexpr size_t kWideChunkBytes = (size_t)1 << 30;
// Seconds per tile point of a pass: both row kernels by the x edge, the column kernel by the
// y edge (measured on the two grids above), and per kernel its launch and first and last waves.
double wide_row_seconds(int n) { return n == 256 ? 5.0e-12 : n == 512 ? 5.2e-12 : n == 1024 ? 5.7e-12 : 5.0e-12; }
double wide_col_seconds(int n) { return n == 256 ? 4.0e-12 : n == 512 ? 4.8e-12 : n == 1024 ? 5.6e-12 : 7.2e-12; }
constexpr double kWideLaunchSeconds = 4.5e-6;
// 1-D: 148 SMs of 8192 points, a few lines alone, and the launch (44.3 M cells 228 us, 10000 10.6)
constexpr double kWide1WaveSeconds = 12e-6, kWide1LeastSeconds = 7.6e-6, kWide1LaunchSeconds = 3e-6;

double wide1_pass_cost(const PlanSpec &sp, const PassSpec &ps);

// FFS_WIDE_TILE: "0" keeps wide tiles off, "512x1024" takes that edge wherever it fits.
// Returns -1 off, 0 the model's choice, 1 forced.
int wide_override(int dim, int tile[2])
{
    const char *env = getenv("FFS_WIDE_TILE");
    if (!env || !*env)
        return 0;
    int v[2] = {0, 0};
    const int got = sscanf(env, "%dx%d", &v[0], &v[1]);
    if (got >= 1 && v[0] == 0)
        return -1;
    if (got != dim)
        return 0;
    for (int d = 0; d < dim; ++d) {
        if (dim == 1 ? v[d] != 1024 && v[d] != 2048 && v[d] != 4096
                     : std::find(std::begin(kWideEdges), std::end(kWideEdges), v[d]) == std::end(kWideEdges))
            return 0;
        tile[d] = v[d];
    }
    return 1;
}

// Tiles of one pass over the exact window (vlo, vhi set): as few per axis as cover it, spread
// evenly.  False when the edge cannot hold the halo.
bool wide_geometry(const PlanSpec &sp, PassSpec *ps)
{
    ps->nitems = 1;
    for (int d = 0; d < 2; ++d) {
        ps->whalo[d] = 0;
        ps->worg[d] = 0;
        ps->wuseful[d] = ps->wnt[d] = 1;
        if (d >= sp.dim)
            continue;
        const int h = sp.radius * ps->tau;
        const int64_t u = sp.wtile[d] - 2 * h, w = ps->vhi[d] - ps->vlo[d];
        if (u < 16 || (sp.dim > 1 && sp.n[d] < 128)) // rows_fwd steps up to 128 cells around a periodic axis at once
            return false;
        if (w <= 0) { // no exact window: the band takes the whole grid
            ps->nitems = 0;
            return true;
        }
        ps->wnt[d] = ceil_div(w, u);
        ps->wuseful[d] = ceil_div(w, ps->wnt[d]);
        ps->whalo[d] = h;
        ps->worg[d] = ps->vlo[d] - h;
        ps->nitems *= ps->wnt[d];
    }
    return true;
}

int wide_chunk(const PlanSpec &sp, int64_t tiles)
{
    if (sp.dim == 1) // (no workspace)
        return 0;
    const int64_t c = (int64_t)(kWideChunkBytes / wide_tile_bytes(sp.wtile));
    return (int)std::max<int64_t>(1, std::min(c, tiles));
}

double wide_pass_cost(const PlanSpec &sp, const PassSpec &ps, int num_sms)
{
    if (sp.dim == 1)
        return wide1_pass_cost(sp, ps);
    const double pts = (double)sp.wtile[0] * sp.wtile[1] * (double)ps.nitems;
    const double chunks = std::ceil((double)ps.nitems / wide_chunk(sp, ps.nitems));
    const double tiles = pts * (wide_row_seconds(sp.wtile[0]) + wide_col_seconds(sp.wtile[1])) +
                         chunks * 3 * kWideLaunchSeconds;
    // the band runs beside the tiles, but what SMs it holds they do not have (0.7 of that shows:
    // Box2D9P 1024^2 / 2048^2 / 4096^2 at T = 32 model 50 / 106 / 301 us, measured 46 / 113 / 303)
    double busy = 0.0;
    const double band = sp.frame ? frame_cost(sp, ps.tau, &busy) : (busy = band_cost(sp, ps, num_sms));
    // boxes of more cells than a block decodes once (2 x 1024) take several times their modelled work beside the tiles'
    // small blocks (2802 x 1554, us, tiles alone / with the band: radius 3, 8 and 11 steps 78 / 198 and 89 / 313, radius
    // 6, 3 steps 72 / 259, modelled work 55, 90 and 28)
    const double share = !sp.frame && ps.band_max_vol > 2048 ? 3.0 : 0.7;
    return std::max(tiles + share * busy, band);
}

// 1-D: seconds of one pass.  An SM holds 8192 complex points (16384 tile cells) at a time.
double wide1_pass_cost(const PlanSpec &sp, const PassSpec &ps)
{
    const double waves = (double)ps.nitems * sp.wtile[0] / (148.0 * 16384);
    // 2^20 cells at T = 64 10.6 us with 2048 (12.8 with 1024, 11.2 with 4096), 16.7 M at T = 32 87 (90, 92)
    const double edge = sp.wtile[0] == 1024 ? 1.08 : sp.wtile[0] == 4096 ? 1.04 : 1.0;
    const double tiles = edge * std::max(waves * kWide1WaveSeconds, kWide1LeastSeconds);
    // the boxes are the launch's last blocks: with more tiles than a wave they start with its last one (1.26 M
    // cells, radius 2, 230 steps of 920 staged cells in 1024-cell tiles: 176 us a pass)
    const double before = std::max(tiles - edge * kWide1LeastSeconds, 0.0);
    return std::max(tiles, before + ps.tau * box1_step(sp, ps.tau, true)) + kWide1LaunchSeconds;
}

double pick_wide1(PlanSpec *sp, int forced)
{
    double best = INFINITY;
    PlanSpec t = *sp;
    t.wide = true;
    for (int passes = 1; passes <= std::min(sp->T, 8); ++passes) {
        const int tau = (sp->T + passes - 1) / passes;
        if ((sp->T + tau - 1) / tau != passes)
            continue;
        for (int edge : {1024, 2048, 4096}) {
            // (a tile wraps around a periodic line at most once)
            if ((forced && edge != forced) || edge > sp->n[0] || 2 * round_even(sp->radius * tau) + 16 > edge)
                continue;
            PassSpec ps;
            t.tile = t.wtile[0] = edge;
            geometry(t, tau, &ps);
            if (band_smem_bytes(band_max_volume(t, ps, band_slabs(t, ps)), (int)t.taps.size()) > kBandSmemLimit ||
                !wide_geometry(t, &ps) || ps.nitems == 0)
                continue;
            const double c = passes * wide1_pass_cost(t, ps);
            if (c < best) {
                best = c;
                sp->wtile[0] = edge;
                sp->tau = tau;
                sp->passes = passes;
                sp->tau_last = sp->T - (passes - 1) * tau;
            }
        }
    }
    return forced && best < INFINITY ? 0.0 : best;
}

// Fills the wide tile, tau and passes of `sp` with the cheapest modelled choice; returns its
// seconds (infinite when no wide tile fits).
double pick_wide(PlanSpec *sp)
{
    double best = INFINITY;
    int forced[2] = {0, 0};
    const int mode = wide_override(sp->dim, forced);
    if (sp->form != FFS_FORM_FP64_FFT || sp->dim > 2 || sp->T == 0 || mode < 0)
        return best;
    if (sp->dim == 1)
        return pick_wide1(sp, mode > 0 ? forced[0] : 0);
    PlanSpec t = *sp;
    t.wide = true;
    t.frame = sp->frame = sp->boundary == FFS_BOUNDARY_FIXED && march_max_tau(sp->radius, sp->star) > 0 && sp->n[0] < 1 << 30 &&
                          sp->n[1] < 1 << 30;
    for (int passes = 1; passes <= std::min(sp->T, 16); ++passes) {
        const int tau = (sp->T + passes - 1) / passes;
        if ((sp->T + tau - 1) / tau != passes)
            continue;
        if (2 * round_even(sp->radius * tau) + 16 > 2048)
            continue;
        PassSpec ps;
        t.tile = 2048;
        geometry(t, tau, &ps);
        if (!t.frame)
            ps.band_max_vol = band_max_volume(t, ps, band_slabs(t, ps));
        if (ps.band_max_vol > 0 && band_smem_bytes(ps.band_max_vol, (int)t.taps.size()) > kBandSmemLimit)
            continue;
        for (int ex : kWideEdges)
            for (int ey : kWideEdges) {
                if (mode > 0 && (ex != forced[0] || ey != forced[1]))
                    continue;
                t.wtile[0] = ex;
                t.wtile[1] = ey;
                if (!wide_geometry(t, &ps) || ps.nitems == 0)
                    continue;
                const double c = passes * wide_pass_cost(t, ps, 148);
                if (c < best) {
                    best = c;
                    sp->wtile[0] = ex;
                    sp->wtile[1] = ey;
                    sp->tau = tau;
                    sp->passes = passes;
                    sp->tau_last = sp->T - (passes - 1) * tau;
                }
            }
    }
    return mode > 0 && best < INFINITY ? 0.0 : best;
}

void make_spectrum_2d(const PlanSpec &sp, int tau, std::vector<double2> *out)
{
    const int n = 64;
    const auto rt = roots(n);
    out->resize(n * n);
    const long double scale = 1.0L / (n * n);
    // position p holds frequency (p >> 3) + 8 * (p & 7) (two radix-8 stages)
    for (int px = 0; px < n; ++px)
        for (int py = 0; py < n; ++py) {
            const int k[3] = {(px >> 3) + 8 * (px & 7), (py >> 3) + 8 * (py & 7), 0};
            CLD s = cpow(symbol(sp, rt, n, k), tau);
            (*out)[px * n + py] = make_double2((double)(s.re * scale), (double)(s.im * scale));
        }
}

// 1D tile of 4096 = 64 x 64 (j = 64a + b): SMEM column position px holds the
// first-stage frequency k1 = k(px), row position py the second-stage k2 = k(py),
// k(p) = (p >> 3) + 8 * (p & 7); full frequency k1 + 64 * k2.
void make_spectrum_1d(const PlanSpec &sp, int tau, std::vector<double2> *out)
{
    const int n = 4096;
    const auto rt = roots(n);
    out->resize(n);
    const long double scale = 1.0L / n;
    for (int px = 0; px < 64; ++px)
        for (int py = 0; py < 64; ++py) {
            const int k1 = (px >> 3) + 8 * (px & 7), k2 = (py >> 3) + 8 * (py & 7);
            const int k[3] = {k1 + 64 * k2, 0, 0};
            CLD s = cpow(symbol(sp, rt, n, k), tau);
            (*out)[px * 64 + py] = make_double2((double)(s.re * scale), (double)(s.im * scale));
        }
}

// 1D butterfly form: the Hermitian half k = 0..2048 at slot k + (k >> 6) (2088 slots); the
// kernel takes k > 2048 as conj S[4096 - k].
void make_spectrum_1d_half(const PlanSpec &sp, int tau, std::vector<double2> *out)
{
    const int n = 4096;
    const auto rt = roots(n);
    out->assign(2088, make_double2(0.0, 0.0));
    const long double scale = 1.0L / n;
    for (int f = 0; f <= n / 2; ++f) {
        const int k[3] = {f, 0, 0};
        CLD s = cpow(symbol(sp, rt, n, k), tau);
        (*out)[f + (f >> 6)] = make_double2((double)(s.re * scale), (double)(s.im * scale));
    }
}

// tcgen05 forms: natural frequency order spec[ky * 64 + kx].
void make_spectrum_2d_natural(const PlanSpec &sp, int tau, std::vector<double2> *out)
{
    const int n = 64;
    const auto rt = roots(n);
    out->resize(n * n);
    const long double scale = 1.0L / (n * n);
    for (int ky = 0; ky < n; ++ky)
        for (int kx = 0; kx < n; ++kx) {
            const int k[3] = {kx, ky, 0};
            CLD s = cpow(symbol(sp, rt, n, k), tau);
            (*out)[ky * n + kx] = make_double2((double)(s.re * scale), (double)(s.im * scale));
        }
}

// Butterfly form: the half kx = 0..32, spec[ky * 33 + kx].  Real weights make the
// symbol Hermitian, S(-k) = conj S(k), so the kernel takes kx > 32 as
// conj spec[(-ky mod 64) * 33 + 64 - kx].
void make_spectrum_2d_half(const PlanSpec &sp, int tau, std::vector<double2> *out)
{
    const int n = 64, h = n / 2 + 1;
    const auto rt = roots(n);
    out->resize(n * h);
    const long double scale = 1.0L / (n * n);
    for (int ky = 0; ky < n; ++ky)
        for (int kx = 0; kx < h; ++kx) {
            const int k[3] = {kx, ky, 0};
            CLD s = cpow(symbol(sp, rt, n, k), tau);
            (*out)[ky * h + kx] = make_double2((double)(s.re * scale), (double)(s.im * scale));
        }
}

// 2D butterfly form on the 128 x 128 tile: the half kx = 0..64, spec[kx * 128 + ky] (a
// column's group reads consecutive ky).
void make_spectrum_2d128(const PlanSpec &sp, int tau, std::vector<double2> *out)
{
    const int n = 128;
    const auto rt = roots(n);
    out->resize((n / 2 + 1) * n);
    const long double scale = 1.0L / (n * n);
    for (int kx = 0; kx <= n / 2; ++kx)
        for (int ky = 0; ky < n; ++ky) {
            const int k[3] = {kx, ky, 0};
            CLD s = cpow(symbol(sp, rt, n, k), tau);
            (*out)[kx * n + ky] = make_double2((double)(s.re * scale), (double)(s.im * scale));
        }
}

// 3D butterfly form: the half kx = 0..8, spec[(kx * 16 + kz) * 16 + ky] (the 32 lines
// (kz, ky) of a warp read 32 consecutive entries per kx); the kernel takes kx > 8 as
// conj spec[(16 - kx, -kz mod 16, -ky mod 16)] (Hermitian symbol).
void make_spectrum_3d_half(const PlanSpec &sp, int tau, std::vector<double2> *out)
{
    const int n = 16, h = n / 2 + 1;
    const auto rt = roots(n);
    out->resize(n * n * h);
    const long double scale = 1.0L / (n * n * n);
    for (int kz = 0; kz < n; ++kz)
        for (int ky = 0; ky < n; ++ky)
            for (int kx = 0; kx < h; ++kx) {
                const int k[3] = {kx, ky, kz};
                CLD s = cpow(symbol(sp, rt, n, k), tau);
                (*out)[(kx * n + kz) * n + ky] = make_double2((double)(s.re * scale), (double)(s.im * scale));
            }
}

// 3D (the other forms): natural frequency order spec[(kz * 16 + ky) * 16 + kx].
void make_spectrum_3d_natural(const PlanSpec &sp, int tau, std::vector<double2> *out)
{
    const int n = 16;
    const auto rt = roots(n);
    out->resize(n * n * n);
    const long double scale = 1.0L / (n * n * n);
    for (int kz = 0; kz < n; ++kz)
        for (int ky = 0; ky < n; ++ky)
            for (int kx = 0; kx < n; ++kx) {
                const int k[3] = {kx, ky, kz};
                CLD s = cpow(symbol(sp, rt, n, k), tau);
                (*out)[(kz * n + ky) * n + kx] = make_double2((double)(s.re * scale), (double)(s.im * scale));
            }
}

// 3D butterfly form on the 32^3 tile: natural order spec[(kz * 32 + ky) * 32 + kx] (the
// cluster kernel reads it along kx, coalesced, for its y lines).
void make_spectrum_3d32(const PlanSpec &sp, int tau, std::vector<double2> *out)
{
    const int n = 32;
    const auto rt = roots(n);
    out->resize(n * n * n);
    const long double scale = 1.0L / (n * n * n);
    for (int kz = 0; kz < n; ++kz)
        for (int ky = 0; ky < n; ++ky)
            for (int kx = 0; kx < n; ++kx) {
                const int k[3] = {kx, ky, kz};
                CLD s = cpow(symbol(sp, rt, n, k), tau);
                (*out)[(kz * n + ky) * n + kx] = make_double2((double)(s.re * scale), (double)(s.im * scale));
            }
}

} // namespace

int frame_steps(const PlanSpec &sp) { return sp.radius == 1 ? 11 : 5; }

size_t frame_cells(const PlanSpec &sp, int tau, int face)
{
    size_t at = 0;
    for (int f = 0; f < face; ++f) { // face 2 d + side: 2 r tau deep along d, the whole other axis
        const int d = f / 2;
        if (!(sp.open_faces >> f & 1))
            at += (size_t)std::min<int64_t>(2ll * sp.radius * tau, sp.n[d]) * sp.n[1 - d];
    }
    return at;
}

std::vector<double2> wide_twiddles(int n, int axis)
{
    const int P = wide_points(n, axis), L = n / P;
    const auto rn = roots(n), rl = roots(L);
    std::vector<double2> tw(n + L);
    for (int k1 = 0; k1 < P; ++k1)
        for (int m = 0; m < L; ++m) {
            const CLD w = rn[(int64_t)k1 * m % n];
            tw[k1 * L + m] = make_double2((double)w.re, (double)w.im);
        }
    for (int m2 = 0; m2 < L / P; ++m2)
        for (int k2 = 0; k2 < P; ++k2) {
            const CLD w = rl[(int64_t)k2 * m2 % L];
            tw[n + P * m2 + k2] = make_double2((double)w.re, (double)w.im);
        }
    return tw;
}

std::vector<double2> wide_roots(int n)
{
    const auto r = roots(n);
    std::vector<double2> out(2 * (size_t)n);
    auto split = [](long double v) {
        const double hi = (double)v;
        return make_double2(hi, (double)(v - hi));
    };
    for (int m = 0; m < n; ++m) {
        out[2 * m] = split(r[m].re);
        out[2 * m + 1] = split(-r[m].im); // exp(+2 pi i m / n)
    }
    return out;
}

namespace {

// Byte offset of (row r, K byte kb) in a K-major no-swizzle tcgen05 operand with KB bytes per row.
size_t operand_offset(int r, int kb, int KB) { return (size_t)(r / 8) * (8 * KB) + (kb / 16) * 128 + (r % 8) * 16 + kb % 16; }

uint16_t bf16_rn(float f) // round to nearest even
{
    uint32_t u;
    memcpy(&u, &f, 4);
    const uint32_t lsb = (u >> 16) & 1u;
    u += 0x7fffu + lsb;
    return (uint16_t)(u >> 16);
}

float bf16_to_f(uint16_t h)
{
    uint32_t u = (uint32_t)h << 16;
    float f;
    memcpy(&f, &u, 4);
    return f;
}

// Balanced base-256 digits of y (|y| <= 64), most significant first: y * 256^(S-1)
// rounded once (exact in long double's 64-bit significand for S <= 8), biased by
// 0x80 per byte so that byte S-1-i is digit i + 128 (the device's digit_bytes).
static void ozaki_digits(long double y, int S, int8_t *d)
{
    const int64_t X = (int64_t)nearbyintl(ldexpl(y, 8 * (S - 1)));
    const uint64_t U = (uint64_t)X + (0x8080808080808080ull >> (8 * (8 - S)));
    for (int i = 0; i < S; ++i)
        d[i] = (int8_t)((int)((U >> (8 * (S - 1 - i))) & 255) - 128);
}

// Real-block DFT-64 matrix with interleaved rows (m = 2f + part), 128 x 128:
// A[2f][x] = Re F, A[2f][64+x] = -Im F, A[2f+1][x] = Im F, A[2f+1][64+x] = Re F, F = w64^(f x).
// Ozaki: `slices` balanced base-256 digits of the entry * 2^6; BF16: hi/mid/lo pieces.
void make_a_slices(PlanSpec *sp)
{
    const auto r64 = roots(64);
    auto entry = [&](int m, int k) -> long double {
        const int f = m >> 1, part = m & 1, half = k >> 6, x = k & 63;
        const CLD w = r64[(f * x) % 64];
        if (part == 0)
            return half == 0 ? w.re : -w.im;
        return half == 0 ? w.im : w.re;
    };
    const int S = sp->slices;
    if (sp->form == FFS_FORM_OZAKI_I8) {
        const int KB = 128, slice = 128 * KB;
        sp->a_slices.assign((size_t)S * slice, 0);
        for (int m = 0; m < 128; ++m)
            for (int k = 0; k < 128; ++k) {
                int8_t d[8];
                ozaki_digits(entry(m, k) * 64.0L, S, d);
                for (int i = 0; i < S; ++i)
                    sp->a_slices[(size_t)i * slice + operand_offset(m, k, KB)] = (unsigned char)d[i];
            }
    } else {
        const int KB = 256, slice = 128 * KB;
        sp->a_slices.assign((size_t)S * slice, 0);
        for (int m = 0; m < 128; ++m)
            for (int k = 0; k < 128; ++k) {
                double r = (double)entry(m, k);
                for (int i = 0; i < S; ++i) {
                    const uint16_t h = bf16_rn((float)r);
                    r -= (double)bf16_to_f(h);
                    memcpy(&sp->a_slices[(size_t)i * slice + operand_offset(m, 2 * k, KB)], &h, 2);
                }
            }
    }
}

// DFT-16 operand of the 3D tcgen05 forms: row n = 32 i + 2 f + part of slice i,
// K element k = 2 x + part_in:  [2f][2x] = Re F, [2f][2x+1] = -Im F,
// [2f+1][2x] = Im F, [2f+1][2x+1] = Re F, F = w16^(f x).  Ozaki: digits of F * 2^6
// (32-byte rows, slices stacked along N); BF16: hi/mid/lo pieces (64-byte rows).
void make_f16_slices(PlanSpec *sp)
{
    const auto r16 = roots(16);
    auto entry = [&](int m, int k) -> long double {
        const int f = m >> 1, po = m & 1, x = k >> 1, pi = k & 1;
        const CLD w = r16[(f * x) % 16];
        if (po == 0)
            return pi == 0 ? w.re : -w.im;
        return pi == 0 ? w.im : w.re;
    };
    const int S = sp->slices;
    if (sp->form == FFS_FORM_OZAKI_I8) {
        const int KB = 32;
        sp->a_slices.assign((size_t)S * 32 * KB, 0);
        for (int m = 0; m < 32; ++m)
            for (int k = 0; k < 32; ++k) {
                int8_t d[8];
                ozaki_digits(entry(m, k) * 64.0L, S, d);
                for (int i = 0; i < S; ++i)
                    sp->a_slices[operand_offset(32 * i + m, k, KB)] = (unsigned char)d[i];
            }
    } else {
        const int KB = 64, slice = 32 * KB;
        sp->a_slices.assign((size_t)S * slice, 0);
        for (int m = 0; m < 32; ++m)
            for (int k = 0; k < 32; ++k) {
                double r = (double)entry(m, k);
                for (int i = 0; i < S; ++i) {
                    const uint16_t h = bf16_rn((float)r);
                    r -= (double)bf16_to_f(h);
                    memcpy(&sp->a_slices[(size_t)i * slice + operand_offset(m, 2 * k, KB)], &h, 2);
                }
            }
    }
}

void make_tables(PlanSpec *sp)
{
    sp->tables.clear();
    auto push = [&](const std::vector<CLD> &r, int count) {
        for (int i = 0; i < count; ++i)
            sp->tables.push_back(make_double2((double)r[i % r.size()].re, (double)r[i % r.size()].im));
    };
    if (sp->dim == 3) { // 16th roots (radix-4 DFT matrices and twiddles)
        push(roots(16), 16);
        return;
    }
    push(roots(8), 8);
    push(roots(64), 64);
    if (sp->dim == 2 && sp->tile == 128) // the 128 x 128 kernel's twiddles w128^m
        push(roots(128), 128);
    if (sp->dim == 1) { // four-step twiddles w4096^m (m < 448) and w512^m (m < 512)
        push(roots(4096), 448);
        push(roots(512), 512);
    }
}

std::mutex g_tune_mu;
std::map<std::string, int> g_tune;
bool g_tune_loaded = false;

void tune_load_locked()
{
    if (g_tune_loaded)
        return;
    g_tune_loaded = true;
    const char *path = getenv("FFS_TUNE_CACHE");
    if (!path)
        return;
    FILE *f = fopen(path, "r");
    if (!f)
        return;
    char key[512];
    int tau;
    while (fscanf(f, "%511s %d", key, &tau) == 2)
        g_tune[key] = tau;
    fclose(f);
}

} // namespace

// Problem class: form, slice count, tile edge, dimension, taps, boundary, T and the
// log2 size of each extent.
std::string tune_key(const PlanSpec &sp)
{
    char buf[256];
    int lg[3];
    for (int d = 0; d < 3; ++d)
        lg[d] = (int)std::lround(std::log2((double)sp.n[d]));
    snprintf(buf, sizeof(buf), "f%d.s%d.t%d.d%d.r%d.k%zu.b%d.o%d.T%d.n%d_%d_%d", (int)sp.form, sp.slices, sp.tile,
             sp.dim, sp.radius, sp.taps.size(), (int)sp.boundary, sp.open_faces, sp.T, lg[0], lg[1], lg[2]);
    return buf;
}

// The same class without the tile edge: key of the measured edge of the butterfly form's one-SM tiles.
std::string tile_key(const PlanSpec &sp)
{
    char buf[256];
    int lg[3];
    for (int d = 0; d < 3; ++d)
        lg[d] = (int)std::lround(std::log2((double)sp.n[d]));
    snprintf(buf, sizeof(buf), "E.f%d.d%d.r%d.k%zu.b%d.o%d.T%d.n%d_%d_%d", (int)sp.form, sp.dim, sp.radius,
             sp.taps.size(), (int)sp.boundary, sp.open_faces, sp.T, lg[0], lg[1], lg[2]);
    return buf;
}

// The same class for the route (one-SM tiles, wide tiles or direct steps).  The automatic form and the
// butterfly form by name have an entry each: only the first may step directly, so a route measured for
// one was not chosen among the other's.
std::string route_key(const PlanSpec &sp, bool automatic)
{
    return (automatic ? "RA." : "R.") + tile_key(sp).substr(2);
}

// The same class without the slice count: key of the calibrated Ozaki slice count.
std::string slice_key(const PlanSpec &sp)
{
    char buf[256];
    int lg[3];
    for (int d = 0; d < 3; ++d)
        lg[d] = (int)std::lround(std::log2((double)sp.n[d]));
    snprintf(buf, sizeof(buf), "S.f%d.d%d.r%d.k%zu.b%d.o%d.T%d.n%d_%d_%d", (int)sp.form, sp.dim, sp.radius,
             sp.taps.size(), (int)sp.boundary, sp.open_faces, sp.T, lg[0], lg[1], lg[2]);
    return buf;
}

int tune_lookup(const std::string &key)
{
    std::lock_guard<std::mutex> lk(g_tune_mu);
    tune_load_locked();
    auto it = g_tune.find(key);
    return it == g_tune.end() ? 0 : it->second;
}

void tune_record(const std::string &key, int tau)
{
    std::lock_guard<std::mutex> lk(g_tune_mu);
    tune_load_locked();
    g_tune[key] = tau;
    if (const char *path = getenv("FFS_TUNE_CACHE")) {
        if (FILE *f = fopen(path, "a")) {
            fprintf(f, "%s %d\n", key.c_str(), tau);
            fclose(f);
        }
    }
}

std::vector<int> tau_candidates(const ffs_problem &p, int count)
{
    ffs_problem q = p;
    q.tau = 1;
    PlanSpec sp;
    std::string why;
    if (build_plan_spec(q, &sp, &why, false) != FFS_OK || sp.T == 0)
        return {};
    std::vector<std::pair<double, int>> c;
    const int tmax = max_tau(sp);
    for (int tau = 1; tau <= tmax; ++tau)
        c.push_back({model_cost(sp, tau), tau});
    std::sort(c.begin(), c.end());
    std::vector<int> out;
    for (int i = 0; i < (int)c.size() && i < count; ++i)
        out.push_back(c[i].second);
    return out;
}

const ShapeDef *find_shape(const char *name)
{
    if (!name)
        return nullptr;
    for (const ShapeDef &s : kShapes)
        if (iequals(s.name, name))
            return &s;
    return nullptr;
}

const ShapeDef *find_shape_id(ffs_shape id)
{
    for (const ShapeDef &s : kShapes)
        if (s.id == id)
            return &s;
    return nullptr;
}

// Default weights, each normalised to sum 1 (Heat-1D is (0.25, 0.5, 0.25)).
std::vector<double> shape_weights(const ShapeDef &sd)
{
    const int r = sd.radius, K = 2 * r + 1;
    int vol = 1;
    for (int d = 0; d < sd.dim; ++d)
        vol *= K;
    std::vector<double> w(vol, 0.0);
    auto at = [&](int dx, int dy, int dz) -> double & {
        const int ry = sd.dim >= 2 ? r : 0, rz = sd.dim >= 3 ? r : 0, Ky = 2 * ry + 1;
        return w[((dz + rz) * Ky + (dy + ry)) * K + (dx + r)];
    };
    switch (sd.id) {
    case FFS_SHAPE_HEAT_1D:
        w = {0.25, 0.5, 0.25};
        break;
    case FFS_SHAPE_1D5P:
        w = {0.1, 0.2, 0.4, 0.2, 0.1};
        break;
    case FFS_SHAPE_1D7P:
        w = {0.05, 0.1, 0.15, 0.4, 0.15, 0.1, 0.05};
        break;
    case FFS_SHAPE_HEAT_2D:
        at(0, 0, 0) = 0.5;
        at(1, 0, 0) = at(-1, 0, 0) = at(0, 1, 0) = at(0, -1, 0) = 0.125;
        break;
    case FFS_SHAPE_BOX2D9P:
        for (double &v : w)
            v = 0.1;
        at(0, 0, 0) = 0.2;
        break;
    case FFS_SHAPE_STAR2D9P:
        at(0, 0, 0) = 0.2;
        at(1, 0, 0) = at(-1, 0, 0) = at(0, 1, 0) = at(0, -1, 0) = 0.125;
        at(2, 0, 0) = at(-2, 0, 0) = at(0, 2, 0) = at(0, -2, 0) = 0.075;
        break;
    case FFS_SHAPE_BOX2D25P:
        for (double &v : w)
            v = 0.04;
        break;
    case FFS_SHAPE_HEAT_3D:
        at(0, 0, 0) = 0.4;
        at(1, 0, 0) = at(-1, 0, 0) = at(0, 1, 0) = at(0, -1, 0) = at(0, 0, 1) = at(0, 0, -1) = 0.1;
        break;
    case FFS_SHAPE_BOX3D27P:
        for (double &v : w)
            v = 0.9 / 26.0;
        at(0, 0, 0) = 0.1;
        break;
    default:
        break;
    }
    return w;
}

ffs_status build_plan_spec(const ffs_problem &p, PlanSpec *out, std::string *why, bool with_data, Route route)
{
    PlanSpec sp;
    auto bad = [&](ffs_status st, const std::string &m) {
        *why = m;
        return st;
    };
    for (int i = 0; i < 6; ++i)
        if (p.reserved[i] != 0)
            return bad(FFS_ERR_INVALID_ARGUMENT, "ffs_problem.reserved must be zero");
    if (p.open_faces < 0 || p.open_faces >= (1 << (2 * std::max(1, std::min(p.dim, 3)))))
        return bad(FFS_ERR_INVALID_ARGUMENT, "open_faces names a face the grid does not have");
    sp.open_faces = p.open_faces;
    if (p.dim < 1 || p.dim > 3)
        return bad(FFS_ERR_INVALID_ARGUMENT, "dim must be 1, 2 or 3");
    sp.dim = p.dim;
    if (p.shape != FFS_SHAPE_CUSTOM) {
        const ShapeDef *sd = find_shape_id(p.shape);
        if (!sd)
            return bad(FFS_ERR_INVALID_ARGUMENT, "unknown shape id");
        if (sd->dim != p.dim)
            return bad(FFS_ERR_INVALID_ARGUMENT, std::string("shape ") + sd->name + " is " +
                                                     std::to_string(sd->dim) + "-D");
        sp.radius = sd->radius;
        sp.weights = shape_weights(*sd);
    } else {
        if (p.radius < 0 || p.radius > 8)
            return bad(FFS_ERR_INVALID_ARGUMENT, "custom radius must be in [0, 8]");
        if (!p.weights)
            return bad(FFS_ERR_INVALID_ARGUMENT, "custom shape needs weights");
        sp.radius = p.radius;
    }
    const int K = 2 * sp.radius + 1;
    size_t nw = 1;
    for (int d = 0; d < p.dim; ++d)
        nw *= K;
    if (p.weights) {
        sp.weights.assign(p.weights, p.weights + nw);
        for (double v : sp.weights)
            if (!std::isfinite(v))
                return bad(FFS_ERR_INVALID_ARGUMENT, "weights must be finite");
    }
    if (sp.weights.size() != nw)
        return bad(FFS_ERR_INTERNAL, "weights size mismatch");
    for (int d = 0; d < 3; ++d) {
        const int64_t e = p.extents[d];
        if (d < p.dim && e < 1)
            return bad(FFS_ERR_INVALID_ARGUMENT, "extents must be >= 1");
        if (d >= p.dim && e != 1 && e != 0)
            return bad(FFS_ERR_INVALID_ARGUMENT, "unused extents must be 1");
        sp.n[d] = d < p.dim ? e : 1;
    }
    if (sp.n[0] > (1ll << 31) || sp.n[1] > (1ll << 31) || sp.n[2] > (1ll << 31))
        return bad(FFS_ERR_INVALID_ARGUMENT, "extent too large");
    sp.cells = (size_t)sp.n[0] * sp.n[1] * sp.n[2];
    if (p.T < 0)
        return bad(FFS_ERR_INVALID_ARGUMENT, "T must be >= 0");
    sp.T = p.T;
    if (p.boundary != FFS_BOUNDARY_PERIODIC && p.boundary != FFS_BOUNDARY_FIXED)
        return bad(FFS_ERR_INVALID_ARGUMENT, "unknown boundary");
    sp.boundary = p.boundary;
    if (p.tau < 0)
        return bad(FFS_ERR_INVALID_ARGUMENT, "tau must be >= 0");
    switch (p.form) {
    case FFS_FORM_AUTO: // the fastest FP64-exact form: the butterfly kernels
    case FFS_FORM_FP64_DMMA:
        sp.form = p.form == FFS_FORM_AUTO ? FFS_FORM_FP64_FFT : FFS_FORM_FP64_DMMA;
        if (p.slices != 0)
            return bad(FFS_ERR_INVALID_ARGUMENT, "slices only apply to the Ozaki and BF16 forms");
        break;
    case FFS_FORM_FP64_FFT:
        sp.form = FFS_FORM_FP64_FFT;
        if (p.slices != 0)
            return bad(FFS_ERR_INVALID_ARGUMENT, "slices only apply to the Ozaki and BF16 forms");
        break;
    case FFS_FORM_OZAKI_I8:
        sp.form = FFS_FORM_OZAKI_I8;
        sp.slices = p.slices; // 0: the calibrated count of the problem class, else the default (below)
        if (p.slices != 0 && (p.slices < 4 || p.slices > 8))
            return bad(FFS_ERR_INVALID_ARGUMENT, "Ozaki slices must be in [4, 8]");
        break;
    case FFS_FORM_BF16X3:
        sp.form = FFS_FORM_BF16X3;
        sp.slices = p.slices == 0 ? 3 : p.slices;
        if (sp.slices < 2 || sp.slices > 3)
            return bad(FFS_ERR_INVALID_ARGUMENT, "BF16 split count must be 2 or 3");
        break;
    default:
        return bad(FFS_ERR_INVALID_ARGUMENT, "unknown form");
    }
    if ((sp.form == FFS_FORM_OZAKI_I8 || sp.form == FFS_FORM_BF16X3) && p.dim == 1)
        return bad(FFS_ERR_UNSUPPORTED, "the Ozaki and BF16 tensor-core forms are available for 2-D and 3-D grids");
    // taps (non-zero weights) for the band kernel
    {
        const int r = sp.radius;
        const int ry = sp.dim >= 2 ? r : 0, rz = sp.dim >= 3 ? r : 0, Ky = 2 * ry + 1;
        for (int dz = -rz; dz <= rz; ++dz)
            for (int dy = -ry; dy <= ry; ++dy)
                for (int dx = -r; dx <= r; ++dx) {
                    const int idx = ((dz + rz) * Ky + (dy + ry)) * K + (dx + r);
                    if (sp.weights[idx] != 0.0)
                        sp.taps.push_back(make_int4(dx, dy, dz, idx));
                }
    }
    sp.star = true;
    for (const int4 &t : sp.taps)
        sp.star &= (t.x != 0) + (t.y != 0) + (t.z != 0) <= 1;
    if (sp.form == FFS_FORM_OZAKI_I8 && sp.slices == 0) { // a calibrated count for this class wins
        const int tuned = tune_lookup(slice_key(sp));
        sp.slices = (tuned >= 4 && tuned <= 8) ? tuned : kDefaultOzakiSlices;
    }
    const int fixed_tile = tile_edge(sp.dim, sp.form);
    const int alt = alt_tile_edge(sp.dim, sp.form); // 0: the form has one edge
    if (p.tile != 0 && p.tile != fixed_tile && !(alt && p.tile == alt))
        return bad(FFS_ERR_UNSUPPORTED, "tile edge not available for this form (1D 4096, 2D 64, 3D 16; the FP64 "
                                        "butterfly form also 128 in 2D and 32 in 3D)");
    sp.tile = p.tile != 0 ? p.tile : fixed_tile;
    const bool edge_open = p.tile == 0 && alt && sp.T > 0;
    if (edge_open)
        sp.tile = pick_tile(sp, p.tau);
    if (sp.T == 0) {
        sp.passes = 0;
        sp.npass_kinds = 0;
        *out = std::move(sp);
        return FFS_OK;
    }
    pick_tau(&sp, p.tau);
    // wide tiles and direct stepping: only where the caller left both the edge and the step count
    // open.  Direct stepping is the automatic form's; the butterfly form asked for by name stays that.
    if (p.tile == 0 && p.tau == 0 && sp.T > 0 && sp.form == FFS_FORM_FP64_FFT) {
        const bool may_step = p.form == FFS_FORM_AUTO && direct_override() != "0";
        auto choose = [&](bool tiles, bool wide, bool direct) { // the cheapest modelled of these that fits
            double best = tiles ? tile_route_cost(sp) : INFINITY;
            PlanSpec w = sp, d = sp;
            if (wide) {
                const double c = pick_wide(&w);
                if (c < best) {
                    best = c;
                    sp = std::move(w);
                    sp.wide = true;
                    sp.tile = sp.wtile[0];
                }
            }
            if (direct) {
                const double c = pick_direct(&d);
                if (c < best) {
                    best = c;
                    sp = std::move(d);
                    sp.direct = true;
                    sp.tile = sp.dim == 1 ? 32 * sp.line_k : sp.dim == 2 ? 128 : 64;
                }
            }
        };
        // a measured choice for the class wins over the model, where it fits this problem
        const int measured = route == kRouteAuto ? tune_lookup(route_key(sp, p.form == FFS_FORM_AUTO)) : 0;
        if (measured != kTilesTuned) {
            if (route == kRouteWide || route == kRouteDirect || measured == kWideTuned || measured == kDirectTuned)
                choose(false, route == kRouteWide || measured == kWideTuned,
                       may_step && (route == kRouteDirect || measured == kDirectTuned));
            if (!sp.wide && !sp.direct && route < kRouteWide)
                choose(true, route != kRouteNoWide, may_step);
        }
    }
    if ((route == kRouteWide && !sp.wide) || (route == kRouteDirect && !sp.direct))
        return bad(FFS_ERR_UNSUPPORTED, "no wide tile or direct stepping for this problem");
    if (!sp.wide && !sp.direct && sp.radius > 0 && sp.tile - 2 * round_even(sp.radius * sp.tau) < 8)
        return bad(FFS_ERR_UNSUPPORTED, "stencil radius too large for the tile");
    sp.npass_kinds = (sp.tau_last != sp.tau) ? 2 : 1;
    sp.last_kind = sp.npass_kinds - 1;
    if (!sp.wide && !sp.direct && sp.dim == 2 && sp.boundary == FFS_BOUNDARY_FIXED &&
        route != kRouteNoWide)
        sp.strips = strips_win(sp);
    sp.est_seconds = 0.0;
    for (int k = 0; k < sp.npass_kinds; ++k) {
        const int tau = k == 0 ? sp.tau : sp.tau_last;
        geometry(sp, tau, &sp.pass[k]);
        if (sp.wide) {
            wide_geometry(sp, &sp.pass[k]);
            sp.wchunk = std::max(sp.wchunk, wide_chunk(sp, sp.pass[k].nitems));
        }
        if (sp.direct)
            sp.pass[k].nitems = 1;
        else if (!sp.frame)
            band_boxes(sp, &sp.pass[k]);
        if (sp.pass[k].band_max_vol > 0 &&
            band_smem_bytes(sp.pass[k].band_max_vol, (int)sp.taps.size()) > kBandSmemLimit)
            return bad(FFS_ERR_UNSUPPORTED, "fixed-boundary band does not fit shared memory at this tau");
        if (with_data && !sp.wide && !sp.direct) { // (wide tiles: the spectrum is made on the device)
            if (sp.dim == 1 && sp.form == FFS_FORM_FP64_FFT)
                make_spectrum_1d_half(sp, tau, &sp.pass[k].spectrum);
            else if (sp.dim == 1)
                make_spectrum_1d(sp, tau, &sp.pass[k].spectrum);
            else if (sp.dim == 2 && sp.form == FFS_FORM_FP64_FFT && sp.tile == 128)
                make_spectrum_2d128(sp, tau, &sp.pass[k].spectrum);
            else if (sp.dim == 2 && sp.form == FFS_FORM_FP64_FFT)
                make_spectrum_2d_half(sp, tau, &sp.pass[k].spectrum);
            else if (sp.dim == 2 && sp.form != FFS_FORM_FP64_DMMA)
                make_spectrum_2d_natural(sp, tau, &sp.pass[k].spectrum);
            else if (sp.dim == 2)
                make_spectrum_2d(sp, tau, &sp.pass[k].spectrum);
            else if (sp.form == FFS_FORM_FP64_FFT && sp.tile == 32)
                make_spectrum_3d32(sp, tau, &sp.pass[k].spectrum);
            else if (sp.form == FFS_FORM_FP64_FFT)
                make_spectrum_3d_half(sp, tau, &sp.pass[k].spectrum);
            else
                make_spectrum_3d_natural(sp, tau, &sp.pass[k].spectrum);
        }
        const int count = k == 0 ? sp.passes - 1 : 1;
        sp.est_seconds += (sp.npass_kinds == 1 ? sp.passes : count) *
                          (sp.direct ? direct_cost(sp, tau)
                           : sp.wide ? wide_pass_cost(sp, sp.pass[k], 148) : pass_cost(sp, sp.pass[k], 148));
    }
    if (with_data && !sp.wide && !sp.direct) {
        make_tables(&sp);
        if (sp.form == FFS_FORM_OZAKI_I8 || sp.form == FFS_FORM_BF16X3) {
            if (sp.dim == 2)
                make_a_slices(&sp);
            else
                make_f16_slices(&sp);
        }
    }
    *out = std::move(sp);
    return FFS_OK;
}

// Sustained host<->device copy rate of one direction while the other is busy
// (pinned memory, PCIe Gen5 x16), for the slab-count model only.
constexpr double kCopyBytesPerSecond = 48e9;
// Fixed cost of one pass of a slab's sub-plan beyond the modelled tile waves:
// launches, the band kernel's latency (about 30 us for tau = 8 whatever the box
// count), and the first and last waves of a launch of a few hundred tiles.
// Measured on Box2D9P slabs of 4096 x 192..1024 cells, tau 8.  Direct steps have no band, and their model has
// the launch.
constexpr double kSlabPassSeconds = 25e-6;
constexpr int kMaxSlabs = 16;
constexpr int64_t kMinSlabBytes = 4ll << 20;

ffs_problem slab_problem(const PlanSpec &sp, int64_t rows, int open)
{
    ffs_problem q{};
    q.dim = sp.dim;
    q.shape = FFS_SHAPE_CUSTOM;
    q.radius = sp.radius;
    for (int d = 0; d < 3; ++d)
        q.extents[d] = sp.n[d];
    q.extents[sp.dim - 1] = rows;
    q.weights = sp.weights.data();
    q.T = sp.T;
    q.boundary = sp.boundary;
    q.form = sp.form;
    q.slices = sp.slices;
    if (sp.direct)
        q.form = FFS_FORM_AUTO; // direct stepping is the automatic form's
    if (!sp.wide && !sp.direct) { // the whole grid's tile edge and fused step count; a slab of a
        q.tau = sp.tau; // grid on wide tiles or stepped directly chooses its own
        q.tile = sp.tile;
    }
    q.open_faces = open;
    return q;
}

// Slab count for one grid (1 = whole grid).  The environment variable
// FFS_HOST_SLABS forces a count (1 disables the slab path).  Otherwise slabs
// are at least 4 r T rows (ghost rows at most half the stepped rows) and 4 MiB,
// at most 16, and the count with the smallest modelled time wins.
SlabModel slab_model(const PlanSpec &sp)
{
    SlabModel m;
    if (sp.dim < 2 || sp.passes == 0 || sp.open_faces != 0 ||
        (sp.boundary != FFS_BOUNDARY_FIXED && sp.boundary != FFS_BOUNDARY_PERIODIC))
        return m;
    const int axis = sp.dim - 1;
    const int64_t n = sp.n[axis];
    const int64_t row = (int64_t)sp.cells / n;
    const int64_t g = (int64_t)sp.radius * sp.T;
    if (row % 2 != 0 || n < 2) // slab views must start on 16-byte boundaries
        return m;
    const double bytes = (double)sp.cells * sizeof(double);
    m.copy = bytes / kCopyBytesPerSecond;
    m.comp = sp.est_seconds;
    int forced = 0;
    if (const char *env = std::getenv("FFS_HOST_SLABS"))
        forced = std::max(0, std::atoi(env));
    auto model_for = [&](int k, SlabModel *out) {
        const int64_t h = (n + k - 1) / k;
        const int kk = (int)((n + h - 1) / h);
        const bool periodic = sp.boundary == FFS_BOUNDARY_PERIODIC;
        const int64_t rows = periodic ? h + 2 * g : std::min<int64_t>(h + 2 * g, n);
        const int open = periodic ? 0 : (3 << (2 * axis));
        ffs_problem q = slab_problem(sp, rows, open);
        PlanSpec ss;
        std::string why;
        if (build_plan_spec(q, &ss, &why, false) != FFS_OK)
            return false;
        out->count = kk;
        out->a = out->c = (double)h * row * sizeof(double) / kCopyBytesPerSecond;
        out->b = ss.est_seconds + (ss.direct ? 0.0 : ss.passes * kSlabPassSeconds);
        return true;
    };
    if (forced > 0) {
        SlabModel f = m;
        f.forced = true;
        if (forced > 1 && model_for((int)std::min<int64_t>(forced, n), &f))
            return f;
        return f;
    }
    SlabModel best = m;
    double best_t = m.whole(1);
    for (int k = 2; k <= kMaxSlabs; ++k) {
        const int64_t h = (n + k - 1) / k;
        if (h < 4 * g || (double)h * row * sizeof(double) < (double)kMinSlabBytes)
            break;
        SlabModel c = m;
        if (!model_for(k, &c))
            continue;
        const double t = c.slabs(1);
        if (t < best_t) {
            best_t = t;
            best = c;
        }
    }
    return best;
}

void fill_plan_info(const PlanSpec &sp, ffs_plan_info *info)
{
    memset(info, 0, sizeof(*info));
    info->dim = sp.dim;
    info->radius = sp.radius;
    info->form = sp.form;
    info->tile = sp.tile;
    info->tau = sp.tau;
    info->tau_last = sp.tau_last;
    info->passes = sp.passes;
    info->slices = sp.slices;
    info->host_slabs = slab_model(sp).count;
    info->model_ms = sp.est_seconds * 1e3;
    if (sp.passes > 0) {
        const PassSpec &ps = sp.pass[0];
        info->halo = ps.halo;
        info->useful = ps.useful;
        info->tiles = sp.wide || (sp.dim == 2 && sp.tile == 128) ? ps.nitems : ps.nitems * 2;
        const double n = sp.tile;
        // dense DFT-GEMM count: 2 directions x d axes x n^(d+1) complex MACs x 8 flops, per complex tile
        const double dense = 2.0 * sp.dim * std::pow(n, sp.dim + 1) * 8.0;
        // executed: sum of the radices of the factorisation per axis (8(d) rule n -> n1 + n2):
        // 1D 4096 = 8.8.8.8 -> 32, 2D 64 = 8.8 -> 16, 3D 16 = 4.4 -> 8 (32 = 4.8 -> 12) complex MACs per element
        const double rsum = sp.dim == 1 ? 32.0 : (sp.dim == 2 ? 16.0 : (sp.tile == 32 ? 12.0 : 8.0));
        const double exec = 2.0 * sp.dim * std::pow(n, sp.dim) * rsum * 8.0;
        info->flops_per_pass = dense * (double)ps.nitems;
        info->exec_flops_per_pass = exec * (double)ps.nitems;
        if (sp.form == FFS_FORM_OZAKI_I8 || sp.form == FFS_FORM_BF16X3) {
            const double products = sp.slices * (sp.slices + 1) / 2.0;
            if (sp.dim == 2) // dense DFT-64 GEMMs: 4 stages x (128 x 64 x 128) MACs per slice product
                info->exec_flops_per_pass = 4.0 * 2.0 * 128 * 64 * 128 * products * (double)ps.nitems;
            else // dense DFT-16 GEMMs: 6 stages x (256 lines x 32 x 32) MACs per slice product
                info->exec_flops_per_pass = 6.0 * 2.0 * 256 * 32 * 32 * products * (double)ps.nitems;
        }
        if (sp.direct) {
            info->tiles = 1;
            info->flops_per_pass = info->exec_flops_per_pass = 2.0 * (double)sp.taps.size() * ps.tau * (double)sp.cells;
        } else if (sp.wide) {
            // per line of n points: 16-point butterflies of 176 (log16 n, the last of lower
            // radix), 15 twiddles of 6 between them; Ny/2 packed rows forward, Nx/2 + 1 columns
            // both ways, u/2 packed rows back; plus the spectrum product and the packing
            auto line = [](double e) { return e * (std::log2(e) * 176 / 64 + (e > 256 ? 2 : 1) * 90 / 16.0); };
            const double nx = sp.wtile[0], ny = sp.wtile[1];
            if (sp.dim == 1) { // both ways and the spectrum, per pair
                info->flops_per_pass = 2.0 * nx * nx * 8.0 * (double)ps.nitems / 2;
                info->exec_flops_per_pass = (2 * line(nx) + 6.0 * nx) * (double)ps.nitems / 2;
            } else {
                info->flops_per_pass = 2.0 * (nx * nx * ny + nx * ny * ny) * 4.0 * (double)ps.nitems;
                info->exec_flops_per_pass = ((ny + (double)ps.wuseful[1]) / 2 * line(nx) + (nx + 2) * line(ny) +
                                             10.0 * (nx / 2 + 1) * ny) *
                                            (double)ps.nitems;
            }
        } else if (sp.form == FFS_FORM_FP64_FFT && sp.dim == 1) {
            // 256 DFT-64 lines per pair (64 rows, 2 x 64 columns, 64 rows) of 8 x (2 x 56 + 7 x 6),
            // two 4096-point twiddle passes (12 per element: table product and multiply), spectrum
            const double line = 8.0 * (2 * 56 + 7 * 6);
            info->exec_flops_per_pass = (256 * line + (2 * 12.0 + 6.0) * 4096) * (double)ps.nitems;
        } else if (sp.form == FFS_FORM_FP64_FFT && sp.dim == 2 && sp.tile == 128) {
            // per FFT-128 line: 8 threads x (DFT-16 of 176 = eight DFT-4 of 16 and eight
            // twiddle products of 6, fifteen w128 twiddles of 6, two DFT-8 of 60); lines per
            // tile: 64 row pairs, 64 columns forward and inverse, u/2 row pairs; plus the
            // spectrum product (6 per point) and the half-spectrum separation (4 per point)
            const double line = 8.0 * (176 + 15 * 6 + 2 * 60);
            info->exec_flops_per_pass = ((64 + 128 + ps.useful / 2.0) * line + 10.0 * 128 * 65) * (double)ps.nitems;
        } else if (sp.form == FFS_FORM_FP64_FFT && sp.dim == 2) {
            // FP64 operations (add = mul = 1, fma = 2) per DFT-64 line: 8 threads x (two DFT-8
            // of 56 + seven twiddle products of 6); lines per pair: 64 rows, 2 x 64 columns and
            // the u wanted rows; plus the spectrum product (6 per element)
            const double line = 8.0 * (2 * 56 + 7 * 6);
            info->exec_flops_per_pass = ((3 * 64 + ps.useful) * line + 6.0 * 64 * 64) * (double)ps.nitems;
        } else if (sp.form == FFS_FORM_FP64_FFT && sp.tile == 32) {
            // per DFT-32 line (4 x 8): eight DFT-4 of 16, 20 twiddle products of 6 (w32^8 is
            // free), four DFT-8 of 60; lines per pair: 1024 each for z, x and y forward and y
            // inverse, 8 u per CTA (32 u) for inverse x, u^2 for inverse z; plus the spectrum
            const double line = 8 * 16 + 20 * 6 + 4 * 60, u = ps.useful;
            info->exec_flops_per_pass = ((4 * 1024 + 32 * u + u * u) * line + 6.0 * 32768) * (double)ps.nitems;
        } else if (sp.form == FFS_FORM_FP64_FFT) {
            // per DFT-16 line: eight DFT-4 of 16 + eight twiddle products of 6 (w16^4 is free);
            // lines per pair: 256 each for x, y, z forward and z inverse, 16 u for inverse y,
            // u^2 for inverse x; plus the spectrum product
            const double line = 8 * 16 + 8 * 6, u = ps.useful;
            info->exec_flops_per_pass = ((4 * 256 + 16 * u + u * u) * line + 6.0 * 4096) * (double)ps.nitems;
        }
        info->hbm_bytes_per_pass = 16.0 * (double)sp.cells;
    }
}

} // namespace ffst

// Describe without allocating (host only).
static ffs_status describe(const ffs_problem *problem, ffs_plan_info *info, ffst::Route route, const char *who)
{
    if (!problem || !info)
        return ffst::set_error(FFS_ERR_INVALID_ARGUMENT, std::string(who) + ": null argument");
    ffst::PlanSpec sp;
    std::string why;
    ffs_status st = ffst::build_plan_spec(*problem, &sp, &why, false, route);
    if (st != FFS_OK)
        return ffst::set_error(st, why);
    ffst::fill_plan_info(sp, info);
    return FFS_OK;
}

extern "C" ffs_status ffs_plan_describe(const ffs_problem *problem, ffs_plan_info *info)
{
    return describe(problem, info, ffst::kRouteAuto, "ffs_plan_describe");
}

extern "C" ffs_status ffs_plan_describe_tiles(const ffs_problem *problem, ffs_plan_info *info)
{
    return describe(problem, info, ffst::kRouteTiles, "ffs_plan_describe_tiles");
}

// FP64 butterfly form on wide tiles (256 .. 2048 cells per axis, a tile too large for one
// SM's shared memory; 1024 .. 4096 in 1-D): the transform of one line.
//
// A line of N = P P R3 points is transformed by L = N / P threads holding P points each,
// thread t points t + L a (a = 0 .. P - 1).  P = 8 for rows of 256 and 512 and columns of 256,
// else 16; R3 = 2, 4, 8 or 16.
//   n = L n1 + m, m = R3 m1 + m2;  k = k1 + P k2 + P P k3
//   1. DFT-P over n1 (thread m = t), times w_N^(m k1), put at (k1, m)
//   2. get (k1, m2) = (t % P, t / P) over m1, DFT-P, times w_L^(m2 k2), put back in place
//   3. get (k1, k2) with k1 + P k2 = t + L g (g < P / R3) over m2, DFT-R3
// Thread t then holds frequencies t + L a', a' = g + (P / R3) k3: the layout of its input
// points, so a forward transform feeds an inverse one with no reordering, and lanes on
// consecutive t read and write consecutive points.  Two exchanges for every length: with 8
// points a thread the lines of 1024 and more would need a third.
// Exchange slot of (k1, m): k1 * (L + 1) + m.  The odd pitch puts 8 consecutive k1 (steps 2
// and 3) and 8 consecutive m (step 1) on distinct 16-byte bank groups; with C columns side by
// side (slot * C + c) the same holds for every C that is a power of two.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "ffs_fft2d128.cuh"

namespace ffst {
namespace wide {

constexpr int kPad = 16;  // complex slots between the two halves of a packed row

template <int N, int PTS>
struct Shape {
    static constexpr int P = PTS;               // points per thread
    static constexpr int L = N / P;             // threads per line
    static constexpr int R3 = N / (P * P);      // radix of the last step
    static constexpr int PITCH = L + 1;         // exchange pitch of k1
    static constexpr int SLOTS = P * PITCH;
};

// DFT-R of x[0..R) in place, natural order.
template <int R, bool INV>
__device__ __forceinline__ void dft_small(double (&xr)[R], double (&xi)[R])
{
    if constexpr (R == 2) {
        const double ar = xr[0], ai = xi[0];
        xr[0] = ar + xr[1];
        xi[0] = ai + xi[1];
        xr[1] = ar - xr[1];
        xi[1] = ai - xi[1];
    } else if constexpr (R == 4) {
        dft32::dft4<0, 1, INV>(xr, xi);
    } else if constexpr (R == 8) {
        dft32::dft8<0, INV>(xr, xi);
    } else if constexpr (R == 16) {
        f128::dft16<INV>(xr, xi);
    }
}

template <bool INV>
__device__ __forceinline__ void twiddle(double &re, double &im, double2 w)
{
    f128::cmul(re, im, w.x, INV ? -w.y : w.y);
}

// One line's transform.  `sm`: the line's exchange slots (column c of C side by side: sm
// already offset by c).  `tw`: w_N^(m k1) at k1 * L + m (k1 < P), then w_L^(m2 k2) at
// N + P m2 + k2.  `sync` makes the line's threads' shared-memory writes visible to each other.
template <int N, bool INV, int C, int P, class Sync>
__device__ __forceinline__ void line_fft(double (&xr)[P], double (&xi)[P], int t, double2 *sm,
                                         const double2 *__restrict__ tw, Sync sync)
{
    using S = Shape<N, P>;
    dft_small<P, INV>(xr, xi);
    sm[t * C] = make_double2(xr[0], xi[0]);
#pragma unroll
    for (int k1 = 1; k1 < P; ++k1) {
        twiddle<INV>(xr[k1], xi[k1], __ldg(tw + k1 * S::L + t));
        sm[(k1 * S::PITCH + t) * C] = make_double2(xr[k1], xi[k1]);
    }
    sync();
    const int base = (t & (P - 1)) * S::PITCH + t / P;
#pragma unroll
    for (int m1 = 0; m1 < P; ++m1) {
        const double2 v = sm[(base + m1 * S::R3) * C];
        xr[m1] = v.x;
        xi[m1] = v.y;
    }
    dft_small<P, INV>(xr, xi);
    if constexpr (S::R3 > 1) {
        const double2 *tw2 = tw + N + P * (t / P);
        sm[base * C] = make_double2(xr[0], xi[0]);
#pragma unroll
        for (int k2 = 1; k2 < P; ++k2) {
            twiddle<INV>(xr[k2], xi[k2], __ldg(tw2 + k2));
            sm[(base + k2 * S::R3) * C] = make_double2(xr[k2], xi[k2]);
        }
        sync();
        constexpr int G = P / S::R3;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int q = t + S::L * g;
            const int b3 = (q & (P - 1)) * S::PITCH + (q / P) * S::R3;
            double ar[S::R3], ai[S::R3];
#pragma unroll
            for (int m2 = 0; m2 < S::R3; ++m2) {
                const double2 v = sm[(b3 + m2) * C];
                ar[m2] = v.x;
                ai[m2] = v.y;
            }
            dft_small<S::R3, INV>(ar, ai);
#pragma unroll
            for (int k3 = 0; k3 < S::R3; ++k3) {
                xr[g + G * k3] = ar[k3];
                xi[g + G * k3] = ai[k3];
            }
        }
    }
}

} // namespace wide
} // namespace ffst

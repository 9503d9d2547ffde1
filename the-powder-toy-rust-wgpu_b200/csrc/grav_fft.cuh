// grav_fft.cuh -- FP32 FFT convolution for the Newtonian gravity solve.
//
// Same maths as `FftBuffers::solve` (crates/tpt-sim/src/gravity_gpu/mod.rs:
// 204-278): the mass grid zero-padded to N1 x N2, forward 2-D DFT, product
// with the kernel spectra, inverse 2-D DFT, real part of the top-left X x Y
// quadrant where the mask is set. The reference pads to next_pow2(2X) x
// next_pow2(2Y) and runs ~62 launches of global-memory radix-2 passes
// (mod.rs:285-335). Any N1 >= 2X - 1, N2 >= 2Y - 1 gives the same linear
// convolution; here they are the next products of small radices
// (grav_fft_mixed.cuh) and the solve is three launches:
//
//   R  rows forward, two real rows as one complex transform, written as the
//      Hermitian halves kx <= N1/2
//   C  per block of columns kx <= N1/2: forward DFT down the column, products,
//      two inverse DFTs, keeping the Y output rows
//   I  rows inverse: gx + i gy of a row is one complex transform
//
// The kernels Kx(d), Ky(d) = scale d / |d|^3 are odd, so their spectra are
// purely imaginary, i a and i b with real a (even in ky) and b (odd in ky),
// and the whole solve is one complex field: with B the mass spectrum,
//   spectrum of gx + i gy at  kx:  B (i a - b)
//   ... at N1 - kx, conjugated and ky reversed:  B (i a + b)
// so a column of the half spectrum yields the two columns kx and (as its
// conjugate) N1 - kx of the field the row inverse takes. The offset N/2 of an
// even length, which breaks the oddness, is never used by the linear
// convolution and is left out of the kernels.
#pragma once

#include "grav_fft_mixed.cuh"

namespace tpt {
namespace gfft {

// One gravity solve's device state (a plan, or one instance of a batch).
struct Job {
    uint32_t X, Y;
    Axis ax, ay;                  // transforms along x and y
    uint32_t nh, nhp;             // columns kept: N1/2 + 1; their row stride (a multiple of 8)
    uint32_t pitch;               // row stride (elements) of mass, mask, gx, gy
    uint32_t rows_f, rows_i, lc;  // per block: row pairs (R), rows (I), log2 of the columns (C)
    const int32_t *mass_i;        // fixed-point mass, or
    const float *mass_f;          // f32 mass (one of the two is set)
    float mass_scale_inv;
    const uint32_t *mask;
    float2 *work;                 // Y x nhp forward row spectra
    float2 *spec;                 // 2 x Y x nhp: columns kx, then the conjugates of columns N1 - kx
    const float2 *kern;           // N2 x nhp kernel spectra (a, b)
    float *gx, *gy;
};

// Per-call inputs/outputs of a one-job launch, so a solve with new pointers
// needs no table upload.
struct JobIO {
    const int32_t *mass_i;
    const float *mass_f;
    const uint32_t *mask;
    float *gx, *gy;
    float mass_scale_inv;
};

// Block -> (job, item) maps, built on the host once per plan/batch.
struct BlockRef {
    uint32_t job;
    uint32_t item;  // first row pair (R), first column (C) or first row (I)
};

}  // namespace gfft
}  // namespace tpt

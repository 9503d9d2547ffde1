// grav_fft.cu -- kernels and plan of the FP32 FFT gravity solve; see
// grav_fft.cuh for the algorithm and grav_fft_mixed.cuh for the transforms.
#include <math.h>

#include <algorithm>
#include <vector>

#include "grav_fft.cuh"
#include "grav_fft_mixed.cuh"
#include "grav_plan.hpp"
#include "pdl.cuh"

namespace tpt {
namespace gfft {

// Threads per block, and the blocks per SM the registers are capped for (80
// registers). What bounds the passes at this size is latency: a block's chain
// of loads (job, grid, twiddles), barriers and instruction fetch, at 18 to 22
// resident warps per SM and 41 to 46% of the issue slots; DRAM at 10 to 21% of
// its rate (64 grids of sides 32 to 512).
// Measured on B200, solve of 256 grids (8.1 M cells, sides 32 to 512):
// 0.392 ms (0.988 ms with one warp per transform, padded to powers of two and
// exchanged by lane shuffles); one 400x225 grid 20.2 us (55.3); one 1200x701
// grid 63.5 us (698 us with radix-2 passes in shared memory). Blocks of about
// 2048 row points and 4096 column points: 1024 and 1024 took 0.554 ms, 2048
// and 2048 0.479, 4096 and 4096 0.464, 8192 and 4096 0.509 (before the grid
// addresses were hoisted out of the radix loops, at 0.456).
constexpr int NT = 128, NT_LARGE = 256, MIN_BLOCKS = 3;
// Columns whose two buffers stay below this run in blocks of NT threads, eight
// to an SM; the larger ones in their own launch, in blocks of NT_LARGE, so
// that the smaller ones are not held to the larger ones' three blocks per SM.
constexpr size_t COL_SMEM_SMALL = 28 * 1024;

extern __shared__ float2 fft_smem[];

// The block's job in shared memory, copied word by word by the block's
// threads: from the table, or (a one-job call) from the kernel's parameters
// with the call's own pointers, which spares two dependent loads.
static_assert(sizeof(Job) % 4 == 0 && sizeof(Job) / 4 <= NT, "one word per thread");
__device__ __forceinline__ const Job &stage_job(const Job *jobs, const BlockRef *refs, const Job &one, uint32_t per_block,
                                                uint32_t &item) {
    __shared__ __align__(16) uint32_t words[sizeof(Job) / 4];
    uint32_t j = 0;
    if (jobs != nullptr) {
        const BlockRef r = refs[blockIdx.x];
        j = r.job;
        item = r.item;
    } else {
        item = blockIdx.x * per_block;
    }
    const uint32_t *src = reinterpret_cast<const uint32_t *>(jobs != nullptr ? jobs + j : &one);
    if (threadIdx.x < sizeof(Job) / 4) words[threadIdx.x] = src[threadIdx.x];
    __syncthreads();
    return *reinterpret_cast<const Job *>(words);
}

// ---- the three passes ------------------------------------------------------------
// In a one-grid solve they are programmatic dependent launches: the next pass's
// blocks are launched as this one's drain, stage their job, and wait for its
// results.
//
// One function per radix and step: blocks of all lengths share them.
template <int R, bool INV> __device__ __noinline__ void row_step2(const Axis &A, uint32_t cnt) {
    step2<R, INV>(fft_smem, A, RowSeq{}, cnt);
}
template <int R> __device__ __noinline__ void col_step2(const Axis &A, uint32_t lc) {
    step2<R, false>(fft_smem, A, ColSeq{lc}, 1u << lc);
}
template <int R> __device__ __noinline__ void pair_step2(const Axis &A, uint32_t lc) {
    step2<R, true>(fft_smem, A, PairSeq{lc, A.sz << lc}, 2u << lc);
}

// Row pairs y = 2 p, 2 p + 1 (p0 <= p < p0 + cnt) as z = m[2p] + i m[2p+1].
template <int R> __device__ __noinline__ void rows_load(const Job &J, uint32_t p0, uint32_t cnt) {
    const uint32_t m = J.ax.m, X = J.X, Y = J.Y, pitch = J.pitch;
    const bool real = J.mass_f != nullptr;
    const uint32_t *mask = J.mask, *mass = real ? (const uint32_t *)J.mass_f : (const uint32_t *)J.mass_i;
    const float inv = J.mass_scale_inv;
    step1<R>(fft_smem, J.ax, RowSeq{}, cnt, [&](uint32_t c, uint32_t j, float2(&v)[R]) {
        const uint32_t y = 2u * (p0 + c);
        const bool two = y + 1u < Y;
        const size_t o = (size_t)y * pitch + j;
        const uint32_t *mk = mask + o, *ms = mass + o, *mk1 = two ? mk + pitch : mk, *ms1 = two ? ms + pitch : ms;
        // mask and mass are requested together, not one after the other's test
        uint32_t on[R], on1[R], raw[R], raw1[R];
#pragma unroll
        for (int a = 0; a < R; ++a) {
            const bool in = j + m * a < X;
            on[a] = in ? load_after_wait(mk + m * a) : 0u;
            raw[a] = in ? load_after_wait(ms + m * a) : 0u;
            on1[a] = in && two ? load_after_wait(mk1 + m * a) : 0u;
            raw1[a] = in ? load_after_wait(ms1 + m * a) : 0u;
        }
#pragma unroll
        for (int a = 0; a < R; ++a) {
            const float f0 = real ? __uint_as_float(raw[a]) : (float)(int32_t)raw[a] * inv;
            const float f1 = real ? __uint_as_float(raw1[a]) : (float)(int32_t)raw1[a] * inv;
            v[a] = make_float2(on[a] != 0u ? f0 : 0.0f, on1[a] != 0u ? f1 : 0.0f);
        }
    });
}
template <int R> __device__ __noinline__ void rows_last(const Job &J, uint32_t cnt) {
    const Axis &A = J.ax;
    for (uint32_t it = threadIdx.x; it < cnt * A.q; it += blockDim.x) {
        uint32_t c, q;
        RowSeq{}.split(it, A.q, A.div_q, c, q);
        const float2 *t;
        float2 *o = RowSeq{}.at(fft_smem, A, c, item_pos(A, q, t));
        float2 w[R];
#pragma unroll
        for (int i = 0; i < R; ++i) w[i] = o[i];
        dft<R>(w);
#pragma unroll
        for (int i = 0; i < R; ++i) o[i] = w[i];
    }
}

// With Z the transform of z, the rows' spectra are (Z[k] + conj Z[n-k]) / 2
// and -i (Z[k] - conj Z[n-k]) / 2; their halves k <= n/2 go to `work`.
__global__ void __launch_bounds__(NT_LARGE, MIN_BLOCKS) k_rows_forward(const Job *jobs, const BlockRef *refs,
                                                             const __grid_constant__ Job one) {
    uint32_t p0;
    const Job &J = stage_job(jobs, refs, one, one.rows_f, p0);
    pdl_release();
    pdl_wait();
    const Axis &A = J.ax;
    const uint32_t cnt = min(J.rows_f, (J.Y + 1) / 2 - p0);
    with_radix(A.r1, [&](auto R) { rows_load<decltype(R)::value>(J, p0, cnt); });
    __syncthreads();
    if (A.r2 > 1) {
        with_radix(A.r2, [&](auto R) { row_step2<decltype(R)::value, false>(A, cnt); });
        __syncthreads();
    }
    with_radix(A.r3, [&](auto R) { rows_last<decltype(R)::value>(J, cnt); });
    __syncthreads();
    // k = q + Q k3 and n - k: item Q - q, element R3 - 1 - k3 (q = 0: item 0, element R3 - k3 mod R3)
    const uint32_t nh = J.nh, nhp = J.nhp, Y = J.Y;
    for (uint32_t it = threadIdx.x; it < cnt * A.q; it += blockDim.x) {
        uint32_t c, q;
        RowSeq{}.split(it, A.q, A.div_q, c, q);
        const float2 *t;
        const float2 *za = RowSeq{}.at(fft_smem, A, c, item_pos(A, q, t));
        const float2 *zb = RowSeq{}.at(fft_smem, A, c, item_pos(A, q ? A.q - q : 0u, t)) + (q ? A.r3 - 1u : 0u);
        const uint32_t y = 2u * (p0 + c);
        float2 *o = J.work + (size_t)y * nhp + q;
        for (uint32_t i = 0; q + A.q * i < nh; ++i, ++za, o += A.q) {
            const float2 a = *za, b = *zb;
            o[0] = make_float2(0.5f * (a.x + b.x), 0.5f * (a.y - b.y));
            if (y + 1 < Y) o[nhp] = make_float2(0.5f * (a.y + b.y), 0.5f * (b.x - a.x));
            zb = q || i ? zb - 1 : zb + (A.r3 - 1u);
        }
    }
}

template <int R> __device__ __noinline__ void cols_load(const Job &J, uint32_t h0, uint32_t lc) {
    const float2 *work = J.work + h0;
    const uint32_t Y = J.Y, nhp = J.nhp, left = J.nh - h0;
    const uint32_t m = J.ay.m;
    const size_t stride = (size_t)m * nhp;
    step1<R>(fft_smem, J.ay, ColSeq{lc}, 1u << lc, [&](uint32_t c, uint32_t j, float2(&v)[R]) {
        const float2 *p = work + (size_t)j * nhp + c;
        const uint32_t rows = c < left ? Y : 0u;
#pragma unroll
        for (int a = 0; a < R; ++a) v[a] = j + m * a < rows ? load_after_wait(p + a * stride) : make_float2(0.0f, 0.0f);
    });
}
// Step 3, the two products and the inverses' first step. The spectrum of a
// column stays in each item's own places while its products are inverted, the
// first into the second buffer, the second in place.
template <int R> __device__ __noinline__ void cols_products(const Job &J, uint32_t h0, uint32_t lc, float2 *S2) {
    const Axis &A = J.ay;
    const ColSeq sq{lc};
    const uint32_t st = sq.step(1), nhp = J.nhp;
    for (uint32_t it = threadIdx.x; it < A.q << lc; it += blockDim.x) {
        uint32_t c, q;
        sq.split(it, 0, 0, c, q);
        if (h0 + c >= J.nh) continue;
        const float2 *t;
        const uint32_t pos = item_pos(A, q, t);
        float2 *o = sq.at(fft_smem, A, c, pos);
        const float2 *kern = J.kern + (size_t)q * nhp + h0 + c;
        const size_t kstep = (size_t)A.q * nhp;
        float2 w[R];
#pragma unroll
        for (int i = 0; i < R; ++i) w[i] = o[i * st];
        dft<R>(w);
#pragma unroll
        for (int i = 0; i < R; ++i) o[i * st] = w[i];
#pragma unroll 1
        for (int f = 0; f < 2; ++f) {
            const float sgn = f ? 1.0f : -1.0f;
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const float2 k = __ldg(kern + i * kstep), s = o[i * st];
                const float b = sgn * k.y;
                w[i] = make_float2(s.x * b - s.y * k.x, s.x * k.x + s.y * b);
            }
            unstep3<R>(f ? o : sq.at(S2, A, c, pos), st, t, w);
        }
    }
}
template <int R> __device__ __noinline__ void cols_store(const Job &J, uint32_t h0, uint32_t lc) {
    const Axis &A = J.ay;
    const uint32_t Y = J.Y, nhp = J.nhp, left = J.nh - h0, m = A.m;
    const size_t stride = (size_t)m * nhp, second = (size_t)Y * nhp;
    float2 *out = J.spec + h0;
    unstep1<R>(fft_smem, A, PairSeq{lc, A.sz << lc}, 2u << lc, [&](uint32_t c, uint32_t j, const float2(&v)[R]) {
        const uint32_t f = c >> lc, col = c - (f << lc);
        float2 *p = out + (f ? second : 0) + (size_t)j * nhp + col;
        const uint32_t rows = col < left ? Y : 0u;
#pragma unroll
        for (int a = 0; a < R; ++a)
            if (j + m * a < rows) p[a * stride] = v[a];
    });
}

// 1 << lc columns of the half spectrum from h0.
__global__ void __launch_bounds__(NT_LARGE, MIN_BLOCKS) k_columns(const Job *jobs, const BlockRef *refs,
                                                             const __grid_constant__ Job one) {
    uint32_t h0;
    const Job &J = stage_job(jobs, refs, one, 1u << one.lc, h0);
    pdl_release();
    const Axis &A = J.ay;
    const uint32_t lc = J.lc;
    float2 *S2 = fft_smem + ((size_t)A.sz << lc);
    pdl_wait();
    with_radix(A.r1, [&](auto R) { cols_load<decltype(R)::value>(J, h0, lc); });
    __syncthreads();
    if (A.r2 > 1) {
        with_radix(A.r2, [&](auto R) { col_step2<decltype(R)::value>(A, lc); });
        __syncthreads();
    }
    with_radix(A.r3, [&](auto R) { cols_products<decltype(R)::value>(J, h0, lc, S2); });
    __syncthreads();
    if (A.r2 > 1) {
        with_radix(A.r2, [&](auto R) { pair_step2<decltype(R)::value>(A, lc); });
        __syncthreads();
    }
    with_radix(A.r1, [&](auto R) { cols_store<decltype(R)::value>(J, h0, lc); });
}

template <int R> __device__ __noinline__ void rows_first(const Job &J, uint32_t y0, uint32_t cnt) {
    const Axis &A = J.ax;
    const size_t nhp = J.nhp, mirror = (size_t)J.Y * nhp;  // the second plane
    for (uint32_t it = threadIdx.x; it < cnt * A.q; it += blockDim.x) {
        uint32_t c, q;
        RowSeq{}.split(it, A.q, A.div_q, c, q);
        const float2 *t, *row = J.spec + (y0 + c) * nhp;
        float2 *o = RowSeq{}.at(fft_smem, A, c, item_pos(A, q, t));
        // frequency q + Q i: stored up to n/2 (Q R / 2), else as its mirror's
        // conjugate; with an odd radix the middle element depends on q
        const float2 *lo = row + q, *hi = row + mirror + (A.n - q);
        float2 w[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const bool direct = R % 2 == 1 && i == R / 2 ? 2u * (q + A.q * i) <= A.n : i < (R + 1) / 2;
            w[i] = load_after_wait(direct ? lo + A.q * i : hi - A.q * i);
            if (!direct) w[i].y = -w[i].y;
        }
        unstep3<R>(o, 1, t, w);
    }
}
template <int R> __device__ __noinline__ void rows_store(const Job &J, uint32_t y0, uint32_t cnt) {
    const uint32_t X = J.X, m = J.ax.m, pitch = J.pitch;
    const uint32_t *mask = J.mask;
    float *gx = J.gx, *gy = J.gy;
    unstep1<R>(fft_smem, J.ax, RowSeq{}, cnt, [&](uint32_t c, uint32_t j, const float2(&v)[R]) {
        const size_t r = (size_t)(y0 + c) * pitch + j;
        const uint32_t *mk = mask + r;
        float *px = gx + r, *py = gy + r;
        uint32_t on[R];
#pragma unroll
        for (int a = 0; a < R; ++a) on[a] = j + m * a < X ? load_after_wait(mk + m * a) : 0u;
#pragma unroll
        for (int a = 0; a < R; ++a)
            if (j + m * a < X) {
                px[m * a] = on[a] != 0u ? v[a].x : 0.0f;
                py[m * a] = on[a] != 0u ? v[a].y : 0.0f;
            }
    });
}

// Rows y0 .. of gx + i gy, masked.
__global__ void __launch_bounds__(NT_LARGE, MIN_BLOCKS) k_rows_inverse(const Job *jobs, const BlockRef *refs,
                                                             const __grid_constant__ Job one) {
    uint32_t y0;
    const Job &J = stage_job(jobs, refs, one, one.rows_i, y0);
    const Axis &A = J.ax;
    const uint32_t cnt = min(J.rows_i, J.Y - y0);
    pdl_wait();
    with_radix(A.r3, [&](auto R) { rows_first<decltype(R)::value>(J, y0, cnt); });
    __syncthreads();
    if (A.r2 > 1) {
        with_radix(A.r2, [&](auto R) { row_step2<decltype(R)::value, true>(A, cnt); });
        __syncthreads();
    }
    with_radix(A.r1, [&](auto R) { rows_store<decltype(R)::value>(J, y0, cnt); });
}

// ---- kernel spectra, FP64 (once per plan) ---------------------------------
// One length-n transform per block in shared memory (natural order in and
// out), Stockham passes of the radices 2, 3, 4 and 5; tw[k] = exp(-2 pi i k / n).
template <int R>
__device__ __forceinline__ void stockham_pass(const double2 *a, double2 *b, int n, int ns, const double2 *__restrict__ tw) {
    const int step = n / R, tstep = n / (ns * R);
    for (int j = threadIdx.x; j < step; j += blockDim.x) {
        const int p = j % ns;
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const double2 w = __ldg(tw + p * r * tstep), x = a[j + r * step];
            v[r] = make_double2(x.x * w.x - x.y * w.y, x.x * w.y + x.y * w.x);
        }
        double2 *o = b + (j - p) * R + p;
#pragma unroll
        for (int k = 0; k < R; ++k) {
            double2 s = v[0];
#pragma unroll
            for (int r = 1; r < R; ++r) {
                const double2 w = __ldg(tw + (r * k % R) * step);
                s.x += v[r].x * w.x - v[r].y * w.y;
                s.y += v[r].x * w.y + v[r].y * w.x;
            }
            o[k * ns] = s;
        }
    }
}
// Returns the buffer that holds the result; ends after a barrier.
__device__ double2 *stockham_f64(double2 *a, double2 *b, int n, const double2 *__restrict__ tw) {
    int rest = n;
    for (int ns = 1; rest > 1;) {
        const int R = rest % 4 == 0 ? 4 : rest % 2 == 0 ? 2 : rest % 3 == 0 ? 3 : 5;
        if (R == 4) stockham_pass<4>(a, b, n, ns, tw);
        else if (R == 2) stockham_pass<2>(a, b, n, ns, tw);
        else if (R == 3) stockham_pass<3>(a, b, n, ns, tw);
        else stockham_pass<5>(a, b, n, ns, tw);
        __syncthreads();
        double2 *t = a;
        a = b;
        b = t;
        ns *= R;
        rest /= R;
    }
    return a;
}

// build_kernel_field_kernel (crates/tpt-sim/src/gravity_gpu/fft.rs:208-237)
// in double, one row: Kx + i Ky of K(d) = scale * d / |d|^3 with d folded into
// (-N/2, N/2) (the offset N/2 left out), transformed along x.
__global__ void spectrum_rows_f64(double2 *out, uint32_t n1, uint32_t n2, double scale, const double2 *tw1) {
    extern __shared__ double2 smd[];
    const uint32_t y = blockIdx.x;
    const double dy = 2 * y < n2 ? (double)y : (double)y - (double)n2;
    for (uint32_t i = threadIdx.x; i < n1; i += blockDim.x) {
        const double dx = 2 * i < n1 ? (double)i : (double)i - (double)n1;
        double2 v = make_double2(0.0, 0.0);
        if (2 * i != n1 && 2 * y != n2 && (dx != 0.0 || dy != 0.0)) {
            const double d = sqrt(dx * dx + dy * dy), inv = scale / (d * d * d);
            v = make_double2(dx * inv, dy * inv);
        }
        smd[i] = v;
    }
    __syncthreads();
    const double2 *s = stockham_f64(smd, smd + n1, (int)n1, tw1);
    for (uint32_t i = threadIdx.x; i < n1; i += blockDim.x) out[(size_t)y * n1 + i] = s[i];
}

// Column kx = blockIdx.x: the transform along y. Both fields' spectra are
// purely imaginary, i a and i b, so that of Kx + i Ky is -b + i a.
__global__ void spectrum_cols_f64(const double2 *rows, uint32_t n1, uint32_t n2, const double2 *tw2, float2 *kern,
                                  uint32_t nhp) {
    extern __shared__ double2 smd[];
    const uint32_t c = blockIdx.x;
    for (uint32_t j = threadIdx.x; j < n2; j += blockDim.x) smd[j] = rows[(size_t)j * n1 + c];
    __syncthreads();
    const double2 *s = stockham_f64(smd, smd + n2, (int)n2, tw2);
    for (uint32_t j = threadIdx.x; j < n2; j += blockDim.x)
        kern[(size_t)j * nhp + c] = make_float2((float)s[j].y, (float)-s[j].x);
}

// ---- lengths and tables --------------------------------------------------------
// Points of a set's row transforms up to which the set is as a single grid
// (see axis_for): two blocks of 1024 points per SM.
constexpr size_t FEW_POINTS = 2 * 148 * 1024;

// The axis of `cells` cells: the shortest even length that holds the linear
// convolution, 2 cells - 1, as a product of two radices or else of three.
// Neighbouring lengths lie within 1.25 of each other (1.07 on average above
// 256), where padding to a power of two costs up to 2 in each direction.
//
// Of the factorings of that length a batch takes two radices before three:
// fewer steps. A set of few points -- one grid, or a batch below FEW_POINTS --
// is a serial chain instead, with fewer work items than threads, and takes the
// smallest radices. Measured on B200, us per solve of one grid, two radices and
// smallest: 153x96 19.2 and 14.8, 300x64 17.4 and 14.2, 400x225 (no factoring in
// two) 19.5; of 16 grids 153x96 26.7 and 22.6, 64x64 22.2 and 16.4, of 4 20.5 and
// 14.4; 64 of 48x48 20.5 and 18.5, 64 of 64x64 (0.5 million points) 24.5 and 22.6;
// 256 of 32x32 (as many) 22.5 and 28.7, 256 of 48x48 35.0 and 41.0, the mixed 256
// grids 402 and 439.
//
// For the same reason such a set takes no radix above 10 in a short transform,
// even where another length is the price: 72 points are 12 x 6, 80 are 5 x 4 x 4.
// One 33x33 grid (72 and 80 points) 14.3 and 11.2 us per solve, 27.4 and 24.0 with
// the air's launches before it, at errors against 64 bits of 1.14e-7 and 0.97e-7.
// (Radix 10 stays: 64 points instead of its 60 gain 0.8 us and lose a third of
// the precision, 1.01e-7 and 1.35e-7.)
//
// The largest radix r1 loads a column and r3, which has the most work items,
// inverts its two products. Rows have it the other way round: their loading
// step takes two rows of masses and masks per item, and is the longest with a
// large radix. 16x16 10.1 -> 8.7 us, 600x400 30.2 -> 26.6, 256 grids 0.402 ->
// 0.392 ms (columns the same way: 1000x900 64.2 -> 69.4 us).
static bool axis_for(uint32_t cells, bool few, bool rows, Axis *out) {
    const uint32_t need = std::max<uint32_t>(2 * cells - 1, 32u), largest = few && need <= 128 ? 10u : 16u;
    Axis best{};
    for (uint32_t r1 : kRadices)
        for (uint32_t r2 = 1; r2 <= r1; ++r2) {
            if (r2 > 1 && std::find(std::begin(kRadices), std::end(kRadices), r2) == std::end(kRadices)) continue;
            for (uint32_t r3 : kRadices) {
                const uint32_t n = r1 * r2 * r3;
                if (r1 > largest || r3 > r1 || n < need || n % 2) continue;
                bool better = best.n == 0 || n < best.n;
                if (n == best.n) {  // r1 is the largest
                    if (few && r1 != best.r1) better = r1 < best.r1;
                    else if (!few && (r2 == 1) != (best.r2 == 1)) better = r2 == 1;
                    else better = r1 + r2 + r3 < best.r1 + best.r2 + best.r3;
                }
                if (better) {
                    best.n = n;
                    best.r1 = r1;
                    best.r2 = r2;
                    best.r3 = r3;
                }
            }
        }
    if (best.n == 0) return false;
    if (rows) std::swap(best.r1, best.r3);
    auto magic = [](uint32_t d) { return (uint32_t)(((1ull << 32) + d - 1) / d); };
    best.m = best.r2 * best.r3;
    best.q = best.r1 * best.r2;
    best.sr = best.r3 | 1u;
    best.sb = (best.r2 * best.sr) | 1u;
    best.sz = best.r1 * best.sb;
    best.div_r1 = magic(best.r1);
    best.div_r3 = magic(best.r3);
    best.div_m = magic(best.m);
    best.div_q = magic(best.q);
    best.div_13 = magic(best.r1 * best.r3);
    *out = best;
    return true;
}

// The fewest work items that a transform has in one step.
static uint32_t fewest_items(const Axis &a) {
    return std::min(std::min(a.m, a.q), a.r2 > 1 ? a.r1 * a.r3 : a.m);
}

// The axis's twiddles (layout: Axis::tw), evaluated in double.
static void fill_twiddles(const Axis &a, std::vector<float2> &t) {
    auto w = [](uint64_t k, uint32_t n) {
        const double p = -2.0 * M_PI * (double)(k % n) / (double)n;
        return make_float2((float)cos(p), (float)sin(p));
    };
    for (uint32_t k = 0; k < a.r1; ++k)
        for (uint32_t j = 0; j < a.m; ++j) t.push_back(w((uint64_t)k * j, a.n));
    if (a.r2 > 1)
        for (uint32_t k = 0; k < a.r2; ++k)
            for (uint32_t j = 0; j < a.r3; ++j) t.push_back(w((uint64_t)k * j, a.m));
}

static int init_kernel_attrs() {
    static bool done = false;
    if (done) return TPT_OK;
    const int most = 227 * 1024;
    const void *fns[] = {(const void *)k_rows_forward, (const void *)k_columns, (const void *)k_rows_inverse,
                         (const void *)spectrum_rows_f64, (const void *)spectrum_cols_f64};
    for (const void *f : fns) {
        cudaFuncAttributes a{};
        TPT_CUDA(cudaFuncGetAttributes(&a, f));
        TPT_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)a.sharedSizeBytes));
    }
    done = true;
    return TPT_OK;
}

// Builds the kernel spectra of an n1 x n2 transform in FP64 and stores them
// rounded. Synchronous.
static int build_spectra(uint32_t n1, uint32_t n2, uint32_t nhp, float2 *kern) {
    auto full_circle = [](uint32_t n) {
        std::vector<double2> t(n);
        for (uint32_t k = 0; k < n; ++k) {
            const double a = -2.0 * M_PI * (double)k / (double)n;
            t[k] = make_double2(cos(a), sin(a));
        }
        return t;
    };
    const double scale = -(double)6.673e-1f / ((double)n1 * (double)n2);
    auto tw1 = full_circle(n1), tw2 = full_circle(n2);
    double2 *buf = nullptr, *t1 = nullptr, *t2 = nullptr;
    cudaError_t e = cudaMalloc(&buf, (size_t)n1 * n2 * sizeof(double2));
    if (e == cudaSuccess) e = cudaMalloc(&t1, n1 * sizeof(double2));
    if (e == cudaSuccess) e = cudaMalloc(&t2, n2 * sizeof(double2));
    if (e == cudaSuccess) e = cudaMemcpy(t1, tw1.data(), n1 * sizeof(double2), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(t2, tw2.data(), n2 * sizeof(double2), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        spectrum_rows_f64<<<n2, 256, 2 * n1 * sizeof(double2)>>>(buf, n1, n2, scale, t1);
        count_launch();
        spectrum_cols_f64<<<n1 / 2 + 1, 256, 2 * n2 * sizeof(double2)>>>(buf, n1, n2, t2, kern, nhp);
        count_launch();
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaDeviceSynchronize();
    }
    cudaFree(buf);
    cudaFree(t1);
    cudaFree(t2);
    if (e != cudaSuccess) TPT_FAIL(e == cudaErrorMemoryAllocation ? TPT_ERR_OUT_OF_MEMORY : TPT_ERR_CUDA,
                                   "gravity spectrum build failed: %s", cudaGetErrorString(e));
    return TPT_OK;
}

// ---- FFT gravity set (one plan or a batch) --------------------------------
int FftSet::create(const std::vector<JobShape> &shapes) {
    int rc = init_kernel_attrs();
    if (rc) return rc;
    destroy();
    const size_t nj = shapes.size();
    jobs_host.assign(nj, Job{});
    size_t work_elems = 0, kern_elems = 0;
    std::vector<size_t> woff(nj), koff(nj);
    struct Size {
        uint32_t n1, n2;
        bool lone;  // a single cell feels no force: a zero kernel, or the transforms' rounding would show
        size_t off;
    };
    std::vector<Size> sizes;     // distinct kernels: the spectra depend on the lengths only
    std::vector<Axis> axes;      // distinct factorings, their twiddle tables
    std::vector<size_t> axes_off;
    std::vector<float2> twh;
    auto axis_index = [&](const Axis &a) {
        return (size_t)(std::find_if(axes.begin(), axes.end(), [&](const Axis &b) {
                            return a.r1 == b.r1 && a.r2 == b.r2 && a.r3 == b.r3;
                        }) - axes.begin());
    };
    auto table = [&](const Axis &a) {
        if (axis_index(a) < axes.size()) return;
        axes.push_back(a);
        axes_off.push_back(twh.size());
        fill_twiddles(a, twh);
    };
    size_t least = 0;  // points of the row transforms, without padding
    for (const JobShape &s : shapes) least += (size_t)s.Y * (2 * s.X - 1);
    const bool few = nj == 1 || least < FEW_POINTS;
    for (size_t j = 0; j < nj; ++j) {
        Job &J = jobs_host[j];
        if (!axis_for(shapes[j].X, few, true, &J.ax) || !axis_for(shapes[j].Y, few, false, &J.ay))
            TPT_FAIL(TPT_ERR_INVALID_DIMS, "gravity grid %ux%u exceeds the longest transform", shapes[j].X, shapes[j].Y);
        J.X = J.pitch = shapes[j].X;
        J.Y = shapes[j].Y;
        J.nh = J.ax.n / 2 + 1;
        J.nhp = (J.nh + 7) / 8 * 8;
        J.mass_scale_inv = 1.0f / 65536.0f;
        woff[j] = work_elems;
        work_elems += (size_t)J.Y * J.nhp;
        const bool lone = J.X == 1 && J.Y == 1;
        auto it = std::find_if(sizes.begin(), sizes.end(),
                               [&](const Size &s) { return s.n1 == J.ax.n && s.n2 == J.ay.n && s.lone == lone; });
        if (it == sizes.end()) {
            sizes.push_back({J.ax.n, J.ay.n, lone, kern_elems});
            koff[j] = kern_elems;
            kern_elems += (size_t)J.ay.n * J.nhp;
        } else {
            koff[j] = it->off;
        }
        table(J.ax);
        table(J.ay);
    }
    TPT_CUDA(cudaMalloc(&work, std::max<size_t>(work_elems, 1) * sizeof(float2)));
    TPT_CUDA(cudaMalloc(&spec, std::max<size_t>(2 * work_elems, 1) * sizeof(float2)));
    TPT_CUDA(cudaMalloc(&kern, std::max<size_t>(kern_elems, 1) * sizeof(float2)));
    TPT_CUDA(cudaMemset(kern, 0, std::max<size_t>(kern_elems, 1) * sizeof(float2)));
    TPT_CUDA(cudaMalloc(&tw, std::max<size_t>(twh.size(), 1) * sizeof(float2)));
    TPT_CUDA(cudaMemcpy(tw, twh.data(), twh.size() * sizeof(float2), cudaMemcpyHostToDevice));
    for (const Size &s : sizes) {
        if (s.lone) continue;  // zeroed above
        rc = build_spectra(s.n1, s.n2, (s.n1 / 2 + 1 + 7) / 8 * 8, kern + s.off);
        if (rc) return rc;
    }
    auto tw_of = [&](const Axis &a) { return tw + axes_off[axis_index(a)]; };
    // Per block about `per` points of rows and twice that of columns (two to
    // four work items per thread in each step: the job's staging and the code
    // fetched serve all of them), fewer while that leaves SMs idle.
    size_t points = 0;
    for (const Job &J : jobs_host) points += (size_t)J.Y * J.ax.n;
    uint32_t per = 2048;
    while (per > 512 && points / per < 2 * 148) per /= 2;
    // The columns of many small grids make blocks enough at any width: 256 grids of
    // 16x16 in twos 18.5 us per solve, in fours 17.1 (23.0 and 17.1 as ordinary
    // launches, the step beside the air 27.5 and 23.0).
    auto few_blocks = [&](uint32_t lc) {
        size_t blocks = 0;
        for (const Job &J : jobs_host) blocks += (J.nh + (1u << lc) - 1) >> lc;
        return points / per < 2 * 148 && blocks < 2 * 148;
    };
    std::vector<BlockRef> list[4];  // rows forward, columns, rows inverse, longer columns
    size_t smem[4] = {};
    for (size_t j = 0; j < nj; ++j) {
        Job &J = jobs_host[j];
        J.work = work + woff[j];
        J.spec = spec + 2 * woff[j];
        J.kern = kern + koff[j];
        J.ax.tw = tw_of(J.ax);
        J.ay.tw = tw_of(J.ay);
        J.rows_f = J.rows_i = std::max<uint32_t>(1u, per / J.ax.n);
        // columns: at least 4 (32-byte pieces of the rows), 2 when there are
        // few blocks or their two buffers would leave one block per SM (two, for
        // one grid: 1200x701 62.5 -> 52.8 us), and 1 when even those would
        // (1500x1500 181 -> 157 us)
        J.lc = 2;
        while (J.lc < 5 && (J.ay.n << (J.lc + 1)) <= 2 * per) ++J.lc;
        auto col_smem = [&J]() { return ((size_t)J.ay.sz << J.lc) * 2 * sizeof(float2); };
        while (J.lc > 1 && (few_blocks(J.lc) || col_smem() > (nj == 1 ? 72u : 100u) * 1024)) --J.lc;
        if (col_smem() > 100 * 1024) J.lc = 0;
        for (uint32_t p = 0; p < (J.Y + 1) / 2; p += J.rows_f) list[0].push_back({(uint32_t)j, p});
        const size_t csm = ((size_t)J.ay.sz << J.lc) * 2 * sizeof(float2);
        const int pc = csm <= COL_SMEM_SMALL ? 1 : 3;
        for (uint32_t h = 0; h < J.nh; h += 1u << J.lc) list[pc].push_back({(uint32_t)j, h});
        for (uint32_t y = 0; y < J.Y; y += J.rows_i) list[2].push_back({(uint32_t)j, y});
        smem[0] = std::max(smem[0], J.rows_f * J.ax.sz * sizeof(float2));
        smem[pc] = std::max(smem[pc], csm);
        smem[2] = std::max(smem[2], J.rows_i * J.ax.sz * sizeof(float2));
    }
    std::vector<BlockRef> all;
    Pass *passes[4] = {&rows, &cols[0], &inv, &cols[1]};
    for (int p = 0; p < 4; ++p) {
        // longest first, blocks of one length together (they run the same code)
        std::stable_sort(list[p].begin(), list[p].end(), [&](const BlockRef &a, const BlockRef &b) {
            const Job &ja = jobs_host[a.job], &jb = jobs_host[b.job];
            return p & 1 ? ja.ay.n > jb.ay.n : ja.ax.n > jb.ax.n;
        });
        passes[p]->first = (uint32_t)all.size();
        passes[p]->blocks = (uint32_t)list[p].size();
        passes[p]->smem = smem[p];
        // the first pass of one grid has few blocks, of a pair of rows each when
        // they are long: a thread for every item (1200x701 67.4 -> 62.5 us)
        const bool few = p == 0 && nj == 1 && list[p].size() < 3 * 148 && fewest_items(jobs_host[0].ax) > NT;
        passes[p]->threads = p == 3 || few ? NT_LARGE : NT;
        all.insert(all.end(), list[p].begin(), list[p].end());
    }
    TPT_CUDA(cudaMalloc(&jobs, std::max<size_t>(nj, 1) * sizeof(Job)));
    TPT_CUDA(cudaMalloc(&refs, std::max<size_t>(all.size(), 1) * sizeof(BlockRef)));
    TPT_CUDA(cudaMemcpy(refs, all.data(), all.size() * sizeof(BlockRef), cudaMemcpyHostToDevice));
    return upload_jobs();
}

int FftSet::upload_jobs() {
    TPT_CUDA(cudaMemcpy(jobs, jobs_host.data(), jobs_host.size() * sizeof(Job), cudaMemcpyHostToDevice));
    return TPT_OK;
}

int FftSet::set_io(size_t j, const int32_t *mass_i, const float *mass_f, float inv, const uint32_t *mask, float *gx,
                   float *gy, uint32_t pitch) {
    Job &J = jobs_host[j];
    J.pitch = pitch;
    bool changed = J.mass_i != mass_i || J.mass_f != mass_f || J.mass_scale_inv != inv || J.mask != mask ||
                   J.gx != gx || J.gy != gy;
    J.mass_i = mass_i;
    J.mass_f = mass_f;
    J.mass_scale_inv = inv;
    J.mask = mask;
    J.gx = gx;
    J.gy = gy;
    return changed ? 1 : 0;
}

int FftSet::launch(cudaStream_t st, const JobIO *io) const {
    if (rows.blocks == 0) return TPT_OK;
    Job one{};
    if (io) {
        one = jobs_host[0];
        one.mass_i = io->mass_i;
        one.mass_f = io->mass_f;
        one.mask = io->mask;
        one.gx = io->gx;
        one.gy = io->gy;
        one.mass_scale_inv = io->mass_scale_inv;
    }
    // Every pass of a one-grid solve is a programmatic dependent of the one
    // before it, the first of the work before the solve: it waits for that to
    // complete, and only its launch overlaps it (a gravity tick of 153x96 cells
    // and 117,500 particles, with its other kernels dependent too, 36.2 -> 29.3
    // us; a solve of 400x225 cells 22.6 -> 20.9). A batch's passes are ordinary
    // launches: blocks that wait take their places among those of the air
    // kernels running beside them. Alone they are 1 to 6 us slower, but a step is
    // faster, us with dependent and ordinary ones: 2 grids of 400x225 33.7 and
    // 30.5, 16 of 64x64 23.5 and 21.8, 64 of 48x48 35.1 and 30.7, 16 of 153x96 43.5 and
    // 37.7, 256 of 24x24 34.6 and 29.7, the mixed 256 grids 815 and 813 (64 of
    // 100x100 94.5 and 95.6).
    auto run = [&](void (*kernel)(const Job *, const BlockRef *, const Job), const Pass &p) -> int {
        if (p.blocks == 0) return TPT_OK;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(p.blocks);
        cfg.blockDim = dim3(p.threads);
        cfg.dynamicSmemBytes = p.smem;
        cfg.stream = st;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at.val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = &at;
        cfg.numAttrs = io ? 1 : 0;
        TPT_CUDA(cudaLaunchKernelEx(&cfg, kernel, io ? (const Job *)nullptr : (const Job *)jobs,
                                    (const BlockRef *)(refs + p.first), one));
        TPT_LAUNCHED();
        return TPT_OK;
    };
    int rc = run(k_rows_forward, rows);
    if (rc == TPT_OK) rc = run(k_columns, cols[1]);
    if (rc == TPT_OK) rc = run(k_columns, cols[0]);
    if (rc == TPT_OK) rc = run(k_rows_inverse, inv);
    return rc;
}

void FftSet::destroy() {
    cudaFree(work);
    cudaFree(spec);
    cudaFree(kern);
    cudaFree(tw);
    cudaFree(jobs);
    cudaFree(refs);
    work = spec = kern = tw = nullptr;
    jobs = nullptr;
    refs = nullptr;
    jobs_host.clear();
    rows = cols[0] = cols[1] = inv = Pass{};
}

}  // namespace gfft
}  // namespace tpt

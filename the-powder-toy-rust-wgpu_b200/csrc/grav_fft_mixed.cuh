// grav_fft_mixed.cuh -- 1-D DFTs of mixed-radix length n = R1 * R2 * R3 for a
// thread block (R2 = 1: two radices), each radix an in-register DFT of one
// thread, the sequence in shared memory between the steps.
//
// With m = R2 * R3 and j = j3 + R3 j2 an index below m, the forward transform
// of x[j + m a] is
//
//   1  DFT over a -> k1, times W_n^(j k1)             m work items
//   2  (R2 > 1) DFT over j2 -> k2, times W_m^(j3 k2)  R1 R3 items
//   3  DFT over j3 -> k3                              Q = R1 R2 items
//
// and leaves X[q + Q k3] in element k3 of item q = k1 + R1 k2: natural
// frequency order, so spectra need no permutation anywhere. The inverse runs
// the steps backwards with conjugate twiddles and is unnormalised. In shared
// memory element (k1, j2, j3) is at k1 * sb + j2 * sr + j3, sr and sb odd, so
// the items of neighbouring threads lie in different banks.
//
// The steps' radices are run-time values of the axis: every length shares the
// code of its radices (4 to 16 points, one function per radix and step). What
// bounds a transform this short is instruction fetch: a first form of this
// file with one function per length and radices up to 32 executed 2700
// instructions once per warp (44 KB of code) and issued on 12% of the cycles,
// 5.7 of 11 stalled warps per issue waiting for instructions; the registers of
// one warp exchanged by lane shuffles, the form before, waited the same way.
#pragma once

#include <utility>

#include "common.cuh"

namespace tpt {
namespace gfft {

// f(integral_constant<int, 0>) .. f(integral_constant<int, N - 1>): loops
// whose index must be a constant (register arrays, twiddle constants).
template <int N, int I = 0, typename F> __device__ __forceinline__ void sfor(F &&f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        sfor<N, I + 1>(f);
    }
}

// ---- constants -----------------------------------------------------------
constexpr double kPi = 3.14159265358979323846;
// sin and cos of |x| <= pi / 4 by their Taylor series (terms below 1e-17)
constexpr double sin_series(double x) {
    double t = x, s = x;
    for (int k = 1; k < 12; ++k) {
        t *= -x * x / (double)((2 * k) * (2 * k + 1));
        s += t;
    }
    return s;
}
constexpr double cos_series(double x) {
    double t = 1.0, s = 1.0;
    for (int k = 1; k < 12; ++k) {
        t *= -x * x / (double)((2 * k - 1) * (2 * k));
        s += t;
    }
    return s;
}
// cos(2 pi k / n), sin(2 pi k / n), reduced to the first octant
constexpr double cos_2pi(int k, int n);
constexpr double sin_2pi(int k, int n) {
    k %= n;
    if (2 * k >= n) return 2 * k == n ? 0.0 : -sin_2pi(n - k, n);
    if (4 * k > n) return 4 * k == n ? 1.0 : (2 * (n - 2 * k) == 0 ? 0.0 : sin_2pi(n - 2 * k, 2 * n));
    if (8 * k <= n) return sin_series(2.0 * kPi * k / n);
    return cos_series(kPi * (n - 4 * k) / (2.0 * n));
}
constexpr double cos_2pi(int k, int n) {
    k %= n;
    if (2 * k > n) k = n - k;
    if (4 * k > n) return 2 * k == n ? -1.0 : -cos_2pi(n - 2 * k, 2 * n);
    if (8 * k <= n) return cos_series(2.0 * kPi * k / n);
    return sin_series(kPi * (n - 4 * k) / (2.0 * n));
}

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * conj(b)
__device__ __forceinline__ float2 cmulcf(float2 a, float2 b) {
    return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}

// a * exp(-2 pi i K / R)
template <int K, int R> __device__ __forceinline__ float2 ctwid(float2 a) {
    constexpr int k = K % R;
    if constexpr (k == 0) {
        return a;
    } else if constexpr (4 * k == R) {
        return make_float2(a.y, -a.x);
    } else if constexpr (2 * k == R) {
        return make_float2(-a.x, -a.y);
    } else if constexpr (4 * k == 3 * R) {
        return make_float2(-a.y, a.x);
    } else if constexpr (8 * k == R) {
        constexpr float h = (float)0.70710678118654752440;
        return make_float2(h * (a.x + a.y), h * (a.y - a.x));
    } else if constexpr (8 * k == 3 * R) {
        constexpr float h = (float)0.70710678118654752440;
        return make_float2(h * (a.y - a.x), -h * (a.x + a.y));
    } else {
        constexpr float c = (float)cos_2pi(k, R), s = (float)sin_2pi(k, R);
        return make_float2(a.x * c + a.y * s, a.y * c - a.x * s);
    }
}

// ---- in-register DFTs, natural order in and out ---------------------------
constexpr int gcd_c(int a, int b) { return b == 0 ? a : gcd_c(b, a % b); }
// x with a x = 1 (mod m)
constexpr int inv_mod(int a, int m) {
    for (int x = 1; x < m; ++x)
        if (a * x % m == 1) return x;
    return 1 % m;
}
// Splitting of a composite radix into P * Q: coprime factors where there are
// any (the Good-Thomas index maps need no twiddles), else 4 x R / 4 or 5 x 5.
constexpr int radix_p(int R) {
    return R % 3 == 0 && R != 3 ? 3 : R % 5 == 0 && R != 5 ? 5 : R % 4 == 0 && R != 4 ? 4 : R % 2 == 0 && R != 2 ? 2 : R;
}

template <int R> __device__ __forceinline__ void dft(float2 (&v)[R]) {
    if constexpr (R == 1) {
    } else if constexpr (R == 2) {
        const float2 a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    } else if constexpr (R == 3) {
        constexpr float s3 = (float)0.86602540378443864676;
        const float2 t = cadd(v[1], v[2]), d = csub(v[1], v[2]);
        const float2 m = make_float2(v[0].x - 0.5f * t.x, v[0].y - 0.5f * t.y);
        v[0] = cadd(v[0], t);
        v[1] = make_float2(m.x + s3 * d.y, m.y - s3 * d.x);
        v[2] = make_float2(m.x - s3 * d.y, m.y + s3 * d.x);
    } else if constexpr (R == 4) {
        const float2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]), d = csub(v[1], v[3]);
        v[0] = cadd(a, c);
        v[2] = csub(a, c);
        v[1] = make_float2(b.x + d.y, b.y - d.x);
        v[3] = make_float2(b.x - d.y, b.y + d.x);
    } else if constexpr (R == 5) {
        constexpr float c1 = (float)cos_2pi(1, 5), c2 = (float)cos_2pi(2, 5), s1 = (float)sin_2pi(1, 5),
                        s2 = (float)sin_2pi(2, 5);
        const float2 a = cadd(v[1], v[4]), b = cadd(v[2], v[3]), d = csub(v[1], v[4]), e = csub(v[2], v[3]);
        const float2 p = make_float2(v[0].x + c1 * a.x + c2 * b.x, v[0].y + c1 * a.y + c2 * b.y);
        const float2 q = make_float2(v[0].x + c2 * a.x + c1 * b.x, v[0].y + c2 * a.y + c1 * b.y);
        const float2 f = make_float2(s1 * d.x + s2 * e.x, s1 * d.y + s2 * e.y);
        const float2 g = make_float2(s2 * d.x - s1 * e.x, s2 * d.y - s1 * e.y);
        v[0] = make_float2(v[0].x + a.x + b.x, v[0].y + a.y + b.y);
        v[1] = make_float2(p.x + f.y, p.y - f.x);
        v[4] = make_float2(p.x - f.y, p.y + f.x);
        v[2] = make_float2(q.x + g.y, q.y - g.x);
        v[3] = make_float2(q.x - g.y, q.y + g.x);
    } else {
        constexpr int P = radix_p(R), Q = R / P;
        static_assert(P < R, "radix");
        constexpr bool coprime = gcd_c(P, Q) == 1;
        float2 t[R];
        // DFT_P of every residue q; t[q + Q k1]
        sfor<Q>([&](auto qi) {
            constexpr int q = decltype(qi)::value;
            float2 u[P];
            sfor<P>([&](auto pi) {
                constexpr int p = decltype(pi)::value;
                u[p] = v[coprime ? (Q * p + P * q) % R : q + Q * p];
            });
            dft<P>(u);
            sfor<P>([&](auto pi) {
                constexpr int p = decltype(pi)::value;
                t[q + Q * p] = ctwid<coprime ? 0 : q * p, R>(u[p]);
            });
        });
        sfor<P>([&](auto pi) {
            constexpr int p = decltype(pi)::value;
            float2 u[Q];
            sfor<Q>([&](auto qi) {
                constexpr int q = decltype(qi)::value;
                u[q] = t[q + Q * p];
            });
            dft<Q>(u);
            sfor<Q>([&](auto qi) {
                constexpr int q = decltype(qi)::value;
                constexpr int k = coprime ? (Q * inv_mod(Q % P, P) * p + P * inv_mod(P % Q, Q) * q) % R : p + P * q;
                v[k] = u[q];
            });
        });
    }
}

// Unnormalised inverse: the forward transform with real and imaginary parts
// exchanged on both sides.
template <int R> __device__ __forceinline__ void idft(float2 (&v)[R]) {
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = make_float2(v[i].y, v[i].x);
    dft<R>(v);
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = make_float2(v[i].y, v[i].x);
}

// ---- block transforms -------------------------------------------------------
// One axis of a job: length, radices and the shared-memory strides.
struct Axis {
    uint32_t n, r1, r2, r3;
    uint32_t m, q;     // R2 R3, R1 R2
    uint32_t sr, sb;   // strides of j2 (R3 made odd) and k1 (R2 sr made odd)
    uint32_t sz;       // one sequence: R1 sb
    uint32_t div_r1, div_r3, div_m, div_q, div_13;  // ceil(2^32 / R1, R3, m, Q, R1 R3)
    const float2 *tw;  // W_n^(j k1) at k1 * m + j, then W_m^(j3 k2) at n + k2 * R3 + j3
};

// x / d for x, d < 2^16 and magic = ceil(2^32 / d), d > 1
__device__ __forceinline__ uint32_t fast_div(uint32_t x, uint32_t magic) { return __umulhi(x, magic); }

// How a block's sequences lie in shared memory: interleaved columns (position
// p of sequence c at (p << lc) + c; neighbouring threads take neighbouring
// columns) or rows one after the other (sz apart; neighbouring threads take
// neighbouring items of a row).
struct ColSeq {
    uint32_t lc;
    __device__ __forceinline__ void split(uint32_t it, uint32_t, uint32_t, uint32_t &c, uint32_t &e) const {
        c = it & ((1u << lc) - 1u);
        e = it >> lc;
    }
    __device__ __forceinline__ float2 *at(float2 *S, const Axis &, uint32_t c, uint32_t pos) const {
        return S + (pos << lc) + c;
    }
    __device__ __forceinline__ uint32_t step(uint32_t stride) const { return stride << lc; }
};
// The columns of both fields: field 0's lie `off` behind field 1's, and its
// items come first. Column c of field f is c + (f << lc).
struct PairSeq {
    uint32_t lc, off;
    __device__ __forceinline__ void split(uint32_t it, uint32_t items, uint32_t, uint32_t &c, uint32_t &e) const {
        const uint32_t half = items << lc, f = it >= half ? 1u : 0u;
        it -= f ? half : 0u;
        c = (it & ((1u << lc) - 1u)) | (f << lc);
        e = it >> lc;
    }
    __device__ __forceinline__ float2 *at(float2 *S, const Axis &, uint32_t c, uint32_t pos) const {
        return S + (pos << lc) + (c & ((1u << lc) - 1u)) + (c >> lc ? 0u : off);
    }
    __device__ __forceinline__ uint32_t step(uint32_t stride) const { return stride << lc; }
};
struct RowSeq {
    __device__ __forceinline__ void split(uint32_t it, uint32_t items, uint32_t magic, uint32_t &c, uint32_t &e) const {
        c = fast_div(it, magic);
        e = it - c * items;
    }
    __device__ __forceinline__ float2 *at(float2 *S, const Axis &A, uint32_t c, uint32_t pos) const {
        return S + c * A.sz + pos;
    }
    __device__ __forceinline__ uint32_t step(uint32_t stride) const { return stride; }
};

// An item's twiddles t[i * stride], requested before its DFT so that their
// latency passes with the data's; radices 12 and 16 have no registers for that
// and load them when they are used.
template <int R> __device__ __forceinline__ void twiddles(float2 (&w)[R], const float2 *t, uint32_t stride) {
    if constexpr (R <= 10) {
#pragma unroll
        for (int i = 0; i < R; ++i) w[i] = __ldg(t + i * stride);
    }
}
template <int R>
__device__ __forceinline__ float2 twiddle(const float2 (&w)[R], const float2 *t, uint32_t stride, int i) {
    return R <= 10 ? w[i] : __ldg(t + i * stride);
}

// Step 1 of `cnt` sequences; load(c, j, v) fills v[a] = x[j + m a] of sequence c.
template <int R, class Seq, class Load>
__device__ __forceinline__ void step1(float2 *S, const Axis &A, const Seq &sq, uint32_t cnt, const Load &load) {
    const uint32_t m = A.m, st = sq.step(A.sb);
    for (uint32_t it = threadIdx.x; it < cnt * m; it += blockDim.x) {
        uint32_t c, j;
        sq.split(it, m, A.div_m, c, j);
        float2 v[R], w[R];
        load(c, j, v);
        twiddles<R>(w, A.tw + j, m);
        dft<R>(v);
        float2 *o = sq.at(S, A, c, j + fast_div(j, A.div_r3) * (A.sr - A.r3));
        o[0] = v[0];
#pragma unroll
        for (int k = 1; k < R; ++k) o[k * st] = cmulf(v[k], twiddle<R>(w, A.tw + j, m, k));
    }
}
// The inverse's last step: store(c, j, v) takes v[a] = x[j + m a].
template <int R, class Seq, class Store>
__device__ __forceinline__ void unstep1(float2 *S, const Axis &A, const Seq &sq, uint32_t cnt, const Store &store) {
    const uint32_t m = A.m, st = sq.step(A.sb);
    for (uint32_t it = threadIdx.x; it < cnt * m; it += blockDim.x) {
        uint32_t c, j;
        sq.split(it, m, A.div_m, c, j);
        const float2 *o = sq.at(S, A, c, j + fast_div(j, A.div_r3) * (A.sr - A.r3));
        float2 v[R];
#pragma unroll
        for (int k = 0; k < R; ++k) v[k] = o[k * st];
        idft<R>(v);
        store(c, j, v);
    }
}
// Step 2, and its inverse (which also takes out step 1's twiddles).
template <int R, bool INV, class Seq>
__device__ __forceinline__ void step2(float2 *S, const Axis &A, const Seq &sq, uint32_t cnt) {
    const uint32_t items = A.r1 * A.r3, st = sq.step(A.sr), r3 = A.r3;
    for (uint32_t it = threadIdx.x; it < cnt * items; it += blockDim.x) {
        uint32_t c, e;
        sq.split(it, items, A.div_13, c, e);
        const uint32_t k1 = fast_div(e, A.div_r3), j3 = e - k1 * r3;
        float2 *o = sq.at(S, A, c, k1 * A.sb + j3);
        const float2 *t = A.tw + (INV ? k1 * A.m : A.n) + j3;
        float2 v[R], w[R];
        twiddles<R>(w, t, r3);
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = o[i * st];
        if (INV) {
            idft<R>(v);
#pragma unroll
            for (int i = 0; i < R; ++i) o[i * st] = cmulcf(v[i], twiddle<R>(w, t, r3, i));
        } else {
            dft<R>(v);
            o[0] = v[0];
#pragma unroll
            for (int i = 1; i < R; ++i) o[i * st] = cmulf(v[i], twiddle<R>(w, t, r3, i));
        }
    }
}
// Position of item q's elements for step 3, and the twiddles its inverse
// applies: step 2's, or step 1's where there is no step 2.
__device__ __forceinline__ uint32_t item_pos(const Axis &A, uint32_t q, const float2 *&t) {
    const uint32_t k2 = fast_div(q, A.div_r1), k1 = q - k2 * A.r1;
    t = A.r2 > 1 ? A.tw + A.n + k2 * A.r3 : A.tw + k1 * A.m;
    return k1 * A.sb + k2 * A.sr;
}
// The inverse's first step of one item: w[k3] = X[q + Q k3] into S.
template <int R> __device__ __forceinline__ void unstep3(float2 *o, uint32_t st, const float2 *t, float2 (&w)[R]) {
    float2 u[R];
    twiddles<R>(u, t, 1);
    idft<R>(w);
#pragma unroll
    for (int i = 0; i < R; ++i) o[i * st] = cmulcf(w[i], twiddle<R>(u, t, 1, i));
}

// The radices: f(integral_constant<int, R>) for the run-time value r.
template <typename F> __device__ __forceinline__ void with_radix(uint32_t r, F &&f) {
    switch (r) {
        case 4: f(std::integral_constant<int, 4>{}); break;
        case 5: f(std::integral_constant<int, 5>{}); break;
        case 6: f(std::integral_constant<int, 6>{}); break;
        case 8: f(std::integral_constant<int, 8>{}); break;
        case 10: f(std::integral_constant<int, 10>{}); break;
        case 12: f(std::integral_constant<int, 12>{}); break;
        case 16: f(std::integral_constant<int, 16>{}); break;
        default: break;
    }
}
constexpr uint32_t kRadices[] = {4, 5, 6, 8, 10, 12, 16};

}  // namespace gfft
}  // namespace tpt

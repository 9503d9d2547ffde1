// air_strip.cuh -- the three passes of an air tick as warp strips.
//
// One warp owns a strip of 26 to 30 columns and walks down its rows: a lane
// holds a column, the 3 to 1 lanes on either side are the stages' halo. A
// stage's y neighbours are the lane's own registers from earlier rows, its x
// neighbours come by shuffles, blocked cells are bits of ballots (one word
// per row, so the tests of a whole 3x3 neighbourhood are a few word
// operations), and nothing is exchanged between warps: no shared memory and
// no barriers. Only the far-advection walks and samples read memory at an
// arbitrary cell (L1 mostly: the rows around were just read).
//
// A 3x3 mean adds its nine taps row by row, so a cell's sum starts when its
// own row arrives (taps of the row above and of its own) and ends with the
// next row; each loaded value is multiplied once per weight, not once per
// tap that uses it. The operations and their order are those of the per-cell
// code in air.cuh, each rounded separately (-fmad=false): the results are the
// same bits.
//
// What bounds the passes is instruction issue and the latency between a warp's
// dependent instructions: on 5.8 M cells they issue on 61% of the cycles with 24
// warps per SM, 43 warp instructions per cell, and their time falls with every
// further resident warp (3 CTAs of 4 warps per SM 0.59 ms, 4 0.49, 5 0.43, 6
// 0.38), so the advection and heat passes are capped at 80 registers: 96 and 108
// (no spills, 5 and 4 CTAs) took 0.392 and 0.418 ms where 80 took 0.376, 72 and
// 64 spill and took 0.413 and 0.460. For the same reason advection and heat are
// two passes: as one (128 registers, 16 warps) 0.60 ms against 0.56.
// The tiles of one thread per cell (32x8 cells and their halo in shared memory,
// air_tiles.cu) execute 58 warp instructions per cell: every tap is a shared
// load with its own mask load, test and product, the halo ring is recomputed
// (1.33 of the cells for the advection, 1.69 for the vorticity), the warps are
// unevenly filled on the rings, and barriers separate the stages. Measured on
// B200, air per tick, tiles and strips: 8.1 M cells in 256 grids 0.613 and 0.454
// ms, 6.1 M in 128 grids 0.440 and 0.347 ms, one 2048x2048 grid 0.378 and 0.246.
#pragma once

#include "air.cuh"
#include "air_launch.hpp"

namespace tpt {
namespace air {

// A lane's bits of a row's word: 1 its left neighbour's, 2 its own, 4 its right
// neighbour's.
__device__ __forceinline__ uint32_t around(uint32_t row, uint32_t lane) {
    return __funnelshift_r(row << 1, row >> 31, lane) & 7u;
}

// What a strip knows of its columns; the words' bit l is lane l.
struct StripCols {
    uint32_t lane;
    int x;
    bool in;               // x in the grid
    uint32_t not_inner;    // x < 1 or x + 1 >= X
    __device__ __forceinline__ StripCols(const AirInst &I, int x0, int halo) {
        lane = threadIdx.x & 31u;
        x = x0 - halo + (int)lane;
        const int X = (int)I.X;
        in = x >= 0 && x < X;
        not_inner = __ballot_sync(~0u, x < 1 || x + 1 >= X);
    }
    __device__ __forceinline__ bool output(int halo) const {
        return in && (int)lane >= halo && (int)lane < 32 - halo;
    }
};

__device__ __forceinline__ float left_of(float v) { return __shfl_up_sync(~0u, v, 1); }
__device__ __forceinline__ float right_of(float v) { return __shfl_down_sync(~0u, v, 1); }

// ---- pass A: pressure and velocity (pressure.rs:173-299) ----------------------
// Rows y0 .. y1 - 1 of the strip at x0. The step that loads row r forms the
// effective velocity of row r - 1, the pressure of row r - 2 and the velocity
// of row r - 3; a name's digit is the age of its row.
__device__ __forceinline__ void strip_a(const StripGrids &P, const AirInst &I, uint32_t off, int x0, int y0, int y1) {
    const StripCols C(I, x0, VELOCITY_HALO);
    const int Y = (int)I.Y;
    const uint32_t pitch = I.pitch, inner = ~C.not_inner, bit = 1u << C.lane;
    const bool rim = C.x < 2 || C.x + 2 >= (int)I.X, mid = (inner & bit) != 0u;
    const uint32_t m_left = __ballot_sync(~0u, C.x >= 2), m_right = __ballot_sync(~0u, C.x + 2 < (int)I.X);
    const bool out = C.output(VELOCITY_HALO);
    const float evx = I.evx, evy = I.evy, ep = I.ep;
    float vx1 = 0.f, vy1 = 0.f, pv1 = 0.f, pv2 = 0.f;
    uint32_t b1 = 0u, b2 = 0u, b3 = 0u, b4 = 0u;
    float ex2 = 0.f, ey2 = 0.f, ex3 = 0.f, ey3 = 0.f, p3 = 0.f, p4 = 0.f;
    uint32_t o = off + (uint32_t)(y0 - 3) * pitch + (uint32_t)C.x;  // row r
    float nvx = 0.f, nvy = 0.f, npv = 0.f;
    uint32_t nb = 0u;
    auto load = [&](int r, uint32_t e) {  // the next row's loads are in flight during a step
        const bool ok = C.in && r >= 0 && r < Y;
        nvx = ok ? load_after_wait(P.vx + e) : 0.f;
        nvy = ok ? load_after_wait(P.vy + e) : 0.f;
        npv = ok ? load_after_wait(P.pv + e) : 0.f;
        nb = ok ? load_after_wait(P.bair + e) : 0u;
    };
    load(y0 - 3, o);
#pragma unroll 1
    for (int r = y0 - 3; r < y1 + 3; ++r, o += pitch) {
        const float vx0 = nvx, vy0 = nvy, pv0 = npv;
        const uint32_t b0 = __ballot_sync(~0u, nb != 0u);
        load(r + 1, o + pitch);
        // effective_vx / vy (pressure.rs:119-157) of row e = r - 1
        const int e = r - 1;
        const bool ein = e >= 1 && e + 1 < Y;
        float ex = vx1, ey = vy1;
        if (e < 2 || e + 2 >= Y || rim) {
            ex = evx + (ex - evx) * 0.9f;
            ey = evy + (ey - evy) * 0.9f;
        }
        // wall_cleared_vx / vy (pressure.rs:43-85)
        const uint32_t clx = ein ? (b1 & inner) | ((b1 << 1) & m_left) | ((b1 >> 1) & m_right) : 0u;
        const uint32_t cly = ((ein ? b1 : 0u) | (e >= 2 ? b2 : 0u) | (e + 2 < Y ? b0 : 0u)) & inner;
        if (clx & bit) ex = 0.0f;
        if (cly & bit) ey = 0.0f;
        // air_pressure_kernel (pressure.rs:186-237) of row p = r - 2
        const int p = r - 2;
        float p2 = pv2;
        if (p < 2 || p + 2 >= Y || rim) p2 = ep + (p2 - ep) * 0.8f;
        const float exl = left_of(ex2), exr = right_of(ex2);
        if (p >= 1 && p + 1 < Y && mid) {
            const float dp = exl - exr + ey3 - ey;
            p2 = ep + (p2 - ep) * 0.9999f + dp * 0.15f;
        }
        // air_velocity_kernel (pressure.rs:260-298) of row v = r - 3
        const int v = r - 3;
        const float pl = left_of(p3), pr = right_of(p3);
        if (v >= y0 && v < Y) {
            float ox = ex3, oy = ey3;
            if (v >= 1 && v + 1 < Y && mid) {
                const float dx = pl - pr, dy = p4 - p2;
                ox = evx + (ox - evx) * 0.999f + dx * 0.2f;
                oy = evy + (oy - evy) * 0.999f + dy * 0.2f;
                // adjacent_blocked_x / y (pressure.rs:92-114)
                if (around(b3, C.lane)) ox = 0.0f;
                if ((b4 | b3 | b2) & bit) oy = 0.0f;
            }
            if (out) {
                const uint32_t w = o - 3u * pitch;
                P.ovx[w] = ox;
                P.ovy[w] = oy;
                P.opv[w] = p3;
            }
        }
        b4 = b3, b3 = b2, b2 = b1, b1 = b0;
        ex3 = ex2, ex2 = ex, ey3 = ey2, ey2 = ey;
        p4 = p3, p3 = p2;
        pv2 = pv1, pv1 = pv0, vx1 = vx0, vy1 = vy0;
    }
}

// |v| as the reference takes it: -0 stays -0
__device__ __forceinline__ float magnitude(float v) { return v < 0.0f ? -v : v; }

// ---- 3x3 means --------------------------------------------------------------
constexpr float kEdge = 0.13533528f, kCorner = 0.01831564f;  // smooth_w

// One row's contribution to the means of one field: the products of the
// lane's value and of its two neighbours with the weights.
struct RowTaps {
    float v, l, r;                      // the lane's value and its neighbours'
    float e, c, lc, le, rc, re;         // times the edge and corner weights
    __device__ __forceinline__ explicit RowTaps(float value) {
        v = value;
        l = left_of(v);
        r = right_of(v);
        e = v * kEdge;
        c = v * kCorner;
        lc = l * kCorner;
        le = l * kEdge;
        rc = r * kCorner;
        re = r * kEdge;
    }
};
// What a field keeps of a row for the next one: the taps the next row's cells
// take from it as the row above, its centre products, and its cells' sums so far.
struct RowState {
    float lc, e, rc, c, s;
};
// Which of a row's three cells around a lane are closed (blocked or not
// interior): a closed cell's tap is the centre's value (advect.rs:205-253).
struct Closed {
    bool l, m, r;
    __device__ __forceinline__ explicit Closed(uint32_t bits) : l(bits & 1u), m(bits & 2u), r(bits & 4u) {}
};
// The sum of the row above's cells, finished with this row's taps.
__device__ __forceinline__ float finish_sum(const RowState &a, const RowTaps &t, const Closed &k) {
    float s = a.s + (k.l ? a.c : t.lc);
    s = s + (k.m ? a.e : t.e);
    return s + (k.r ? a.c : t.rc);
}
// This row's sums begun: the row above (ka its closed cells), then its own.
__device__ __forceinline__ void start_sum(RowState &a, const RowTaps &t, const Closed &ka, const Closed &k) {
    float s = 0.0f + (ka.l ? t.c : a.lc);
    s = s + (ka.m ? t.e : a.e);
    s = s + (ka.r ? t.c : a.rc);
    s = s + (k.l ? t.e : t.le);
    s = s + t.v;
    s = s + (k.r ? t.e : t.re);
    a = RowState{t.lc, t.e, t.rc, t.c, s};
}
// Two values in one register pair, for the two components of a velocity: one
// instruction adds or multiplies both, each rounded as the single ones are.
struct Pair {
    unsigned long long v;
    __device__ __forceinline__ Pair() : v(0ull) {}
    __device__ __forceinline__ Pair(float a, float b) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b)); }
    __device__ __forceinline__ void get(float &a, float &b) const { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
};
__device__ __forceinline__ Pair add2(Pair a, Pair b) {
    Pair r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ Pair mul2(Pair a, float w) {
    Pair r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(Pair(w, w).v));
    return r;
}
struct RowTaps2 {
    float lx, ly, rx, ry;  // the neighbours' values
    Pair v, e, c, lc, le, rc, re;
    __device__ __forceinline__ RowTaps2(float x, float y) {
        lx = left_of(x), ly = left_of(y), rx = right_of(x), ry = right_of(y);
        const Pair l(lx, ly), r(rx, ry);
        v = Pair(x, y);
        e = mul2(v, kEdge), c = mul2(v, kCorner);
        lc = mul2(l, kCorner), le = mul2(l, kEdge);
        rc = mul2(r, kCorner), re = mul2(r, kEdge);
    }
};
struct RowState2 {
    Pair lc, e, rc, c, s;
};
__device__ __forceinline__ Pair finish_sum(const RowState2 &a, const RowTaps2 &t, const Closed &k) {
    Pair s = add2(a.s, k.l ? a.c : t.lc);
    s = add2(s, k.m ? a.e : t.e);
    return add2(s, k.r ? a.c : t.rc);
}
__device__ __forceinline__ void start_sum(RowState2 &a, const RowTaps2 &t, const Closed &ka, const Closed &k) {
    Pair s = add2(Pair(), ka.l ? t.c : a.lc);
    s = add2(s, ka.m ? t.e : a.e);
    s = add2(s, ka.r ? t.c : a.rc);
    s = add2(s, k.l ? t.e : t.le);
    s = add2(s, t.v);
    s = add2(s, k.r ? t.e : t.re);
    a = RowState2{t.lc, t.e, t.rc, t.c, s};
}

// Three sums over kSmoothWsum: div_by_const's correction step (exact_div.cuh)
// with one test for all three. A sum that starts at +0 is never -0, so zeros
// take the short way too.
__device__ __forceinline__ bool needs_division(float s) {
    const uint32_t b = __float_as_uint(s) & 0x7FFFFFFFu;
    return b != 0u && b - 0x0D800000u > 0x7F7FFFFFu - 0x0D800000u;  // below 2^-100, infinite or NaN
}
__device__ __forceinline__ float short_mean(float s) {
    const float q = __fmul_rn(s, kSmoothWsumRcp);
    return __fmaf_rn(__fmaf_rn(-q, kSmoothWsum, s), kSmoothWsumRcp, q);
}
__device__ __forceinline__ void means_of(float &a, float &b, float &c) {
    if (needs_division(a) || needs_division(b) || needs_division(c)) {
        a = div_by_const(a, kSmoothWsum, kSmoothWsumRcp);
        b = div_by_const(b, kSmoothWsum, kSmoothWsumRcp);
        c = div_by_const(c, kSmoothWsum, kSmoothWsumRcp);
    } else {
        a = short_mean(a);
        b = short_mean(b);
        c = short_mean(c);
    }
}

// The convection direction (heat.rs:182-251) before its per-cell weight: for
// all but radial gravity the same in every cell.
__device__ __forceinline__ void convection_dir(const AirInst &I, int x, int y, float &convx, float &convy) {
    float gxv = 0.0f, gyv = 0.0f;
    if (I.gmode == 0u) {
        gyv = 1.0f;
    } else if (I.gmode == 2u) {
        const float rx = (float)I.X * 0.5f - ((float)x + 0.5f);
        const float ry = (float)I.Y * 0.5f - ((float)y + 0.5f);
        const float rd = sqrtf(rx * rx + ry * ry);
        if (rd > 0.0f) {
            gxv = rx / rd;
            gyv = ry / rd;
        }
    } else if (I.gmode == 3u) {
        gxv = I.cgx;
        gyv = I.cgy;
    }
    convx = 0.0f - gxv;
    convy = 0.0f - gyv;
    if (I.conv == 2u) {
        const float gm = sqrtf(convx * convx + convy * convy);
        if (gm > 10.0f) {
            convx /= 0.1f * gm;
            convy /= 0.1f * gm;
        }
    }
}

// far_advect_target (air.cuh; advect.rs:66-152) with the cell's and the
// limits' float forms, which a strip converts once.
template <typename B>
__device__ __forceinline__ void far_target(float x, float y, float dx, float dy, float limx, float limy, B &&blocked,
                                           float &otx, float &oty) {
    const float ex = dx * 0.7f, ey = dy * 0.7f;
    float tx = x - ex, ty = y - ey;
    if ((fabsf(ex) > 1.0f || fabsf(ey) > 1.0f) && tx >= 2.0f && tx < limx && ty >= 2.0f && ty < limy) {
        const float abs_dx = fabsf(dx), abs_dy = fabsf(dy);
        const bool along = abs_dx > abs_dy;
        const float slope = along ? 0.0f - dy / abs_dx : 0.0f - dx / abs_dy;
        const float sx = along ? (dx < 0.0f ? 1.0f : -1.0f) : slope;
        const float sy = along ? slope : (dy < 0.0f ? 1.0f : -1.0f);
        const int limit = along ? (int)fabsf(ex) : (int)fabsf(ey);
        const int X = (int)limx + 2, Y = (int)limy + 2;
        float wx = x, wy = y;
        for (int step = 0; step < limit; ++step) {
            wx += sx;
            wy += sy;
            const int cx = (int)(wx + 0.5f), cy = (int)(wy + 0.5f);
            bool hit = true;
            if (cx >= 0 && cy >= 0 && cx < X && cy < Y) hit = blocked(cx, cy);
            if (hit) {
                tx = wx - sx;
                ty = wy - sy;
                break;
            }
        }
    }
    otx = tx;
    oty = ty;
}

// clampf(v, -256, 256) of an arithmetic result (its NaN is the canonical one)
__device__ __forceinline__ float clamp_speed(float v) {
    asm("max.NaN.f32 %0, %0, 0fC3800000;\n\tmin.NaN.f32 %0, %0, 0f43800000;" : "+f"(v));
    return v;
}

// Where a backtrace lands: its cell, the weights, and whether the cell lies in
// [lo, X - hi) x [lo, Y - hi) -- for a truncated coordinate and a fraction that
// must not be negative, whether the coordinate itself does (lo >= 0).
struct Landing {
    uint32_t g;  // element of the cell, or of the instance's first cell
    float fx, fy;
    bool ok;
    __device__ __forceinline__ Landing(float tx, float ty, float lo, float endx, float endy, uint32_t off, uint32_t pitch,
                                       bool wanted) {
        ok = wanted && tx >= lo && tx < endx && ty >= lo && ty < endy;
        const int i = (int)tx, j = (int)ty;
        fx = tx - (float)i;
        fy = ty - (float)j;
        g = off + (ok ? (uint32_t)j * pitch + (uint32_t)i : 0u);
    }
    __device__ __forceinline__ float blend(float v00, float v10, float v01, float v11) const {
        const float w00 = (1.0f - fx) * (1.0f - fy);
        const float w10 = fx * (1.0f - fy);
        const float w01 = (1.0f - fx) * fy;
        const float w11 = fx * fy;
        return v00 * w00 + v10 * w10 + v01 * w01 + v11 * w11;
    }
};

// ---- pass B1: smoothing, advection, vorticity, fans (advect.rs:174-360) ---------
// Rows y0 .. y1 - 1 of the strip at x0. The step that loads row r of the
// velocity pass's output finishes the means and the vorticity of row r - 1
// and advects row a = r - 2, whose samples are requested at the step's start.
// The advected velocity goes to `ou` / `ov` where the heat pass follows (which
// reads its neighbours), else to vx / vy; the pressure to pv.
__device__ __forceinline__ void strip_advect(const StripGrids &P, const AirInst &I, float *__restrict__ ou,
                                             float *__restrict__ ov, uint32_t off, int x0, int y0, int y1) {
    const StripCols C(I, x0, ADVECT_HALO);
    const int Y = (int)I.Y;
    const uint32_t pitch = I.pitch, lane = C.lane;
    const bool out = C.output(ADVECT_HALO), deep = C.x > 1 && C.x + 2 < (int)I.X;
    const float xf = (float)C.x, limx = (float)I.X - 2.0f, limy = (float)I.Y - 2.0f, vk = I.vk;
    const bool confine = I.vcoef > 0.0f && deep;
    uint32_t o = off + (uint32_t)(y0 - 2) * pitch + (uint32_t)C.x;  // row r

    RowState2 sv{};                          // means of row r - 1
    RowState sp{};
    uint32_t bk1 = 0u, bk2 = 0u, cl1 = 7u;   // blocked and closed cells around the lane, rows r - 1, r - 2
    float vx1 = 0.f, vx2 = 0.f, dvy1 = 0.f;  // ovx of rows r - 1, r - 2; y part of row r - 1's vorticity
    Pair mv2;                                // sums of row r - 2
    float mp2 = 0.f;
    float w2 = 0.f, w3 = 0.f;                // vorticity of rows r - 2, r - 3
    float nvx = 0.f, nvy = 0.f, npv = 0.f;
    uint32_t nb = 0u, nw = 0u;
    auto load = [&](int r, uint32_t e) {  // the next step's loads are in flight during a step
        const bool ok = C.in && r >= 0 && r < Y, okw = out && r - 2 >= 0 && r - 2 < Y;
        nvx = ok ? load_after_wait(P.ovx + e) : 0.f;
        nvy = ok ? load_after_wait(P.ovy + e) : 0.f;
        npv = ok ? load_after_wait(P.opv + e) : 0.f;
        nb = ok ? load_after_wait(P.bair + e) : 0u;
        nw = okw ? load_after_wait(P.wall + (e - 2u * pitch)) : 0u;
    };
    load(y0 - 2, o);
#pragma unroll 1
    for (int r = y0 - 2; r < y1 + 2; ++r, o += pitch) {
        const float vx0 = nvx, vy0 = nvy, pv0 = npv;
        const uint32_t wall2 = nw;
        const uint32_t row0 = __ballot_sync(~0u, nb != 0u), bk0 = around(row0, lane);
        load(r + 1, o + pitch);
        const int a = r - 2;
        const bool mine = out && a >= y0 && a < Y;
        // backtrace of row a (advect.rs:255-280)
        float nx, ny, np = mp2;
        mv2.get(nx, ny);
        means_of(nx, ny, np);
        float tx = -1.f, ty = -1.f;
        if (mine)
            far_target(xf, (float)a, nx, ny, limx, limy,
                       [&](int cx, int cy) -> bool {
                           return load_after_wait(P.bair + (off + (uint32_t)cy * pitch + (uint32_t)cx)) != 0u;
                       },
                       tx, ty);
        const Landing q(tx, ty, 2.0f, limx - 1.0f, limy - 1.0f, off, pitch, mine && !(bk2 & 2u));
        // both rows of the sample: cells of the grid in any case (it has two rows and columns)
        const float *q0 = P.ovx + q.g, *q1 = P.ovy + q.g;
        const float a00 = load_after_wait(q0), a10 = load_after_wait(q0 + 1), a01 = load_after_wait(q0 + pitch), a11 = load_after_wait(q0 + pitch + 1);
        const float b00 = load_after_wait(q1), b10 = load_after_wait(q1 + 1), b01 = load_after_wait(q1 + pitch), b11 = load_after_wait(q1 + pitch + 1);
        // the means of row r - 1 get this row's taps, row r's begin (advect.rs:192-253)
        const uint32_t cl0 = around(row0 | C.not_inner | (r < 1 || r + 1 >= Y ? ~0u : 0u), lane);
        const Closed k0(cl0), k1(cl1);
        const RowTaps2 tv(vx0, vy0);
        const RowTaps tpv(pv0);
        const Pair mv1 = finish_sum(sv, tv, k0);
        const float mp1 = finish_sum(sp, tpv, k0);
        start_sum(sv, tv, k1, k0);
        start_sum(sp, tpv, k1, k0);
        // vorticity_bmap (advect.rs:10-42) of row r - 1
        float w1 = 0.0f;
        if (deep && r - 1 > 1 && r + 1 < Y) {
            float dvxdy = vx0 - vx2;
            if ((bk0 | bk1 | bk2) & 2u) dvxdy = 0.0f;
            w1 = (dvy1 - dvxdy) * 0.5f;
        }
        dvy1 = tv.ry - tv.ly;
        if (bk0) dvy1 = 0.0f;
        const float wl = left_of(w2), wr = right_of(w2);
        if (mine) {
            if (q.ok) {  // advect.rs:280-295
                nx = nx * 0.7f + 0.3f * q.blend(a00, a10, a01, a11);
                ny = ny * 0.7f + 0.3f * q.blend(b00, b10, b01, b11);
            }
            if (confine && a > 1 && a + 2 < Y) {  // advect.rs:297-328
                const float dwx = (magnitude(wr) - magnitude(wl)) * 0.5f;
                const float dwy = (magnitude(w1) - magnitude(w3)) * 0.5f;
                const float norm = sqrtf(dwx * dwx + dwy * dwy) + 0.001f;
                nx += vk * dwy / norm * w2;
                ny += vk * (0.0f - dwx) / norm * w2;
            }
            const uint32_t w = o - 2u * pitch;
            if (wall2 == 5u) {  // WL_FAN, advect.rs:331-334
                nx += load_after_wait(P.fvx + w);
                ny += load_after_wait(P.fvy + w);
            }
            nx = clamp_speed(nx);
            ny = clamp_speed(ny);
            np = clamp_speed(np);
            if (I.air_mode != 0u) {
                if (I.air_mode == 1u || I.air_mode == 3u) np = 0.0f;
                if (I.air_mode == 2u || I.air_mode == 3u) nx = ny = 0.0f;
            }
            P.pv[w] = np;
            if (I.aheat) {
                ou[w] = nx;
                ov[w] = ny;
            } else {
                P.vx[w] = nx;
                P.vy[w] = ny;
            }
        }
        vx2 = vx1, vx1 = vx0;
        w3 = w2, w2 = w1;
        mv2 = mv1, mp2 = mp1;
        bk2 = bk1, bk1 = bk0, cl1 = cl0;
    }
}

// ---- pass B2: heat, convection (heat.rs:31-253), masks (settle.rs:50-93) --------
// Rows y0 .. y1 - 1 of the strip at x0. The step that loads row r finishes the
// means of row r - 1 and writes row h = r - 2, whose samples are requested at
// the step's start. `iu` / `iv` hold the advected velocity, vx / vy get the
// convected one; STORED (NoUpdate) reads vx / vy and writes ovx / ovy, so that
// no warp writes a cell another may still read. MASKS: also rebuilds the masks
// of its rows (a batch; the one-grid step has a settle pass).
template <bool MASKS, bool STORED>
__device__ __forceinline__ void strip_heat(const StripGrids &P, const AirInst &I, const float *__restrict__ iu,
                                           const float *__restrict__ iv, uint32_t off, int x0, int y0, int y1,
                                           uint32_t lag) {
    const StripCols C(I, x0, HEAT_HALO);
    const int Y = (int)I.Y;
    const uint32_t pitch = I.pitch, lane = C.lane;
    const bool out = C.output(HEAT_HALO), side = C.x < 2 || C.x + 2 >= (int)I.X;
    const float xf = (float)C.x, limx = (float)I.X - 2.0f, limy = (float)I.Y - 2.0f, amb = I.amb;
    const bool radial = I.gmode == 2u;
    uint32_t o = off + (uint32_t)(y0 - 1) * pitch + (uint32_t)C.x;  // row r
    float convx, convy;
    convection_dir(I, C.x, 0, convx, convy);

    RowState sh{};                                      // means of row r - 1
    RowState2 sv{};
    uint32_t hb1 = 0u, hb2 = 0u, hc1 = 7u;              // heat-blocked / closed cells around the lane
    float mh2 = 0.f;                                    // sums of row r - 2
    Pair mv2;
    float nh = 0.f, nu = 0.f, nv = 0.f;
    uint32_t nbh = 0u;
    auto load = [&](int r, uint32_t e) {  // the next step's loads are in flight during a step
        const bool ok = C.in && r >= 0 && r < Y;
        nu = ok ? load_after_wait((STORED ? P.vx : iu) + e) : 0.f;
        nv = ok ? load_after_wait((STORED ? P.vy : iv) + e) : 0.f;
        nh = ok ? load_after_wait(P.hv + e) : 0.f;
        nbh = ok ? load_after_wait(P.bairh + e) : 0u;
    };
    load(y0 - 1, o);
#pragma unroll 1
    for (int r = y0 - 1; r < y1 + 2; ++r, o += pitch) {
        const float u0 = nu, v0 = nv, h0 = nh;
        const uint32_t row0 = __ballot_sync(~0u, (nbh & 0x8u) != 0u), hb0 = around(row0, lane);
        load(r + 1, o + pitch);
        const int h = r - 2;
        const bool mine = out && h >= y0 && h < Y;
        const uint32_t w = o - 2u * pitch;
        // row h's own words again (in L1), instead of registers that hold them for two steps
        float h2 = 0.f, nx = 0.f, ny = 0.f;
        uint32_t mw = 0u, me = 0u, ma = 0u, mb = 0u;  // the mask rebuild's
        if (mine) {
            h2 = load_after_wait(P.hv + w);
            nx = load_after_wait((STORED ? P.vx : iu) + w);
            ny = load_after_wait((STORED ? P.vy : iv) + w);
            if (MASKS) {
                mw = load_after_wait(P.wall + w);
                me = P.emap[w];
                ma = load_after_wait(P.eair + w);
                mb = load_after_wait(P.eairh + w);
            }
        }
        // backtrace of row h (heat.rs:105-130)
        float dh = mh2, svx, svy;
        mv2.get(svx, svy);
        means_of(dh, svx, svy);
        float tx = -1.f, ty = -1.f;
        if (mine)
            far_target(xf, (float)h, svx, svy, limx, limy,
                       [&](int cx, int cy) -> bool {
                           return (load_after_wait(P.bairh + (off + (uint32_t)cy * pitch + (uint32_t)cx)) & 0x8u) != 0u;
                       },
                       tx, ty);
        const bool here = (hb2 & 2u) != 0u;
        const Landing q(tx, ty, 0.0f, limx + 1.0f, limy + 1.0f, off, pitch, mine && !here);
        const float *q0 = P.hv + q.g;
        const uint32_t *qb = P.bairh + q.g;
        const float t00 = load_after_wait(q0), t10 = load_after_wait(q0 + 1), t01 = load_after_wait(q0 + pitch), t11 = load_after_wait(q0 + pitch + 1);
        const uint32_t c00 = load_after_wait(qb), c10 = load_after_wait(qb + 1), c01 = load_after_wait(qb + pitch), c11 = load_after_wait(qb + pitch + 1);
        // the means of row r - 1 get this row's taps, row r's begin (heat.rs:46-104)
        const uint32_t hc0 = around(row0 | C.not_inner | (r < 1 || r + 1 >= Y ? ~0u : 0u), lane);
        const Closed k0(hc0), k1(hc1);
        const RowTaps th(h0);
        const RowTaps2 tv(u0, v0);
        const float mh1 = finish_sum(sh, th, k0);
        const Pair mv1 = finish_sum(sv, tv, k0);
        start_sum(sh, th, k1, k0);
        start_sum(sv, tv, k1, k0);
        if (mine) {
            if (q.ok) {
                const float s = q.blend((c00 & 0x8u) ? dh : t00, (c10 & 0x8u) ? dh : t10, (c01 & 0x8u) ? dh : t01,
                                        (c11 & 0x8u) ? dh : t11);
                dh = dh * 0.7f + 0.3f * s;
            }
            if (here) dh = h2;
            dh = clampf(dh, 0.0f, 9999.0f);
            const bool rim = h < 2 || h + 2 >= Y || side;
            if (rim) dh = amb;
            if (!rim) {  // convection (heat.rs:182-251)
                if (radial) convection_dir(I, C.x, h, convx, convy);
                if (I.conv == 1u) {
                    const float weight =
                        div_by_const((h2 - load_after_wait(P.hv + (w - 1u))) * convx + (h2 - load_after_wait(P.hv + (w - pitch))) * convy,
                                     kConvLegacy, kConvLegacyRcp);
                    if (weight > 0.0f && !(load_after_wait(P.bairh + (w - pitch)) & 0x8u)) {
                        nx += weight * convx;
                        ny += weight * convy;
                    }
                } else if (I.conv == 2u) {
                    float weight = div_by_const(h2 - amb, kConvBouss, kConvBoussRcp);
                    if (weight > 0.01f) weight = 0.01f;
                    nx += weight * convx;
                    ny += weight * convy;
                }
                nx = clampf(nx, -256.0f, 256.0f);
                ny = clampf(ny, -256.0f, 256.0f);
            }
            P.hv_out[w] = dh;
            (STORED ? P.ovx : P.vx)[w] = nx;
            (STORED ? P.ovy : P.vy)[w] = ny;
            if (MASKS) {
                const uint32_t raw = emap_seen(me, lag), next = raw != 0u ? raw - 1u : 0u;
                if (next != me) P.emap[w] = next;
                uint32_t ba, bh;
                masks_of(mw, raw, ma, mb, ba, bh);
                P.bair_out[w] = ba;
                P.bairh_out[w] = bh;
            }
        }
        hb2 = hb1, hb1 = hb0, hc1 = hc0;
        mh2 = mh1, mv2 = mv1;
    }
}

}  // namespace air
}  // namespace tpt

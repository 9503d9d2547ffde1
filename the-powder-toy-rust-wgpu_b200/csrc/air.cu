// air.cu -- the one-grid air step (tpt_air_step and its static-scratch
// variant): tiles, or warp strips for a large grid. Compiled with -fmad=false: see air.cuh.
#include <algorithm>

#include "air_strip.cuh"
#include "air_launch.hpp"

namespace tpt {
namespace air {

// What bounds a tick of one grid of up to a few hundred thousand cells is its
// serial chain: three launches, and in each the barriers, the ring cells that
// a thread takes one after the other, and the walk of the advection.
//
// The kernels are programmatic dependent launches: each waits for the one
// before it to complete before it touches memory, and starts as soon as that
// one's blocks exit, or, the settle pass, have staged their tile. (Releasing
// pass B from pass A's staging as well puts its blocks unevenly beside those
// still running: 401x225 16.7 -> 20.0 us.)
//
// A block has more threads than its tile has cells: pass A's +2 ring has 432
// cells and pass B's +1 ring 340, and each ring is one turn instead of two.
// Measured on B200, us per tick in a graph, before (256 threads, ordinary
// launches) and now: 16x16 10.9 and 8.1, 64x48 16.3 and 11.4, 153x96 18.5 and
// 13.4, 300x200 18.6 and 14.3, 401x225 20.2 and 16.7, 512x512 32.0 and 27.7,
// 590x590 39.8 and 35.4; as strips, launches alone: 1024x1024 84.8 and 76.9,
// 2048x2048 249.5 and 244.7 in calls back to back.
constexpr int NT_A = 448, NT_B = 384;
static_assert(NT_A >= (TX + 4) * (TY + 4) && NT_B >= (TX + 2) * (TY + 2), "a ring is one turn");

template <typename... Args>
static int launch_pdl(void (*kernel)(Args...), dim3 grid, unsigned block, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    TPT_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
    TPT_LAUNCHED();
    return TPT_OK;
}

// Pass A of one tile, staged by plain loads (the caller's grids may have any
// row length, so no TMA).
__global__ void __launch_bounds__(NT_A) k_pressure_velocity(const AirInst I) {
    __shared__ LayoutA1 S;
    pdl_wait();
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY;
    stage_flag<3, NT_A>(S.b, I.bair, 0xFFFFFFFFu, I, x0, y0);
    stage<float, 2, NT_A>(S.vx, I.vx, I, x0, y0);
    stage<float, 2, NT_A>(S.vy, I.vy, I, x0, y0);
    stage<float, 1, NT_A>(S.pv, I.pv, I, x0, y0);
    __syncthreads();
    pass_a<NT_A>(I, x0, y0, S);
}

// Pass B of one tile.
__global__ void __launch_bounds__(NT_B, 5) k_advect_heat(const AirInst I) {
    __shared__ LayoutB1 S;
    pdl_wait();
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY;
    if (I.air_mode != 4u) {
        stage_flag<3, NT_B>(S.b, I.bair, 0xFFFFFFFFu, I, x0, y0);
        stage<float, 3, NT_B>(S.ovx, I.ovx, I, x0, y0);
        stage<float, 3, NT_B>(S.ovy, I.ovy, I, x0, y0);
        stage<float, 2, NT_B>(S.opv, I.opv, I, x0, y0);
    } else {
        stage<float, 1, NT_B>(S.nvx, I.vx, I, x0, y0);
        stage<float, 1, NT_B>(S.nvy, I.vy, I, x0, y0);
    }
    if (I.aheat) {
        stage_flag<1, NT_B>(S.bh, I.bairh, 0x8u, I, x0, y0);
        stage<float, 1, NT_B>(S.hv, I.hv, I, x0, y0);
    }
    __syncthreads();
    pdl_release();
    pass_b<NT_B>(I, x0, y0, S);
}

// The same tick as warp strips (air_strip.cuh): warp w takes strip w % strips of
// row block w / strips. Strips need fewer instructions per cell, but a warp
// walks its rows one after the other: below about 300,000 cells the tiles, a
// thread per cell, are done sooner. Measured on B200, us per tick, tiles and
// strips: 401x225 16.4 and 24.1, 512x512 27.8 and 28.8, 590x590 35.7 and 33.7,
// 700x600 40.3 and 37.8, 1024x1024 87.1 and 76.5, 2048x2048 360 and 245.
constexpr size_t STRIP_MIN_CELLS = 300000;
struct OneGrid {
    StripGrids P;
    AirInst I;
    uint32_t strips, rows;  // strips across the grid, rows per block
};
__device__ __forceinline__ bool strip_of(const OneGrid &G, int width, int &x0, int &y0, int &y1) {
    const uint32_t w = blockIdx.x * (blockDim.x / 32u) + threadIdx.x / 32u, b = w / G.strips;
    x0 = (int)((w - b * G.strips) * (uint32_t)width);
    y0 = (int)(b * G.rows);
    y1 = min(y0 + (int)G.rows, (int)G.I.Y);
    return y0 < (int)G.I.Y;
}
__global__ void __launch_bounds__(STRIP_WARPS * 32, 8) k_strip_velocity(const __grid_constant__ OneGrid G) {
    pdl_wait();
    int x0, y0, y1;
    if (strip_of(G, strip_width(PASS_VELOCITY), x0, y0, y1)) strip_a(G.P, G.I, 0u, x0, y0, y1);
}
__global__ void __launch_bounds__(STRIP_WARPS * 32, 6) k_strip_advect(const __grid_constant__ OneGrid G) {
    pdl_wait();
    int x0, y0, y1;
    // into vx / vy, free since the velocity pass read them
    if (strip_of(G, strip_width(PASS_ADVECT), x0, y0, y1)) strip_advect(G.P, G.I, G.P.vx, G.P.vy, 0u, x0, y0, y1);
}
__global__ void __launch_bounds__(STRIP_WARPS * 32, 6) k_strip_heat(const __grid_constant__ OneGrid G) {
    pdl_wait();
    int x0, y0, y1;
    // from vx / vy into ovx / ovy; the settle pass copies them back
    if (strip_of(G, strip_width(PASS_HEAT), x0, y0, y1))
        strip_heat<false, true>(G.P, G.I, nullptr, nullptr, 0u, x0, y0, y1, 0u);
}

// What the settle pass reads of a cell, all of it requested before anything is
// written: an ordinary load stays behind the stores before it. Measured on B200
// at 2048x2048, whose words fit L2, us: the masks alone 15.9 (19.2 with loads
// between the stores, 15.4 by the read-only path, which is not for memory that
// the launch before may write), a whole step with heat 228 (243 and 239).
struct Settled {
    MaskWords m;
    float hv = 0.0f, vx = 0.0f, vy = 0.0f;
    __device__ __forceinline__ Settled(const AirInst &I, size_t g, bool copy_v) : m(I, g) {
        if (I.aheat) hv = load_after_wait(I.hv_out + g);
        if (copy_v) {
            vx = load_after_wait(I.ovx + g);
            vy = load_after_wait(I.ovy + g);
        }
    }
};

// Settle pass: new heat -> hv, convected velocity -> vx/vy where the heat pass
// left it in ovx/ovy (`copy_v`), wall masks (settle.rs:50-93) and the optional
// HotAir pass (settle.rs:118-161). The grid is dense here (pitch == X).
__global__ void k_settle(const AirInst I, const uint32_t *__restrict__ pmap, const uint32_t *__restrict__ props,
                         uint32_t nprops, uint32_t xres, uint32_t yres, bool copy_v) {
    pdl_wait();
    const size_t n = (size_t)I.X * I.Y, step = (size_t)gridDim.x * blockDim.x;
    size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    copy_v = copy_v && I.aheat;
    for (; g < n; g += step) {
        const Settled c(I, g, copy_v);
        if (I.aheat) {
            I.hv[g] = c.hv;
            if (copy_v) {
                I.vx[g] = c.vx;
                I.vy[g] = c.vy;
            }
        }
        uint32_t ba, bh;
        masks_cell(I, g, c.m, ba, bh);
        I.bair_out[g] = ba;
        I.bairh_out[g] = bh;
        if (pmap != nullptr) {
            const uint32_t cx = (uint32_t)(g % I.X), cy = (uint32_t)(g / I.X);
            float pv = I.pv[g];
            bool touched = false;
            for (uint32_t dy = 0; dy < 4; ++dy)
                for (uint32_t dx = 0; dx < 4; ++dx) {
                    uint32_t px = cx * 4 + dx, py = cy * 4 + dy;
                    if (px >= xres || py >= yres) continue;
                    uint32_t e = load_after_wait(pmap + (size_t)py * xres + px);
                    if (e == 0u) continue;
                    uint32_t ty = e & 0x1FFu;
                    if (ty >= nprops) continue;  // guard: no row for this id
                    float hot = __uint_as_float(__ldg(props + (size_t)ty * 32 + 11));
                    if (hot == 0.0f) continue;
                    touched = true;
                    if (ty == 10u || ty == 97u) {  // PT_GAS / PT_NBLE
                        if (pv < 3.5f) pv += 4.0f * hot * (3.5f - pv);
                    } else {
                        pv += 4.0f * hot;
                    }
                }
            if (touched) I.pv[g] = pv;
        }
    }
}

static StripGrids one_grid(const AirInst &I) {
    StripGrids g{};
    g.pv = I.pv, g.vx = I.vx, g.vy = I.vy, g.opv = I.opv, g.ovx = I.ovx, g.ovy = I.ovy;
    g.hv = I.hv, g.hv_out = I.hv_out;
    g.bair = I.bair, g.bairh = I.bairh;
    g.wall = I.wall;
    g.fvx = I.fvx, g.fvy = I.fvy;
    return g;
}

int launch_single(const AirInst &I, const uint32_t *pmap, const uint32_t *props, uint32_t nprops, uint32_t xres,
                  uint32_t yres, cudaStream_t st) {
    const size_t n = (size_t)I.X * I.Y;
    const bool strips = n >= STRIP_MIN_CELLS && I.X >= 3 && I.Y >= 3;
    if (strips) {
        OneGrid G{one_grid(I), I, 0u, 0u};
        auto run = [&](void (*kernel)(const OneGrid), int pass) -> int {
            const uint32_t w = (uint32_t)strip_width(pass);
            G.strips = (I.X + w - 1) / w;
            // about three strips per resident warp, of 4 to 32 rows
            const size_t fit = (size_t)G.strips * I.Y / (3 * 148 * 24);
            G.rows = (uint32_t)std::min<size_t>(32, std::max<size_t>(4, fit));
            const uint32_t warps = G.strips * ((I.Y + G.rows - 1) / G.rows);
            return launch_pdl(kernel, dim3((warps + STRIP_WARPS - 1) / STRIP_WARPS), STRIP_WARPS * 32, st, (const OneGrid)G);
        };
        int rc = TPT_OK;
        if (I.air_mode != 4u) {
            rc = run(k_strip_velocity, PASS_VELOCITY);
            if (rc == TPT_OK) rc = run(k_strip_advect, PASS_ADVECT);
        }
        if (rc == TPT_OK && I.aheat) rc = run(k_strip_heat, PASS_HEAT);
        if (rc) return rc;
    } else {
        dim3 grid((I.X + TX - 1) / TX, (I.Y + TY - 1) / TY);
        int rc = TPT_OK;
        if (I.air_mode != 4u) rc = launch_pdl(k_pressure_velocity, grid, NT_A, st, (const AirInst)I);
        if (rc == TPT_OK && (I.air_mode != 4u || I.aheat)) rc = launch_pdl(k_advect_heat, grid, NT_B, st, (const AirInst)I);
        if (rc) return rc;
    }
    unsigned blocks = (unsigned)std::min<size_t>((n + 255) / 256, 148 * 16);
    return launch_pdl(k_settle, dim3(blocks), 256, st, (const AirInst)I, pmap, props, nprops, xres, yres,
                      I.aheat && (strips || I.air_mode == 4u));
}

// ---- air step with library-owned scratch (no allocation) ------------------
// The step needs four grids of scratch (new pressure, the two new velocity
// components and the new heat). tpt_air_step takes them from the caller;
// this variant takes them from one array that lives in the library's device
// image, so a call allocates nothing. Every device that loads the library
// holds the array (4 MiB) until the process exits.
static __device__ __align__(256) float g_static_scratch[4 * (size_t)TPT_STATIC_SCRATCH_MAX_CELLS];

// Device address of g_static_scratch in the current device's context. The
// name is a host-side stand-in in host code, so the address is looked up
// with the device current. It is looked up on every call rather than cached:
// the lookup allocates nothing, and a cached address would go stale when the
// context is torn down and recreated (cudaDeviceReset, or a primary-context
// reset through the driver API), leaving kernels to write through a pointer
// of the old context.
static int static_scratch(float **out) {
    int dev = 0;
    TPT_CUDA(cudaGetDevice(&dev));
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
    if (e != cudaSuccess || p == nullptr)
        TPT_FAIL(TPT_ERR_CUDA, "cudaGetSymbolAddress(static scratch) failed on device %d: %s", dev,
                 cudaGetErrorString(e));
    *out = static_cast<float *>(p);
    return TPT_OK;
}

}  // namespace air
}  // namespace tpt

extern "C" int tpt_air_step_static_scratch(const tpt_air_params *params, const tpt_air_bufs *b,
                                           tpt_stream_t stream) {
    using namespace tpt;
    if (!params || !b) TPT_FAIL(TPT_ERR_NULL_POINTER, "tpt_air_step_static_scratch: params or bufs is NULL");
    const tpt_air_params &p = *params;
    if (p.air_mode > 4u || p.convection_mode > 2u || p.gravity_mode > 3u || p.aheat_enable > 1u)
        TPT_FAIL(TPT_ERR_INVALID_ARG, "tpt_air_step_static_scratch: enum field out of range");
    if (p.xcells == 0 || p.ycells == 0) return TPT_OK;
    const size_t n = (size_t)p.xcells * p.ycells;
    if (p.xcells > TPT_MAX_CELLS_PER_SIDE || p.ycells > TPT_MAX_CELLS_PER_SIDE || n > TPT_STATIC_SCRATCH_MAX_CELLS)
        TPT_FAIL(TPT_ERR_INVALID_DIMS,
                 "tpt_air_step_static_scratch: grid %ux%u = %zu cells exceeds the static scratch of %u cells "
                 "(use tpt_air_step with caller-owned scratch)",
                 p.xcells, p.ycells, n, (unsigned)TPT_STATIC_SCRATCH_MAX_CELLS);
    if (!b->pv || !b->vx || !b->vy || !b->hv || !b->block_air || !b->block_airh || !b->wall_bmap || !b->wall_emap ||
        !b->fan_vx || !b->fan_vy)
        TPT_FAIL(TPT_ERR_NULL_POINTER, "tpt_air_step_static_scratch: a required grid pointer is NULL");
    if (b->pmap && (!b->elem_props || b->xres == 0 || b->yres == 0))
        TPT_FAIL(TPT_ERR_INVALID_ARG, "tpt_air_step_static_scratch: pmap given without elem_props / xres / yres");
    int rc = require_sm100();
    if (rc) return rc;
    float *s = nullptr;
    rc = air::static_scratch(&s);
    if (rc) return rc;
    // Every scratch cell the step reads is written earlier in the same step,
    // so nothing has to be cleared between calls.
    AirInst I = make_air_inst(p);
    I.pv = b->pv;
    I.vx = b->vx;
    I.vy = b->vy;
    I.hv = b->hv;
    I.opv = s;
    I.ovx = s + n;
    I.ovy = s + 2 * n;
    I.ohv = s + 3 * n;
    I.bair = b->block_air;
    I.bairh = b->block_airh;
    I.wall = b->wall_bmap;
    I.emap = b->wall_emap;
    I.eair = b->elem_block_air;
    I.eairh = b->elem_block_airh;
    I.fvx = b->fan_vx;
    I.fvy = b->fan_vy;
    I.bair_out = b->block_air;
    I.bairh_out = b->block_airh;
    I.hv_out = I.ohv;
    return air::launch_single(I, b->pmap, b->elem_props, b->n_elements, b->xres, b->yres, (cudaStream_t)stream);
}

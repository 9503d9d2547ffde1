// air_strips.cu -- a large batch's air tick in the tile form: three launches of
// warp strips (air_strip.cuh). The velocity pass writes opv/ovx/ovy; the
// advection pass reads them, writes pv and the advected velocity (to vx/vy,
// or, where the heat pass follows, to the other parity's ovx/ovy, which are
// free during the tick); the heat pass reads that velocity's neighbours,
// convects it into vx/vy, and rebuilds the masks, with heat and masks in
// ping-pong halves. Compiled with -fmad=false: see air.cuh.
#include <algorithm>

#include "air_strip.cuh"
#include "air_launch.hpp"

namespace tpt {
namespace air {

// Warps take strips one at a time: from an atomic counter, or (queue == null)
// strided statically. Each pass's counter is cleared by the launch of the
// pass before it.
__device__ __forceinline__ uint32_t next_strip(uint32_t *queue, uint32_t t) {
    if (queue == nullptr) return t + gridDim.x * (blockDim.x / 32u);
    uint32_t n = 0;
    if ((threadIdx.x & 31u) == 0u) n = atomicAdd(queue, 1u);
    return __shfl_sync(~0u, n, 0);
}
__device__ __forceinline__ uint32_t first_strip(uint32_t *queue) {
    return queue == nullptr ? blockIdx.x * (blockDim.x / 32u) + threadIdx.x / 32u : next_strip(queue, 0u);
}

__global__ void __launch_bounds__(STRIP_WARPS * 32, 8)
    kb_pressure_velocity(const __grid_constant__ StripGrids P, const AirInst *__restrict__ insts,
                         const StripRef *__restrict__ strips, uint32_t nstrips, uint32_t *queue, uint32_t *reset) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *reset = 0u;
    for (uint32_t t = first_strip(queue); t < nstrips; t = next_strip(queue, t)) {
        const StripRef s = strips[t];
        const AirInst I = insts[2 * s.inst];
        if (I.air_mode == 4u) continue;  // NoUpdate
        strip_a(P, I, (uint32_t)(I.wall - P.wall), s.x0, s.y0, s.y0 + s.rows);
    }
}

// `su` / `sv`: the advected velocity's place where the heat pass follows.
__global__ void __launch_bounds__(STRIP_WARPS * 32, 6)
    kb_advect(const __grid_constant__ StripGrids P, float *su, float *sv, const AirInst *__restrict__ insts,
              const StripRef *__restrict__ strips, uint32_t nstrips, uint32_t *queue, uint32_t *reset) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *reset = 0u;
    for (uint32_t t = first_strip(queue); t < nstrips; t = next_strip(queue, t)) {
        const StripRef s = strips[t];
        const AirInst I = insts[2 * s.inst];
        if (I.air_mode == 4u) continue;  // NoUpdate
        strip_advect(P, I, su, sv, (uint32_t)(I.wall - P.wall), s.x0, s.y0, s.y0 + s.rows);
    }
}

// The masks of an instance without ambient heat. The batch's launches are
// ordinary ones, and nothing writes what they read this way: as ordinary loads,
// which stay behind the row before's stores, the step of 64 grids of 400x225
// without heat took 255 us where it takes 234.
__device__ __forceinline__ void strip_masks(const StripGrids &P, const AirInst &I, uint32_t off, int x0, int y0, int y1,
                                            uint32_t lag) {
    const StripCols C(I, x0, HEAT_HALO);
    if (!C.output(HEAT_HALO)) return;
    for (int y = y0; y < y1; ++y) {
        const uint32_t w = off + (uint32_t)y * I.pitch + (uint32_t)C.x, me = P.emap[w];
        const uint32_t raw = emap_seen(me, lag), next = raw != 0u ? raw - 1u : 0u;
        if (next != me) P.emap[w] = next;
        uint32_t ba, bh;
        masks_of(__ldg(P.wall + w), raw, __ldg(P.eair + w), __ldg(P.eairh + w), ba, bh);
        P.bair_out[w] = ba;
        P.bairh_out[w] = bh;
    }
}

__global__ void __launch_bounds__(STRIP_WARPS * 32, 6)
    kb_heat_masks(const __grid_constant__ StripGrids P, const float *su, const float *sv,
                  const AirInst *__restrict__ insts, const StripRef *__restrict__ strips, uint32_t nstrips,
                  uint32_t emap_lag, uint32_t *queue, uint32_t *reset) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *reset = 0u;
    for (uint32_t t = first_strip(queue); t < nstrips; t = next_strip(queue, t)) {
        const StripRef s = strips[t];
        const AirInst I = insts[2 * s.inst];
        const uint32_t off = (uint32_t)(I.wall - P.wall);
        if (I.aheat && I.air_mode != 4u)
            strip_heat<true, false>(P, I, su, sv, off, s.x0, s.y0, s.y0 + s.rows, emap_lag);
        else if (I.aheat)
            strip_heat<true, true>(P, I, su, sv, off, s.x0, s.y0, s.y0 + s.rows, emap_lag);
        else
            strip_masks(P, I, off, s.x0, s.y0, s.y0 + s.rows, emap_lag);
    }
}

// NoUpdate + ambient heat writes its convected velocity to ovx/ovy; a batch
// with such an instance copies it back after the B passes.
__global__ void kb_noupdate_settle(const __grid_constant__ StripGrids P, const AirInst *__restrict__ insts,
                                   const StripRef *__restrict__ strips, uint32_t nstrips) {
    const uint32_t warps = gridDim.x * (blockDim.x / 32u);
    for (uint32_t t = blockIdx.x * (blockDim.x / 32u) + threadIdx.x / 32u; t < nstrips; t += warps) {
        const StripRef s = strips[t];
        const AirInst I = insts[2 * s.inst];
        if (!(I.air_mode == 4u && I.aheat)) continue;
        const uint32_t x = s.x0 + (threadIdx.x & 31u), off = (uint32_t)(I.wall - P.wall);
        if (x >= s.x0 + (uint32_t)strip_width(PASS_HEAT) || x >= I.X) continue;
        for (uint32_t y = s.y0; y < (uint32_t)s.y0 + s.rows; ++y) {
            const uint32_t g = off + y * I.pitch + x;
            P.vx[g] = P.ovx[g];
            P.vy[g] = P.ovy[g];
        }
    }
}

// ---- host side --------------------------------------------------------------
const TileShape *const *tile_shapes() {
    static const TileShape *const all[TILE_SHAPES] = {&tile_shape_s32x8, &tile_shape_s64x8, &tile_shape_s32x16,
                                                      &tile_shape_s64x16};
    return all;
}

const TileShape *tile_shape(uint32_t tx, uint32_t ty) {
    for (int k = 0; k < TILE_SHAPES; ++k)
        if (tile_shapes()[k]->tx == tx && tile_shapes()[k]->ty == ty) return tile_shapes()[k];
    return nullptr;
}

int read_errors(uint32_t *out) {  // the strips and the sweep form have no waits
    uint32_t all = 0;
    int frc = read_fused_errors(&all);
    if (frc) return frc;
    for (int k = 0; k < TILE_SHAPES; ++k) {
        uint32_t v = 0;
        int rc = tile_shapes()[k]->read_errors(&v);
        if (rc) return rc;
        all |= v;
    }
    *out = all;
    return TPT_OK;
}

// Rows of all strips across the grids.
static uint64_t strip_rows_total(const std::vector<std::pair<uint32_t, uint32_t>> &grids, uint32_t w) {
    uint64_t total = 0;
    for (const auto &g : grids) total += (uint64_t)((g.first + w - 1) / w) * g.second;
    return total;
}

// Rows per strip: the shape's, or what makes three strips per resident warp
// where that is less, down to 4 (a small batch is bound by how long one warp
// walks).
uint32_t strip_rows(int pass, const std::vector<std::pair<uint32_t, uint32_t>> &grids, uint32_t rows,
                    uint32_t resident) {
    const uint64_t fit = strip_rows_total(grids, (uint32_t)strip_width(pass)) / (3ull * std::max<uint32_t>(resident, 1u));
    return std::max<uint32_t>(4u, (uint32_t)std::min<uint64_t>(fit, rows));
}

// A strip of h rows takes h + 3 to h + 6 steps, so tall strips spend the least
// on their halo, but a launch's last strips must be short for its warps to end
// together: the first half of the cells is cut into strips of twice `rows`, the
// last quarter into half of them.
void plan_strips(int pass, const std::vector<std::pair<uint32_t, uint32_t>> &grids, uint32_t rows,
                 std::vector<StripRef> &out) {
    const uint32_t w = (uint32_t)strip_width(pass);
    const uint64_t total = strip_rows_total(grids, w);
    uint64_t done = 0;
    for (uint32_t i = 0; i < (uint32_t)grids.size(); ++i) {
        const uint32_t X = grids[i].first, Y = grids[i].second;
        const uint32_t h = 2 * done < total ? 2 * rows : 4 * done < 3 * total ? rows : std::max<uint32_t>(4u, rows / 2);
        const uint32_t n = (Y + h - 1) / h;  // of equal heights, to a row
        for (uint32_t k = 0; k < n; ++k) {
            const uint32_t y0 = (uint32_t)((uint64_t)Y * k / n), y1 = (uint32_t)((uint64_t)Y * (k + 1) / n);
            for (uint32_t x0 = 0; x0 < X; x0 += w)
                out.push_back({i, (uint16_t)x0, (uint16_t)y0, (uint16_t)(y1 - y0), 0});
        }
        done += (uint64_t)((X + w - 1) / w) * Y;
    }
}

int strip_occupancy(int occupancy[STRIP_PASSES]) {
    const int n = STRIP_WARPS * 32;
    TPT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(occupancy + PASS_VELOCITY, kb_pressure_velocity, n, 0));
    TPT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(occupancy + PASS_ADVECT, kb_advect, n, 0));
    TPT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(occupancy + PASS_HEAT, kb_heat_masks, n, 0));
    return TPT_OK;
}

// the counter a pass takes its strips from, and the one it clears
static uint32_t *queue_of(const StripLaunch &s, int pass) { return s.use_queue ? s.queues + pass : nullptr; }
static uint32_t *reset_of(const StripLaunch &s, int pass) { return s.queues + (pass + 1) % STRIP_PASSES; }

int launch_strips_a(const StripLaunch &s, uint32_t parity, cudaStream_t st) {
    const int k = PASS_VELOCITY;
    kb_pressure_velocity<<<s.grid[k], STRIP_WARPS * 32, 0, st>>>(s.grids[parity], s.insts, s.strips[k], s.nstrips[k],
                                                             queue_of(s, k), reset_of(s, k));
    TPT_LAUNCHED();
    return TPT_OK;
}

int launch_strips_settle(const StripLaunch &s, uint32_t parity, cudaStream_t st) {
    const int k = PASS_HEAT;
    kb_noupdate_settle<<<s.grid[k], STRIP_WARPS * 32, 0, st>>>(s.grids[parity], s.insts, s.strips[k], s.nstrips[k]);
    TPT_LAUNCHED();
    return TPT_OK;
}

int launch_strips_b(const StripLaunch &s, uint32_t parity, uint32_t emap_lag, bool any_noupdate_heat, cudaStream_t st) {
    const StripGrids &other = s.grids[parity ^ 1u];
    int k = PASS_ADVECT;
    kb_advect<<<s.grid[k], STRIP_WARPS * 32, 0, st>>>(s.grids[parity], other.ovx, other.ovy, s.insts, s.strips[k],
                                                  s.nstrips[k], queue_of(s, k), reset_of(s, k));
    TPT_LAUNCHED();
    k = PASS_HEAT;
    kb_heat_masks<<<s.grid[k], STRIP_WARPS * 32, 0, st>>>(s.grids[parity], other.ovx, other.ovy, s.insts, s.strips[k],
                                                      s.nstrips[k], emap_lag, queue_of(s, k), reset_of(s, k));
    TPT_LAUNCHED();
    return any_noupdate_heat ? launch_strips_settle(s, parity, st) : TPT_OK;
}

}  // namespace air
}  // namespace tpt

// field3d_batch.cu -- the batched form of the 3-D sandbox's field step
// (crates/tpt-sim/src/voxel3d/{air,gravity}.rs) on sm_100a: every world of a
// call in each launch, one launch per Jacobi sweep index.
//
//   prep    grid-wide, once: per air world the pv update, the velocity
//           snapshot, the sweeps' divergence and a 4-bit pin mask per x-quad
//           (world face or solid > 0.5); per gravity world the source
//           4*pi*G*rho. None of these changes during the sweeps, which the
//           reference recomputes in every sweep.
//   sweep s one launch per sweep index: the air sweep of every world while
//           s < air iterations and the gravity sweep of every world while
//           s < 24, side by side in the same grid. A thread updates x-quads
//           (4 cells, a float4); the x neighbours outside the quad come from
//           the adjacent lanes.
//   finish  grid-wide, once: the air advection, the gravity force and the
//           mass clear.
//
// Every launch is a programmatic dependent launch: it waits for the previous
// grid's completion and memory (griddepcontrol.wait), then lets the next one
// start (griddepcontrol.launch_dependents), so that a launch's latency
// overlaps the grid before it. As the release comes after the wait, a grid
// that runs knows every grid before its predecessor complete, and may load
// what those wrote, and its predecessor does not write, before its own wait:
// a sweep after the first its source and pins, the finishing pass the
// temperature and solid fields (all past L1, which an earlier step may have
// filled). That took the step of one world from 65.0 to 57.4 us, of eight
// from 248 to 239; releasing before the wait, without early loads, 65.0; after
// it, without them, 62.8. The fields of a world stay in L2 (1 MiB each) across
// the sweeps.
#include "field3d.hpp"
#include "field3d_cell.cuh"
#include "pdl.cuh"

namespace tpt {
namespace vox {

namespace {

constexpr int QUADS = CELLS / 4;
constexpr int PBLOCK = 128;             // quads per block of the passes around the sweeps
constexpr int PBLOCKS = QUADS / PBLOCK;
// Worlds from which a sweep's thread takes two quads (see k_b_sweep).
constexpr uint32_t MANY_WORLDS = 4;
static_assert(TPT_VOX_GRAV_ITERATIONS % 2 == 0, "an even sweep count leaves the last sweep in grav_potential");

// Which field block z of a launch works on: bit f of `fields` (f = 0 air,
// 1 gravity) marks the fields in the grid, in that order.
__device__ __forceinline__ int field_of(uint32_t fields, int z) {
    return (fields & 1u) ? z : 1;
}

// The passes around the sweeps move every field of a world once and are bound
// by DRAM when the worlds are many. A thread takes a quad, so a field's
// neighbours are five float4 loads and two shuffles instead of 28 word loads:
// the whole step with the layouts below, 1 / 2 / 4 / 8 worlds, went from 65 /
// 104 / 165 / 284 us to 65 / 96 / 149 / 248 (without the early loads).

// A quad's neighbourhood of one field: its cells, the quads beside it in z and
// y (zero outside the world) and the cells before and after it in x, from the
// adjacent lanes (unused at the world's faces).
struct Quad {
    float4 c, zm, zp, ym, yp;
    float l, r;
    __device__ __forceinline__ float xm(int k) const { return k == 0 ? l : f4(c, k - 1); }
    __device__ __forceinline__ float xp(int k) const { return k == 3 ? r : f4(c, k + 1); }
};
__device__ __forceinline__ void quad_x(Quad &q) {
    q.l = __shfl_up_sync(0xFFFFFFFFu, q.c.w, 1, 16);
    q.r = __shfl_down_sync(0xFFFFFFFFu, q.c.x, 1, 16);
}
// L2: past L1.
template <bool L2 = false>
__device__ __forceinline__ float4 load4(const float *a) {
    return L2 ? __ldcg(reinterpret_cast<const float4 *>(a)) : ld4(a);
}
template <bool L2 = false>
__device__ __forceinline__ Quad load_quad(const float *a, int i0, int y, int z) {
    Quad q;
    q.c = load4<L2>(a + i0);
    q.zm = z > 0 ? load4<L2>(a + i0 - SZ) : zero4();
    q.zp = z + 1 < N ? load4<L2>(a + i0 + SZ) : zero4();
    q.ym = y > 0 ? load4<L2>(a + i0 - SY) : zero4();
    q.yp = y + 1 < N ? load4<L2>(a + i0 + SY) : zero4();
    quad_x(q);
    return q;
}

__global__ void __launch_bounds__(PBLOCK) k_b_prep(const __grid_constant__ Batch B) {
    pdl_wait();
    pdl_release();
    const BWorld &w = B.w[blockIdx.y];
    const int f = field_of(B.fields, blockIdx.z);
    const int q = blockIdx.x * PBLOCK + threadIdx.x;
    const int i0 = 4 * q, x0 = i0 & 63, z = (i0 >> 6) & 63, y = i0 >> 12;
    if (f == 1) {
        const int4 m = *reinterpret_cast<const int4 *>(w.mass + i0);
        st4(w.src + i0, make_float4(grav_source(m.x), grav_source(m.y), grav_source(m.z), grav_source(m.w)));
        return;
    }
    const bool row = y > 0 && z > 0 && y < N - 1 && z < N - 1;  // off the y and z faces
    const bool row_rim = y < 2 || y >= N - 2 || z < 2 || z >= N - 2;
    Quad vx;
    vx.c = ld4(w.vx + i0);
    const float4 vy = ld4(w.vy + i0), vz = ld4(w.vz + i0), solid = ld4(w.solid + i0);
    const int4 pv = *reinterpret_cast<const int4 *>(w.pv + i0);
    const float4 ym = row ? ld4(w.vy + i0 - SY) : zero4(), yp = row ? ld4(w.vy + i0 + SY) : zero4();
    const float4 zm = row ? ld4(w.vz + i0 - SZ) : zero4(), zp = row ? ld4(w.vz + i0 + SZ) : zero4();
    quad_x(vx);
    const int32_t pvs[4] = {pv.x, pv.y, pv.z, pv.w};
    int32_t pn[4];
    float4 div;
    uint32_t pins = 0u;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int x = x0 + k;
        const bool inner = row && x > 0 && x < N - 1, rim = row_rim || x < 2 || x >= N - 2;
        const float xm = vx.xm(k), xp = vx.xp(k);
        const float dp = (xm - xp) + (f4(ym, k) - f4(yp, k)) + (f4(zm, k) - f4(zp, k));
        const float d = 0.5f * ((xp - xm) + (f4(yp, k) - f4(ym, k)) + (f4(zp, k) - f4(zm, k)));
        f4set(div, k, inner ? d : 0.0f);
        pn[k] = pv_update(pvs[k], rim, dp);  // the rim holds every cell outside `inner`
        if (!inner || f4(solid, k) > 0.5f) pins |= 1u << k;
    }
    st4(w.snap + i0, vx.c);
    st4(w.snap + CELLS + i0, vy);
    st4(w.snap + 2 * CELLS + i0, vz);
    st4(w.div + i0, div);
    *reinterpret_cast<int4 *>(w.pv + i0) = make_int4(pn[0], pn[1], pn[2], pn[3]);
    w.pin[q] = (uint8_t)pins;
}

// One sweep. A thread takes the quads of YPT planes, one above the other, and
// a block BZ rows in z: the quads beside its own in y and z are its own in
// other threads' loads, or on the way into L1 for them. What bounds it is L1
// and the latency of one dependent round to L2, where the fields stay; of the
// layouts, (YPT, BZ, threads), measured on B200 as whole field steps with 12
// air sweeps and 30% of the bricks listed, before the early loads and the
// passes below, us for 1 / 2 / 4 / 8 worlds:
//
//   (1, 16, 256), a strip of 16 rows  66 / 108 / 177 / 310
//   (1, 4, 256)                       65 / 104 / 167 / 295   below 4 worlds
//   (2, 8, 128)                       67 / 109 / 165 / 284   from 4 worlds on
//   (2, 8, 256)                       73 / 106 / 166 / 292
//   (4, 8, 128)                       80 / 121 / 172 / 298
//
// Two quads a thread load 4 quads each instead of 5 but leave few warps when
// the worlds are few. Several sweeps per launch over tiles with halo rows in
// shared memory were slower for every number of worlds (two sweeps: 68 / 120 /
// 194 / 363 at best): the halo's redundant cells and the shared-memory traffic
// outweigh the launches.
template <int YPT, int BZ, int THREADS>
__global__ void __launch_bounds__(THREADS) k_b_sweep(const __grid_constant__ Batch B, uint32_t s) {
    constexpr int BY = THREADS / 16 / BZ * YPT;  // planes of a block
    const BWorld &w = B.w[blockIdx.y];
    const int f = field_of(B.fields, blockIdx.z);
    const int x0 = 4 * (threadIdx.x & 15), row = threadIdx.x >> 4;
    const int z = (int)(blockIdx.x % (N / BZ)) * BZ + row % BZ;
    const int y0 = (int)(blockIdx.x / (N / BZ)) * BY + row / BZ * YPT;
    const int i0 = y0 * SY + z * SZ + x0;
    const bool even = (s & 1u) == 0u;
    const float *S;
    float *T;
    if (f == 0) {
        S = even ? w.p : w.p_tmp;  // odd sweeps (1-based) write p_tmp, even ones p
        T = even ? w.p_tmp : w.p;
    } else {
        S = even ? w.pot : w.pot_tmp;
        T = even ? w.pot_tmp : w.pot;
    }
    const float *source = f == 0 ? w.div : w.src;
    float4 c[YPT + 2], zm[YPT], zp[YPT], sr[YPT];
    uint32_t pn[YPT];
    auto load_source = [&]() {
#pragma unroll
        for (int j = 0; j < YPT; ++j) {
            sr[j] = __ldcg(reinterpret_cast<const float4 *>(source + i0 + j * SY));
            pn[j] = f == 0 ? __ldcg(w.pin + ((i0 + j * SY) >> 2)) : 0u;
        }
    };
    if (s > 0) load_source();  // the first sweep's predecessor is the pass that writes it
    pdl_wait();
    pdl_release();
    if (s == 0) load_source();
    c[0] = y0 > 0 ? ld4(S + i0 - SY) : zero4();
#pragma unroll
    for (int j = 0; j < YPT; ++j) c[j + 1] = ld4(S + i0 + j * SY);
    c[YPT + 1] = y0 + YPT < N ? ld4(S + i0 + YPT * SY) : zero4();
#pragma unroll
    for (int j = 0; j < YPT; ++j) {
        zm[j] = z > 0 ? ld4(S + i0 + j * SY - SZ) : zero4();
        zp[j] = z + 1 < N ? ld4(S + i0 + j * SY + SZ) : zero4();
    }
#pragma unroll
    for (int j = 0; j < YPT; ++j) {
        const int y = y0 + j;
        const float l = __shfl_up_sync(0xFFFFFFFFu, c[j + 1].w, 1, 16);
        const float r = __shfl_down_sync(0xFFFFFFFFu, c[j + 1].x, 1, 16);
        float4 out;
        if (f == 0) {
            const uint32_t pins = pn[j];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float xm = k == 0 ? l : f4(c[j + 1], k - 1), xp = k == 3 ? r : f4(c[j + 1], k + 1);
                f4set(out, k, air_sweep_cell(xm, xp, f4(zm[j], k), f4(zp[j], k), f4(c[j], k), f4(c[j + 2], k),
                                             f4(sr[j], k), (pins >> k) & 1u));
            }
        } else {
            const bool face = y == 0 || z == 0 || y == N - 1 || z == N - 1;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int x = x0 + k;
                const float xm = k == 0 ? l : f4(c[j + 1], k - 1), xp = k == 3 ? r : f4(c[j + 1], k + 1);
                f4set(out, k, grav_sweep_cell(xm, xp, f4(zm[j], k), f4(zp[j], k), f4(c[j], k), f4(c[j + 2], k),
                                              f4(sr[j], k), f4(c[j + 1], k), face || x == 0 || x == N - 1));
            }
        }
        st4(T + i0 + j * SY, out);
    }
}

__global__ void __launch_bounds__(PBLOCK) k_b_finish(const __grid_constant__ Batch B) {
    const BWorld &w = B.w[blockIdx.y];
    const int f = field_of(B.fields, blockIdx.z);
    const int i0 = 4 * (int)(blockIdx.x * PBLOCK + threadIdx.x), x0 = i0 & 63, z = (i0 >> 6) & 63, y = i0 >> 12;
    if (f == 1) {
        pdl_wait();
        pdl_release();
        // gravity_force_kernel (gravity.rs:199-224) on the last sweep, then
        // gravity_clear_kernel (gravity.rs:112-118) when asked
        const Quad u = load_quad(w.pot, i0, y, z);
        const bool face = y == 0 || z == 0 || y == N - 1 || z == N - 1;
        float4 fx, fy, fz;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const bool boundary = face || x0 + k == 0 || x0 + k == N - 1;
            const float seed = seed_f32(f4(u.c, k), 0.0f);
            f4set(fx, k, boundary ? seed : (u.xm(k) - u.xp(k)) * 0.5f);
            f4set(fz, k, boundary ? seed : (f4(u.zm, k) - f4(u.zp, k)) * 0.5f);
            f4set(fy, k, boundary ? seed : (f4(u.ym, k) - f4(u.yp, k)) * 0.5f);
        }
        st4(w.fx + i0, fx);
        st4(w.fy + i0, fy);
        st4(w.fz + i0, fz);
        if (B.clear_mass) *reinterpret_cast<int4 *>(w.mass + i0) = make_int4(0, 0, 0, 0);
        return;
    }
    // air_advect_kernel (air_kernel.rs:414-536) from the snapshot
    const float4 solid = __ldcg(reinterpret_cast<const float4 *>(w.solid + i0));
    const Quad t = load_quad<true>(w.temp, i0, y, z);
    float4 buoy;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float lt = nb_average(f4(t.c, k), t.xm(k), t.xp(k), f4(t.zm, k), f4(t.zp, k), f4(t.ym, k), f4(t.yp, k),
                                    x0 + k, y, z);
        f4set(buoy, k, (lt - kAmbient) * kBuoyancy);
    }
    pdl_wait();
    pdl_release();
    const Quad p = load_quad((B.air_iters & 1u) ? w.p_tmp : w.p, i0, y, z);  // the last sweep's buffer
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const Quad v = load_quad(w.snap + (size_t)a * CELLS, i0, y, z);
        float4 out;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int x = x0 + k;
            const float pc = f4(p.c, k);
            const float grad = a == 0   ? pressure_grad(p.xm(k), p.xp(k), pc, x)
                               : a == 1 ? pressure_grad(f4(p.ym, k), f4(p.yp, k), pc, y)
                                        : pressure_grad(f4(p.zm, k), f4(p.zp, k), pc, z);
            const float o = advect_cell(f4(v.c, k), v.xm(k), v.xp(k), f4(v.zm, k), f4(v.zp, k), f4(v.ym, k),
                                        f4(v.yp, k), a, grad, a == 1 ? f4(buoy, k) : 0.0f, x, y, z);
            f4set(out, k, f4(solid, k) > 0.5f ? 0.0f : o);
        }
        st4((a == 0 ? w.vx : a == 1 ? w.vy : w.vz) + i0, out);
    }
}

template <typename... Args>
int launch_pdl(void (*kernel)(Args...), dim3 grid, dim3 block, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    TPT_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
    TPT_LAUNCHED();
    return TPT_OK;
}

// One sweep of the `nf` fields of B, YPT quads a thread.
template <int YPT, int BZ, int THREADS>
int launch_sweep(const Batch &B, uint32_t nf, uint32_t s, cudaStream_t st) {
    return launch_pdl(k_b_sweep<YPT, BZ, THREADS>, dim3(QUADS / YPT / THREADS, B.n, nf), dim3(THREADS), st, B, s);
}

}  // namespace

int launch_batch(Batch &b, cudaStream_t st) {
    if (b.n == 0 || (b.fields & 3u) == 0u) return TPT_OK;
    const uint32_t nf = (b.fields & 1u) + ((b.fields >> 1) & 1u);
    int rc = launch_pdl(k_b_prep, dim3(PBLOCKS, b.n, nf), dim3(PBLOCK), st, (const Batch)b);
    if (rc) return rc;
    const uint32_t air = (b.fields & 1u) ? b.air_iters : 0u, grav = (b.fields & 2u) ? TPT_VOX_GRAV_ITERATIONS : 0u;
    const uint32_t sweeps = air > grav ? air : grav;
    Batch bs = b;
    for (uint32_t s = 0; s < sweeps; ++s) {
        bs.fields = (s < air ? 1u : 0u) | (s < grav ? 2u : 0u);
        const uint32_t n = (bs.fields & 1u) + ((bs.fields >> 1) & 1u);
        rc = b.n < MANY_WORLDS ? launch_sweep<1, 4, 256>(bs, n, s, st) : launch_sweep<2, 8, 128>(bs, n, s, st);
        if (rc) return rc;
    }
    return launch_pdl(k_b_finish, dim3(PBLOCKS, b.n, nf), dim3(PBLOCK), st, (const Batch)b);
}

}  // namespace vox
}  // namespace tpt

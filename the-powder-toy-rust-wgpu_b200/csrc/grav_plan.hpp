// grav_plan.hpp -- host-side objects of the gravity solve.
#pragma once

#include <vector>

#include "grav_fft.cuh"

namespace tpt {

struct JobShape {
    uint32_t X, Y;
};

namespace gfft {

// A set of independent FP32 FFT gravity solves (one plan = one job; a batch
// = one job per instance) that run as three launches.
struct FftSet {
    // One launch: its blocks (a range of `refs`) and dynamic shared memory.
    struct Pass {
        uint32_t first = 0, blocks = 0, threads = 0;
        size_t smem = 0;
    };
    std::vector<Job> jobs_host;
    Job *jobs = nullptr;
    BlockRef *refs = nullptr;
    float2 *work = nullptr, *spec = nullptr, *kern = nullptr, *tw = nullptr;
    Pass rows, cols[2], inv;  // rows forward, columns (small and large shared memory), rows inverse

    int create(const std::vector<JobShape> &shapes);
    // Points job j at its inputs/outputs; returns 1 if anything changed
    // (the caller then re-uploads with upload_jobs()).
    int set_io(size_t j, const int32_t *mass_i, const float *mass_f, float inv, const uint32_t *mask, float *gx,
               float *gy, uint32_t pitch);
    int upload_jobs();
    // io != null: a one-job set solving on per-call pointers.
    int launch(cudaStream_t st, const JobIO *io = nullptr) const;
    // Launches of one solve.
    uint32_t launches() const {
        uint32_t n = 0;
        for (const Pass *p : {&rows, &cols[0], &cols[1], &inv}) n += p->blocks > 0 ? 1u : 0u;
        return n;
    }
    void destroy();
    ~FftSet() { destroy(); }
};

}  // namespace gfft
}  // namespace tpt

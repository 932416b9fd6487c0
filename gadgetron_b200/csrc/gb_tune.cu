// Autotuner for the tiling of the gridding/degridding kernels.
//
// The best tile shape and coil group depend on the trajectory density (dense
// radial centres favour small tiles, which split work finely; uniform
// trajectories favour large tiles, which re-read fewer halo cells), on the
// kernel width and on the number of coils.  For a preprocessed plan this
// re-bins the trajectory for each candidate, times one gridding and one
// degridding pass on `nb` batches with CUDA events -- as the normal operator
// runs them (its sample workspace layout), since the
// CG-SENSE iteration is where the convolutions' time goes -- and keeps the
// fastest.
// Results are cached per (D, N, mos, W, frames, samples within 5%, batches)
// so later plans of the same shape skip the timing.
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "gb_internal.cuh"
#include "gb_ops.hpp"

namespace gb {

namespace {

struct TuneKey {
    int D, N0, N1, N2, m0, m1, m2, F, nb;
    float W;
    int64_t msize;
    bool operator<(const TuneKey &o) const {
        return std::tie(D, N0, N1, N2, m0, m1, m2, F, nb, W, msize) <
               std::tie(o.D, o.N0, o.N1, o.N2, o.m0, o.m1, o.m2, o.F, o.nb, o.W, o.msize);
    }
};

struct TuneResult {
    int tile[kMaxD];
    int cg;
};

std::mutex g_tune_mu;
std::map<TuneKey, TuneResult> g_tune_cache;

std::vector<TuneResult> candidates(const NufftPlan &p) {
    std::vector<TuneResult> out;
    std::vector<std::vector<int>> shapes;
    if (p.D == 1) shapes = {{256, 1, 1}, {512, 1, 1}, {1024, 1, 1}};
    if (p.D == 2) shapes = {{16, 16, 1}, {32, 16, 1}, {16, 32, 1}, {32, 32, 1}, {8, 32, 1}, {32, 8, 1}};
    if (p.D == 3) shapes = {{8, 8, 4}, {8, 8, 8}, {16, 8, 8}, {8, 16, 8}, {16, 16, 4}};
    for (const auto &s : shapes)
        for (int cg : {4, 8, 16}) {
            TuneResult r{};
            for (int d = 0; d < kMaxD; d++) r.tile[d] = s[d];
            r.cg = cg;
            out.push_back(r);
        }
    return out;
}

bool try_tiling(NufftPlan &p, const TuneResult &r) {
    try {
        plan_set_tiling(p, r.tile, r.cg);
        return true;
    } catch (...) {
        return false;
    }
}

struct Event {
    cudaEvent_t e = nullptr;
    Event() { GB_CUDA(cudaEventCreate(&e)); }
    ~Event() { cudaEventDestroy(e); }
    Event(const Event &) = delete;
};

// Milliseconds of one gridding and one degridding of nb batches in the plan's
// tiling.
float time_tiling(NufftPlan &p, float2 *samples, float2 *grid, int nb, const std::vector<uint64_t> &offs,
                  const Event &e0, const Event &e1, cudaStream_t st) {
    plan_preprocess(p, p.traj_copy.get(), (uint64_t)p.Mtot, (uint32_t)(offs.size() - 1), offs.data(), p.prep_mode, st);
    launch_grid_prepare(p, nb, st);
    const SampleLayout lay = normal_op_layout(p, nb);
    for (int pass = 0; pass < 2; pass++) {   // the first pass untimed (module loading, caches)
        if (pass) GB_CUDA(cudaEventRecord(e0.e, st));
        launch_grid(p, samples, grid, nb, lay, nullptr, true, false, st);
        launch_degrid(p, grid, samples, nb, lay, nullptr, 1, true, false, st);
    }
    GB_CUDA(cudaEventRecord(e1.e, st));
    GB_CUDA(cudaEventSynchronize(e1.e));
    float ms = 0.f;
    GB_CUDA(cudaEventElapsedTime(&ms, e0.e, e1.e));
    return ms;
}

}  // namespace

void plan_autotune(NufftPlan &p, int nb, cudaStream_t st) {
    if (!p.prepped) fail(GB_ERR_NOT_PREPROCESSED, "autotune needs a preprocessed plan");
    if (nb <= 0) fail(GB_ERR_INVALID_ARGUMENT, "number of batches must be positive");
    const TuneKey key{p.D, (int)p.N[0], (int)p.N[1], (int)p.N[2], (int)p.mos[0], (int)p.mos[1], (int)p.mos[2],
                      (int)p.F, nb, p.W, (int64_t)(std::log((double)p.Mtot) / std::log(1.05))};
    const int64_t M = p.Mtot;
    const uint32_t F = p.F;
    const std::vector<uint64_t> offs(p.frame_off.begin(), p.frame_off.end());
    const TuneResult start{{p.tiling.tile[0], p.tiling.tile[1], p.tiling.tile[2]}, p.tiling.cg};
    TuneResult best = start;
    bool cached = false;
    {
        std::lock_guard<std::mutex> lock(g_tune_mu);
        auto it = g_tune_cache.find(key);
        if (it != g_tune_cache.end()) {
            best = it->second;
            cached = true;
        }
    }
    if (!cached) {
        DevBuf<float2> samples, grid;
        const size_t ns = (size_t)il_stride_for(nb) * M;   // room for either sorted layout
        samples.ensure(ns);
        grid.ensure((size_t)nb * F * p.kp.G);
        GB_CUDA(cudaMemsetAsync(samples.get(), 0, ns * sizeof(float2), st));
        Event e0, e1;
        float best_ms = 1e30f;
        for (const TuneResult &c : candidates(p)) {
            try {
                plan_set_tiling(p, c.tile, c.cg);
                const float ms = time_tiling(p, samples.get(), grid.get(), nb, offs, e0, e1, st);
                if (ms < best_ms) {
                    best_ms = ms;
                    best = c;
                }
            } catch (...) {
                // a tiling that this plan does not take, or has no room for; an
                // error that outlasts the launch shows in the preprocess below
            }
        }
        std::lock_guard<std::mutex> lock(g_tune_mu);
        g_tune_cache[key] = best;
    }
    if (!try_tiling(p, best)) {
        plan_set_tiling(p, start.tile, start.cg);
        best = start;
    }
    plan_preprocess(p, p.traj_copy.get(), (uint64_t)M, F, offs.data(), p.prep_mode, st);
}

}  // namespace gb

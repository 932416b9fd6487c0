// Iterative density compensation estimate with a Jinc-shaped kernel
// (estimate_dcw, toolboxes/mri/sdc/SDC.hpp:19-80 and gpu/cuSDC.cu): starting
// from w = 1 (or the caller's weights), `iterations` times
//     grid = NC2C(w)            (gridding of the real weights),
//     t    = C2NC(grid)         (degridding back to the samples),
//     w    = t == 0 ? 0 : w / t
// on an oversampled grid of size round_up_32(N * os_factor) per dimension.
//
// The kernel is JincKernel (toolboxes/nfft/ConvolutionKernel.{h,hpp}):
// radius R = 0.96960938 * kernel_width, width 2R; the weight of a cell at
// offset u from the sample is 0 if any |u_d| > R, else with
// r = sqrt(sum u_d^2) / R: 0 if r >= 0.96960938, else the reference's
// degree-5 polynomial fit sum c_k r^k clipped at 0.  Cells and coordinates
// follow the gridding convention of the KB path: s = k mos + mos / 2 (float,
// as fma(k, mos, (mos + pad) / 2) - pad / 2 with pad = 2 ceil(R)), taps
// [ceil(s - R), floor(s + R)] per dimension, periodic wrap.
//
// It is a setup computation (once per trajectory), so the gridding here is a
// per-sample scatter with float atomics (the sum order per cell is not fixed,
// unlike the CG-loop gridding) and the degridding a per-sample gather.  A warp
// serves one sample, its lanes spread over the footprint's taps row by row (up
// to 11^D at width 5.5; neighbouring lanes hit neighbouring cells, so an atomic
// instruction covers a few 32-byte sectors), each tap with a square root and a
// degree-5 polynomial; everything of a tap that does not depend on the lane's
// cell is formed once per sample, and the dimension is a template parameter so
// that the footprint stays in registers.  The degridding sums the lanes'
// partial sums in a fixed butterfly order and clears the grid of the next
// iteration on the side (two grids in turn).  49152 samples, width 5.5, 512^2:
// 125 -> 53 us an iteration (footprint arrays indexed by a runtime dimension
// lived in local memory before); bound by instruction issue (85 %).  The grids and the
// trajectory-range flag are kept per device between calls.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <utility>

#include "gb_internal.cuh"

namespace gb {

namespace {

// JincKernel constants (the reference's polynomial fit and normalised radius;
// ConvolutionKernel.h)
constexpr float kJincNormRadius = 0.96960938f;
constexpr float kJc0 = 0.999923599661866f, kJc1 = 0.014023570134078f, kJc2 = -2.969947516849635f,
                kJc3 = 0.891173008769047f, kJc4 = 2.326043034495162f, kJc5 = -1.270644932677047f;

struct SdcArgs {
    int D;
    int mos[3];
    float half_mos_pad[3];   // (mos + pad) / 2
    float hp;                // pad / 2
    float radius, inv_R;
    float d2_limit;          // squared distances of a disc's cells lie below it
    int64_t M;
};

// Smallest d2 outside the disc, i.e. with !(sqrtf(d2) / R < kJincNormRadius):
// the root and the quotient are correctly rounded and monotone, so the
// reference's rule is a threshold on d2, found by bisection over the floats.
float jinc_limit(float R) {
    auto outside = [R](uint32_t bits) {
        float d2;
        std::memcpy(&d2, &bits, sizeof(d2));
        return !(std::sqrt(d2) / R < kJincNormRadius);
    };
    uint32_t in = 0u, out = 0x7f800000u;   // 0 and infinity; positive floats order as their bits
    while (out - in > 1u) {
        const uint32_t mid = in + (out - in) / 2u;
        (outside(mid) ? out : in) = mid;
    }
    float limit;
    std::memcpy(&limit, &out, sizeof(limit));
    return limit;
}

// Weight of a cell at squared distance d2 from the sample (the any-|u_d| > R
// rule of the reference cuts nothing that the radius below does not).  The
// polynomial is 6.6e-4 where the disc ends, so which cells are inside is
// decided exactly as by sqrtf(d2) / R < kJincNormRadius; with the once more
// rounded sqrtf(d2) * (1 / R) one tap in 7 million (width 4) changes sides and
// moves a weight by up to 5e-4.  The polynomial's r is the product corrected by
// its remainder: half an ulp (and 1e-6 of one) from the quotient.  Direct passes
// of 300000 samples, width 5.5, 10 iterations: 2.74 ms with a division, 2.65 so.
__device__ __forceinline__ float jinc_weight(float d2, const SdcArgs &a) {
    if (!(d2 < a.d2_limit)) return 0.f;
    const float root = sqrtf(d2), q = root * a.inv_R;
    const float r = fmaf(fmaf(-q, a.radius, root), a.inv_R, q);
    // the reference's sum c0 + c1 r + ... + c5 r^5 in its order, the powers
    // formed by products (within a few ulp of pow(r, k))
    const float r2 = r * r, r3 = r2 * r, r4 = r2 * r2, r5 = r4 * r;
    float v = kJc0 + kJc1 * r + kJc2 * r2 + kJc3 * r3 + kJc4 * r4 + kJc5 * r5;
    return v < 0.f ? 0.f : v;
}

__device__ __forceinline__ int wrap_cell(int c, int m) { return c < 0 ? c + m : (c >= m ? c - m : c); }

// Visits this lane's share of the footprint cells of sample j (tap t =
// lane, lane + 32, ... in z, y, x order), calling f(cell_index, weight) for
// the nonzero weights.
template <int D, class F>
__device__ __forceinline__ void for_footprint_lane(const SdcArgs &a, const float *traj, int64_t j, int lane,
                                                   F &&f) {
    float s[D];
    int lo[D], n[D];
    int taps = 1;
#pragma unroll
    for (int d = 0; d < D; d++) {
        s[d] = fmaf(traj[j * D + d], (float)a.mos[d], a.half_mos_pad[d]) - a.hp;
        lo[d] = (int)ceilf(s[d] - a.radius);
        const int hi = (int)floorf(s[d] + a.radius);
        n[d] = hi >= lo[d] ? hi - lo[d] + 1 : 0;
        taps *= n[d];
    }
    if (lane >= taps) return;
    // tap coordinates of t, stepped by 32 taps per round without divisions
    int tx = lane % n[0], ty = lane / n[0], tz = 0;
    if (D > 2) {
        tz = ty / n[1 % D];
        ty -= tz * n[1 % D];
    }
    for (int t = lane; t < taps; t += 32) {
        const int cx = lo[0] + tx;
        float u = s[0] - (float)cx;
        float d2 = u * u;
        int64_t idx = wrap_cell(cx, a.mos[0]);
        if (D > 1) {
            const int cy = lo[1 % D] + ty;
            u = s[1 % D] - (float)cy;
            d2 = fmaf(u, u, d2);
            int64_t row = wrap_cell(cy, a.mos[1]);
            if (D > 2) {
                const int cz = lo[2 % D] + tz;
                u = s[2 % D] - (float)cz;
                d2 = fmaf(u, u, d2);
                row += (int64_t)wrap_cell(cz, a.mos[2]) * a.mos[1];
            }
            idx += row * a.mos[0];
        }
        const float w = jinc_weight(d2, a);
        if (w != 0.f) f(idx, w);
        tx += 32;
        while (tx >= n[0]) {
            tx -= n[0];
            if (++ty == n[1 % D] && D > 2) {
                ty = 0;
                ++tz;
            }
        }
    }
}

template <int D>
__global__ void __launch_bounds__(256) k_sdc_grid(SdcArgs a, const float *__restrict__ traj,
                                                  const float *__restrict__ w, float *__restrict__ grid) {
    const int64_t j = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (j >= a.M) return;
    const float v = w[j];
    for_footprint_lane<D>(a, traj, j, threadIdx.x & 31,
                          [&](int64_t idx, float wt) { atomicAdd(&grid[idx], wt * v); });
}

// w <- w / C2NC(grid); `clear` (G cells) is zeroed for the next iteration.
template <int D>
__global__ void __launch_bounds__(256) k_sdc_degrid_update(SdcArgs a, const float *__restrict__ traj,
                                                           const float *__restrict__ grid, float *__restrict__ w,
                                                           float *__restrict__ clear, int64_t G) {
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t i = i0; i < G; i += (int64_t)gridDim.x * blockDim.x) clear[i] = 0.f;
    const int64_t j = i0 >> 5;
    if (j >= a.M) return;   // whole warps leave together (blockDim is a multiple of 32)
    const int lane = threadIdx.x & 31;
    float t = 0.f;
    for_footprint_lane<D>(a, traj, j, lane, [&](int64_t idx, float wt) { t += wt * grid[idx]; });
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) w[j] = t == 0.f ? 0.f : w[j] / t;
}

// `two`: two grids in turn; one, cleared by itself, otherwise
template <int D>
void sdc_iterations(const SdcArgs &a, const float *traj, float *w, float *grid, int64_t G, bool two, int iterations,
                    cudaStream_t st) {
    const unsigned int tb = 256;
    const unsigned int wb = (unsigned int)((a.M + (tb / 32) - 1) / (tb / 32));   // one warp per sample
    float *cur = grid, *next = two ? grid + G : grid;
    for (int it = 0; it < iterations; it++) {
        if (it == 0 || !two) GB_CUDA(cudaMemsetAsync(cur, 0, (size_t)G * sizeof(float), st));
        k_sdc_grid<D><<<wb, tb, 0, st>>>(a, traj, w, cur); note_launch();
        k_sdc_degrid_update<D><<<wb, tb, 0, st>>>(a, traj, cur, w, next, two && it + 1 < iterations ? G : 0); note_launch();
        std::swap(cur, next);
    }
}

// ---- 2D, footprints of at most 128 taps: weights evaluated once per call.
//
// The weights do not change between iterations, so they are laid into a table
// of 128 floats per sample (tap t = lane + 32 r of a cap x cap square from the
// sample's first cell, zero outside the disc) that every iteration reads back
// from L2: four coalesced loads per lane take the place of the square roots and
// polynomials that bound the direct passes.  A tap that rounding may put beyond
// the square lies at |u| = R, where the weight is zero.  Width 5.5, 512^2, 10
// iterations, without / with the table, us a call: 16384 samples 275 / 241, 49152 536 /
// 355, 262144 2302 / 1334, 524288 4471 / 2483; bound now by the L2 atomics and gathers of the
// footprints.  The table pays at every size; kSdcTableSamples bounds the scratch
// kept between calls (128 MiB).  Above it, for one iteration (nothing to reuse),
// for other dimensions and for wider kernels, every pass evaluates the weights.
constexpr int kSdcRounds = 4;
constexpr int64_t kSdcTableSamples = (int64_t)1 << 18;

struct SdcTaps {
    int tx[kSdcRounds], ty[kSdcRounds];
};

__device__ __forceinline__ SdcTaps sdc_lane_taps(int cap, int lane) {
    SdcTaps q;
#pragma unroll
    for (int r = 0; r < kSdcRounds; r++) {
        const int t = lane + 32 * r;
        q.ty[r] = t / cap;
        q.tx[r] = t - q.ty[r] * cap;
    }
    return q;
}

// Position and first cell of sample j along dimension d.
__device__ __forceinline__ float sdc_pos(const SdcArgs &a, const float *traj, int64_t j, int d, int &lo) {
    const float s = fmaf(traj[j * 2 + d], (float)a.mos[d], a.half_mos_pad[d]) - a.hp;
    lo = (int)ceilf(s - a.radius);
    return s;
}

__global__ void __launch_bounds__(256) k_sdc_table(SdcArgs a, int cap, const float *__restrict__ traj,
                                                   float *__restrict__ tab) {
    const int64_t j = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (j >= a.M) return;
    const int lane = threadIdx.x & 31;
    const SdcTaps q = sdc_lane_taps(cap, lane);
    int lo[2];
    const float s0 = sdc_pos(a, traj, j, 0, lo[0]), s1 = sdc_pos(a, traj, j, 1, lo[1]);
    const int n0 = (int)floorf(s0 + a.radius) - lo[0] + 1, n1 = (int)floorf(s1 + a.radius) - lo[1] + 1;
#pragma unroll
    for (int r = 0; r < kSdcRounds; r++) {
        float w = 0.f;
        if (q.tx[r] < n0 && q.ty[r] < n1) {
            const float u = s0 - (float)(lo[0] + q.tx[r]), v = s1 - (float)(lo[1] + q.ty[r]);
            w = jinc_weight(fmaf(v, v, u * u), a);
        }
        tab[j * (32 * kSdcRounds) + 32 * r + lane] = w;
    }
}

// Calls f(cell, weight) for this lane's taps of sample j with nonzero weight.
template <class F>
__device__ __forceinline__ void sdc_table_taps(const SdcArgs &a, const SdcTaps &q, const float *traj,
                                               const float *tab, int64_t j, int lane, F &&f) {
    float w[kSdcRounds];
#pragma unroll
    for (int r = 0; r < kSdcRounds; r++) w[r] = __ldg(tab + j * (32 * kSdcRounds) + 32 * r + lane);
    int lo[2];
    sdc_pos(a, traj, j, 0, lo[0]);
    sdc_pos(a, traj, j, 1, lo[1]);
#pragma unroll
    for (int r = 0; r < kSdcRounds; r++) {
        if (w[r] != 0.f) {
            const int cx = wrap_cell(lo[0] + q.tx[r], a.mos[0]), cy = wrap_cell(lo[1] + q.ty[r], a.mos[1]);
            f((int64_t)cy * a.mos[0] + cx, w[r]);
        }
    }
}

__global__ void __launch_bounds__(256) k_sdc_table_grid(SdcArgs a, int cap, const float *__restrict__ traj,
                                                        const float *__restrict__ tab, const float *__restrict__ w,
                                                        float *__restrict__ grid) {
    const int lane = threadIdx.x & 31;
    const SdcTaps q = sdc_lane_taps(cap, lane);
    for (int64_t j = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; j < a.M; j += (int64_t)gridDim.x * 8) {
        const float v = w[j];
        sdc_table_taps(a, q, traj, tab, j, lane, [&](int64_t idx, float wt) { atomicAdd(&grid[idx], wt * v); });
    }
}

__global__ void __launch_bounds__(256) k_sdc_table_update(SdcArgs a, int cap, const float *__restrict__ traj,
                                                          const float *__restrict__ tab,
                                                          const float *__restrict__ grid, float *__restrict__ w,
                                                          float *__restrict__ clear, int64_t G) {
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t i = i0; i < G; i += (int64_t)gridDim.x * blockDim.x) clear[i] = 0.f;
    const int lane = threadIdx.x & 31;
    const SdcTaps q = sdc_lane_taps(cap, lane);
    for (int64_t j = i0 >> 5; j < a.M; j += (int64_t)gridDim.x * 8) {
        float t = 0.f;
        sdc_table_taps(a, q, traj, tab, j, lane, [&](int64_t idx, float wt) { t += wt * grid[idx]; });
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) w[j] = t == 0.f ? 0.f : w[j] / t;
    }
}

// Taps per dimension of the table's square; 0 when the table does not apply.
int sdc_table_cap(const SdcArgs &a, bool two, int iterations) {
    const int cap = (int)std::floor(2.f * a.radius) + 1;
    return (a.D == 2 && cap * cap <= 32 * kSdcRounds && a.M <= kSdcTableSamples && two && iterations > 1)
               ? cap
               : 0;
}

void sdc_table_iterations(const SdcArgs &a, int cap, const float *traj, float *w, float *grid, float *tab, int64_t G,
                          int iterations, cudaStream_t st) {
    const unsigned int all = (unsigned int)((a.M + 7) / 8);   // one warp per sample
    const unsigned int blocks = std::min(all, (unsigned int)kSMs * 16u);    // a few samples per warp
    k_sdc_table<<<all, 256, 0, st>>>(a, cap, traj, tab); note_launch();
    float *cur = grid, *next = grid + G;
    GB_CUDA(cudaMemsetAsync(cur, 0, (size_t)G * sizeof(float), st));
    for (int it = 0; it < iterations; it++) {
        k_sdc_table_grid<<<blocks, 256, 0, st>>>(a, cap, traj, tab, w, cur); note_launch();
        k_sdc_table_update<<<blocks, 256, 0, st>>>(a, cap, traj, tab, cur, w, next, it + 1 < iterations ? G : 0);
        note_launch();
        std::swap(cur, next);
    }
}

// Scratch kept per device between calls; the mutex is held for a whole call.
// Beyond the one grid a call needs it keeps at most the table of
// kSdcTableSamples samples (128 MiB) and a second grid of kSdcTwoGrids cells (64 MiB;
// a larger grid is cleared by a copy engine pass that costs little beside its iteration).
constexpr int64_t kSdcTwoGrids = (int64_t)1 << 24;
struct SdcScratch {
    std::mutex mu;
    DevBuf<unsigned int> bad;
    DevBuf<float> grid, table;
};

__global__ void k_fill(float *p, int64_t n, float v) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}

__global__ void k_traj_range(const float *traj, int64_t n, unsigned int *bad) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const float v = traj[i];
        if (!(v >= -0.5f && v <= 0.5f)) atomicOr(bad, 1u);
    }
}

}  // namespace

void sdc_estimate_dcw(int D, const uint64_t *N, float os_factor, int iterations, float kernel_width,
                      const float *traj, int64_t M, const float *initial, float *dcw, cudaStream_t st) {
    if (D < 1 || D > 3 || !N || !traj || !dcw || M <= 0 || iterations < 0)
        fail(GB_ERR_INVALID_ARGUMENT, "invalid density estimation arguments");
    if (!(os_factor >= 1.f) || !(kernel_width > 0.f)) fail(GB_ERR_INVALID_ARGUMENT, "invalid oversampling or width");
    SdcArgs a{};
    a.D = D;
    a.M = M;
    a.radius = kJincNormRadius * kernel_width;
    if (2.f * a.radius < 1.8f) fail(GB_ERR_INVALID_ARGUMENT, "Kernel width must be equal to or larger than 1.8.");
    a.inv_R = 1.f / a.radius;
    a.d2_limit = jinc_limit(a.radius);
    const int pad = 2 * (int)std::ceil(a.radius);
    a.hp = (float)(pad / 2);
    int64_t G = 1;
    for (int d = 0; d < 3; d++) a.mos[d] = 1;
    for (int d = 0; d < D; d++) {
        if (N[d] == 0) fail(GB_ERR_INVALID_ARGUMENT, "invalid matrix size");
        // vector_td<size_t>(vector_td<REAL>(N) * os), rounded up to a multiple of 32
        size_t m = (size_t)((float)N[d] * os_factor);
        m = ((m + 31) / 32) * 32;
        if (m > (1u << 20)) fail(GB_ERR_INVALID_ARGUMENT, "matrix size too large");
        a.mos[d] = (int)m;
        a.half_mos_pad[d] = (float)((m + pad) >> 1);
        G *= (int64_t)m;
    }
    const unsigned int tb = 256;
    const unsigned int sb = (unsigned int)((M + tb - 1) / tb);
    int dev = 0;
    GB_CUDA(cudaGetDevice(&dev));
    SdcScratch &sc = device_scratch<SdcScratch>(dev);
    std::lock_guard<std::mutex> lock(sc.mu);
    {
        sc.bad.ensure(1);
        GB_CUDA(cudaMemsetAsync(sc.bad.get(), 0, sizeof(unsigned int), st));
        const int64_t nt = M * D;
        k_traj_range<<<(unsigned int)((nt + tb - 1) / tb), tb, 0, st>>>(traj, nt, sc.bad.get()); note_launch();
        unsigned int hb = 0;
        GB_CUDA(cudaMemcpyAsync(&hb, sc.bad.get(), sizeof(hb), cudaMemcpyDeviceToHost, st));
        GB_CUDA(cudaStreamSynchronize(st));
        if (hb) fail(GB_ERR_TRAJECTORY_RANGE, "trajectory out of range [-1/2, 1/2]");
    }
    if (initial) {
        if (initial != dcw) GB_CUDA(cudaMemcpyAsync(dcw, initial, M * sizeof(float), cudaMemcpyDeviceToDevice, st));
    } else {
        k_fill<<<sb, tb, 0, st>>>(dcw, M, 1.f); note_launch();
    }
    // two grids in turn up to kSdcTwoGrids cells; where they or the table do not
    // fit, one grid and the direct passes
    const bool two = G <= kSdcTwoGrids && sc.grid.try_ensure(2 * (size_t)G);
    if (!two) sc.grid.ensure((size_t)G);
    const int cap = sdc_table_cap(a, two, iterations);
    if (cap > 0 && sc.table.try_ensure((size_t)M * 32 * kSdcRounds))
        sdc_table_iterations(a, cap, traj, dcw, sc.grid.get(), sc.table.get(), G, iterations, st);
    else if (D == 1) sdc_iterations<1>(a, traj, dcw, sc.grid.get(), G, two, iterations, st);
    else if (D == 2) sdc_iterations<2>(a, traj, dcw, sc.grid.get(), G, two, iterations, st);
    else sdc_iterations<3>(a, traj, dcw, sc.grid.get(), G, two, iterations, st);
    GB_CUDA(cudaGetLastError());
    GB_CUDA(cudaStreamSynchronize(st));   // the grids are free for the next call on return
}

}  // namespace gb

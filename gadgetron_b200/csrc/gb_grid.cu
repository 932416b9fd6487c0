// Gridding (NC2C), degridding (C2NC) and trajectory-gradient kernels.
//
// Reference kernels these replace:
//   NC2C  toolboxes/nfft/gpu/ConvolverNC2C_standard.cuh:229-355 (+ the wrap
//         pass :358-477 and the cell/sample pair sort of
//         toolboxes/nfft/gpu/cuGriddingConvolution.cu:361-422)
//   C2NC  toolboxes/nfft/gpu/ConvolverC2NC.cuh:78-122,228-307 (+ the coil-
//         fastest permute of cuGriddingConvolution.cu:329-334)
//
// Arithmetic kept identical to the reference: taps run over
// [ceil(s - W/2), floor(s + W/2)] per dimension, each tap's weight is the
// product over dimensions of the 1D Kaiser-Bessel value of |s - cell|
// (zero beyond W/2, non-finite weights dropped), and the periodic wrap maps a
// tap to (cell mod mos).  s is the padded-grid coordinate and the cell is folded
// by -pad/2; the reference's C2NC starts from s - pad/2 (ConvolverC2NC.cuh:239-241),
// which gives the same taps of nonzero weight.
//
// The 2D and 3D kernels for the usual tiles are in gb_brick.cu (gridding) and
// gb_degrid.cu (degridding, trajectory gradient); the kernels here serve 1D
// plans, tiles that the bricks do not divide and kernels of fewer than 4 taps:
//   * gridding is output-driven per tile: a CTA owns a tile of the
//     oversampled grid, each thread owns CPT cells and accumulates a group of
//     CG coils in registers; a warp covers an 8x4 patch of cells so that a
//     sample footprint lights up a dense block of lanes.  Samples touching the
//     tile are staged 64 at a time in shared memory (positions -> separable
//     weights, values with the density weights folded in).  No atomics: the
//     result is bit-reproducible.  Tiles with long sample lists are split
//     over several CTAs whose partial tiles are summed in a fixed order by
//     the last CTA to finish.
//   * degridding stages the home tile plus a halo of pad/2 cells, coil
//     fastest, in shared memory; a warp serves 32 / (lanes per sample) samples
//     at once with the separable weights staged per warp.
// In all of them the centring checkerboard of the centred FFT ((-1)^(sum of
// cell coordinates), cuNDFFT.cu:6-36) is folded into the weights or the stores
// (sign_fold), and the density weights into the sample loads (gridding) or
// stores (degridding).
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "gb_conv.cuh"
#include "gb_internal.cuh"
#include "gb_ops.hpp"

namespace gb {

// --------------------------------------------------------------- NC2C -----

// Shared-memory stage of one chunk of kChunk samples for the gridding kernel.
template <int CG>
struct GridStage {
    float w[kChunk][3][kWMax];   // separable weights (checkerboard folded in)
    float2 v[kChunk][CG];        // sample values (density weights folded in)
    int a[kChunk][3];            // tile-local start of the footprint (wrapped)
    int n[kChunk][3];            // taps per dimension
    uint32_t mask[kChunk];       // warps whose cell patches the footprint overlaps
};

template <int CG, int CPT, bool COMP>
__global__ void __launch_bounds__(kThreads)
k_grid_nc2c(ConvArgs a, const float2 *__restrict__ samples, float2 *__restrict__ grid) {
    const KParams &k = a.k;
    const int item_idx = blockIdx.x;
    const int grp = blockIdx.y;
    const int b0 = grp * CG;
    const WorkItem it = a.items[item_idx];
    const int f = it.f, tx = it.tx, ty = it.ty, tz = it.tz;
    const int org[3] = {tx * k.tile[0], ty * k.tile[1], tz * k.tile[2]};

    __shared__ GridStage<CG> stage[2];
    __shared__ int s_last;

    // Cell ownership: warp patches of PX x PY cells.
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int PX = (k.D == 1) ? 32 : 8;
    const int PY = (k.D == 1) ? 1 : 4;
    const int npx = k.tile[0] / PX, npy = k.tile[1] / PY;
    int lc[CPT][3];
#pragma unroll
    for (int c = 0; c < CPT; c++) {
        int q = warp + 8 * c;
        int qx = q % npx, qy = (q / npx) % npy, qz = q / (npx * npy);
        lc[c][0] = qx * PX + (lane % PX);
        lc[c][1] = qy * PY + (lane / PX);
        lc[c][2] = qz;
    }

    float acc[CPT][CG][2];
    float cmp[COMP ? CPT : 1][COMP ? CG : 1][2];
#pragma unroll
    for (int c = 0; c < CPT; c++)
#pragma unroll
        for (int q = 0; q < CG; q++) {
            acc[c][q][0] = acc[c][q][1] = 0.f;
            if (COMP) cmp[c][q][0] = cmp[c][q][1] = 0.f;
        }

    // Staging work per thread: weight entries (sample, dim, tap), value
    // entries (sample, coil) and, for threads < kChunk, one sample's
    // footprint and warp mask.  Raw global values are prefetched into
    // registers one chunk ahead so their latency overlaps the accumulation.
    constexpr int kWE = (kChunk * 3 * kWMax + kThreads - 1) / kThreads;
    constexpr int kVE = (kChunk * CG + kThreads - 1) / kThreads;
    float pw[kWE], pt[kWE];
    float2 pv[kVE];
    float pd[kVE];
    float ps[3];

    auto prefetch = [&](int base, int cnt) {
#pragma unroll
        for (int q = 0; q < kWE; q++) {
            const int e = threadIdx.x + q * kThreads;
            const int i = e / (3 * kWMax), d = (e / kWMax) % 3;
            pw[q] = 0.f;
            pt[q] = 0.f;
            if (e < kChunk * 3 * kWMax && i < cnt && d < k.D) {
                const uint32_t si = a.list[base + i];
                pw[q] = a.pos[(int64_t)d * a.Mtot + si];
                pt[q] = a.wtab[((int64_t)si * k.D + d) * kWMax + (e % kWMax)];
            }
        }
#pragma unroll
        for (int q = 0; q < kVE; q++) {
            const int e = threadIdx.x + q * kThreads;
            const int i = e / CG, c = e % CG;
            pv[q] = make_float2(0.f, 0.f);
            pd[q] = 1.f;
            if (e < kChunk * CG && i < cnt && b0 + c < a.nb) {
                const uint32_t si = a.list[base + i];
                const uint32_t j = a.perm[si];
                const int64_t idx = (a.layout == LAYOUT_SORTED) ? (int64_t)si : (int64_t)j;
                pv[q] = samples[(int64_t)(b0 + c) * a.Mtot + idx];
                if (a.dcw) pd[q] = a.dcw[j];
            }
        }
        if (threadIdx.x < kChunk) {
            const int i = threadIdx.x;
            for (int d = 0; d < 3; d++)
                ps[d] = (i < cnt && d < k.D) ? a.pos[(int64_t)d * a.Mtot + a.list[base + i]] : 0.f;
        }
    };

    auto stage_chunk = [&](GridStage<CG> &S, int cnt) {
#pragma unroll
        for (int q = 0; q < kWE; q++) {
            const int e = threadIdx.x + q * kThreads;
            if (e >= kChunk * 3 * kWMax) break;
            const int i = e / (3 * kWMax), d = (e / kWMax) % 3, t = e % kWMax;
            float w = 0.f;
            if (i < cnt) {
                if (d < k.D) {
                    const int lo = (int)ceilf(pw[q] - k.radius);
                    w = pt[q];   // zero beyond the footprint
                    if (a.sign_fold) w *= sign_of((lo + t - k.hw) & 1);   // parity of (p - hw) mod mos (mos even)
                } else {
                    w = (t == 0) ? 1.f : 0.f;
                }
            }
            S.w[i][d][t] = w;
        }
#pragma unroll
        for (int q = 0; q < kVE; q++) {
            const int e = threadIdx.x + q * kThreads;
            if (e >= kChunk * CG) break;
            const int i = e / CG, c = e % CG;
            float2 v = pv[q];
            if (a.dcw) {
                v.x = pd[q] * v.x;
                v.y = pd[q] * v.y;
            }
            S.v[i][c] = v;
        }
        if (threadIdx.x < kChunk) {
            const int i = threadIdx.x;
            uint32_t m = 0;
            if (i < cnt) {
                int lo[3], hi[3];
                for (int d = 0; d < 3; d++) {
                    int a_ = 0, n = 1;
                    if (d < k.D) {
                        const float s = ps[d];
                        const int l = (int)ceilf(s - k.radius);
                        n = min((int)floorf(s + k.radius) - l + 1, kWMax);
                        a_ = wrapmod(l - k.hw - org[d], k.mos[d]);
                    }
                    S.a[i][d] = a_;
                    S.n[i][d] = n;
                    const int T = k.tile[d];
                    if (k.ntiles[d] == 1) {   // footprint may wrap inside the tile
                        lo[d] = 0;
                        hi[d] = T - 1;
                    } else {
                        const int st = (a_ < T) ? a_ : a_ - k.mos[d];
                        lo[d] = max(st, 0);
                        hi[d] = min(st + n - 1, T - 1);
                    }
                }
                for (int w = 0; w < 8; w++)
                    for (int c = 0; c < CPT; c++) {
                        const int q = w + 8 * c;
                        const int x0 = (q % npx) * PX, y0 = ((q / npx) % npy) * PY, z0 = q / (npx * npy);
                        if (x0 <= hi[0] && x0 + PX - 1 >= lo[0] && y0 <= hi[1] && y0 + PY - 1 >= lo[1] &&
                            z0 <= hi[2] && z0 >= lo[2])
                            m |= 1u << w;
                    }
            }
            S.mask[i] = m;
        }
    };

    int cur = 0;
    if (it.begin < it.end) {
        const int cnt0 = min(kChunk, it.end - it.begin);
        prefetch(it.begin, cnt0);
        stage_chunk(stage[0], cnt0);
    }
    __syncthreads();
    for (int base = it.begin; base < it.end; base += kChunk) {
        const int cnt = min(kChunk, it.end - base);
        const int nbase = base + kChunk;
        const int ncnt = nbase < it.end ? min(kChunk, it.end - nbase) : 0;
        if (ncnt > 0) prefetch(nbase, ncnt);
        GridStage<CG> &S = stage[cur];
        for (int half = 0; half < kChunk / 32; half++) {
        uint32_t bits = __ballot_sync(0xffffffffu, half * 32 + lane < cnt &&
                                                       ((S.mask[half * 32 + lane] >> warp) & 1u));
        while (bits) {
            const int i = half * 32 + __ffs(bits) - 1;
            bits &= bits - 1;
            const int a0 = S.a[i][0], a1 = S.a[i][1], a2 = S.a[i][2];
            const int n0 = S.n[i][0], n1 = S.n[i][1], n2 = S.n[i][2];
#pragma unroll
            for (int c = 0; c < CPT; c++) {
                int o0 = lc[c][0] - a0; if (o0 < 0) o0 += k.mos[0];
                int o1 = lc[c][1] - a1; if (o1 < 0) o1 += k.mos[1];
                int o2 = lc[c][2] - a2; if (o2 < 0) o2 += k.mos[2];
                if (o0 < n0 && o1 < n1 && o2 < n2) {
                    const float w = (S.w[i][0][o0] * S.w[i][1][o1]) * S.w[i][2][o2];
#pragma unroll
                    for (int q = 0; q < CG; q++) {
                        const float2 v = S.v[i][q];
                        if (COMP) {
                            float y0 = w * v.x - cmp[c][q][0];
                            float t0 = acc[c][q][0] + y0;
                            cmp[c][q][0] = (t0 - acc[c][q][0]) - y0;
                            acc[c][q][0] = t0;
                            float y1 = w * v.y - cmp[c][q][1];
                            float t1 = acc[c][q][1] + y1;
                            cmp[c][q][1] = (t1 - acc[c][q][1]) - y1;
                            acc[c][q][1] = t1;
                        } else {
                            acc[c][q][0] = fmaf(w, v.x, acc[c][q][0]);
                            acc[c][q][1] = fmaf(w, v.y, acc[c][q][1]);
                        }
                    }
                }
            }
        }
        }
        if (ncnt > 0) stage_chunk(stage[cur ^ 1], ncnt);
        __syncthreads();
        cur ^= 1;
    }

    bool cell_ok[CPT];
#pragma unroll
    for (int c = 0; c < CPT; c++)
        cell_ok[c] = lc[c][0] < k.tile[0] && lc[c][1] < k.tile[1] && lc[c][2] < k.tile[2];
    auto cell_index = [&](int c) -> int64_t {   // address of the cell within its batch
        const int gx = org[0] + lc[c][0], gy = org[1] + lc[c][1], gz = org[2] + lc[c][2];
        return (int64_t)gz * a.kl.s_z + (int64_t)gy * a.kl.s_y + gx;
    };
    if (it.split < 0) {
#pragma unroll
        for (int c = 0; c < CPT; c++) {
            if (!cell_ok[c]) continue;
            const int64_t g = cell_index(c);
#pragma unroll
            for (int q = 0; q < CG; q++) {
                if (b0 + q >= a.nb) break;
                float2 *o = grid + ((int64_t)(b0 + q) * a.F + f) * a.kl.s_bf + g;
                float2 v = make_float2(acc[c][q][0], acc[c][q][1]);
                if (a.accumulate) { float2 old = *o; v.x += old.x; v.y += old.y; }
                *o = v;
            }
        }
        return;
    }
    // Split tile: write this chunk's partial, the last CTA reduces in order.
    const SplitInfo si = a.splits[it.split];
    const int cells = kThreads * CPT;
    auto part = [&](int slot) -> float2 * {
        return a.partials + ((int64_t)slot * a.ncg + grp) * (int64_t)CG * cells;
    };
    {
        float2 *pp = part(si.first_slot + it.chunk);
#pragma unroll
        for (int c = 0; c < CPT; c++)
#pragma unroll
            for (int q = 0; q < CG; q++)
                pp[(int64_t)q * cells + c * kThreads + threadIdx.x] = make_float2(acc[c][q][0], acc[c][q][1]);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int *ctr = a.counters + (int64_t)it.split * a.ncg + grp;
        unsigned int old = atomicAdd(ctr, 1u);
        s_last = (old == (unsigned int)(si.nchunks - 1));
        if (s_last) *ctr = 0u;   // ready for the next launch
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
#pragma unroll
    for (int c = 0; c < CPT; c++) {
        if (!cell_ok[c]) continue;
        const int64_t g = cell_index(c);
#pragma unroll
        for (int q = 0; q < CG; q++) {
            if (b0 + q >= a.nb) break;
            float sr = 0.f, sim = 0.f, cr = 0.f, ci = 0.f;
            for (int ch = 0; ch < si.nchunks; ch++) {
                const float2 v = __ldcg(&part(si.first_slot + ch)[(int64_t)q * cells + c * kThreads + threadIdx.x]);
                if (COMP) {
                    float y0 = v.x - cr, t0 = sr + y0; cr = (t0 - sr) - y0; sr = t0;
                    float y1 = v.y - ci, t1 = sim + y1; ci = (t1 - sim) - y1; sim = t1;
                } else {
                    sr += v.x;
                    sim += v.y;
                }
            }
            float2 *o = grid + ((int64_t)(b0 + q) * a.F + f) * a.kl.s_bf + g;
            float2 v = make_float2(sr, sim);
            if (a.accumulate) { float2 old = *o; v.x += old.x; v.y += old.y; }
            *o = v;
        }
    }
}

// ------------------------------------------ reference fold (3D, opt-in) --
//
// GB_FLAG_REFERENCE_FOLD.  The reference grids onto a padded grid and folds
// the ring back in wrap_image_kernel (ConvolverNC2C_standard.cuh:394-437):
// for each nonempty combination of dimensions it tries the 2^d wrap
// directions and adds the first periodic image whose dimensions all wrap.
// It tests whether dimension i (1-based) belongs to a combination with
// `i & combination` (:411-413), which for i = 3 looks at bits 0|1 instead of
// bit 2.  ref_fold_mult() restates that loop: how many times the periodic
// image at shift sigma (per dimension -1, 0, +1) is added to a cell in state
// st (per dimension 0 inside, 1 within the ring width of the low face, 2 of
// the high face).  It is 1 everywhere in 1D and 2D, and in 3D differs from 1
// only on cells within the ring width of a z face.  The periodic gridding
// counts every image once, so after it k_ref_fold_fix adds (mult - 1) times
// each wrapped tap's contribution (float atomics: few taps -- only samples
// whose footprint crosses the grid's edge have wrapped taps).
__device__ int ref_fold_mult(int D, const int *st, const int *sigma) {
    bool zero = true;
    for (int d = 0; d < D; d++) zero &= sigma[d] == 0;
    if (zero) return 1;
    int count = 0;
    for (int comb = 1; comb < (1 << D); comb++) {
        int nd = 0;
        for (int i = 0; i < D; i++) nd += (comb & (1 << i)) != 0;
        for (int sel = 0; sel < (1 << nd); sel++) {
            int stride[kMaxD] = {0, 0, 0}, wraps = 0, skipped = 0;
            for (int i = 1; i <= D; i++) {
                if (i & comb) {
                    if (i & (sel << skipped)) {
                        if (st[i - 1] == 2) { stride[i - 1] = -1; wraps++; }
                    } else {
                        if (st[i - 1] == 1) { stride[i - 1] = 1; wraps++; }
                    }
                } else {
                    skipped++;
                }
            }
            if (wraps == nd) {
                bool same = true;
                for (int d = 0; d < D; d++) same &= stride[d] == sigma[d];
                count += same ? 1 : 0;
                break;
            }
        }
    }
    return count;
}

// One thread per sorted sample; samples whose footprint stays inside the
// grid return at once.
__global__ void k_ref_fold_fix(ConvArgs a, const float2 *__restrict__ samples, float2 *__restrict__ grid) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const KParams &k = a.k;
    if (j >= a.Mtot) return;
    int lo[3], n[3];
    bool crosses = false;
    for (int d = 0; d < 3; d++) {
        const float s = a.pos[(int64_t)d * a.Mtot + j];
        lo[d] = (int)ceilf(s - k.radius);
        n[d] = min((int)floorf(s + k.radius) - lo[d] + 1, kWMax);
        const int u0 = lo[d] - k.hw, u1 = u0 + n[d] - 1;
        crosses |= u0 < 0 || u1 >= k.mos[d];
    }
    if (!crosses) return;
    const int f = (int)(a.home_key[j] / (uint32_t)k.ntiles_total);
    const uint32_t jo = a.perm[j];
    const float dw = a.dcw ? a.dcw[jo] : 1.f;
    const float *wt = a.wtab + j * 3 * kWMax;
    for (int tz = 0; tz < n[2]; tz++)
        for (int ty = 0; ty < n[1]; ty++)
            for (int tx = 0; tx < n[0]; tx++) {
                const int t[3] = {tx, ty, tz};
                int sigma[3], st[3], co[3];
                bool wrapped = false;
                for (int d = 0; d < 3; d++) {
                    const int u = lo[d] + t[d] - k.hw;
                    sigma[d] = u < 0 ? -1 : (u >= k.mos[d] ? 1 : 0);
                    co[d] = u - sigma[d] * k.mos[d];
                    st[d] = co[d] < k.hw ? 1 : (co[d] >= k.mos[d] - k.hw ? 2 : 0);
                    wrapped |= sigma[d] != 0;
                }
                if (!wrapped) continue;
                const int m = ref_fold_mult(3, st, sigma) - 1;
                if (m == 0) continue;
                float w = wt[tx] * (wt[kWMax + ty] * wt[2 * kWMax + tz]);
                if (a.sign_fold && ((co[0] + co[1] + co[2]) & 1)) w = -w;
                w *= (float)m * dw;
                const int64_t cell = (int64_t)co[2] * a.kl.s_z + (int64_t)co[1] * a.kl.s_y + co[0];
                for (int b = 0; b < a.nb; b++) {
                    float2 v;
                    if (a.layout == LAYOUT_SORTED_IL) v = samples[j * a.il_stride + b];
                    else if (a.layout == LAYOUT_SORTED) v = samples[(int64_t)b * a.Mtot + j];
                    else v = samples[(int64_t)b * a.Mtot + jo];
                    float *o = reinterpret_cast<float *>(grid + ((int64_t)b * a.F + f) * a.kl.s_bf + cell);
                    atomicAdd(o, w * v.x);
                    atomicAdd(o + 1, w * v.y);
                }
            }
}

static void launch_ref_fold_fix(const NufftPlan &p, const ConvArgs &a, const float2 *samples, float2 *grid,
                                cudaStream_t st) {
    if (!(p.flags & GB_FLAG_REFERENCE_FOLD) || p.D != 3 || p.Mtot == 0) return;
    k_ref_fold_fix<<<(unsigned)((p.Mtot + 255) / 256), 256, 0, st>>>(a, samples, grid); ::gb::note_launch();
    GB_CUDA(cudaGetLastError());
}

// --------------------------------------------------------------- C2NC -----

// Staged region of a home tile: tile + pad/2 cells on each side.
__host__ __device__ __forceinline__ int region_dim(const KParams &k, int d) {
    return d < k.D ? k.tile[d] + 2 * k.hw : 1;
}

// Per-warp staging area of the degridding kernel: separable weights (and
// their derivatives), region-local footprint starts and tap counts for the
// SPW samples a warp serves at once.
template <int SPW, bool GRAD>
struct DegridStage {
    float w[SPW][3][kWMax];
    float dw[GRAD ? SPW : 1][3][kWMax];
    int rs[SPW][3];
    int n[SPW][3];
};

template <int CG>
struct DegridShape {
    static constexpr int CPL = (CG >= 2) ? 2 : 1;   // coils per lane
    static constexpr int LPS = CG / CPL;            // lanes per sample
    static constexpr int SPW = 32 / LPS;            // samples per warp pass
};

// Degridding: a CTA stages its home tile plus a halo of pad/2 cells (coil
// fastest, so one sample's coil group is one contiguous row of CG complex
// values) and serves a range of the tile's home samples.  A warp serves SPW
// samples at once: LPS lanes per sample, CPL coils per lane, one 16-byte
// shared-memory load and 4 FMAs per tap per lane.
template <int CG, bool COMP, bool GRAD>
__global__ void __launch_bounds__(kThreads)
k_degrid_c2nc(ConvArgs a, const float2 *__restrict__ grid, float2 *__restrict__ out,
              const float2 *__restrict__ gweights, float *__restrict__ gout) {
    using Sh = DegridShape<CG>;
    constexpr int CPL = Sh::CPL, LPS = Sh::LPS, SPW = Sh::SPW;
    using Stage = DegridStage<SPW, GRAD>;
    extern __shared__ float4 smem_raw[];
    const KParams &k = a.k;
    const WorkItem it = a.items[blockIdx.x];
    const int f = it.f, tx = it.tx, ty = it.ty, tz = it.tz;
    const int org[3] = {tx * k.tile[0], ty * k.tile[1], tz * k.tile[2]};
    // the gradient sums its coil groups in turn, the degridding runs one per CTA
    for (int grp = GRAD ? 0 : (int)blockIdx.y; grp < (GRAD ? a.ncg : (int)blockIdx.y + 1); grp++) {
    const int b0 = grp * CG;
    if (GRAD && grp > 0) __syncthreads();   // the region is no longer read
    const int R0 = region_dim(k, 0), R1 = region_dim(k, 1), R2 = region_dim(k, 2);
    const int cellsR = R0 * R1 * R2;
    const int h0 = k.D > 0 ? k.hw : 0, h1 = k.D > 1 ? k.hw : 0, h2 = k.D > 2 ? k.hw : 0;
    float2 *tile_s = reinterpret_cast<float2 *>(smem_raw);
    Stage *stages = reinterpret_cast<Stage *>(tile_s + (((size_t)cellsR * CG + 1) & ~(size_t)1));

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // Stage the region, coil fastest: a warp per region row, lanes over
    // (x, coil) with coil fastest (conflict-free shared stores); the periodic
    // wrap needs one conditional per coordinate (|offset| < mos).
    {
        const int rowElems = R0 * CG;
        const int gx0 = org[0] - h0;
        for (int row = warp; row < R1 * R2; row += 8) {
            const int ry = row % R1, rz = row / R1;
            int gy = org[1] - h1 + ry;
            gy = gy < 0 ? gy + k.mos[1] : (gy >= k.mos[1] ? gy - k.mos[1] : gy);
            int gz = org[2] - h2 + rz;
            gz = gz < 0 ? gz + k.mos[2] : (gz >= k.mos[2] ? gz - k.mos[2] : gz);
            const int64_t rowoff = (int64_t)f * a.kl.s_bf + (int64_t)gz * a.kl.s_z + (int64_t)gy * a.kl.s_y;
            float2 *dst = tile_s + (size_t)row * rowElems;
            for (int e = lane; e < rowElems; e += 32) {
                const int c = e % CG;          // CG is a power of two
                const int rx = e / CG;
                int gx = gx0 + rx;
                gx = gx < 0 ? gx + k.mos[0] : (gx >= k.mos[0] ? gx - k.mos[0] : gx);
                // asynchronous 8-byte copy global -> shared (all of a thread's
                // copies in flight at once); coils beyond nb are zero-filled
                const bool in = b0 + c < a.nb;
                const float2 *src = in ? &grid[(int64_t)(b0 + c) * a.F * a.kl.s_bf + rowoff + gx] : grid;
                const unsigned saddr = (unsigned)__cvta_generic_to_shared(dst + e);
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(saddr), "l"(src),
                             "r"(in ? 8 : 0)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();

    const int sl = lane / LPS, ll = lane % LPS;
    Stage &S = stages[warp];
    const bool D3 = k.D > 2;

    for (int base = it.begin + warp * SPW; base < it.end; base += 8 * SPW) {
        // Separable weights of the warp's SPW samples, (sample, dim, tap) over lanes.
        for (int e = lane; e < SPW * 3 * kWMax; e += 32) {
            const int s = e / (3 * kWMax), d = (e / kWMax) % 3, t = e % kWMax;
            const int i = base + s;
            float w = 0.f, dw = 0.f;
            if (i < it.end && d < k.D) {
                const float sp = a.pos[(int64_t)d * a.Mtot + i];
                int n;
                const int lo = first_tap(k, sp, n);
                n = min(n, kWMax);
                if (t < n) {
                    const int g = lo + t;
                    const float diff = sp - (float)(g + k.hw);   // exact
                    // tap t of the sample's table row is the weight of |diff|
                    w = GRAD ? kb_weight_1d(fabsf(diff), k.mos_f[d], k.one_over_W, k.beta[d], k.radius)
                             : a.wtab[((int64_t)i * k.D + d) * kWMax + t];
                    if (GRAD) {
                        dw = kb_deriv_1d(fabsf(diff), k.mos_f[d], k.one_over_W, k.beta[d], k.radius);
                        dw = (diff < 0.f) ? -dw : dw;
                    }
                    if (a.sign_fold) {
                        const float sg = sign_of(wrapmod(g, k.mos[d]));
                        w *= sg;
                        dw *= sg;
                    }
                }
                if (t == 0) {
                    const int od = d == 0 ? org[0] : (d == 1 ? org[1] : org[2]);
                    S.rs[s][d] = wrapmod(lo - od + k.hw, k.mos[d]);
                    S.n[s][d] = n;
                }
            } else if (i < it.end) {
                w = (t == 0) ? 1.f : 0.f;
                if (t == 0) { S.rs[s][d] = 0; S.n[s][d] = 1; }
            } else if (t == 0) {
                S.rs[s][d] = 0;
                S.n[s][d] = 0;
            }
            S.w[s][d][t] = w;
            if (GRAD) S.dw[s][d][t] = dw;
        }
        __syncwarp();

        const int i = base + sl;
        const int rs0 = S.rs[sl][0], rs1 = S.rs[sl][1], rs2 = S.rs[sl][2];
        const int n0 = S.n[sl][0], n1 = S.n[sl][1], n2 = S.n[sl][2];
        float wx[kWMax], dwx[GRAD ? kWMax : 1];
#pragma unroll
        for (int t = 0; t < kWMax; t++) {
            const bool in = (t < n0) && (rs0 + t < R0);
            wx[t] = in ? S.w[sl][0][t] : 0.f;
            if (GRAD) dwx[t] = in ? S.dw[sl][0][t] : 0.f;
        }
        float acc[CPL][2], cmp[COMP ? CPL : 1][2];
        float gacc[GRAD ? CPL : 1][3][2];
#pragma unroll
        for (int c = 0; c < CPL; c++) {
            acc[c][0] = acc[c][1] = 0.f;
            if (COMP) cmp[c][0] = cmp[c][1] = 0.f;
            if (GRAD)
                for (int d = 0; d < 3; d++) gacc[c][d][0] = gacc[c][d][1] = 0.f;
        }
        for (int tzi = 0; tzi < n2; tzi++) {
            const int rz = rs2 + tzi;
            if (rz >= R2) break;
            const float wz = S.w[sl][2][tzi];
            const float dwz = GRAD ? S.dw[sl][2][tzi] : 0.f;
            for (int tyi = 0; tyi < n1; tyi++) {
                const int ry = rs1 + tyi;
                if (ry >= R1) break;
                const float wy = S.w[sl][1][tyi];
                const float dwy = GRAD ? S.dw[sl][1][tyi] : 0.f;
                const float2 *row = tile_s + ((size_t)(rz * R1 + ry) * R0 + rs0) * CG + ll * CPL;
#pragma unroll
                for (int t = 0; t < kWMax; t++) {
                    if (GRAD) {
                        if (wx[t] == 0.f && dwx[t] == 0.f) continue;
                    } else if (wx[t] == 0.f) {
                        continue;
                    }
                    float2 v[CPL];
                    if (CPL == 2) {
                        const float4 q = *reinterpret_cast<const float4 *>(row + t * CG);
                        v[0] = make_float2(q.x, q.y);
                        v[CPL - 1] = make_float2(q.z, q.w);
                    } else {
                        v[0] = row[t * CG];
                    }
                    if (GRAD) {
                        const float ax = (dwx[t] * wy) * wz, ay = (wx[t] * dwy) * wz, az = (wx[t] * wy) * dwz;
#pragma unroll
                        for (int c = 0; c < CPL; c++) {
                            gacc[c][0][0] = fmaf(ax, v[c].x, gacc[c][0][0]);
                            gacc[c][0][1] = fmaf(ax, v[c].y, gacc[c][0][1]);
                            gacc[c][1][0] = fmaf(ay, v[c].x, gacc[c][1][0]);
                            gacc[c][1][1] = fmaf(ay, v[c].y, gacc[c][1][1]);
                            gacc[c][2][0] = fmaf(az, v[c].x, gacc[c][2][0]);
                            gacc[c][2][1] = fmaf(az, v[c].y, gacc[c][2][1]);
                        }
                    } else {
                        float w = wx[t] * wy;
                        if (D3) w *= wz;
#pragma unroll
                        for (int c = 0; c < CPL; c++) {
                            if (COMP) {
                                float y0 = w * v[c].x - cmp[c][0];
                                float s0 = acc[c][0] + y0;
                                cmp[c][0] = (s0 - acc[c][0]) - y0;
                                acc[c][0] = s0;
                                float y1 = w * v[c].y - cmp[c][1];
                                float s1 = acc[c][1] + y1;
                                cmp[c][1] = (s1 - acc[c][1]) - y1;
                                acc[c][1] = s1;
                            } else {
                                acc[c][0] = fmaf(w, v[c].x, acc[c][0]);
                                acc[c][1] = fmaf(w, v[c].y, acc[c][1]);
                            }
                        }
                    }
                }
            }
        }
        const bool valid = i < it.end;
        const uint32_t j = valid ? a.perm[i] : 0u;
        const int64_t idx = (a.layout != LAYOUT_ORIGINAL) ? (int64_t)i : (int64_t)j;
        if (!GRAD) {
            if (valid) {
                float scale = 1.f;
                if (a.dcw) {
                    const float dw2 = a.dcw[j];
                    scale = (a.dcw_pow == 2) ? dw2 * dw2 : dw2;
                }
#pragma unroll
                for (int c = 0; c < CPL; c++) {
                    const int coil = b0 + ll * CPL + c;
                    if (coil >= a.nb) {
                        if (a.layout == LAYOUT_SORTED_IL && coil < a.il_stride)   // the row's padding
                            out[idx * a.il_stride + coil] = make_float2(0.f, 0.f);
                        break;
                    }
                    float2 val = make_float2(acc[c][0], acc[c][1]);
                    if (a.dcw) {
                        if (a.dcw_pow == 2) {
                            const float dw2 = a.dcw[j];
                            val.x = (val.x * dw2) * dw2;
                            val.y = (val.y * dw2) * dw2;
                        } else {
                            val.x *= scale;
                            val.y *= scale;
                        }
                    }
                    float2 *o = (a.layout == LAYOUT_SORTED_IL) ? out + idx * a.il_stride + coil
                                                            : out + (int64_t)coil * a.Mtot + idx;
                    if (a.accumulate) { const float2 ov = *o; val.x += ov.x; val.y += ov.y; }
                    *o = val;
                }
            }
        } else {
            float r[3] = {0.f, 0.f, 0.f};
            if (valid) {
#pragma unroll
                for (int c = 0; c < CPL; c++) {
                    const int coil = b0 + ll * CPL + c;
                    if (coil >= a.nb) break;
                    const float2 v = gweights[(int64_t)coil * a.Mtot + idx];
                    for (int d = 0; d < 3; d++) r[d] += v.x * gacc[c][d][0] - v.y * gacc[c][d][1];
                }
            }
#pragma unroll
            for (int off = 1; off < LPS; off <<= 1)
                for (int d = 0; d < 3; d++) r[d] += __shfl_xor_sync(0xffffffffu, r[d], off);
            if (valid && ll == 0) {
                float scale = 1.f;
                if (a.dcw) scale = (a.dcw_pow == 2) ? a.dcw[j] * a.dcw[j] : a.dcw[j];
                float *gp = gout + (int64_t)j * k.D;
                for (int d = 0; d < k.D; d++) {
                    const float v = r[d] * k.mos_f[d] * scale;
                    gp[d] = grp > 0 ? gp[d] + v : v;
                }
            }
        }
        __syncwarp();
    }
    }
}

// ------------------------------------------------------------ launchers ---

static ConvArgs make_args(NufftPlan &p, int nb, SampleLayout layout, const float *dcw,
                          int dcw_pow, bool sign_fold, bool accumulate) {
    ConvArgs a{};
    a.k = p.kp;
    a.pos = p.pos_sorted.get();
    a.wtab = p.wtab.get();
    a.kl = klayout_standard(p.kp);
    a.prows = p.pair_rows.get();
    a.prng = p.pair_rng;
    a.prow_floats = p.pair_row_stride;
    a.perm = p.perm.get();
    a.Mtot = p.Mtot;
    a.F = (int)p.F;
    a.nb = nb;
    a.layout = layout;
    a.il_stride = il_stride_for(nb);
    a.home_key = p.pp_key_sorted.get();
    a.dcw = dcw;
    a.dcw_pow = dcw_pow;
    a.sign_fold = sign_fold ? 1 : 0;
    a.accumulate = accumulate ? 1 : 0;
    return a;
}

int choose_cg(int requested, int nb) {
    int cg = requested;
    if (cg != 1 && cg != 2 && cg != 4 && cg != 8 && cg != 16) cg = 8;
    while (cg > 1 && cg / 2 >= nb) cg /= 2;
    return cg;
}

static GridCfg grid_config(const NufftPlan &p, int nb) {
    const KParams &k = p.kp;
    GridCfg c{};
    const int cells = k.tile[0] * k.tile[1] * k.tile[2];
    c.cpt = (cells + kThreads - 1) / kThreads;
    if (!brick_config(p, nb, c)) {
        const bool comp = (p.flags & GB_FLAG_COMPENSATED) != 0;
        c.cg = choose_cg(p.tiling.cg, nb);
        if (c.cpt * c.cg > (comp ? 16 : 32)) c.cg = std::max(1, (comp ? 16 : 32) / c.cpt);
    }
    c.ncg = (nb + c.cg - 1) / c.cg;
    c.part_elems = (int64_t)c.cg * (c.brick ? cells : kThreads * c.cpt);
    return c;
}

template <int CG, int CPT, bool COMP>
static void grid_dispatch(const ConvArgs &a, dim3 g, const float2 *s, float2 *o, cudaStream_t st) {
    k_grid_nc2c<CG, CPT, COMP><<<g, kThreads, 0, st>>>(a, s, o); ::gb::note_launch();
}

template <int CG, bool COMP>
static void grid_dispatch_cpt(int cpt, const ConvArgs &a, dim3 g, const float2 *s, float2 *o,
                              cudaStream_t st) {
    switch (cpt) {
        case 1: grid_dispatch<CG, 1, COMP>(a, g, s, o, st); break;
        case 2: grid_dispatch<CG, 2, COMP>(a, g, s, o, st); break;
        case 4: grid_dispatch<CG, 4, COMP>(a, g, s, o, st); break;
        default: fail(GB_ERR_INTERNAL, "unsupported cells per thread");
    }
}

// Launches the gridding kernel selected by `c` over all work items.
static void grid_dispatch_cfg(const GridCfg &c, const NufftPlan &p, const ConvArgs &a, const float2 *samples,
                              float2 *grid, cudaStream_t st) {
    dim3 g(a.n_items, c.ncg);
    if (c.brick) {
        launch_grid_brick(c, p, a, samples, grid, st);
    } else if (p.flags & GB_FLAG_COMPENSATED) {
        switch (c.cg) {
            case 1: grid_dispatch_cpt<1, true>(c.cpt, a, g, samples, grid, st); break;
            case 2: grid_dispatch_cpt<2, true>(c.cpt, a, g, samples, grid, st); break;
            case 4: grid_dispatch_cpt<4, true>(c.cpt, a, g, samples, grid, st); break;
            case 8: grid_dispatch_cpt<8, true>(c.cpt, a, g, samples, grid, st); break;
            default: grid_dispatch_cpt<16, true>(c.cpt, a, g, samples, grid, st); break;
        }
    } else {
        switch (c.cg) {
            case 1: grid_dispatch_cpt<1, false>(c.cpt, a, g, samples, grid, st); break;
            case 2: grid_dispatch_cpt<2, false>(c.cpt, a, g, samples, grid, st); break;
            case 4: grid_dispatch_cpt<4, false>(c.cpt, a, g, samples, grid, st); break;
            case 8: grid_dispatch_cpt<8, false>(c.cpt, a, g, samples, grid, st); break;
            default: grid_dispatch_cpt<16, false>(c.cpt, a, g, samples, grid, st); break;
        }
    }
    GB_CUDA(cudaGetLastError());
}

// Counters and partial tiles of the split tiles for one launch (null without
// splits), grown where they have to be.
struct SplitScratch {
    unsigned int *counters = nullptr;
    float2 *partials = nullptr;
};

static SplitScratch take_split_scratch(NufftPlan &p, const GridCfg &c, cudaStream_t st) {
    SplitScratch g;
    if (p.n_splits == 0) return g;
    const size_t ctr = ((size_t)p.n_splits * c.ncg * c.groups * sizeof(unsigned int) + 255) & ~(size_t)255;
    const size_t part = (size_t)p.n_slots * c.ncg * c.part_elems * sizeof(float2);
    if (ctr > p.grid_ctr_bytes) {   // the partial tiles move: nothing recorded earlier may share the allocation
        p.grid_ws.release();
        p.grid_ctr_bytes = ctr;
    }
    if (p.grid_ws.ensure(p.grid_ctr_bytes + part)) p.grid_ctr_clean = false;
    if (!p.grid_ctr_clean) {
        GB_CUDA(cudaMemsetAsync(p.grid_ws.get(), 0, p.grid_ctr_bytes, st));
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        GB_CUDA(cudaStreamIsCapturing(st, &cs));
        p.grid_ctr_clean = cs == cudaStreamCaptureStatusNone;   // a captured clear has not run yet
    }
    g.counters = reinterpret_cast<unsigned int *>(p.grid_ws.get());
    g.partials = reinterpret_cast<float2 *>(p.grid_ws.get() + p.grid_ctr_bytes);
    return g;
}

// Allocates the gridding scratch for `nb` batches (must run outside stream
// capture).
void launch_grid_prepare(NufftPlan &p, int nb, cudaStream_t st) { take_split_scratch(p, grid_config(p, nb), st); }

// Coils from which the adjoint lays the caller's samples into rows (2D, 3D).
// Adjoint in us, gathering / with rows: 49152 samples on 512^2, 5 coils 43.5 / 46.5, 8
// coils 48.4 / 50.2, 12 coils 62.0 / 59.8, 16 coils 69.2 / 65.0; 873 samples, 8 coils 22.8 /
// 24.8; 2.56 M samples on 192^3, 5 coils 1773 / 1686, 8 coils 1969 / 1866.
constexpr int kIlMinCoils[2] = {9, 5};

// The caller's samples are one plane per coil: from kIlMinCoils coils on they
// are first laid into sorted coil-interleaved rows (density weights folded in),
// so that a hit loads its coils as one run instead of one sector per coil.
// Only for coil pairs per lane (a coil group of 1 can be asked for with any
// coil count).  0: no rows.
size_t grid_row_elems(const NufftPlan &p, int nb) {
    if (nb < kIlMinCoils[p.D == 3]) return 0;
    const GridCfg c = grid_config(p, nb);
    return c.brick && c.cg >= 2 ? (size_t)il_stride_for(nb) * p.Mtot : 0;
}

void launch_grid(NufftPlan &p, const float2 *samples, float2 *grid, int nb, SampleLayout layout,
                 const float *dcw, bool sign_fold, bool accumulate, cudaStream_t st, const KLayout *kl, float2 *rows) {
    if (!p.prepped) fail(GB_ERR_NOT_PREPROCESSED, "preprocess has not been called");
    const GridCfg c = grid_config(p, nb);
    if (layout == LAYOUT_SORTED_IL && (!c.brick || dcw))
        fail(GB_ERR_INTERNAL, "interleaved samples need the brick gridding kernel and no density weights");
    if (p.n_grd_items == 0) return;
    const ConvArgs orig = make_args(p, nb, layout, dcw, 1, sign_fold, accumulate);
    const float2 *src = samples;
    SampleLayout lay = layout;
    if (rows && layout == LAYOUT_ORIGINAL && grid_row_elems(p, nb) > 0) {
        launch_samples_il(p, samples, dcw, nb, rows, st);
        src = rows;
        lay = LAYOUT_SORTED_IL;
    }
    const SplitScratch ws = take_split_scratch(p, c, st);
    ConvArgs a = make_args(p, nb, lay, lay == layout ? dcw : nullptr, 1, sign_fold, accumulate);
    if (kl) a.kl = *kl;
    a.list = p.grid_list.get();
    a.items = p.grd_items.get();
    a.n_items = p.n_grd_items;
    a.splits = p.splits.get();
    a.ncg = c.ncg;
    a.part_elems = c.part_elems;
    a.partials = ws.partials;
    a.counters = ws.counters;
    grid_dispatch_cfg(c, p, a, src, grid, st);
    ConvArgs fix = orig;
    fix.kl = a.kl;
    launch_ref_fold_fix(p, fix, samples, grid, st);
}

// The sample workspace layout of E^H E: interleaved rows when the brick
// gridding runs on coil pairs.
SampleLayout normal_op_layout(const NufftPlan &p, int nb) {
    const GridCfg c = grid_config(p, nb);
    return c.brick && c.cg >= 2 ? LAYOUT_SORTED_IL : LAYOUT_SORTED;
}

// Scratch (split-tile partial tiles and their counters) that a gridding launch
// needs for `nb` batches, in elements, with the fine or the coarse chunks.
void grid_scratch_need(const NufftPlan &p, int nb, bool coarse, size_t *partial_elems, size_t *counter_elems) {
    const GridCfg c = grid_config(p, nb);
    const int slots = coarse ? p.n_coarse_slots : p.n_slots;
    *partial_elems = p.n_splits > 0 ? (size_t)slots * c.ncg * c.part_elems : 0;
    *counter_elems = p.n_splits > 0 ? (size_t)p.n_splits * c.ncg * c.groups : 0;
}

// Partial-tile elements by which the fixed-scratch entry point accepts a call:
// long chunks, the batches rounded up to the plan's coil group (with compensated
// sums, to a group whose sums fit the cell kernel's registers).  The forms may
// take larger groups; such a call then runs on fewer batches at a time.
size_t grid_scratch_accepted(const NufftPlan &p, int nb) {
    const KParams &k = p.kp;
    const int cells = k.tile[0] * k.tile[1] * k.tile[2], cpt = (cells + kThreads - 1) / kThreads;
    int cg = choose_cg(p.tiling.cg, nb);
    if (p.flags & GB_FLAG_COMPENSATED) cg = std::min(cg, std::max(1, 16 / cpt));
    return p.n_splits > 0 ? (size_t)p.n_coarse_slots * ((nb + cg - 1) / cg * cg) * cells : 0;
}

// The gridding launch of launch_grid with caller-provided scratch: no device
// allocation.  `counters` must hold counter_elems zeros on entry (the kernel
// leaves them zero again when it completes).
void launch_grid_external_scratch(NufftPlan &p, const float2 *samples, float2 *grid, int nb, bool accumulate,
                                  bool coarse, float2 *partials, unsigned int *counters, cudaStream_t st) {
    if (!p.prepped) fail(GB_ERR_NOT_PREPROCESSED, "preprocess has not been called");
    const GridCfg c = grid_config(p, nb);
    ConvArgs a = make_args(p, nb, LAYOUT_ORIGINAL, nullptr, 1, false, accumulate);
    a.list = p.grid_list.get();
    a.ncg = c.ncg;
    a.part_elems = c.part_elems;
    a.partials = partials;
    a.counters = counters;
    if (p.n_grd_items == 0) return;
    const WorkItem *items = p.grd_items.get();
    auto run = [&](const WorkItem *first, int n, const SplitInfo *splits) {
        if (n == 0) return;
        a.items = first;
        a.n_items = n;
        a.splits = splits;
        grid_dispatch_cfg(c, p, a, samples, grid, st);
    };
    if (coarse) {
        run(items + p.n_grd_items, p.n_coarse_items, p.splits.get() + p.n_splits);
        run(items + (p.n_grd_items - p.n_light_items), p.n_light_items, p.splits.get());
    } else {
        run(items, p.n_grd_items, p.splits.get());
    }
    launch_ref_fold_fix(p, a, samples, grid, st);
}

template <int CG, bool GRAD>
static size_t degrid_smem_t(const KParams &k) {
    const size_t tile = (((size_t)region_dim(k, 0) * region_dim(k, 1) * region_dim(k, 2) * CG + 1) & ~(size_t)1) *
                        sizeof(float2);
    return tile + 8 * sizeof(DegridStage<DegridShape<CG>::SPW, GRAD>);
}

static size_t degrid_smem(const KParams &k, int cg, bool grad = false) {
    switch (cg) {
        case 1: return grad ? degrid_smem_t<1, true>(k) : degrid_smem_t<1, false>(k);
        case 2: return grad ? degrid_smem_t<2, true>(k) : degrid_smem_t<2, false>(k);
        case 4: return grad ? degrid_smem_t<4, true>(k) : degrid_smem_t<4, false>(k);
        case 8: return grad ? degrid_smem_t<8, true>(k) : degrid_smem_t<8, false>(k);
        default: return grad ? degrid_smem_t<16, true>(k) : degrid_smem_t<16, false>(k);
    }
}

template <int CG, bool COMP, bool GRAD>
static void degrid_launch(const ConvArgs &a, dim3 g, size_t smem, const float2 *grid, float2 *out,
                          const float2 *gw, float *gout, cudaStream_t st) {
    auto kern = k_degrid_c2nc<CG, COMP, GRAD>;
    if (smem > 48 * 1024)
        GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<g, kThreads, smem, st>>>(a, grid, out, gw, gout); ::gb::note_launch();
}

template <bool COMP, bool GRAD>
static void degrid_dispatch(int cg, const ConvArgs &a, dim3 g, size_t smem, const float2 *grid,
                            float2 *out, const float2 *gw, float *gout, cudaStream_t st) {
    switch (cg) {
        case 1: degrid_launch<1, COMP, GRAD>(a, g, smem, grid, out, gw, gout, st); break;
        case 2: degrid_launch<2, COMP, GRAD>(a, g, smem, grid, out, gw, gout, st); break;
        case 4: degrid_launch<4, COMP, GRAD>(a, g, smem, grid, out, gw, gout, st); break;
        case 8: degrid_launch<8, COMP, GRAD>(a, g, smem, grid, out, gw, gout, st); break;
        default: degrid_launch<16, COMP, GRAD>(a, g, smem, grid, out, gw, gout, st); break;
    }
}

static int degrid_cg(NufftPlan &p, int nb, bool grad = false) {
    int cg = choose_cg(p.tiling.cg, nb);
    while (cg > 1 && degrid_smem(p.kp, cg, grad) > 200 * 1024) cg /= 2;
    if (degrid_smem(p.kp, cg, grad) > 220 * 1024) fail(GB_ERR_INVALID_ARGUMENT, "tile too large for shared memory");
    return cg;
}

void launch_degrid(NufftPlan &p, const float2 *grid, float2 *samples, int nb, SampleLayout layout,
                   const float *dcw, int dcw_pow, bool sign_fold, bool accumulate, cudaStream_t st,
                   const KLayout *kl) {
    if (!p.prepped) fail(GB_ERR_NOT_PREPROCESSED, "preprocess has not been called");
    int cg = degrid_cg(p, nb);
    const bool comp = (p.flags & GB_FLAG_COMPENSATED) != 0;
    // 12 coils (or a multiple of 12): one group of 12 for the table kernel
    // instead of a group of 16 with 4 empty coil slots
    if (nb % 12 == 0 && nb % 16 != 0 && cg >= 8 && degrid_table_ok(p, 12)) cg = 12;
    const int ncg = (nb + cg - 1) / cg;
    ConvArgs a = make_args(p, nb, layout, dcw, dcw_pow, sign_fold, accumulate);
    if (kl) a.kl = *kl;
    a.items = p.deg_items.get();
    a.n_items = p.n_deg_items;
    if (p.n_deg_items == 0) return;
    if (degrid_table_ok(p, cg)) {
        launch_degrid_table(p, a, cg, ncg, comp, grid, samples, st);
        return;
    }
    dim3 g(p.n_deg_items, ncg);
    const size_t smem = degrid_smem(p.kp, cg);
    if (comp)
        degrid_dispatch<true, false>(cg, a, g, smem, grid, samples, nullptr, nullptr, st);
    else
        degrid_dispatch<false, false>(cg, a, g, smem, grid, samples, nullptr, nullptr, st);
    GB_CUDA(cudaGetLastError());
}

// Every sample has one home item, so every gradient is written; the coil
// groups of an item are summed by its CTA in turn.
void launch_traj_grad(NufftPlan &p, const float2 *grid, const float2 *weights, int nb,
                      const float *dcw, float *grad, bool sign_fold, cudaStream_t st, const KLayout *kl) {
    if (!p.prepped) fail(GB_ERR_NOT_PREPROCESSED, "preprocess has not been called");
    const int cg = degrid_cg(p, nb, true);
    const int ncg = (nb + cg - 1) / cg;
    ConvArgs a = make_args(p, nb, LAYOUT_ORIGINAL, dcw, 1, sign_fold, false);
    if (kl) a.kl = *kl;
    a.items = p.deg_items.get();
    a.n_items = p.n_deg_items;
    a.ncg = ncg;
    if (p.n_deg_items == 0) return;
    if (grad_table_ok(p, cg)) {
        launch_grad_table(p, a, cg, grid, weights, grad, st);
        return;
    }
    degrid_dispatch<false, true>(cg, a, dim3(p.n_deg_items), degrid_smem(p.kp, cg, true), grid, nullptr, weights, grad,
                                 st);
    GB_CUDA(cudaGetLastError());
}

}  // namespace gb

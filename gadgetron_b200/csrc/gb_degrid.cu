// Degridding (C2NC) from the per-trajectory weight table, and the trajectory
// gradient, 2D and 3D.
//
// Reference kernel: toolboxes/nfft/gpu/ConvolverC2NC.cuh:78-122,228-307 (+ the
// coil-fastest permute of cuGriddingConvolution.cu:329-334).  The gradient has
// no reference counterpart.
//
// A CTA stages its home tile plus a halo of pad/2 cells, coils of a cell
// adjacent, in shared memory; a warp then serves 32 / (lanes per sample)
// samples at once, a lane one coil pair of a sample (with 1 or 2 coils: a
// sample per lane).  Each lane reads its sample's tap weights from the table
// into registers one pass ahead and runs a fully unrolled NT x NT (x NT) tap
// nest: one shared load and the multiply-adds per tap.  NT is the largest tap
// count a footprint can have, floor(W) + 1; a footprint has NT or NT - 1 taps
// per dimension, and the last one is skipped where it has NT - 1: nothing outside
// the footprint is ever read, and no cell is read with a weight of zero (which
// would make a NaN of an infinite one).  Against re-reading the tap before it with
// weight zero: 278 -> 262 us (1.13 M samples in 23 frames, 5 coils, 512^2, W 5.5).
//
// Before, 1 and 2 coils and compensated sums went through k_degrid_c2nc, which
// evaluates and stages the weights per warp and predicates every tap: 28.4 ->
// 7.7 us (32768 radial samples, 1 coil, 256^2 grid), 156 -> 65 us (98304 spiral
// samples, 32 coils, compensated, 640^2).
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "gb_conv.cuh"

namespace gb {

// Staged region of a home tile: tile + pad/2 cells on each side.
__host__ __device__ __forceinline__ int region_dim_t(const KParams &k, int d) {
    return d < k.D ? k.tile[d] + 2 * k.hw : 1;
}

template <int CG>
struct TableShape {
    static constexpr int CPL = (CG >= 2) ? 2 : 1;   // coils per lane
    static constexpr int LPS = CG / CPL;            // lanes per sample
    static constexpr int SPW = 32 / LPS;            // samples per warp pass
};

// Staged cell stride in float2.  2D, 4 coils and more: an odd number of
// 16-byte chunks (conflict-free staging stores; the region copy is a large
// share of a 2D item's work) -- except 12 coils, whose unpadded region lets 4
// CTAs share an SM.  3D, and 1 or 2 coils: unpadded.
__host__ __device__ constexpr int cell_stride(int cg, bool d3) {
    return (d3 || cg == 12 || cg <= 2) ? cg : cg + 2;
}

// Region staging through registers.  Thread e of the CTA takes cells e, e +
// kThreads, ... of the region in x-fastest order (every load instruction is a
// coalesced run of one coil plane, no idle lanes at row ends), loads all CG
// coils of UC cells before storing any (the loads in flight cover the memory
// latency), then stores each cell's coils as 16-byte chunks (with padded
// cells, the chunks that a warp stores at once fall into different banks).
template <int CG, bool D3>
__device__ __forceinline__ void stage_region(const ConvArgs &a, int f, int b0, int org0, int org1, int org2,
                                             const float2 *__restrict__ grid, float2 *tile_s) {
    constexpr int CS = cell_stride(CG, D3);
    constexpr int UC = CG <= 4 ? 2 : 1;   // cells in flight per thread
    const KParams &k = a.k;
    const int R0 = region_dim_t(k, 0), R1 = region_dim_t(k, 1), R2 = region_dim_t(k, 2);
    const int ncell = R0 * R1 * R2;
    const int gx0 = org0 - k.hw, gy0 = org1 - k.hw, gz0 = org2 - (D3 ? k.hw : 0);
    const int64_t pstride = (int64_t)a.F * a.kl.s_bf;
    const float2 *fbase = grid + (int64_t)b0 * pstride + (int64_t)f * a.kl.s_bf;
    for (int e0 = threadIdx.x; e0 < ncell; e0 += UC * kThreads) {
        float2 v[UC][CG];
#pragma unroll
        for (int u = 0; u < UC; u++) {
            const int e = e0 + u * kThreads;
            const int row = e / R0, xo = e - row * R0;
            const int rz = row / R1, ry = row - rz * R1;
            int gx = gx0 + xo, gy = gy0 + ry, gz = gz0 + rz;
            gx = gx < 0 ? gx + k.mos[0] : (gx >= k.mos[0] ? gx - k.mos[0] : gx);
            gy = gy < 0 ? gy + k.mos[1] : (gy >= k.mos[1] ? gy - k.mos[1] : gy);
            gz = gz < 0 ? gz + k.mos[2] : (gz >= k.mos[2] ? gz - k.mos[2] : gz);
            const float2 *src = fbase + (int64_t)gz * a.kl.s_z + (int64_t)gy * a.kl.s_y + gx;
            const bool in = e < ncell;
#pragma unroll
            for (int c = 0; c < CG; c++)
                v[u][c] = (in && b0 + c < a.nb) ? __ldg(src + c * pstride) : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < UC; u++) {
            const int e = e0 + u * kThreads;
            if (e < ncell) {
                if (CG == 1) {
                    tile_s[e] = v[u][0];
                } else {
                    float4 *cell = reinterpret_cast<float4 *>(tile_s + (size_t)e * CS);
#pragma unroll
                    for (int q = 0; q < CG / 2; q++)
                        cell[q] = make_float4(v[u][2 * q].x, v[u][2 * q].y, v[u][(2 * q + 1) % CG].x,
                                              v[u][(2 * q + 1) % CG].y);
                }
            }
        }
    }
}

// Per-sample inputs of one pass (loaded a pass ahead).
struct TapRaw {
    float sp[3];
    float4 t0[3], t1[3];
    uint32_t j;
    float dw;
};

template <int CG, int NT, bool D3>
__device__ __forceinline__ void load_taps(const ConvArgs &a, const WorkItem &it, int bs, bool need_j, TapRaw &r) {
    using Sh = TableShape<CG>;
    constexpr int D = D3 ? 3 : 2;
    const int sl = (threadIdx.x & 31) / Sh::LPS;
    const int i = bs + sl;
    // idle lanes (past the item's end; the 2 spare lanes of coil group 12) load a valid row
    const int ic = (sl < Sh::SPW && i < it.end) ? i : it.begin;
#pragma unroll
    for (int d = 0; d < D; d++) {
        r.sp[d] = a.pos[(int64_t)d * a.Mtot + ic];
        const float4 *trow = reinterpret_cast<const float4 *>(a.wtab + ((int64_t)ic * D + d) * kWMax);
        r.t0[d] = __ldg(trow);
        r.t1[d] = NT > 4 ? __ldg(trow + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    r.j = need_j ? a.perm[ic] : (uint32_t)ic;
    r.dw = a.dcw ? a.dcw[r.j] : 1.f;
}

// Footprint of a pass's sample: region-local start rs, tap counts n (0 for an
// idle lane, at least NT - 1 otherwise), weights w with the checkerboard
// folded in, and the checkerboard sign s0 of the first tap.
template <int NT, bool D3>
__device__ __forceinline__ void unpack_taps(const ConvArgs &a, const TapRaw &r, bool valid, int org0, int org1,
                                            int org2, int (&rs)[3], int (&n)[3], float (&w)[3][NT], float (&s0)[3]) {
    const KParams &k = a.k;
    constexpr int D = D3 ? 3 : 2;
    rs[2] = 0;
    n[2] = 1;
    s0[2] = 1.f;
#pragma unroll
    for (int t = 0; t < NT; t++) w[2][t] = (t == 0) ? 1.f : 0.f;
#pragma unroll
    for (int d = 0; d < D; d++) {
        int taps;
        const int lo = first_tap(k, r.sp[d], taps);
        n[d] = valid ? min(taps, NT) : 0;
        const int od = d == 0 ? org0 : (d == 1 ? org1 : org2);
        int x = lo - od + k.hw;   // region-local start, |x| < 2 mos
        x = x < 0 ? x + k.mos[d] : (x >= k.mos[d] ? x - k.mos[d] : x);
        rs[d] = x;
        n[d] = min(n[d], region_dim_t(k, d) - x);   // the footprint lies inside the region; keep reads there
        const float tv[8] = {r.t0[d].x, r.t0[d].y, r.t0[d].z, r.t0[d].w, r.t1[d].x, r.t1[d].y, r.t1[d].z, r.t1[d].w};
        // centring checkerboard: (-1)^(cell) with cell = lo + t (mos even)
        s0[d] = (a.sign_fold && (lo & 1)) ? -1.f : 1.f;
#pragma unroll
        for (int t = 0; t < NT; t++) w[d][t] = (a.sign_fold && (t & 1)) ? -s0[d] * tv[t] : s0[d] * tv[t];
    }
}

__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }

// Degridding.  COMP: compensated sums (each lane's, in tap order).
// Bound by its shared loads (one 16-byte load per tap and coil pair) on long
// items, by the region copy and the latency of a pass on short ones.
template <int CG, int NT, bool D3, bool COMP>
__global__ void __launch_bounds__(kThreads, D3 ? 2 : (COMP ? 2 : (CG == 12 || CG <= 2 ? 4 : 3)))
k_degrid_table(ConvArgs a, const float2 *__restrict__ grid, float2 *__restrict__ out) {
    using Sh = TableShape<CG>;
    constexpr int CPL = Sh::CPL, LPS = Sh::LPS, SPW = Sh::SPW;
    constexpr int CS = cell_stride(CG, D3);
    extern __shared__ float4 smem_raw[];
    const KParams &k = a.k;
    const WorkItem it = a.items[blockIdx.x];
    const int b0 = (int)blockIdx.y * CG;
    const int org0 = it.tx * k.tile[0], org1 = it.ty * k.tile[1], org2 = it.tz * k.tile[2];
    const int R0 = region_dim_t(k, 0), R1 = region_dim_t(k, 1);
    float2 *tile_s = reinterpret_cast<float2 *>(smem_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sl = lane / LPS, ll = lane % LPS;
    const bool lane_ok = sl < SPW;
    const bool need_j = a.layout == LAYOUT_ORIGINAL || a.dcw;

    TapRaw cur, nxt;
    int base = it.begin + warp * SPW;
    if (base < it.end) load_taps<CG, NT, D3>(a, it, base, need_j, cur);
    stage_region<CG, D3>(a, it.f, b0, org0, org1, org2, grid, tile_s);
    __syncthreads();

    for (; base < it.end; base += 8 * SPW) {
        const int i = base + sl;
        const bool valid = lane_ok && i < it.end;
        if (base + 8 * SPW < it.end) load_taps<CG, NT, D3>(a, it, base + 8 * SPW, need_j, nxt);
        int rs[3], n[3];
        float w[3][NT], s0[3];
        unpack_taps<NT, D3>(a, cur, valid, org0, org1, org2, rs, n, w, s0);
        // (re, im) of each of the lane's coils, packed FP32x2 multiply-adds
        float2 acc[CPL], cmp[CPL];
#pragma unroll
        for (int c = 0; c < CPL; c++) acc[c] = cmp[c] = make_float2(0.f, 0.f);
        const float2 *base_s = tile_s + (((size_t)rs[2] * R1 + rs[1]) * R0 + rs[0]) * CS + ll * CPL;
        const bool full_x = n[0] >= NT, full_y = n[1] >= NT;   // tap NT - 1 along x and y
        auto tap = [&](float2 wv, float2 v, int c) {
            if (COMP) {
                const float2 t = __ffma2_rn(wv, v, neg2(cmp[c]));
                const float2 s = __fadd2_rn(acc[c], t);
                cmp[c] = __fadd2_rn(__fadd2_rn(s, neg2(acc[c])), neg2(t));
                acc[c] = s;
            } else {
                acc[c] = __ffma2_rn(wv, v, acc[c]);
            }
        };
        // Tap nest of NTT taps per dimension; NT - 1 when every sample of the
        // warp has fewer than NT in every dimension (W an even integer: NT only
        // at exact-integer positions).
        auto nest = [&](auto ntc) {
            constexpr int NTT = decltype(ntc)::value;
#pragma unroll
            for (int tz = 0; tz < (D3 ? NTT : 1); tz++) {
                if (tz < n[2]) {
#pragma unroll
                    for (int ty = 0; ty < NTT; ty++) {
                        if (ty == NT - 1 && !full_y) continue;
                        const float wyz = D3 ? w[1][ty] * w[2][tz] : w[1][ty];
                        const float2 *row = base_s + (size_t)tz * R1 * R0 * CS + ty * R0 * CS;
#pragma unroll
                        for (int t = 0; t < NTT; t++) {
                            if (t == NT - 1 && !full_x) continue;
                            const float wv = w[0][t] * wyz;
                            const float2 wv2 = make_float2(wv, wv);
                            const float2 *cell = row + t * CS;
                            if (CPL == 2) {
                                const float4 q = *reinterpret_cast<const float4 *>(cell);
                                tap(wv2, make_float2(q.x, q.y), 0);
                                tap(wv2, make_float2(q.z, q.w), CPL - 1);
                            } else {
                                tap(wv2, *cell, 0);
                            }
                        }
                    }
                }
            }
        };
        const bool shorter = (NT > 4 && 2 * k.hw < NT) &&
                             __all_sync(0xffffffffu, n[0] < NT && n[1] < NT && n[2] < NT);
        if (shorter)
            nest(std::integral_constant<int, (NT > 4 ? NT - 1 : NT)>{});
        else
            nest(std::integral_constant<int, NT>{});
        if (valid) {
            const int64_t idx = (a.layout != LAYOUT_ORIGINAL) ? (int64_t)i : (int64_t)cur.j;
            const float dw = cur.dw;
#pragma unroll
            for (int c = 0; c < CPL; c++) {
                const int coil = b0 + ll * CPL + c;
                if (coil >= a.nb) {
                    if (a.layout == LAYOUT_SORTED_IL && coil < a.il_stride)   // the row's padding
                        out[idx * a.il_stride + coil] = make_float2(0.f, 0.f);
                    break;
                }
                float2 val = acc[c];
                if (a.dcw) {
                    if (a.dcw_pow == 2) {
                        val.x = (val.x * dw) * dw;
                        val.y = (val.y * dw) * dw;
                    } else {
                        val.x *= dw;
                        val.y *= dw;
                    }
                }
                float2 *o = (a.layout == LAYOUT_SORTED_IL) ? out + idx * a.il_stride + coil
                                                            : out + (int64_t)coil * a.Mtot + idx;
                if (a.accumulate) { const float2 ov = *o; val.x += ov.x; val.y += ov.y; }
                *o = val;
            }
        }
        cur = nxt;
    }
}

// Trajectory gradient: grad[j][d] = mos_d dcw_j sum_b Re(g[b][j] sum_taps
// d phi/d s_d * grid[b][tap]).  Per tap the lane first contracts its coils
// with the caller's weights (s = Re sum g v, kept as an FP32x2 pair that is
// added up at the end), so the three derivative sums cost two packed
// multiply-adds per tap and a few per row instead of six multiply-adds per
// coil.  The derivative weights are evaluated once per sample and tap by the
// lanes of the warp and kept in shared memory; the coil groups of an item
// follow one another in its CTA and add up in the output (no partial arrays, no
// allocation and no synchronisation of the call).  83.5 -> 33 us (49152 radial
// samples, 16 coils, 512^2 grid), 528 -> 252 us (320000 kooshball samples, 8
// coils, 96^3: one CTA per SM there, bound by the latency of its few warps).
template <int CG, int NT, bool D3>
__global__ void __launch_bounds__(kThreads, 2)
k_traj_grad(ConvArgs a, const float2 *__restrict__ grid, const float2 *__restrict__ gweights, float *__restrict__ gout) {
    using Sh = TableShape<CG>;
    constexpr int CPL = Sh::CPL, LPS = Sh::LPS, SPW = Sh::SPW;
    constexpr int CS = cell_stride(CG, D3), D = D3 ? 3 : 2;
    extern __shared__ float4 smem_raw[];
    const KParams &k = a.k;
    const WorkItem it = a.items[blockIdx.x];
    const int org0 = it.tx * k.tile[0], org1 = it.ty * k.tile[1], org2 = it.tz * k.tile[2];
    const int R0 = region_dim_t(k, 0), R1 = region_dim_t(k, 1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sl = lane / LPS, ll = lane % LPS;
    float *dwt = reinterpret_cast<float *>(smem_raw) + warp * (SPW * D * kWMax);   // [sample][dim][tap]
    float2 *tile_s = reinterpret_cast<float2 *>(reinterpret_cast<float *>(smem_raw) + 8 * SPW * D * kWMax);

    for (int grp = 0; grp < a.ncg; grp++) {
        const int b0 = grp * CG;
        if (grp > 0) __syncthreads();   // the region is no longer read
        stage_region<CG, D3>(a, it.f, b0, org0, org1, org2, grid, tile_s);
        __syncthreads();
        for (int base = it.begin + warp * SPW; base < it.end; base += 8 * SPW) {
            const int i = base + sl;
            const bool valid = i < it.end;
            TapRaw cur;
            load_taps<CG, NT, D3>(a, it, base, true, cur);
            float2 gw[CPL];   // (re, -im) of the caller's weights
#pragma unroll
            for (int c = 0; c < CPL; c++) {
                const int coil = b0 + ll * CPL + c;
                gw[c] = make_float2(0.f, 0.f);
                if (valid && coil < a.nb) {
                    const float2 g = gweights[(int64_t)coil * a.Mtot + cur.j];
                    gw[c] = make_float2(g.x, -g.y);
                }
            }
            __syncwarp();   // the derivative weights of the last pass are no longer read
            for (int e = lane; e < SPW * D * kWMax; e += 32) {
                const int s = e / (D * kWMax), d = (e / kWMax) % D, t = e % kWMax;
                float dw = 0.f;
                if (base + s < it.end) {
                    const float sp = a.pos[(int64_t)d * a.Mtot + base + s];
                    int n;
                    const int lo = first_tap(k, sp, n);
                    if (t < min(n, NT)) {
                        const float diff = sp - (float)(lo + k.hw + t);
                        dw = kb_deriv_1d(fabsf(diff), k.mos_f[d], k.one_over_W, k.beta[d], k.radius);
                        if (diff < 0.f) dw = -dw;
                        if (a.sign_fold && ((lo + t) & 1)) dw = -dw;
                    }
                }
                dwt[e] = dw;
            }
            __syncwarp();
            int rs[3], n[3];
            float w[3][NT], s0[3];
            unpack_taps<NT, D3>(a, cur, valid, org0, org1, org2, rs, n, w, s0);
            const float *dws = dwt + sl * (D * kWMax);
            float dx[NT];
#pragma unroll
            for (int t = 0; t < NT; t++) dx[t] = dws[t];
            const float2 *base_s = tile_s + (((size_t)rs[2] * R1 + rs[1]) * R0 + rs[0]) * CS + ll * CPL;
            const bool full_x = n[0] >= NT, full_y = n[1] >= NT;
            float2 r[3] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
            for (int tz = 0; tz < (D3 ? NT : 1); tz++) {
                if (tz >= n[2]) continue;
                const float wz = D3 ? w[2][tz] : 1.f, dz = D3 ? dws[2 * kWMax + tz] : 0.f;
                const float2 *slice = base_s + (size_t)tz * R1 * R0 * CS;
#pragma unroll
                for (int ty = 0; ty < NT; ty++) {
                    if (ty == NT - 1 && !full_y) continue;
                    const float2 *row = slice + ty * R0 * CS;
                    float2 A = make_float2(0.f, 0.f), B = make_float2(0.f, 0.f);   // sums with the weights, the derivatives
#pragma unroll
                    for (int t = 0; t < NT; t++) {
                        if (t == NT - 1 && !full_x) continue;
                        const float2 *cell = row + t * CS;
                        float2 s;
                        if (CPL == 2) {
                            const float4 q = *reinterpret_cast<const float4 *>(cell);
                            s = __ffma2_rn(gw[CPL - 1], make_float2(q.z, q.w), __fmul2_rn(gw[0], make_float2(q.x, q.y)));
                        } else {
                            s = __fmul2_rn(gw[0], *cell);
                        }
                        A = __ffma2_rn(make_float2(w[0][t], w[0][t]), s, A);
                        B = __ffma2_rn(make_float2(dx[t], dx[t]), s, B);
                    }
                    const float wy = w[1][ty], dy = dws[kWMax + ty];
                    const float cx = wy * wz, cy = dy * wz;
                    r[0] = __ffma2_rn(make_float2(cx, cx), B, r[0]);
                    r[1] = __ffma2_rn(make_float2(cy, cy), A, r[1]);
                    if (D3) {
                        const float cz = wy * dz;
                        r[2] = __ffma2_rn(make_float2(cz, cz), A, r[2]);
                    }
                }
            }
            float g[3] = {r[0].x + r[0].y, r[1].x + r[1].y, r[2].x + r[2].y};
#pragma unroll
            for (int off = 1; off < LPS; off <<= 1)
#pragma unroll
                for (int d = 0; d < D; d++) g[d] += __shfl_xor_sync(0xffffffffu, g[d], off);
            if (valid && ll == 0) {
                float *gp = gout + (int64_t)cur.j * D;
#pragma unroll
                for (int d = 0; d < D; d++) {
                    const float v = g[d] * k.mos_f[d] * cur.dw;
                    gp[d] = grp > 0 ? gp[d] + v : v;
                }
            }
        }
    }
}

// ------------------------------------------------------------- dispatch ---

static size_t region_smem(const KParams &k, int cg) {
    return (size_t)region_dim_t(k, 0) * region_dim_t(k, 1) * region_dim_t(k, 2) * cell_stride(cg, k.D == 3) *
           sizeof(float2);
}

static int table_taps(const NufftPlan &p) { return (int)std::floor(p.W) + 1; }   // most taps per dimension

// Whether the table kernel serves coil group cg: 2D and 3D, 4 to 8 taps, the
// region within shared memory.
bool degrid_table_ok(const NufftPlan &p, int cg) {
    const int nt = table_taps(p);
    return p.D >= 2 && nt >= 4 && nt <= kWMax && region_smem(p.kp, cg) <= 220 * 1024;
}

static size_t grad_smem(const KParams &k, int cg) {
    const int spw = cg >= 2 ? 32 / (cg / 2) : 32;
    return region_smem(k, cg) + (size_t)8 * spw * k.D * kWMax * sizeof(float);
}

bool grad_table_ok(const NufftPlan &p, int cg) {
    const int nt = table_taps(p);
    return p.D >= 2 && nt >= 4 && nt <= kWMax && cg != 12 && grad_smem(p.kp, cg) <= 220 * 1024;
}

template <int CG, int NT, bool D3, bool COMP>
static void table_launch(const ConvArgs &a, dim3 g, size_t smem, const float2 *grid, float2 *out, cudaStream_t st) {
    auto kern = k_degrid_table<CG, NT, D3, COMP>;
    if (smem > 48 * 1024)
        GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<g, kThreads, smem, st>>>(a, grid, out); note_launch();
}

template <int CG, int NT, bool D3>
static void grad_launch(const ConvArgs &a, size_t smem, const float2 *grid, const float2 *w, float *out,
                        cudaStream_t st) {
    auto kern = k_traj_grad<CG, NT, D3>;
    if (smem > 48 * 1024)
        GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<(unsigned)a.n_items, kThreads, smem, st>>>(a, grid, w, out); note_launch();
}

#define GB_TAPS(CALL)            \
    switch (nt) {                \
        case 4: CALL(4); break;  \
        case 5: CALL(5); break;  \
        case 6: CALL(6); break;  \
        case 7: CALL(7); break;  \
        default: CALL(8); break; \
    }

template <int CG, bool D3, bool COMP>
static void table_taps_dispatch(int nt, const ConvArgs &a, dim3 g, size_t smem, const float2 *grid, float2 *out,
                                cudaStream_t st) {
#define GB_CALL(N) table_launch<CG, N, D3, COMP>(a, g, smem, grid, out, st)
    GB_TAPS(GB_CALL)
#undef GB_CALL
}

template <int CG, bool D3>
static void grad_taps_dispatch(int nt, const ConvArgs &a, size_t smem, const float2 *grid, const float2 *w, float *out,
                               cudaStream_t st) {
#define GB_CALL(N) grad_launch<CG, N, D3>(a, smem, grid, w, out, st)
    GB_TAPS(GB_CALL)
#undef GB_CALL
}

template <bool D3, bool COMP>
static void table_group_dispatch(int cg, int nt, const ConvArgs &a, dim3 g, size_t smem, const float2 *grid,
                                 float2 *out, cudaStream_t st) {
    switch (cg) {
        case 1: table_taps_dispatch<1, D3, COMP>(nt, a, g, smem, grid, out, st); break;
        case 2: table_taps_dispatch<2, D3, COMP>(nt, a, g, smem, grid, out, st); break;
        case 4: table_taps_dispatch<4, D3, COMP>(nt, a, g, smem, grid, out, st); break;
        case 8: table_taps_dispatch<8, D3, COMP>(nt, a, g, smem, grid, out, st); break;
        case 12: table_taps_dispatch<12, D3, COMP>(nt, a, g, smem, grid, out, st); break;
        default: table_taps_dispatch<16, D3, COMP>(nt, a, g, smem, grid, out, st); break;
    }
}

void launch_degrid_table(const NufftPlan &p, const ConvArgs &a, int cg, int ncg, bool comp, const float2 *grid,
                         float2 *out, cudaStream_t st) {
    const int nt = table_taps(p);
    const size_t smem = region_smem(p.kp, cg);
    const dim3 g((unsigned)a.n_items, (unsigned)ncg);
    if (p.D == 3) {
        if (comp) table_group_dispatch<true, true>(cg, nt, a, g, smem, grid, out, st);
        else table_group_dispatch<true, false>(cg, nt, a, g, smem, grid, out, st);
    } else {
        if (comp) table_group_dispatch<false, true>(cg, nt, a, g, smem, grid, out, st);
        else table_group_dispatch<false, false>(cg, nt, a, g, smem, grid, out, st);
    }
    GB_CUDA(cudaGetLastError());
}

template <bool D3>
static void grad_group_dispatch(int cg, int nt, const ConvArgs &a, size_t smem, const float2 *grid, const float2 *w,
                                float *out, cudaStream_t st) {
    switch (cg) {
        case 1: grad_taps_dispatch<1, D3>(nt, a, smem, grid, w, out, st); break;
        case 2: grad_taps_dispatch<2, D3>(nt, a, smem, grid, w, out, st); break;
        case 4: grad_taps_dispatch<4, D3>(nt, a, smem, grid, w, out, st); break;
        case 8: grad_taps_dispatch<8, D3>(nt, a, smem, grid, w, out, st); break;
        default: grad_taps_dispatch<16, D3>(nt, a, smem, grid, w, out, st); break;
    }
}

void launch_grad_table(const NufftPlan &p, const ConvArgs &a, int cg, const float2 *grid, const float2 *w, float *out,
                       cudaStream_t st) {
    const size_t smem = grad_smem(p.kp, cg);
    if (p.D == 3) grad_group_dispatch<true>(cg, table_taps(p), a, smem, grid, w, out, st);
    else grad_group_dispatch<false>(cg, table_taps(p), a, smem, grid, w, out, st);
    GB_CUDA(cudaGetLastError());
}

}  // namespace gb

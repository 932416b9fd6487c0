// Gridding (NC2C), 2D and 3D: one warp per brick of cells.
//
// Reference kernels this replaces:
//   toolboxes/nfft/gpu/ConvolverNC2C_standard.cuh:229-355 (+ the wrap pass
//   :358-477 and the cell/sample pair sort of
//   toolboxes/nfft/gpu/cuGriddingConvolution.cu:361-422)
//
// A tile of the oversampled grid is cut into bricks; a warp owns one brick for
// one coil group and walks the tile's sample list alone: it tests 32 samples
// at a time against its brick (one ballot over the packed footprint ranges) and
// queues the hits; batches of queued hits are staged into a small ring of the
// warp's own shared memory by asynchronous copies (coil values, and the x, y, z
// weights of the brick from the sample's pair row -- weights laid over the
// tile, zero outside the footprint) two batches ahead of the one being summed.
// A lane is a (few coils, x column[, y block]) of the brick and keeps YC x ZC
// cells of 1 to 4 coils in registers; a hit costs it a few shared loads and
// packed FP32x2 multiply-adds over pairs of y cells.  Warps never wait for one
// another inside a list (only the chunks of a split tile meet, through a
// counter), and a lane's cells go straight from registers to the grid.  No
// atomics on the grid; per-cell sums follow the list order: results are
// bit-reproducible.
//
// What bounds it, and what was tried: loading a hit's operands straight from
// L2 one hit ahead left every warp waiting on that latency (118 us for the
// launch below against 36 us); one staged hit per copy spent 115 instructions
// a hit on staging, batches of 4 to 8 spend about 15.  Now 16 coils in 2D (wide
// form, 1.13 M samples on 384^2) issue on 55 % of the cycles with the shared-memory
// pipe at 41 %, 85 instructions a hit, and wait on their few warps' chains; 3D is
// issue- and latency-bound at 16 warps per SM (64 accumulators a lane).  Launch
// times before (a CTA per tile staging chunks through registers or a producer
// warp) and after:
//   32768 radial samples, 1 coil, 256^2 grid           63.6 -> 17 us
//   98304 spiral samples, 32 coils, compensated, 640^2  411 -> 140 us
//   5.12 M kooshball samples, 32 coils, 192^3          13.2 -> 7.5 ms
//   1.13 M samples in 23 frames, 12 coils, 512^2        485 -> 364 us
//   the same, 16 coils / 18 coils                       499 -> 448 / 935 -> 839 us
//   49152 radial samples, 16 coils, 512^2                37 -> 35 us
//   46000 samples, 16 coils, 96^2                       203 -> 43 us
//
// A zero weight times an infinity would put a NaN into cells the footprint
// does not touch, so a brick whose sums came out non-finite is summed again
// with the zero-weight cells skipped (the values of finite data never change).
#include <algorithm>
#include <type_traits>

#include "gb_conv.cuh"

namespace gb {

// CPL coils per lane, LPC lanes over the coils of a group, XL x YL lanes over
// the columns, YC x ZC cells per lane, at most NT threads (warps * 32) per CTA,
// MB resident CTAs asked of the register allocation, at most CTA bricks per CTA
// (a CTA's slot is held until its slowest brick is done -- samples crowd -- so a
// tile of more bricks is spread over several CTAs).
template <int CPL_, int LPC_, int XL_, int YL_, int YC_, int ZC_, bool D3_, int NT_, int MB_, int CTA_ = 4>
struct BrickShape {
    static constexpr int CPL = CPL_, LPC = LPC_, XL = XL_, YL = YL_, YC = YC_, ZC = ZC_, NT = NT_, MB = MB_, CTA = CTA_;
    static constexpr bool D3 = D3_;
    static constexpr int CG = CPL * LPC, BX = XL, BY = YL * YC, BZ = ZC, YP = YC / 2, V = 2 * CPL;
    static constexpr int NACC = ZC * YP * V;   // float2 accumulators of a lane
    // A staged hit, in 16-byte chunks: coil values, x, y and z weights of the
    // brick (x and z from the aligned group of 4 that holds them).
    static constexpr int VC = (CG * 8 + 15) / 16, XC = (BX + 3) / 4, YCH = BY / 4, ZCH = D3 ? 1 : 0;
    static constexpr int WCH = XC + YCH + ZCH, WL = WCH <= 4 ? 4 : 8;       // weight chunks, lanes staging them
    static constexpr int SLOT = VC + WCH + 1;                               // one more: the density weight
    static constexpr int UH = NACC > 16 ? 1 : 2;                            // hits summed together
    static constexpr int HB = CG >= 12 ? 4 : 8;                             // hits staged together
    static_assert(32 * CTA <= NT, "a CTA's bricks fit its threads");
    static_assert(LPC * XL * YL == 32 && YC % 2 == 0 && BY % 4 == 0, "a brick fills a warp");
};

constexpr int kBrickDepth = 3;    // batches of hits in the ring of a warp
constexpr int kBrickQueue = 64;   // pending hits of a warp
constexpr int kBrickMax = 16;     // bricks per tile
// Warps up to which bricks share their lists among several warps (and the narrow
// form takes 2 bricks per CTA).  Gridding in us at 0 / 888 / 1776 / 3552: 4096 samples on 128^2, 1
// coil 15.9 / 13.3 / 13.2 / 12.8, 16 coils 23.0 / 19.7 / 18.2 / 18.4; 16384 samples on 256^2, 1 coil 17.0 /
// 17.2 / 15.2 / 15.0.
constexpr int kBrickFillWarps = kSMs * 12;
constexpr int kBrickWideWarps = kSMs * 24 * 4;   // narrow-form warps from which the wide forms are taken
constexpr int64_t kBrick3DWidePairs = 4 << 20;   // pairs from which 8 coils in 3D take four slices
constexpr int kBrickWideList = 512;     // average list up to which they are

// Asynchronous copy of BYTES to shared memory; zeros instead when !full.
template <int BYTES>
__device__ __forceinline__ void cp_async(void *dst, const void *src, bool full) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(d), "l"(src), "n"(BYTES), "r"(full ? BYTES : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

__device__ __forceinline__ float2 f2neg(float2 a) { return make_float2(-a.x, -a.y); }

// Compensated sum += v.
__device__ __forceinline__ void comp_add(float2 &sum, float2 &err, float2 v) {
    const float2 t = __fadd2_rn(v, f2neg(err));
    const float2 n = __fadd2_rn(sum, t);
    err = __fadd2_rn(__fadd2_rn(n, f2neg(sum)), f2neg(t));
    sum = n;
}

template <class S, bool COMP, bool IL>
__global__ void __launch_bounds__(S::NT, COMP ? (S::MB + 1) / 2 : S::MB)
k_grid_brick(ConvArgs a, const float2 *__restrict__ samples, float2 *__restrict__ grid) {
    constexpr int CPL = S::CPL, LPC = S::LPC, YC = S::YC, ZC = S::ZC, YP = S::YP, V = S::V;
    constexpr bool D3 = S::D3;
    constexpr int VC = S::VC, XC = S::XC, YCH = S::YCH, WCH = S::WCH, WL = S::WL, SLOT = S::SLOT, HB = S::HB;
    constexpr int DEPTH = kBrickDepth;
    // [warps][DEPTH][HB][SLOT] staged hits, [warps][kBrickQueue] pending hits;
    // afterwards the sums of list parts
    extern __shared__ float4 brick_sm[];
    __shared__ int s_last;
    const KParams &k = a.k;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int b0 = (int)blockIdx.y * S::CG;
    // a tile's bricks are spread over `groups` CTAs of 1 << lcta bricks
    const int groups = 1 << (a.lbricks - a.lcta), group = (int)blockIdx.x & (groups - 1);
    const WorkItem it = a.items[blockIdx.x >> (a.lbricks - a.lcta)];
    const int T0 = k.tile[0], T1 = k.tile[1];
    // `parts` warps share a brick: part p takes blocks p, p + parts, ... of the list
    const int nbricks = 1 << a.lcta, parts = 1 << a.lparts;   // bricks of this CTA
    const int slot_id = warp & (nbricks - 1), part_id = warp >> a.lcta;
    const int brick = (group << a.lcta) + slot_id;
    const int bx = brick & ((1 << a.lbx) - 1), by = (brick >> a.lbx) & ((1 << a.lby) - 1), bz = brick >> (a.lbx + a.lby);
    const int x0 = bx * S::BX, y0 = by * S::BY, z0 = bz * S::BZ;   // the brick within the tile
    const int cp = lane % LPC, lx = (lane / LPC) % S::XL, ly = lane / (LPC * S::XL);
    const int coil = b0 + CPL * cp;
    const bool coil_ok = coil < a.nb;
    float4 *ring = brick_sm + warp * (DEPTH * HB * SLOT);
    uint2 *queue = reinterpret_cast<uint2 *>(brick_sm + (blockDim.x >> 5) * (DEPTH * HB * SLOT)) + warp * kBrickQueue;

    float2 acc[ZC][YP][V];                                    // [z][y pair][re, im of each coil]
    float2 cmp[COMP ? ZC : 1][COMP ? YP : 1][COMP ? V : 1];

    // This lane's weight chunk when staging (WL lanes per hit).
    const int wch = lane % WL;
    const int woff = wch < XC ? (x0 & ~3) + 4 * wch
                              : (wch < XC + YCH ? T0 + y0 + 4 * (wch - XC) : T0 + T1 + (z0 & ~3));
    const float *wsrc = a.prows + woff;

    auto pass = [&](auto safe_c) {
        constexpr bool SAFE = decltype(safe_c)::value;
#pragma unroll
        for (int z = 0; z < ZC; z++)
#pragma unroll
            for (int y = 0; y < YP; y++)
#pragma unroll
                for (int c = 0; c < V; c++) {
                    acc[z][y][c] = make_float2(0.f, 0.f);
                    if (COMP) cmp[z][y][c] = make_float2(0.f, 0.f);
                }
        // values of coils beyond nb are never staged: zero them once
        for (int e = lane; e < DEPTH * HB * SLOT; e += 32) ring[e] = make_float4(0.f, 0.f, 0.f, 0.f);
        // Blocks of 32 list entries: the next block's entries are loaded
        // while the current block's hits are staged and summed.
        const int bstep = 32 * parts;
        uint32_t p_id = 0;
        uint2 p_rg = make_uint2(0u, 0u);
        int next = it.begin + 32 * part_id;
        int q_head = 0, q_tail = 0;   // pending hits (sample, pair) in the queue
        auto fetch = [&](int b) {
            if (b + lane >= it.end) return;
            p_rg = __ldg(a.prng + b + lane);
            p_id = __ldg(a.list + b + lane);
            if (!IL && a.layout == LAYOUT_ORIGINAL) p_id = __ldg(a.perm + p_id);
        };
        fetch(next);
        // Stages the next (at most HB) hits into batch `t`; returns how many.
        auto stage = [&](int t) -> int {
            while (q_tail - q_head < HB && next < it.end) {
                const int xlo = p_rg.x & 0xff, xhi = (p_rg.x >> 8) & 0xff;
                const int ylo = (p_rg.x >> 16) & 0xff, yhi = p_rg.x >> 24;
                bool hit = next + lane < it.end && xlo < x0 + S::BX && xhi >= x0 && ylo < y0 + S::BY && yhi >= y0;
                if (D3) hit = hit && (int)(p_rg.y & 0xff) < z0 + S::BZ && (int)((p_rg.y >> 8) & 0xff) >= z0;
                const uint32_t bits = __ballot_sync(0xffffffffu, hit);
                if (hit)
                    queue[(q_tail + __popc(bits & ((1u << lane) - 1u))) % kBrickQueue] =
                        make_uint2(p_id, (uint32_t)(next + lane));
                q_tail += __popc(bits);
                next += bstep;
                fetch(next);
            }
            __syncwarp();   // the queue is visible; the batch summed before may be overwritten
            const int n = min(HB, q_tail - q_head);
            float4 *batch = ring + t * (HB * SLOT);
            if (n > 0) {
#pragma unroll
                for (int e0 = 0; e0 < HB * WL; e0 += 32) {   // weights, zero for the missing hits of a short batch
                    const int h = (e0 + lane) / WL;
                    if (h < HB && wch < WCH) {
                        const uint32_t pair = queue[(q_head + (h < n ? h : 0)) % kBrickQueue].y;
                        cp_async<16>(batch + h * SLOT + VC + wch, wsrc + (int64_t)pair * a.prow_floats, h < n);
                    }
                }
                if (IL) {
#pragma unroll
                    for (int e0 = 0; e0 < HB * VC; e0 += 32) {
                        const int h = (e0 + lane) / VC, c = (e0 + lane) % VC;
                        if (h < n && b0 + 2 * c < a.nb) {
                            const uint32_t id = queue[(q_head + h) % kBrickQueue].x;
                            cp_async<16>(batch + h * SLOT + c, samples + (int64_t)id * a.il_stride + b0 + 2 * c, true);
                        }
                    }
                } else {
#pragma unroll
                    for (int e0 = 0; e0 < HB * S::CG; e0 += 32) {
                        const int h = (e0 + lane) / S::CG, c = (e0 + lane) % S::CG;
                        if (h < n && b0 + c < a.nb) {
                            const uint32_t id = queue[(q_head + h) % kBrickQueue].x;
                            cp_async<8>(reinterpret_cast<float2 *>(batch + h * SLOT) + c,
                                        samples + (int64_t)(b0 + c) * a.Mtot + id, true);
                        }
                    }
                    if (a.dcw && lane < n) {
                        const uint32_t id = queue[(q_head + lane) % kBrickQueue].x;
                        const uint32_t j = a.layout == LAYOUT_ORIGINAL ? id : __ldg(a.perm + id);
                        cp_async<4>(batch + lane * SLOT + VC + WCH, a.dcw + j, true);
                    }
                }
                q_head += n;
            }
            cp_async_commit();
            return n;
        };
        auto add = [&](const float4 *slot) {
            const float *wf = reinterpret_cast<const float *>(slot + VC);
            float v[V];
            if (CPL % 2 == 0) {
#pragma unroll
                for (int c = 0; c < CPL / 2; c++) {
                    const float4 q = slot[cp * (CPL / 2) + c];
                    v[(4 * c) % V] = q.x;
                    v[(4 * c + 1) % V] = q.y;
                    v[(4 * c + 2) % V] = q.z;
                    v[(4 * c + 3) % V] = q.w;
                }
            } else {
#pragma unroll
                for (int c = 0; c < CPL; c++) {
                    const float2 q = reinterpret_cast<const float2 *>(slot)[cp * CPL + c];
                    v[2 * c] = q.x;
                    v[2 * c + 1] = q.y;
                }
            }
            if (!IL && a.dcw) {
                const float dw = *reinterpret_cast<const float *>(slot + VC + WCH);
#pragma unroll
                for (int c = 0; c < V; c++) v[c] = dw * v[c];
            }
            const float wx = wf[(x0 & 3) * (S::BX < 4) + lx];
            // Row pairs the footprint misses are skipped where they are the
            // same for every lane (a lane's column is the whole brick): 2.1 of 4
            // are met at W = 5.5.
            constexpr bool SKIP = !D3 && !COMP && S::YL == 1;
            float2 wxy[YP];
            float pair_w[SKIP ? YP : 1];
            const float2 wx2 = make_float2(wx, wx);
            if (YC % 4 == 0) {
#pragma unroll
                for (int q = 0; q < YC / 4; q++) {
                    const float4 w = reinterpret_cast<const float4 *>(slot + VC + XC)[ly * (YC / 4) + q];
                    if (SKIP) {   // weights are not negative
                        pair_w[(2 * q) % (SKIP ? YP : 1)] = fmaxf(w.x, w.y);
                        pair_w[(2 * q + 1) % (SKIP ? YP : 1)] = fmaxf(w.z, w.w);
                    }
                    wxy[2 * q] = __fmul2_rn(make_float2(w.x, w.y), wx2);
                    wxy[(2 * q + 1) % YP] = __fmul2_rn(make_float2(w.z, w.w), wx2);
                }
            } else {
#pragma unroll
                for (int y = 0; y < YP; y++)
                    wxy[y] = __fmul2_rn(reinterpret_cast<const float2 *>(wf + 4 * XC + ly * YC)[y], wx2);
            }
            float wzs[4] = {1.f, 1.f, 1.f, 1.f};
            if (D3) {
                const float4 w = slot[VC + XC + YCH];
                wzs[0] = w.x;
                wzs[1] = w.y;
                wzs[2] = w.z;
                wzs[3] = w.w;
                if (S::BZ < 4 && (z0 & 2)) {
                    wzs[0] = w.z;
                    wzs[1] = w.w;
                }
            }
            float2 vd[V];
#pragma unroll
            for (int c = 0; c < V; c++) vd[c] = make_float2(v[c], v[c]);
#pragma unroll
            for (int z = 0; z < ZC; z++) {
                const float wz = wzs[z];
                if (ZC > 2 && wz == 0.f) continue;   // a slice the footprint misses (the same for every lane)
#pragma unroll
                for (int y = 0; y < YP; y++) {
                    if (SKIP && pair_w[y % (SKIP ? YP : 1)] == 0.f) continue;
                    const float2 w = D3 ? __fmul2_rn(wxy[y], make_float2(wz, wz)) : wxy[y];
#pragma unroll
                    for (int c = 0; c < V; c++) {
                        float2 &t = acc[z][y][c];
                        float2 n;
                        if (COMP) {
                            float2 &e = cmp[z][y][c];
                            const float2 u = __ffma2_rn(w, vd[c], f2neg(e));
                            n = __fadd2_rn(t, u);
                            const float2 ne = __fadd2_rn(__fadd2_rn(n, f2neg(t)), f2neg(u));
                            if (!SAFE) e = ne;
                            else {
                                if (w.x != 0.f) e.x = ne.x;
                                if (w.y != 0.f) e.y = ne.y;
                            }
                        } else {
                            n = __ffma2_rn(w, vd[c], t);
                        }
                        if (!SAFE) t = n;
                        else {
                            if (w.x != 0.f) t.x = n.x;
                            if (w.y != 0.f) t.y = n.y;
                        }
                    }
                }
            }
        };
        // DEPTH - 1 batches are in flight (an empty group stands for a batch
        // past the end); where registers allow, hits are summed in pairs, a
        // missing second one with zero weights.
        int cnt[DEPTH];
#pragma unroll
        for (int t = 0; t < DEPTH - 1; t++) cnt[t] = stage(t);
        bool live = cnt[0] > 0;
        while (live) {
#pragma unroll
            for (int t = 0; t < DEPTH; t++) {
                if (!live) break;
                cp_async_wait<DEPTH - 2>();
                cnt[(t + DEPTH - 1) % DEPTH] = stage((t + DEPTH - 1) % DEPTH);
                const float4 *slot = ring + t * (HB * SLOT);
#pragma unroll 1
                for (int h = 0; h < cnt[t]; h += S::UH, slot += S::UH * SLOT) {
#pragma unroll
                    for (int u = 0; u < S::UH; u++) add(slot + u * SLOT);
                }
                live = cnt[(t + 1) % DEPTH] > 0;
            }
        }
        cp_async_wait<0>();
        __syncwarp();
    };
    pass(std::false_type{});
    float2 odd = make_float2(0.f, 0.f);   // stays 0 while every sum is finite
#pragma unroll
    for (int z = 0; z < ZC; z++)
#pragma unroll
        for (int y = 0; y < YP; y++)
#pragma unroll
            for (int c = 0; c < V; c++) odd = __ffma2_rn(acc[z][y][c], make_float2(0.f, 0.f), odd);
    if (__any_sync(0xffffffffu, !(odd.x + odd.y == 0.f))) pass(std::true_type{});

    if (parts > 1) {
        // The first part's warp adds the other parts' sums in order.
        __syncthreads();   // the rings are free
        float4 *sums = brick_sm;
        constexpr int N4 = S::NACC / 2;
        if (part_id > 0) {
            float4 *o = sums + ((part_id - 1) * nbricks + slot_id) * (N4 * 32) + lane;
            int q = 0;
#pragma unroll
            for (int z = 0; z < ZC; z++)
#pragma unroll
                for (int y = 0; y < YP; y++)
#pragma unroll
                    for (int c = 0; c < V; c += 2, q++)
                        o[q * 32] = make_float4(acc[z][y][c].x, acc[z][y][c].y, acc[z][y][c + 1].x, acc[z][y][c + 1].y);
        }
        __syncthreads();
        if (part_id == 0) {
            for (int p = 1; p < parts; p++) {
                const float4 *o = sums + ((p - 1) * nbricks + slot_id) * (N4 * 32) + lane;
                int q = 0;
#pragma unroll
                for (int z = 0; z < ZC; z++)
#pragma unroll
                    for (int y = 0; y < YP; y++)
#pragma unroll
                        for (int c = 0; c < V; c += 2, q++) {
                            const float4 w = o[q * 32];
                            if (COMP) {
                                comp_add(acc[z][y][c], cmp[z][y][c], make_float2(w.x, w.y));
                                comp_add(acc[z][y][c + 1], cmp[z][y][c + 1], make_float2(w.z, w.w));
                            } else {
                                acc[z][y][c] = __fadd2_rn(acc[z][y][c], make_float2(w.x, w.y));
                                acc[z][y][c + 1] = __fadd2_rn(acc[z][y][c + 1], make_float2(w.z, w.w));
                            }
                        }
            }
        }
    }

    if (it.split >= 0) {
        // Chunk of a split tile: write the partial bricks; the CTA of this
        // group that arrives last sums the partials in chunk order.
        const SplitInfo si = a.splits[it.split];
        auto part = [&](int slot) -> float4 * {
            return reinterpret_cast<float4 *>(a.partials + ((int64_t)slot * a.ncg + blockIdx.y) * a.part_elems) +
                   32 * brick + lane;
        };
        const int nthr = 32 * nbricks * groups;   // lanes of the whole tile
        if (part_id == 0) {
            float4 *pp = part(si.first_slot + it.chunk);
#pragma unroll
            for (int z = 0; z < ZC; z++)
#pragma unroll
                for (int y = 0; y < YP; y++)
#pragma unroll
                    for (int c = 0; c < V; c += 2) {
                        *pp = make_float4(acc[z][y][c].x, acc[z][y][c].y, acc[z][y][c + 1].x, acc[z][y][c + 1].y);
                        pp += nthr;
                    }
        }
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned int *ctr = a.counters + ((int64_t)it.split * a.ncg + blockIdx.y) * groups + group;
            const unsigned int old = atomicAdd(ctr, 1u);
            s_last = (old == (unsigned int)(si.nchunks - 1));
            if (s_last) *ctr = 0u;   // ready for the next launch
        }
        __syncthreads();
        if (!s_last || part_id > 0) return;
        __threadfence();
#pragma unroll
        for (int z = 0; z < ZC; z++)
#pragma unroll
            for (int y = 0; y < YP; y++)
#pragma unroll
                for (int c = 0; c < V; c++) {
                    acc[z][y][c] = make_float2(0.f, 0.f);
                    if (COMP) cmp[z][y][c] = make_float2(0.f, 0.f);
                }
#pragma unroll 2
        for (int ch = 0; ch < si.nchunks; ch++) {
            const float4 *pp = part(si.first_slot + ch);
#pragma unroll
            for (int z = 0; z < ZC; z++)
#pragma unroll
                for (int y = 0; y < YP; y++)
#pragma unroll
                    for (int c = 0; c < V; c += 2) {
                        const float4 q = __ldcg(pp);
                        pp += nthr;
                        const float2 two[2] = {make_float2(q.x, q.y), make_float2(q.z, q.w)};
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            if (COMP) comp_add(acc[z][y][c + h], cmp[z][y][c + h], two[h]);
                            else acc[z][y][c + h] = __fadd2_rn(acc[z][y][c + h], two[h]);
                        }
                    }
        }
    }

    // Out: a lane's cells go straight to the grid (the x lanes of a coil are
    // neighbours, so a store instruction writes whole 32-byte sectors).
    if (!coil_ok || part_id > 0) return;
    if (a.accumulate && it.begin == it.end && it.split < 0) return;
    const int gx = it.tx * T0 + x0 + lx, gy0 = it.ty * T1 + y0 + ly * YC, gz0 = it.tz * k.tile[2] + z0;
    const float s0 = (a.sign_fold && ((gx + gy0 + gz0) & 1)) ? -1.f : 1.f;
    const float s1 = a.sign_fold ? -s0 : s0;
    const int64_t plane = (int64_t)a.F * a.kl.s_bf;   // from coil to coil
    float2 *cell = grid + (int64_t)coil * plane + (int64_t)it.f * a.kl.s_bf + (int64_t)gz0 * a.kl.s_z +
                   (int64_t)gy0 * a.kl.s_y + gx;
#pragma unroll
    for (int z = 0; z < ZC; z++) {
        const float2 sg = (z & 1) ? make_float2(s1, s0) : make_float2(s0, s1);
#pragma unroll
        for (int c = 0; c < CPL; c++) {
            if (c > 0 && coil + c >= a.nb) break;
            float2 *o = cell + c * plane + (int64_t)z * a.kl.s_z;
#pragma unroll
            for (int y = 0; y < YP; y++) {
                const float2 re = __fmul2_rn(acc[z][y][2 * c], sg), im = __fmul2_rn(acc[z][y][2 * c + 1], sg);
                float2 v0 = make_float2(re.x, im.x), v1 = make_float2(re.y, im.y);
                float2 *o1 = o + a.kl.s_y;
                if (a.accumulate) {
                    const float2 p0 = *o, p1 = *o1;
                    v0 = make_float2(v0.x + p0.x, v0.y + p0.y);
                    v1 = make_float2(v1.x + p1.x, v1.y + p1.y);
                }
                *o = v0;
                *o1 = v1;
                o = o1 + a.kl.s_y;
            }
        }
    }
}

// CT coils x 1024 / CT samples per block through shared memory: the planes are
// read along the samples, the rows written along the coils.
template <int CT>
__global__ void __launch_bounds__(256) k_samples_il(const float2 *__restrict__ samples, const float *__restrict__ dcw,
                                                    const uint32_t *__restrict__ perm, int64_t M, int nb, int il,
                                                    float2 *__restrict__ rows) {
    constexpr int SB = 1024 / CT;   // samples per block
    __shared__ float2 t[CT][SB + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t i0 = (int64_t)blockIdx.x * SB;
    const int c0 = (int)blockIdx.y * CT;
    uint32_t j[SB / 32];
    float w[SB / 32];
#pragma unroll
    for (int g = 0; g < SB / 32; g++) {
        const int64_t i = i0 + 32 * g + lane;
        j[g] = i < M ? perm[i] : 0u;
        w[g] = dcw && i < M ? dcw[j[g]] : 1.f;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int ct = warp + 8 * (q % (CT / 8)), g = q / (CT / 8);
        const int c = c0 + ct;
        float2 v = make_float2(0.f, 0.f);
        if (i0 + 32 * g + lane < M && c < nb) {
            v = samples[(int64_t)c * M + j[g]];
            if (dcw) v = make_float2(w[g] * v.x, w[g] * v.y);
        }
        t[ct][32 * g + lane] = v;
    }
    __syncthreads();
    const int cn = min(CT, il - c0);
    for (int e = threadIdx.x; e < SB * cn; e += 256) {
        const int r = e / cn, c = e - r * cn;
        if (i0 + r < M) rows[(i0 + r) * il + c0 + c] = t[c][r];
    }
}

void launch_samples_il(const NufftPlan &p, const float2 *samples, const float *dcw, int nb, float2 *rows,
                       cudaStream_t st) {
    const int il = il_stride_for(nb);
    auto go = [&](auto kern, int ct) {
        const dim3 g((unsigned)((p.Mtot + 1024 / ct - 1) / (1024 / ct)), (unsigned)((il + ct - 1) / ct));
        kern<<<g, 256, 0, st>>>(samples, dcw, p.perm.get(), p.Mtot, nb, il, rows); note_launch();
    };
    if (il <= 8) go(k_samples_il<8>, 8);
    else if (il <= 16) go(k_samples_il<16>, 16);
    else go(k_samples_il<32>, 32);
    GB_CUDA(cudaGetLastError());
}

// ------------------------------------------------------------- dispatch ---
//
// The lanes left over by the coils of a group run along x (then y), so that a
// group of any size fills the warp.  A brick of 8 x 8 cells is met by 2.4
// times as many (sample, brick) pairs as there are samples at W = 5.5, one of
// 4 x 8 by 3.3 times.  16 coils in 2D have two forms: the wide one (4 coils per
// lane, 4 bricks to a tile of 16 x 16) runs fewer instructions and serves launches
// of many tiles with short lists; the narrow one (2 coils per lane, 8 bricks) has
// shorter chains and serves small launches and long lists.  12 coils have a
// wide form of their own (3 per lane, no idle lanes).
// Gridding in us, 96 x 512 radial samples a frame on 512^2, wide / narrow:
//   1 frame, 16 coils 39.4 / 35.1; 2 frames 49.9 / 53.9; 4 frames 85.5 / 98.9; 23: 457 / 535
//   1 frame, 12 coils 37.1 / 34.1; 2 frames 46.5 / 50.0; 4 frames 70.2 / 90.7; 23: 370 / 489
// so the line lies between 1 and 2 frames of 1024 tiles.  On 96^2 with 46000
// samples a frame (2000 to a tile) the narrow form is the faster one at 23 frames:
// 264 against 306 us (16 coils), 484 against 552 (18).
// A CTA of one brick for the wide forms: its slot is free when its brick is done
// (4 bricks per CTA: 470 us for the 23 frames above with 16 coils, 378 with 12).  The narrow form
// takes 8 bricks per CTA where lists are short (they share the list's reads: 35.1
// against 37.9 us for 1 frame) and 2 where they are long (96^2, 1 frame: 59 against 166 us) or
// where that lets several warps share a brick's list (10400 samples on 192 x 128: 24 against 32 us).
// 3D bricks of 16 and 32 coils are four slices thick, of the others two (W = 4
// meets 2.5 of two: 80 % of the slices computed are hit).  8 coils have both: two
// slices leave registers for 24 warps per SM instead of 16, four have fewer
// (sample, brick) pairs.  Gridding of 5 coils, two / four slices, us: 64000 samples on 96^3 71 / 79,
// 256000 on 64^3 205 / 276, 768000 on 160^3 (2 M pairs) 438 / 459, 2.56 M on 192^3 (6.7 M pairs) 1309 /
// 1194.  One brick per CTA here too, two with 32 coils (2.56 M samples, 16 coils, 4 / 2 / 1: 2143 /
// 2050 / 2005; 32 coils 4232 / 4222 / 4293).
using Brick2D16 = BrickShape<2, 8, 4, 1, 8, 1, false, 256, 3, 8>;
// Compensated; 8 CTAs per SM instead of 6: 11.52 -> 11.40 ms per refined solve at
// 512^2 -> 640^2, 32 coils.
using Brick2D16C = BrickShape<2, 8, 4, 1, 8, 1, false, 128, 8>;
using Brick2D16W = BrickShape<4, 4, 8, 1, 8, 1, false, 128, 4, 1>;
using Brick2D12 = BrickShape<3, 4, 8, 1, 8, 1, false, 128, 5, 1>;
using Brick2D8 = BrickShape<2, 4, 8, 1, 8, 1, false, 256, 3>;
using Brick2D4 = BrickShape<2, 2, 8, 2, 4, 1, false, 512, 2>;
using Brick2D2 = BrickShape<2, 1, 8, 4, 2, 1, false, 512, 2>;
using Brick2D1 = BrickShape<1, 1, 8, 4, 2, 1, false, 512, 2>;
using Brick3D32 = BrickShape<2, 16, 2, 1, 4, 4, true, 128, 4, 2>;
using Brick3D16 = BrickShape<2, 8, 4, 1, 4, 4, true, 128, 4, 1>;
using Brick3D8 = BrickShape<2, 4, 8, 1, 4, 2, true, 128, 6, 1>;
using Brick3D8W = BrickShape<2, 4, 8, 1, 4, 4, true, 128, 4, 1>;
using Brick3D16C = BrickShape<2, 8, 4, 1, 4, 2, true, 128, 4>;    // compensated
using Brick3D8C = BrickShape<2, 4, 8, 1, 4, 2, true, 128, 4>;
using Brick3D4 = BrickShape<2, 2, 8, 2, 4, 2, true, 256, 3>;
using Brick3D2 = BrickShape<2, 1, 8, 4, 2, 2, true, 256, 3>;
using Brick3D1 = BrickShape<1, 1, 8, 4, 2, 2, true, 256, 4>;

// Calls f(shape, compensated) for the form of coil group cg; false for a group
// that has none.
template <class F>
static bool with_brick(int D, int cg, bool comp, bool wide, F &&f) {
    using P = std::false_type;   // plain sums
    using C = std::true_type;    // compensated sums
#define GB_EITHER(S) (comp ? f(S{}, C{}) : f(S{}, P{}))
    if (D == 2) {
        switch (cg) {
            case 16:
                if (comp) f(Brick2D16C{}, C{});
                else if (wide) f(Brick2D16W{}, P{});
                else f(Brick2D16{}, P{});
                return true;
            case 12:
                if (!comp) f(Brick2D12{}, P{});
                return !comp;
            case 8: GB_EITHER(Brick2D8); return true;
            case 4: GB_EITHER(Brick2D4); return true;
            case 2: GB_EITHER(Brick2D2); return true;
            default: GB_EITHER(Brick2D1); return true;
        }
    }
    switch (cg) {
        case 32:
            if (!comp) f(Brick3D32{}, P{});
            return !comp;
        case 16:
            if (comp) f(Brick3D16C{}, C{});
            else f(Brick3D16{}, P{});
            return true;
        case 8:
            if (comp) f(Brick3D8C{}, C{});
            else if (wide) f(Brick3D8W{}, P{});
            else f(Brick3D8{}, P{});
            return true;
        case 4: GB_EITHER(Brick3D4); return true;
        case 2: GB_EITHER(Brick3D2); return true;
        default: GB_EITHER(Brick3D1); return true;
    }
#undef GB_EITHER
}

// Cuts the plan's tile into the bricks of the form: bricks per tile, and CTAs a
// tile's bricks are spread over; false when the form does not divide the tile.
static bool cut_tile(const KParams &k, int cg, bool comp, bool wide, GridCfg &c) {
    int n = 0;
    with_brick(k.D, cg, comp, wide, [&](auto shape, auto) {
        using S = decltype(shape);
        if (k.tile[0] % S::BX || k.tile[1] % S::BY || k.tile[2] % S::BZ) return;
        n = (k.tile[0] / S::BX) * (k.tile[1] / S::BY) * (k.tile[2] / S::BZ);
        // tile extents are powers of two (a tile holds a divisor of 256 cells, 512 or 1024)
        if (n > kBrickMax || (n & (n - 1)) != 0) n = 0;
        c.groups = std::max(1, n / S::CTA);
    });
    if (!n) return false;
    c.brick = true;
    c.cg = cg;
    c.wide = wide;
    c.nbricks = n;
    return true;
}

bool brick_config(const NufftPlan &p, int nb, GridCfg &c) {
    const KParams &k = p.kp;
    if (k.D < 2 || p.pair_row_stride <= 0 || p.pair_row_stride != pair_row_floats(k)) return false;
    const bool comp = (p.flags & GB_FLAG_COMPENSATED) != 0;
    const int cg = choose_cg(p.tiling.cg, nb);
    // 3D, more than 16 coils: one group of 32 visits a sample's bricks once
    // instead of twice
    if (k.D == 3 && cg == 16 && nb > 16 && cut_tile(k, 32, comp, false, c)) return true;
    if (k.D == 2 && cg == 16 && !comp) {
        const int64_t avg = p.total_pairs / std::max<int64_t>(1, (int64_t)p.F * k.ntiles_total);
        const bool twelve = nb % 12 == 0 && nb % 16 != 0;
        if (!cut_tile(k, cg, comp, false, c)) return false;
        const int64_t warps = (int64_t)p.n_grd_items * ((nb + cg - 1) / cg) * c.nbricks;
        if (warps >= kBrickWideWarps && avg <= kBrickWideList) {
            GridCfg w = c;
            if ((twelve && cut_tile(k, 12, comp, false, w)) || cut_tile(k, cg, comp, true, w)) c = w;
        } else if (avg > kBrickWideList || warps < kBrickFillWarps) {
            c.groups = std::max(1, c.nbricks / 2);
        }
        return true;
    }
    return cut_tile(k, cg, comp, k.D == 3 && p.total_pairs >= kBrick3DWidePairs, c);
}

template <class S, bool COMP>
static void brick_launch(const GridCfg &c, const ConvArgs &args, const float2 *samples, float2 *grid, cudaStream_t st) {
    ConvArgs a = args;
    const int cta = c.nbricks / c.groups;   // bricks per CTA
    // Warps per brick: one when the bricks alone fill the GPU, more (each with
    // its share of the list) when the launch is small and bound by its longest
    // list.  Powers of two, as the tile's extents.
    int parts = 1;
    while (2 * parts * cta * 32 <= S::NT && (int64_t)a.n_items * c.ncg * c.nbricks * parts < kBrickFillWarps)
        parts *= 2;
    auto log2i = [](int v) {
        int l = 0;
        while ((1 << l) < v) l++;
        return l;
    };
    a.lbx = log2i(a.k.tile[0] / S::BX);
    a.lby = log2i(a.k.tile[1] / S::BY);
    a.lbricks = log2i(c.nbricks);
    a.lcta = log2i(cta);
    a.lparts = log2i(parts);
    const int warps = cta * parts;
    if (32 * warps > S::NT) fail(GB_ERR_INTERNAL, "more bricks per CTA than the gridding kernel has warps");
    const dim3 g((unsigned)(a.n_items * c.groups), (unsigned)c.ncg);
    const size_t ring = (size_t)warps * (kBrickDepth * S::HB * S::SLOT * 16 + kBrickQueue * sizeof(uint2));
    const size_t smem = std::max(ring, (size_t)(warps - cta) * S::NACC * 32 * 8);
    auto go = [&](auto kern) {
        if (smem > 48 * 1024)
            GB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<g, 32 * warps, smem, st>>>(a, samples, grid); note_launch();
    };
    if constexpr (S::CPL >= 2) {
        if (a.layout == LAYOUT_SORTED_IL) {
            go(k_grid_brick<S, COMP, true>);
            return;
        }
    }
    go(k_grid_brick<S, COMP, false>);
}

void launch_grid_brick(const GridCfg &c, const NufftPlan &p, const ConvArgs &a, const float2 *samples, float2 *grid,
                       cudaStream_t st) {
    const bool comp = (p.flags & GB_FLAG_COMPENSATED) != 0;
    if (a.layout == LAYOUT_SORTED_IL && (c.cg < 2 || a.dcw))
        fail(GB_ERR_INTERNAL, "interleaved samples need a coil pair per lane and carry their density weights");
    with_brick(p.kp.D, c.cg, comp, c.wide, [&](auto shape, auto comp_c) {
        brick_launch<decltype(shape), decltype(comp_c)::value>(c, a, samples, grid, st);
    });
    GB_CUDA(cudaGetLastError());
}

}  // namespace gb

// Persistent tile-queue blend for sm_103a.
//
// One warp renders one tile at a time; every lane owns a (BX/8) x (BY/4)
// block of pixels (8 x 4 lanes over the tile, csrc/cuda_rasterizer/
// render.cu:1736-1737).  Warps take tiles from a per-launch atomic queue in
// the caller's workspace (no module-global counter, so concurrent launches on
// different workspaces are safe); with few tiles a CTA takes one tile.  The
// Gaussians of a tile are consumed in batches of 32.  k_blend, which renders
// almost everything, holds the next batch in registers and blends in paired
// FP32; k_render is the scalar form for the general shader, the
// distance-thresholded and the split renders, and stages batches with cp.async
// or (GSR_RENDER_TMA=1) 1-D TMA bulk copies completed on an mbarrier, whose
// waits are bounded: on expiry the warp records a timeout in the status word
// and stops.
//
// The blend of each Gaussian-pixel pair is the reference's arithmetic
// (pixel_shader_axis_shared_16x16 / pixel_shader, render.cu:228-271 and
// 216-226): alpha = ex2.approx.ftz(power) with no 0.99 clamp and no 1/255
// skip, front-to-back compositing, and a whole-tile exit once every pixel of
// the tile has T < 1e-4, checked every CADENCE Gaussians.  Output is the
// truncating uint8 encode of render.cu:375-394.
#include <atomic>
#include <cstdlib>
#include <cstring>

#include "f32x2.cuh"
#include "gsr_internal.h"

namespace gsr {
namespace {

constexpr int kRenderWarps = 4;
constexpr int kBatch = 32;

struct WarpRing {
    float4 con[2][kBatch];
    float4 rgbd[2][kBatch];
    float4 xy2[2][kBatch];  // 16-byte pair holding the Gaussian's centre
    uint32_t sel[2][kBatch];
    uint64_t bar[2];
};

struct RenderParams {
    int n_host;
    const int32_t* d_num;
    long long cap;
    int W, H, gx, tiles, P;  // quad renders: gx and tiles count quads
    int items;               // work items: tiles, or 4 per quad
    const float2* xy;
    const float4* rgbd;
    const float4* con;
    const uint64_t* keys;
    const uint32_t* vals;
    const int2* ranges;
    float3 bg;
    uchar3* out;
    uint32_t* queue;
    uint32_t* status;
    const RenderView* views;  // batched render: per-view blocks (nullptr: one view)
    int n_views;
};

__device__ __forceinline__ uint8_t encode8(float x) { return (uint8_t)fminf(fmaxf(0.0f, x * 255.0f), 255.0f); }

// Final colour of a pixel: C + T' bg with T' = 0 once T < 1e-4; background
// only for a tile without Gaussians (render.cu:375-394, 1845-1858).
__device__ __forceinline__ uchar3 encode_px(const float (&c)[3], float t, bool any, float3 bg)
{
    if (t < 0.0001f) t = 0.0f;
    uchar3 o;
    if (any) {
        o.x = encode8(c[0] + t * bg.x);
        o.y = encode8(c[1] + t * bg.y);
        o.z = encode8(c[2] + t * bg.z);
    } else {
        o.x = encode8(bg.x);
        o.y = encode8(bg.y);
        o.z = encode8(bg.z);
    }
    return o;
}

// First index in keys[lo, hi) whose tile id is > t (UPPER) or >= t (!UPPER);
// warp-cooperative 32-way search, log32(n) rounds.
template <bool UPPER>
__device__ __forceinline__ int warp_bound(const uint64_t* keys, int lo, int hi, uint32_t t, unsigned lane)
{
    while (hi - lo > 32) {
        const int step = (hi - lo + 31) >> 5;
        const int p = lo + ((int)lane + 1) * step - 1;
        bool pred = false;
        if (p < hi) {
            const uint32_t kt = (uint32_t)(keys[p] >> 32);
            pred = UPPER ? (kt <= t) : (kt < t);
        }
        const int c = __popc(__ballot_sync(GSR_FULL_MASK, pred));
        const int nlo = c == 0 ? lo : lo + c * step;  // first probe that failed is p_c
        const int nhi = min(hi, lo + (c + 1) * step);
        lo = nlo;
        hi = nhi;
    }
    const int p = lo + (int)lane;
    bool pred = false;
    if (p < hi) {
        const uint32_t kt = (uint32_t)(keys[p] >> 32);
        pred = UPPER ? (kt <= t) : (kt < t);
    }
    return lo + __popc(__ballot_sync(GSR_FULL_MASK, pred));
}

// Stage the next Gaussians of the tile's list, from position `pos` on, into
// ring half `b`, and advance `pos` past them; returns how many were staged.
// Per-tile lists: the next min(32, end - pos).  QUAD: the quad's list is
// scanned from `pos` on until 32 values with bit `sub_bit` set (the
// Gaussians of this warp's tile of the quad) are staged, in list order, or
// the list ends -- so a batch is as full as in a per-tile list.
template <bool TMA, bool QUAD = false>
__device__ __forceinline__ int stage_batch(WarpRing& R, int b, const RenderParams& p, int& pos, int end,
                                           unsigned lane, bool& bad, uint32_t sub_bit = 0u)
{
    __syncwarp();
    if (TMA) fence_proxy_async_smem();
    if (QUAD) {
        static_assert(!QUAD || !TMA, "quad renders stage with cp.async");
        int filled = 0;
        while (filled < kBatch && pos < end) {
            const int cnt = min(kBatch, end - pos);
            uint32_t v = 0u;
            if ((int)lane < cnt) v = __ldg(p.vals + pos + lane);
            const bool hit = (int)lane < cnt && (v & sub_bit) != 0u;
            const unsigned hits = __ballot_sync(GSR_FULL_MASK, hit);
            const int room = kBatch - filled;
            const int rank = __popc(hits & lanemask_lt());
            uint32_t gid = v & kQuadGidMask;
            if (hit && rank < room) {
                if (gid < (uint32_t)p.P) {
                    const int slot = filled + rank;
                    cp_async_16(&R.con[b][slot], p.con + gid);
                    cp_async_16(&R.rgbd[b][slot], p.rgbd + gid);
                    cp_async_8(&R.xy2[b][slot], p.xy + gid);
                    R.sel[b][slot] = 0u;
                } else {  // index outside the feature arrays: a transparent stand-in
                    bad = true;
                    const int slot = filled + rank;
                    R.con[b][slot] = make_float4(0.f, 0.f, 0.f, -1e30f);
                    R.rgbd[b][slot] = make_float4(0.f, 0.f, 0.f, 0.f);
                    R.xy2[b][slot] = make_float4(0.f, 0.f, 0.f, 0.f);
                    R.sel[b][slot] = 0u;
                }
            }
            const int n = __popc(hits);
            if (n <= room) {
                pos += cnt;
                filled += n;
            } else {
                // the batch is full: resume right after its last Gaussian
                pos += __ffs(__ballot_sync(GSR_FULL_MASK, hit && rank == room - 1));
                filled = kBatch;
            }
        }
        cp_async_commit();
        return filled;
    }
    const int cnt = min(kBatch, end - pos);
    pos += cnt;
    const int base = pos - cnt;
    uint32_t gid = 0;
    bool ok = (int)lane < cnt;
    if (ok) {
        gid = __ldg(p.vals + base + lane);
        if (gid >= (uint32_t)p.P) {  // index outside the feature arrays: skip it
            ok = false;
            bad = true;
        }
    }
    const bool pair_ok = ok && (gid | 1u) < (uint32_t)p.P;
    if (TMA) {
        const uint32_t tx = 32u * __popc(__ballot_sync(GSR_FULL_MASK, ok)) + 16u * __popc(__ballot_sync(GSR_FULL_MASK, pair_ok));
        if (lane == 0) mbar_arrive_expect_tx(&R.bar[b], tx);
        __syncwarp();
        if (ok) {
            tma_bulk_g2s(&R.con[b][lane], p.con + gid, 16, &R.bar[b]);
            tma_bulk_g2s(&R.rgbd[b][lane], p.rgbd + gid, 16, &R.bar[b]);
            if (pair_ok) {
                tma_bulk_g2s(&R.xy2[b][lane], p.xy + (gid & ~1u), 16, &R.bar[b]);
                R.sel[b][lane] = gid & 1u;
            } else {
                const float2 v = __ldg(p.xy + gid);
                R.xy2[b][lane] = make_float4(v.x, v.y, 0.f, 0.f);
                R.sel[b][lane] = 0u;
            }
        }
        if (!ok && (int)lane < cnt) {  // skipped index: a fully transparent stand-in
            R.con[b][lane] = make_float4(0.f, 0.f, 0.f, -1e30f);
            R.rgbd[b][lane] = make_float4(0.f, 0.f, 0.f, 0.f);
            R.xy2[b][lane] = make_float4(0.f, 0.f, 0.f, 0.f);
            R.sel[b][lane] = 0u;
        }
    } else {
        if (ok) {
            cp_async_16(&R.con[b][lane], p.con + gid);
            cp_async_16(&R.rgbd[b][lane], p.rgbd + gid);
            cp_async_8(&R.xy2[b][lane], p.xy + gid);
            R.sel[b][lane] = 0u;
        } else if ((int)lane < cnt) {
            R.con[b][lane] = make_float4(0.f, 0.f, 0.f, -1e30f);
            R.rgbd[b][lane] = make_float4(0.f, 0.f, 0.f, 0.f);
            R.xy2[b][lane] = make_float4(0.f, 0.f, 0.f, 0.f);
            R.sel[b][lane] = 0u;
        }
        cp_async_commit();
    }
    return cnt;
}

// Wait until ring half `b` is filled.  Returns false on timeout.
template <bool TMA>
__device__ __forceinline__ bool wait_batch(WarpRing& R, int b, uint32_t& phase_bits)
{
    bool ok = true;
    if (TMA) {
        ok = mbar_wait_bounded(&R.bar[b], (phase_bits >> b) & 1u);
        phase_bits ^= 1u << b;
    } else {
        cp_async_wait_all();
    }
    __syncwarp();
    return ok;
}

// SHADER 0: pixel_shader_axis_shared_16x16 (render.cu:228-271)
// SHADER 1: pixel_shader (render.cu:216-226)
template <int TX, int TY, int SHADER, bool DT>
__device__ __forceinline__ void shade(float (&C)[TY][TX][3], float (&T)[TY][TX], int ox, int oy, int cb, int rb,
                                      float2 xy, float4 co, float3 rgb)
{
    if (SHADER == 0) {
        float xs[TX], xc[TX];
#pragma unroll
        for (int j = 0; j < TX; j++) {
            float dx = xy.x - (float)(ox + cb + j);
            xs[j] = co.x * dx * dx;
            xc[j] = co.y * dx;
        }
        float yd[TY], ys[TY];
#pragma unroll
        for (int i = 0; i < TY; i++) {
            float dy = xy.y - (float)(oy + rb + i);
            yd[i] = dy;
            ys[i] = co.z * dy * dy;
        }
#pragma unroll
        for (int i = 0; i < TY; i++)
#pragma unroll
            for (int j = 0; j < TX; j++) {
                float power = fmaf(xc[j], yd[i], co.w + xs[j] + ys[i]);
                if (DT && !(power >= -7.994353375f)) continue;
                float alpha = ex2_approx_ftz(power);
                float weight = alpha * T[i][j];
                C[i][j][0] += rgb.x * weight;
                C[i][j][1] += rgb.y * weight;
                C[i][j][2] += rgb.z * weight;
                T[i][j] -= weight;
            }
    } else {
#pragma unroll
        for (int i = 0; i < TY; i++)
#pragma unroll
            for (int j = 0; j < TX; j++) {
                float dx = xy.x - (float)(ox + cb + j);
                float dy = xy.y - (float)(oy + rb + i);
                float power = co.w + co.x * dx * dx + co.z * dy * dy + co.y * dx * dy;
                float alpha = ex2_approx_ftz(power);
                C[i][j][0] += rgb.x * (alpha * T[i][j]);
                C[i][j][1] += rgb.y * (alpha * T[i][j]);
                C[i][j][2] += rgb.z * (alpha * T[i][j]);
                T[i][j] -= alpha * T[i][j];
            }
    }
}

// RANGE_MODE 0: ranges[] given; 1: warp search in the sorted keys.
// EXIT 0: the tile stops when all its pixels are saturated; EXIT 1: the top
// and bottom halves (8 rows each, lanes 0-15 and 16-31) stop independently,
// as the reference's two-warp split kernels do (renderCUDAWarpSplit,
// render.cu:4115-4357; renderCUDA32x16Split, render.cu:3859-4106).
// QUAD: the keys name 2x2 groups of 16x16 tiles (ranges and key ids count
// quads); each of a quad's four tiles is a work item of its own, whose warp
// blends, in list order, only the Gaussians whose value has that tile's bit,
// which is exactly the tile's per-tile list; the exit count runs over them.
template <int BX, int BY, int CADENCE, int SHADER, bool DT, int RANGE_MODE, bool TMA, bool BATCH, int EXIT = 0,
          bool QUAD = false>
__global__ __launch_bounds__(kRenderWarps * 32) void k_render(const RenderParams p)
{
    static_assert(!QUAD || (BX == 16 && BY == 16 && EXIT == 0 && !TMA), "quad renders: 16x16 tiles");
    constexpr int TX = BX / 8, TY = BY / 4;
    __shared__ WarpRing rings[kRenderWarps];
    const unsigned lane = threadIdx.x & 31u;
    const int warp = threadIdx.x >> 5;
    WarpRing& R = rings[warp];
    if (TMA) {
        if (lane == 0) {
            mbar_init(&R.bar[0], 1);
            mbar_init(&R.bar[1], 1);
            fence_mbar_init();
        }
        __syncwarp();
    }
    long long nl = p.d_num ? (long long)*p.d_num : (long long)p.n_host;
    const int n = (int)max(0LL, min(nl, p.cap));
    const int cb = (int)(lane & 7u) * TX;
    const int rb = (int)(lane >> 3) * TY;
    uint32_t phase_bits = 0;
    bool bad = false;
    bool timed_out = false;

    int item = blockIdx.x * kRenderWarps + warp;
    while (item < p.items) {
        const int tile = QUAD ? (item >> 2) : item;  // key tile id (a quad's id for QUAD)
        const int sub = item & 3;                     // QUAD: which tile of the quad
        // per-view geometry (batched renders); the single-view kernel reads
        // its parameters directly
        int W = 0, H = 0, gx = p.gx, ltile = tile;
        float3 bg = make_float3(0.f, 0.f, 0.f);
        uchar3* out = nullptr;
        if (BATCH) {
            // the view holding this global tile: last tile_base <= tile
            int lo = 0, hi = p.n_views - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (__ldg(&p.views[mid].tile_base) <= tile) lo = mid;
                else hi = mid - 1;
            }
            const RenderView& v = p.views[lo];
            W = v.W;
            H = v.H;
            gx = max(1, v.gx);
            ltile = tile - v.tile_base;
            bg = make_float3(v.bg[0], v.bg[1], v.bg[2]);
            out = reinterpret_cast<uchar3*>(v.out);
        }
        const int ox = QUAD ? (ltile % gx) * 32 + (sub & 1) * 16 : (ltile % gx) * BX;
        const int oy = QUAD ? (ltile / gx) * 32 + (sub >> 1) * 16 : (ltile / gx) * BY;
        if (QUAD && (ox >= (BATCH ? W : p.W) || oy >= (BATCH ? H : p.H))) {
            // a quad's tile beyond the image edge has no pixels and no Gaussians
            int next = 0;
            if (lane == 0) next = (int)atomicAdd(p.queue, 1u) + (int)gridDim.x * kRenderWarps;
            item = __shfl_sync(GSR_FULL_MASK, next, 0);
            continue;
        }
        const uint32_t sub_bit = QUAD ? (1u << (kQuadShift + sub)) : 0u;
        int start, end;
        if (RANGE_MODE == 0) {
            int2 r = make_int2(0, 0);
            if (lane == 0) r = __ldg(p.ranges + tile);
            // ranges come from the caller: keep them inside [0, n]
            start = min(max(__shfl_sync(GSR_FULL_MASK, r.x, 0), 0), n);
            end = min(max(__shfl_sync(GSR_FULL_MASK, r.y, 0), start), n);
        } else {
            start = warp_bound<false>(p.keys, 0, n, (uint32_t)tile, lane);
            end = warp_bound<true>(p.keys, start, n, (uint32_t)tile, lane);
        }
        float T[TY][TX];
        float C[TY][TX][3];
#pragma unroll
        for (int i = 0; i < TY; i++)
#pragma unroll
            for (int j = 0; j < TX; j++) {
                T[i][j] = 1.0f;
                C[i][j][0] = C[i][j][1] = C[i][j][2] = 0.0f;
            }
        const int total = end - start;
        bool blended_any = false;  // QUAD: the tile's own list is not empty
        if (total > 0) {
            int cur = 0;
            int scan = start;  // next list position to stage from
            int staged = stage_batch<TMA, QUAD>(R, 0, p, scan, end, lane, bad, sub_bit);
            int processed = 0;
            bool half_done = false;  // EXIT 1: this lane's half has stopped
            while (staged > 0) {
                const int bsize = staged;
                if (!wait_batch<TMA>(R, cur, phase_bits)) {
                    timed_out = true;
                    break;
                }
                const int nsize = scan < end ? stage_batch<TMA, QUAD>(R, cur ^ 1, p, scan, end, lane, bad, sub_bit)
                                             : 0;
                staged = nsize;
                blended_any = true;
                bool exit_now = false;
                for (int g = 0; g < bsize; g++) {
                    const float4 co = R.con[cur][g];
                    const float4 cd = R.rgbd[cur][g];
                    const float4 x2 = R.xy2[cur][g];
                    const float2 xy = R.sel[cur][g] ? make_float2(x2.z, x2.w) : make_float2(x2.x, x2.y);
                    if (EXIT == 0 || !half_done)
                        shade<TX, TY, SHADER, DT>(C, T, ox, oy, cb, rb, xy, co, make_float3(cd.x, cd.y, cd.z));
                    ++processed;
                    if (processed % CADENCE == 0) {
                        bool sat = true;
#pragma unroll
                        for (int i = 0; i < TY; i++)
#pragma unroll
                            for (int j = 0; j < TX; j++) sat = sat && T[i][j] < 0.0001f;
                        if (EXIT == 0) {
                            if (__all_sync(GSR_FULL_MASK, sat)) {
                                exit_now = true;
                                break;
                            }
                        } else {
                            const unsigned m = __ballot_sync(GSR_FULL_MASK, sat);
                            const bool lo = (m & 0xFFFFu) == 0xFFFFu, hi = (m >> 16) == 0xFFFFu;
                            if (lo && hi) {
                                exit_now = true;
                                break;
                            }
                            half_done = half_done || (lane < 16u ? lo : hi);
                        }
                    }
                }
                cur ^= 1;
                if (exit_now) {
                    // consume the batch already in flight so the ring is idle
                    if (nsize > 0 && !wait_batch<TMA>(R, cur, phase_bits)) timed_out = true;
                    break;
                }
            }
        }
        if (timed_out) break;
#pragma unroll
        for (int i = 0; i < TY; i++)
#pragma unroll
            for (int j = 0; j < TX; j++) {
                const int px = ox + cb + j, py = oy + rb + i;
                const bool any = QUAD ? blended_any : total > 0;
                if (BATCH) {
                    if (px < W && py < H) out[(size_t)py * W + px] = encode_px(C[i][j], T[i][j], any, bg);
                } else {
                    if (px < p.W && py < p.H) p.out[(size_t)py * p.W + px] = encode_px(C[i][j], T[i][j], any, p.bg);
                }
            }
        int next = 0;
        if (lane == 0) next = (int)atomicAdd(p.queue, 1u) + (int)gridDim.x * kRenderWarps;
        item = __shfl_sync(GSR_FULL_MASK, next, 0);
    }
    if (timed_out && lane == 0) record_error(p.status, kErrTimeout);
    if (__any_sync(GSR_FULL_MASK, bad) && lane == 0) record_error(p.status, kErrBadInput);
    if (TMA && timed_out) {
        // give copies still in flight a bounded chance to land before exit
        mbar_wait_bounded(&R.bar[0], (phase_bits >> 0) & 1u);
        mbar_wait_bounded(&R.bar[1], (phase_bits >> 1) & 1u);
    }
}

// ---------------------------------------------------------------------------
// The blend with paired FP32 (shader 0, even tile widths, whole-tile exit).
//
// The scalar kernel above is bound by instruction issue: 12.9 thread
// instructions per pixel and Gaussian at 70% issue.  Here the two columns of a
// lane go through one fma.rn.f32x2, which gives each pixel the bits of the
// scalar form (power = fma(b dx, dy, fma(c dy, dy, fma(a dx, dx, w))), C =
// fma(rgb, alpha T, C), T - alpha T).  A paired instruction holds the FMA pipe
// for two cycles, so it saves issue slots and not FMA work: a Gaussian costs a
// warp 72 FMA cycles, 32 MUFU cycles and about 70 issue slots, and the FMA
// pipe bounds the kernel.  The rows' terms, the same for both columns, are
// scalar (as pairs they cost 8 FMA cycles more: 2429 against 2192 us per
// frame of 20 M Gaussians at 7680x4320).  Four CTAs per SM at 120 registers:
// five at 96 are slower (2623 us), as the Gaussians in flight per warp hide
// more than another warp does.
//
// A batch's records are loaded into registers one batch ahead and its list
// values one chunk before that, so neither load is waited for.  With DUP a
// record's scalars are stored twice, so a broadcast read is an operand pair;
// the kernels that split a tile over warps read every record four times and
// store them once (5 instead of 9 shared-memory wavefronts per read).
template <bool DUP>
struct BlendRing {
    float4 xyab[kBatch * (DUP ? 2 : 1)];  // x y a b, or x x y y and a a b b
    float4 cwrg[kBatch * (DUP ? 2 : 1)];  // c w r g
    float2 bl[kBatch];                    // b b
    uint32_t gid[kBatch];
    uint32_t ids[2 * kBatch];  // QUAD: list values of this tile not yet in a batch
    int at[2 * kBatch];        // QUAD: their list positions
};

// One Gaussian's record as operand pairs.
struct PairRecord {
    f32x2 x, y, a, b, c, w, r, g, bl;
};

template <bool DUP>
__device__ __forceinline__ PairRecord read_record(const BlendRing<DUP>& R, int k)
{
    PairRecord q;
    if (DUP) {
        const ulonglong2 xy = *reinterpret_cast<const ulonglong2*>(&R.xyab[2 * k]);
        const ulonglong2 ab = *reinterpret_cast<const ulonglong2*>(&R.xyab[2 * k + 1]);
        const ulonglong2 cw = *reinterpret_cast<const ulonglong2*>(&R.cwrg[2 * k]);
        const ulonglong2 rg = *reinterpret_cast<const ulonglong2*>(&R.cwrg[2 * k + 1]);
        q.x = xy.x;
        q.y = xy.y;
        q.a = ab.x;
        q.b = ab.y;
        q.c = cw.x;
        q.w = cw.y;
        q.r = rg.x;
        q.g = rg.y;
        q.bl = *reinterpret_cast<const f32x2*>(&R.bl[k]);
    } else {
        const float4 u = R.xyab[k], v = R.cwrg[k];
        const float bl = R.bl[k].x;
        q.x = pair(u.x, u.x);
        q.y = pair(u.y, u.y);
        q.a = pair(u.z, u.z);
        q.b = pair(u.w, u.w);
        q.c = pair(v.x, v.x);
        q.w = pair(v.y, v.y);
        q.r = pair(v.z, v.z);
        q.g = pair(v.w, v.w);
        q.bl = pair(bl, bl);
    }
    return q;
}

struct Features {
    const float2* xy;
    const float4* con;
    const float4* rgbd;
    const uint32_t* vals;
    uint32_t P;
};

// Reads the list positions [start, end) in batches of up to 32 Gaussians, one
// per lane, from the front or (REV) from the back.  QUAD: the quad's list is
// compacted to the values with bit `sub_bit` set, in that order, through the
// ring's ids; otherwise a batch is the next 32 values.
template <bool QUAD, bool REV, bool DUP>
struct Feed {
    int pos, end;     // next list position to take, and where the list stops
    uint32_t ahead;   // the lane's list value of the next chunk
    int head, tail;   // QUAD: taken and stored ids
    uint32_t sub_bit;
    // the batch in registers
    int n, where;     // its size; the lane's list position
    uint32_t gid;     // feature row, ~0 outside the feature arrays
    float2 xy;
    float4 con, rgbd;
    float3 mid;       // REV: taken off the stored colours (centre())

    __device__ __forceinline__ int left() const { return REV ? pos - end : end - pos; }
    __device__ __forceinline__ int mine(unsigned lane) const { return REV ? pos - 1 - (int)lane : pos + (int)lane; }

    __device__ __forceinline__ void open(const Features& f, int start, int stop, uint32_t bit, unsigned lane)
    {
        pos = REV ? stop : start;
        end = REV ? start : stop;
        head = tail = 0;
        sub_bit = bit;
        ahead = (int)lane < left() ? f.vals[mine(lane)] : 0u;
    }

    __device__ __forceinline__ void fetch(BlendRing<DUP>& R, const Features& f, unsigned lane, bool& bad)
    {
        uint32_t v = 0u;
        if (QUAD) {
            while (tail - head < kBatch && left() > 0) {
                const bool hit = (int)lane < left() && (ahead & sub_bit) != 0u;
                const unsigned m = __ballot_sync(GSR_FULL_MASK, hit);
                if (hit) {
                    const int slot = (tail + __popc(m & lanemask_lt())) & (2 * kBatch - 1);
                    R.ids[slot] = ahead;
                    R.at[slot] = mine(lane);
                }
                tail += __popc(m);
                pos += REV ? -kBatch : kBatch;
                ahead = (int)lane < left() ? f.vals[mine(lane)] : 0u;
            }
            __syncwarp();
            n = min(kBatch, tail - head);
            if ((int)lane < n) {
                const int slot = (head + (int)lane) & (2 * kBatch - 1);
                v = R.ids[slot] & kQuadGidMask;
                where = R.at[slot];
            }
            head += n;
            __syncwarp();
        } else {
            n = max(0, min(kBatch, left()));
            v = ahead;
            where = mine(lane);
            pos += REV ? -n : n;
            ahead = (int)lane < left() ? f.vals[mine(lane)] : 0u;
        }
        if ((int)lane < n) {
            if (v < f.P) {
                gid = v;
                xy = f.xy[v];
                con = f.con[v];
                rgbd = f.rgbd[v];
            } else {  // index outside the feature arrays: a transparent stand-in
                bad = true;
                gid = 0xFFFFFFFFu;
                xy = make_float2(0.f, 0.f);
                con = make_float4(0.f, 0.f, 0.f, -1e30f);
                rgbd = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    }

    // The backward's colours relative to that of the first batch's first
    // Gaussian, the farthest one blended (0 if that is not finite).
    __device__ __forceinline__ void centre()
    {
        auto of_lane0 = [](float v) {
            v = __shfl_sync(GSR_FULL_MASK, v, 0);
            return fabsf(v) < 1e30f ? v : 0.0f;
        };
        mid = n > 0 ? make_float3(of_lane0(rgbd.x), of_lane0(rgbd.y), of_lane0(rgbd.z)) : make_float3(0.f, 0.f, 0.f);
    }

    __device__ __forceinline__ void store(BlendRing<DUP>& R, unsigned lane) const
    {
        if ((int)lane < n) {
            const float r = REV ? rgbd.x - mid.x : rgbd.x, g = REV ? rgbd.y - mid.y : rgbd.y,
                        b = REV ? rgbd.z - mid.z : rgbd.z;
            if (DUP) {
                R.xyab[2 * lane] = make_float4(xy.x, xy.x, xy.y, xy.y);
                R.xyab[2 * lane + 1] = make_float4(con.x, con.x, con.y, con.y);
                R.cwrg[2 * lane] = make_float4(con.z, con.z, con.w, con.w);
                R.cwrg[2 * lane + 1] = make_float4(r, r, g, g);
            } else {
                R.xyab[lane] = make_float4(xy.x, xy.y, con.x, con.y);
                R.cwrg[lane] = make_float4(con.z, con.w, r, g);
            }
            R.bl[lane] = make_float2(b, b);
            if (REV) R.gid[lane] = gid;  // the backward's gradient row
        }
    }
};

// A lane's TY x TX pixels: transmittance and colour, columns in pairs.
template <int TX, int TY>
struct Pixels {
    f32x2 T[TY][TX / 2], C[TY][TX / 2][3];
    f32x2 ncol[TX / 2];  // minus the pixels' coordinates
    float nrow[TY];

    __device__ __forceinline__ void reset(int x0, int y0)
    {
#pragma unroll
        for (int j = 0; j < TX / 2; j++) ncol[j] = pair(-(float)(x0 + 2 * j), -(float)(x0 + 2 * j + 1));
#pragma unroll
        for (int i = 0; i < TY; i++) {
            nrow[i] = -(float)(y0 + i);
#pragma unroll
            for (int j = 0; j < TX / 2; j++) {
                T[i][j] = pair(1.0f, 1.0f);
                C[i][j][0] = C[i][j][1] = C[i][j][2] = pair(0.0f, 0.0f);
            }
        }
    }

    __device__ __forceinline__ void blend(const PairRecord& q)
    {
        f32x2 xw[TX / 2], xb[TX / 2];
#pragma unroll
        for (int j = 0; j < TX / 2; j++) {
            const f32x2 dx = add2(q.x, ncol[j]);
            xw[j] = fma2(mul2(q.a, dx), dx, q.w);
            xb[j] = mul2(q.b, dx);
        }
        const f32x2 minus1 = pair(-1.0f, -1.0f);
#pragma unroll
        for (int i = 0; i < TY; i++) {
            const float y = __fadd_rn(lo_of(q.y), nrow[i]), cy = __fmul_rn(lo_of(q.c), y);
            const f32x2 dy = pair(y, y), cdy = pair(cy, cy);
#pragma unroll
            for (int j = 0; j < TX / 2; j++) {
                const f32x2 alpha = ex2_2(fma2(xb[j], dy, fma2(cdy, dy, xw[j])));
                const f32x2 w = mul2(alpha, T[i][j]);
                C[i][j][0] = fma2(q.r, w, C[i][j][0]);
                C[i][j][1] = fma2(q.g, w, C[i][j][1]);
                C[i][j][2] = fma2(q.bl, w, C[i][j][2]);
                T[i][j] = fma2(w, minus1, T[i][j]);
            }
        }
    }

    // every pixel below the exit transmittance (a NaN is not)
    __device__ __forceinline__ bool saturated() const
    {
        float m = 0.0f;
#pragma unroll
        for (int i = 0; i < TY; i++)
#pragma unroll
            for (int j = 0; j < TX / 2; j++) m = max_nan(m, max_nan(lo_of(T[i][j]), hi_of(T[i][j])));
        return m < 0.0001f;
    }
};

// Blends the list positions [start, end) front to back, up to the whole-tile
// exit checked every CADENCE Gaussians.  Returns whether the tile has a
// Gaussian; `last` is the list position of the last one blended.  SPLIT > 1:
// the CTA's warps each hold a strip of the tile's rows and exit together.
template <int TX, int TY, int CADENCE, bool QUAD, int SPLIT>
__device__ __forceinline__ bool blend_list(Pixels<TX, TY>& px, BlendRing<SPLIT == 1>& R, const Features& f, int start,
                                           int end, uint32_t sub_bit, unsigned lane, bool& bad, int& last)
{
    static_assert(kBatch % CADENCE == 0, "the exit checks fall on the same Gaussian of every full batch");
    Feed<QUAD, false, SPLIT == 1> feed;
    feed.open(f, start, end, sub_bit, lane);
    feed.fetch(R, f, lane, bad);
    bool any = false;
    while (feed.n > 0) {
        const int n = feed.n, where = feed.where;
        __syncwarp();
        feed.store(R, lane);
        __syncwarp();
        feed.fetch(R, f, lane, bad);
        any = true;
        int done = n;
        bool stop = false;
        for (int g0 = 0; g0 < n; g0 += CADENCE) {
            if (g0 + CADENCE <= n) {
#pragma unroll 2
                for (int g = g0; g < g0 + CADENCE; g++) px.blend(read_record(R, g));
                const bool sat = px.saturated();
                if (SPLIT > 1 ? __syncthreads_and(sat) != 0 : __all_sync(GSR_FULL_MASK, sat) != 0) {
                    done = g0 + CADENCE;
                    stop = true;
                    break;
                }
            } else {
                for (int g = g0; g < n; g++) px.blend(read_record(R, g));
            }
        }
        last = __shfl_sync(GSR_FULL_MASK, where, done - 1);
        if (stop) break;
    }
    __syncwarp();
    return any;
}

// A render of few tiles, where a tile per warp would not even fill the warps
// that fit on the GPU at once (4 CTAs of 4 per SM), takes a tile per CTA, four
// rows to a warp: each tile's chain of Gaussians is then a quarter of the work
// per step.  With more tiles the fourfold record reads cost more than the
// shorter chains give.  Training steps, render backward, tile per warp against
// tile per CTA: 1900 tiles 408 / 294 us, 2400 tiles 339 / 274 us, 3600 tiles
// 362 / 522 us, 28800 tiles 1873 / 3698 us; the forwards cross at the same
// place.
static bool split_tiles(long long tiles) { return tiles <= 16LL * device_sm_count(); }

// Persistent render, a tile per warp; with SPLIT = 4 a tile per CTA and no
// queue.
//
// 32x16 tiles need three CTAs per SM (162 to 168 registers): left to itself the
// compiler takes 196, two CTAs fit, and where tiles are many the kernel falls
// behind k_render (four CTAs); at four CTAs it spills.  Render alone, k_render /
// two / three / four CTAs: 20 M Gaussians at 7680x4320 3964 / 4290 / 3799 / 4109
// us, 3 M at 3840x2160 127 / 137 / 111 / 123, 500 k at 1271x717 144 / 162 / 128 /
// 146, 100 k at 800x600 174 / 146 / 127 / 183.  32x32 tiles (255 registers, two
// CTAs, some bytes spilled) beat k_render throughout: 8325 / 6333, 156 / 124 (at
// 3840x2160), 709 / 365 (at 800x600).
template <int BX, int BY, int CADENCE, int RANGE_MODE, bool BATCH, bool QUAD, int SPLIT>
__global__ __launch_bounds__(kRenderWarps * 32, BX * BY == 256 ? 4 : BX * BY == 512 ? 3 : 1)
void k_blend(const RenderParams p)
{
    static_assert(!QUAD || (BX == 16 && BY == 16), "quad renders: 16x16 tiles");
    static_assert(SPLIT == 1 || (SPLIT == kRenderWarps && BY == 16), "a tile per warp, or per CTA");
    constexpr int TX = BX / 8, TY = BY / 4 / SPLIT;
    __shared__ BlendRing<SPLIT == 1> rings[kRenderWarps];
    const unsigned lane = threadIdx.x & 31u;
    const int warp = threadIdx.x >> 5;
    BlendRing<SPLIT == 1>& R = rings[warp];
    chain_wait();
    chain_ready();
    const long long nl = p.d_num ? (long long)*p.d_num : (long long)p.n_host;
    const int n = (int)max(0LL, min(nl, p.cap));
    const int cb = (int)(lane & 7u) * TX;
    const int rb = (SPLIT > 1 ? warp * (BY / SPLIT) : 0) + (int)(lane >> 3) * TY;
    const Features f{p.xy, p.con, p.rgbd, p.vals, (uint32_t)p.P};
    bool bad = false;

    int item = SPLIT > 1 ? (int)blockIdx.x : (int)blockIdx.x * kRenderWarps + warp;
    while (item < p.items) {
        const int tile = QUAD ? (item >> 2) : item;  // key tile id (a quad's id for QUAD)
        const int sub = item & 3;                     // QUAD: which tile of the quad
        int W = p.W, H = p.H, gx = p.gx, ltile = tile;
        float3 bg = p.bg;
        uchar3* out = p.out;
        if (BATCH) {
            // the view holding this global tile: last tile_base <= tile
            int lo = 0, hi = p.n_views - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (p.views[mid].tile_base <= tile) lo = mid;
                else hi = mid - 1;
            }
            const RenderView& v = p.views[lo];
            W = v.W;
            H = v.H;
            gx = max(1, v.gx);
            ltile = tile - v.tile_base;
            bg = make_float3(v.bg[0], v.bg[1], v.bg[2]);
            out = reinterpret_cast<uchar3*>(v.out);
        }
        const int ox = QUAD ? (ltile % gx) * 32 + (sub & 1) * 16 : (ltile % gx) * BX;
        const int oy = QUAD ? (ltile / gx) * 32 + (sub >> 1) * 16 : (ltile / gx) * BY;
        if (!QUAD || (ox < W && oy < H)) {  // a quad's tile beyond the image edge has no pixels
            int start, end;
            if (RANGE_MODE == 0) {
                const int2 r = p.ranges[tile];
                // ranges come from the caller: keep them inside [0, n]
                start = min(max(r.x, 0), n);
                end = min(max(r.y, start), n);
            } else {
                start = warp_bound<false>(p.keys, 0, n, (uint32_t)tile, lane);
                end = warp_bound<true>(p.keys, start, n, (uint32_t)tile, lane);
            }
            Pixels<TX, TY> px;
            px.reset(ox + cb, oy + rb);
            int last = 0;
            const bool any = blend_list<TX, TY, CADENCE, QUAD, SPLIT>(
                px, R, f, start, end, QUAD ? (1u << (kQuadShift + sub)) : 0u, lane, bad, last);
#pragma unroll
            for (int i = 0; i < TY; i++)
#pragma unroll
                for (int j = 0; j < TX; j++) {
                    const int x = ox + cb + j, y = oy + rb + i;
                    auto half = [&](f32x2 v) { return (j & 1) ? hi_of(v) : lo_of(v); };
                    const float c[3] = {half(px.C[i][j / 2][0]), half(px.C[i][j / 2][1]), half(px.C[i][j / 2][2])};
                    if (x < W && y < H) out[(size_t)y * W + x] = encode_px(c, half(px.T[i][j / 2]), any, bg);
                }
        }
        if (SPLIT > 1) break;
        int next = 0;
        if (lane == 0) next = (int)atomicAdd(p.queue, 1u) + (int)gridDim.x * kRenderWarps;
        item = __shfl_sync(GSR_FULL_MASK, next, 0);
    }
    if (__any_sync(GSR_FULL_MASK, bad) && lane == 0) record_error(p.status, kErrBadInput);
}

template <int BX, int BY, int CADENCE, int RANGE_MODE, bool BATCH, bool QUAD = false>
cudaError_t launch_blend(const RenderParams& p, cudaStream_t stream)
{
    if constexpr (BX == 16 && BY == 16) {
        if (split_tiles(p.items)) {
            return launch_chained(k_blend<BX, BY, CADENCE, RANGE_MODE, BATCH, QUAD, kRenderWarps>, p.items,
                                  kRenderWarps * 32, 0, stream, p);
        }
    }
    auto kern = k_blend<BX, BY, CADENCE, RANGE_MODE, BATCH, QUAD, 1>;
    // per device; host threads may race to fill it with the same value
    static std::atomic<int> per_sm_cache[kMaxDevices];
    const int dev = current_device();
    if (dev < 0) return cudaErrorInvalidDevice;
    int per_sm = per_sm_cache[dev].load(std::memory_order_relaxed);
    if (per_sm == 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kRenderWarps * 32, 0) != cudaSuccess ||
            per_sm < 1)
            per_sm = 1;
        per_sm_cache[dev].store(per_sm, std::memory_order_relaxed);
    }
    const int grid = max(1, min(device_sm_count() * per_sm, div_up(p.items, kRenderWarps)));
    return launch_chained(kern, grid, kRenderWarps * 32, 0, stream, p);
}

template <int BX, int BY, int CADENCE, int SHADER, bool DT, int RANGE_MODE, bool TMA, bool BATCH = false,
          int EXIT = 0, bool QUAD = false>
cudaError_t launch_variant(const RenderParams& p, cudaStream_t stream)
{
    auto kern = k_render<BX, BY, CADENCE, SHADER, DT, RANGE_MODE, TMA, BATCH, EXIT, QUAD>;
    // per device; host threads may race to fill it with the same value
    static std::atomic<int> per_sm_cache[kMaxDevices];
    const int dev = current_device();
    if (dev < 0) return cudaErrorInvalidDevice;
    int per_sm = per_sm_cache[dev].load(std::memory_order_relaxed);
    if (per_sm == 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kRenderWarps * 32, 0) != cudaSuccess ||
            per_sm < 1)
            per_sm = 1;
        per_sm_cache[dev].store(per_sm, std::memory_order_relaxed);
    }
    const int warps_needed = p.items;
    int grid = device_sm_count() * per_sm;
    grid = max(1, min(grid, div_up(warps_needed, kRenderWarps)));
    kern<<<grid, kRenderWarps * 32, 0, stream>>>(p);
    return cudaGetLastError();
}

// TMA staging, the distance-thresholded and the split renders, the general
// shader (SH 1) and 24-wide tiles (three columns a lane) take the scalar kernel;
// the rest take the paired one, the faster of the two at every size measured (see
// k_blend).
template <int BX, int BY, int CADENCE, int SHADER, int RANGE_MODE>
cudaError_t launch_whole(bool tma, const RenderParams& p, cudaStream_t stream)
{
    if (tma) return launch_variant<BX, BY, CADENCE, SHADER, false, RANGE_MODE, true>(p, stream);
    if constexpr (SHADER == 0 && BX % 16 == 0) return launch_blend<BX, BY, CADENCE, RANGE_MODE, false>(p, stream);
    else return launch_variant<BX, BY, CADENCE, SHADER, false, RANGE_MODE, false>(p, stream);
}

template <int BX, int BY>
cudaError_t dispatch_shape(int variant, bool tma, const RenderParams& p, cudaStream_t stream)
{
    constexpr int SH = (BX == 16 && BY == 16) ? 0 : 1;
    // FUSED/DEFAULT find their ranges in-kernel unless ranges were supplied
    // (the same [lower, upper) bounds, so the same image)
    const bool ranges = p.ranges != nullptr;
    switch (variant) {
    case GSR_RENDER_PERSISTENT_RANGES: return launch_whole<BX, BY, 8, 0, 0>(tma, p, stream);
    case GSR_RENDER_PERSISTENT_FUSED:
        return ranges ? launch_whole<BX, BY, 16, 0, 0>(tma, p, stream) : launch_whole<BX, BY, 16, 0, 1>(tma, p, stream);
    case GSR_RENDER_DEFAULT:
        return ranges ? launch_whole<BX, BY, 2, SH, 0>(tma, p, stream) : launch_whole<BX, BY, 2, SH, 1>(tma, p, stream);
    case GSR_RENDER_RANGES_CADENCE2: return launch_whole<BX, BY, 2, SH, 0>(tma, p, stream);
    case GSR_RENDER_DT:
        return tma ? launch_variant<BX, BY, 8, 0, true, 0, true>(p, stream)
                   : launch_variant<BX, BY, 8, 0, true, 0, false>(p, stream);
    case GSR_RENDER_SPLIT:  // axis-shared shader at every tile width, per-half exit
        if (BY != 16) return cudaErrorInvalidValue;
        if (ranges) return launch_variant<BX, BY, 2, 0, false, 0, false, false, 1>(p, stream);
        return launch_variant<BX, BY, 2, 0, false, 1, false, false, 1>(p, stream);
    default:
        return cudaErrorInvalidValue;
    }
}

// Quad renders (16x16 tiles, keys per 2x2 group of tiles): the paired kernel, but
// for the distance-thresholded render.
template <bool BATCH>
cudaError_t dispatch_quad(int variant, const RenderParams& p, cudaStream_t stream)
{
    const bool ranges = p.ranges != nullptr;
    switch (variant) {
    case GSR_RENDER_PERSISTENT_RANGES: return launch_blend<16, 16, 8, 0, BATCH, true>(p, stream);
    case GSR_RENDER_PERSISTENT_FUSED:
        if (ranges || BATCH) return launch_blend<16, 16, 16, 0, BATCH, true>(p, stream);
        return launch_blend<16, 16, 16, 1, false, true>(p, stream);
    case GSR_RENDER_DEFAULT:
        if (ranges || BATCH) return launch_blend<16, 16, 2, 0, BATCH, true>(p, stream);
        return launch_blend<16, 16, 2, 1, false, true>(p, stream);
    case GSR_RENDER_RANGES_CADENCE2: return launch_blend<16, 16, 2, 0, BATCH, true>(p, stream);
    case GSR_RENDER_DT: return launch_variant<16, 16, 8, 0, true, 0, false, BATCH, 0, true>(p, stream);
    default: return cudaErrorInvalidValue;
    }
}

// Batched renders: ranges always precomputed, never staged by TMA, 16x16,
// 32x16 and 32x32 tiles.
template <int BX, int BY>
cudaError_t dispatch_batch(int variant, const RenderParams& p, cudaStream_t stream)
{
    constexpr int SH = (BX == 16 && BY == 16) ? 0 : 1;
    switch (variant) {
    case GSR_RENDER_PERSISTENT_RANGES: return launch_blend<BX, BY, 8, 0, true>(p, stream);
    case GSR_RENDER_PERSISTENT_FUSED: return launch_blend<BX, BY, 16, 0, true>(p, stream);
    case GSR_RENDER_DEFAULT:
    case GSR_RENDER_RANGES_CADENCE2:
        if constexpr (SH == 0) return launch_blend<BX, BY, 2, 0, true>(p, stream);
        else return launch_variant<BX, BY, 2, SH, false, 0, false, true>(p, stream);
    case GSR_RENDER_DT: return launch_variant<BX, BY, 8, 0, true, 0, false, true>(p, stream);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

static cudaError_t launch_prepared(const RenderArgs& a, RenderParams& p, cudaStream_t stream);

static bool use_render_tma()
{
    // in the scalar kernel per-thread cp.async staging measured faster than
    // per-lane 16-byte bulk copies (28 vs 48 us at 1080p, 2.5 vs 3.6 ms at 8K), and
    // k_blend stages neither way: bulk copies only on request (read once,
    // thread-safe initialisation)
    static const bool tma = [] {
        const char* e = getenv("GSR_RENDER_TMA");
        return e && strcmp(e, "1") == 0;
    }();
    return tma;
}

// ---------------------------------------------------------------------------
// Differentiable render (no counterpart in the reference): the forward of the
// persistent lite render (16x16 tiles, exit check every 8 Gaussians, same
// per-pixel arithmetic through shade<>) writing a float image, each pixel's
// final transmittance and each tile's number of blended Gaussians; and its
// backward, which walks every tile's list in reverse.

namespace {

constexpr int kTrainWarps = 4;
constexpr int kTrainCadence = 8;

// Where tile (tx, ty) of `view` finds its list: its own range, or with quad
// keys its quad's range, whose entries carry the bit `qbit` when they
// belong to this tile.
template <bool QUAD>
__device__ __forceinline__ int train_list(int view, int tile, int tx, int ty, int gx, int gy, uint32_t& qbit)
{
    qbit = 0u;
    if (!QUAD) return tile;
    const int qgx = quad_cols(gx), qpv = qgx * quad_cols(gy);
    qbit = 1u << (kQuadShift + ((tx & 1) | ((ty & 1) << 1)));
    return view * qpv + (ty >> 1) * qgx + (tx >> 1);
}

// The tile (or strip of a tile) of a warp of the training kernels.
template <bool QUAD, int SPLIT>
struct TrainTile {
    int tile, start, stop, ox, oy, cb, rb;
    size_t pix0;
    uint32_t qbit;

    __device__ __forceinline__ bool open(const TrainRenderArgs& a, unsigned lane, int warp)
    {
        // tile: global over the views; lt: within its view
        const int gx = (a.W + 15) / 16, gy = (a.H + 15) / 16, tiles = gx * gy;
        tile = SPLIT > 1 ? (int)blockIdx.x : (int)blockIdx.x * kTrainWarps + warp;
        if (tile >= tiles * max(a.n_views, 1)) return false;
        const int view = tile / tiles, lt = tile - view * tiles;
        pix0 = (size_t)view * a.W * a.H;
        const int n = (int)max(0LL, min((long long)*a.d_num, a.cap));
        const int tx = lt % gx, ty = lt / gx;
        ox = tx * 16;
        oy = ty * 16;
        cb = (int)(lane & 7u) * 2;
        rb = (SPLIT > 1 ? warp * (16 / SPLIT) : 0) + (int)(lane >> 3) * (4 / SPLIT);
        const int2 rg = a.ranges[train_list<QUAD>(view, tile, tx, ty, gx, gy, qbit)];
        start = min(max(rg.x, 0), n);
        stop = min(max(rg.y, start), n);
        return true;
    }
};

template <bool QUAD, int SPLIT>
__global__ __launch_bounds__(kTrainWarps * 32, 4) void k_render_train(const TrainRenderArgs a)
{
    static_assert(SPLIT == 1 || SPLIT == kTrainWarps, "a tile per warp, or per CTA");
    constexpr int TY = 4 / SPLIT;
    __shared__ BlendRing<SPLIT == 1> rings[kTrainWarps];
    const unsigned lane = threadIdx.x & 31u;
    const int warp = threadIdx.x >> 5;
    TrainTile<QUAD, SPLIT> t;
    if (!t.open(a, lane, warp)) return;
    const Features f{a.xy, a.con, a.rgbd, a.vals, (uint32_t)a.P};
    Pixels<2, TY> px;
    px.reset(t.ox + t.cb, t.oy + t.rb);
    bool bad = false;
    int last = 0;
    const bool any =
        blend_list<2, TY, kTrainCadence, QUAD, SPLIT>(px, rings[warp], f, t.start, t.stop, t.qbit, lane, bad, last);
    // list positions up to the last Gaussian blended: what the backward replays
    if (lane == 0 && (SPLIT == 1 || warp == 0)) a.n_tile[t.tile] = any ? last - t.start + 1 : 0;
#pragma unroll
    for (int i = 0; i < TY; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int x = t.ox + t.cb + j, y = t.oy + t.rb + i;
            if (x >= a.W || y >= a.H) continue;
            auto half = [&](f32x2 v) { return j ? hi_of(v) : lo_of(v); };
            const size_t o = t.pix0 + (size_t)y * a.W + x;
            const float T = half(px.T[i][0]), tt = T < 0.0001f ? 0.0f : T;
            a.T_final[o] = T;
            a.image[3 * o + 0] = half(px.C[i][0][0]) + tt * a.bg[0];
            a.image[3 * o + 1] = half(px.C[i][0][1]) + tt * a.bg[1];
            a.image[3 * o + 2] = half(px.C[i][0][2]) + tt * a.bg[2];
        }
}

// One step of a spread sum: lanes whose bit `d` is set keep b and send a, the
// others keep a and send b.
__device__ __forceinline__ float spread(float a, float b, bool up, int d)
{
    return (up ? b : a) + __shfl_xor_sync(GSR_FULL_MASK, up ? a : b, d);
}

// Sums of sixteen values over the warp in 16 shuffles: at each of the first
// four steps a lane keeps half of its partial sums and sends the other half
// to its partner.  Lane l returns the total of v[l >> 1].
__device__ __forceinline__ float warp_sum16_spread(const float (&v)[16], unsigned lane)
{
    float h[8], q[4], p[2];
#pragma unroll
    for (int k = 0; k < 8; k++) h[k] = spread(v[k], v[k + 8], (lane & 16u) != 0u, 16);
#pragma unroll
    for (int k = 0; k < 4; k++) q[k] = spread(h[k], h[k + 4], (lane & 8u) != 0u, 8);
#pragma unroll
    for (int k = 0; k < 2; k++) p[k] = spread(q[k], q[k + 2], (lane & 4u) != 0u, 4);
    const float t = spread(p[0], p[1], (lane & 2u) != 0u, 2);
    return t + __shfl_xor_sync(GSR_FULL_MASK, t, 1);
}

// Sums of two values: lane l returns the total of v[l >> 4].
__device__ __forceinline__ float warp_sum2_spread(float a, float b, unsigned lane)
{
    float t = spread(a, b, (lane & 16u) != 0u, 16);
#pragma unroll
    for (int d = 8; d > 0; d >>= 1) t += __shfl_xor_sync(GSR_FULL_MASK, t, d);
    return t;
}

// A lane's TY x 2 pixels of the reverse walk, columns in pairs.  R . G is
// carried as one number per pixel: the walk only needs the colour behind a
// Gaussian through its product with the pixel's gradient.  All colours, R's
// too, are relative to the list's farthest one (Feed::centre): (c - R) . G is
// then a difference of products as small as the colours' differences, and does
// not cancel where neighbours along a ray have nearly one colour.
template <int TY>
struct BackPixels {
    f32x2 T[TY], RG[TY], G[TY][3];
    f32x2 ncol, nrow[TY];

    // The sums of one Gaussian over the lane's pixels: gradients of its conic
    // (xx, xy, yy) and log2 opacity, centre (x, y), then colour (r, g | b).
    // T goes from behind the Gaussian to before it, RG from behind it to
    // composited with it.
    __device__ __forceinline__ void step(const PairRecord& q, float* v8, float& blue)
    {
        const f32x2 minus1 = pair(-1.0f, -1.0f), one = pair(1.0f, 1.0f);
        // the forward's per-pixel power, term for term (Pixels::blend)
        const f32x2 dx = add2(q.x, ncol);
        const f32x2 xw = fma2(mul2(q.a, dx), dx, q.w);
        const f32x2 xb = mul2(q.b, dx);
        // dx depends on the column only and dy on the row only, so the conic
        // and centre gradients need three sums per column over this lane's
        // rows: of dp, dp dy and dp dy^2
        const f32x2 zero = pair(0.0f, 0.0f);
        f32x2 s0 = zero, s1 = zero, s2 = zero, gr = zero, gg = zero, gb = zero;
#pragma unroll
        for (int i = 0; i < TY; i++) {
            const f32x2 dy = add2(q.y, nrow[i]);
            const f32x2 alpha = ex2_2(fma2(xb, dy, fma2(mul2(q.c, dy), dy, xw)));
            float m0, m1, t0, t1, a0, a1;
            split(fma2(alpha, minus1, one), m0, m1);  // 1 - alpha
            split(T[i], t0, t1);
            split(mul2(T[i], pair(rcp_approx_ftz(m0), rcp_approx_ftz(m1))), a0, a1);
            const f32x2 Tb = pair(m0 > 0.0f ? fminf(1.0f, a0) : t0, m1 > 0.0f ? fminf(1.0f, a1) : t1);
            T[i] = Tb;
            const f32x2 w = mul2(alpha, Tb);
            // (c - R) . G
            const f32x2 d = fma2(RG[i], minus1, fma2(q.bl, G[i][2], fma2(q.g, G[i][1], mul2(q.r, G[i][0]))));
            RG[i] = fma2(alpha, d, RG[i]);  // (alpha c + (1 - alpha) R) . G
            gr = fma2(w, G[i][0], gr);
            gg = fma2(w, G[i][1], gg);
            gb = fma2(w, G[i][2], gb);
            // d power of this pixel, without its factor ln 2 (applied to the totals)
            const f32x2 dp = mul2(d, w);
            const f32x2 dpy = mul2(dp, dy);
            s0 = add2(s0, dp);
            s1 = add2(s1, dpy);
            s2 = fma2(dpy, dy, s2);
        }
        // d power / d (conic x, y, z, w) = (dx^2, dx dy, dy^2, 1);
        // d power / d centre = (2 a dx + b dy, 2 c dy + b dx)
        const f32x2 x0 = mul2(dx, s0);
        const f32x2 xx = mul2(dx, x0), xy = mul2(dx, s1);
        const float a = lo_of(q.a), b = lo_of(q.b), c = lo_of(q.c);
        const float sx = lo_of(x0) + hi_of(x0), sy = lo_of(s1) + hi_of(s1);
        v8[0] = lo_of(xx) + hi_of(xx);
        v8[1] = lo_of(xy) + hi_of(xy);
        v8[2] = lo_of(s2) + hi_of(s2);
        v8[3] = lo_of(s0) + hi_of(s0);
        v8[4] = fmaf(2.0f * a, sx, b * sy);
        v8[5] = fmaf(2.0f * c, sy, b * sx);
        v8[6] = lo_of(gr) + hi_of(gr);
        v8[7] = lo_of(gg) + hi_of(gg);
        blue = lo_of(gb) + hi_of(gb);
    }
};

// Reverse traversal of each tile's blended Gaussians.  With T_after the
// transmittance behind Gaussian i and alpha_i recomputed bit for bit,
// T_before = T_after / (1 - alpha_i) (1 - alpha is exact once alpha >= 1/2);
// R, the colour composited behind i per unit transmittance, starts at bg (or
// 0 where the forward dropped the background term) and follows
// R <- alpha c + (1 - alpha) R.  Then
//   dL/dc_i     = sum_px alpha_i T_before dL/dC
//   dL/dalpha_i = T_before (c_i - R) . dL/dC,   d alpha/d power = alpha ln 2
// and the power's derivatives give the conic/opacity and centre gradients.
//
// The kernel is bound by the FMA pipe and instruction issue: the pixels go in
// column pairs (see Pixels), and the 9 sums of two Gaussians at a time are
// reduced over the warp together, sixteen of them spread over the lanes
// (warp_sum16_spread), which leaves each lane pair with one total to add:
// eight consecutive floats of each Gaussian's 12-float record (grad_rec), or
// entries of the three arrays.
template <bool QUAD, int SPLIT>
__global__ __launch_bounds__(kTrainWarps * 32, 4) void k_render_backward(const TrainRenderArgs a)
{
    static_assert(SPLIT == 1 || SPLIT == kTrainWarps, "a tile per warp, or per CTA");
    constexpr int TY = 4 / SPLIT;
    __shared__ BlendRing<SPLIT == 1> rings[kTrainWarps];
    const unsigned lane = threadIdx.x & 31u;
    const int warp = threadIdx.x >> 5;
    BlendRing<SPLIT == 1>& R = rings[warp];
    TrainTile<QUAD, SPLIT> t;
    if (!t.open(a, lane, warp)) return;
    const int count = min(max(__ldg(a.n_tile + t.tile), 0), t.stop - t.start);
    const Features f{a.xy, a.con, a.rgbd, a.vals, (uint32_t)a.P};
    bool bad = false;
    Feed<QUAD, true, SPLIT == 1> feed;
    feed.open(f, t.start, t.start + count, t.qbit, lane);
    // the pixels' loads travel with the list's
    BackPixels<TY> px;
    px.ncol = pair(-(float)(t.ox + t.cb), -(float)(t.ox + t.cb + 1));
#pragma unroll
    for (int i = 0; i < TY; i++) {
        float T[2], g[2][3];
        const int y = t.oy + t.rb + i;
        px.nrow[i] = pair(-(float)y, -(float)y);
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int x = t.ox + t.cb + j;
            const bool in = x < a.W && y < a.H;
            const size_t o = in ? t.pix0 + (size_t)y * a.W + x : 0;
            T[j] = in ? __ldg(a.T_final + o) : 1.0f;
#pragma unroll
            for (int ch = 0; ch < 3; ch++) g[j][ch] = in ? __ldg(a.grad_image + 3 * o + ch) : 0.0f;
        }
        px.T[i] = pair(T[0], T[1]);
#pragma unroll
        for (int ch = 0; ch < 3; ch++) px.G[i][ch] = pair(g[0][ch], g[1][ch]);
    }
    feed.fetch(R, f, lane, bad);
    feed.centre();
    // R . G behind everything: the background's, or 0 where the forward dropped it
    const float3 m = feed.mid, bg = make_float3(a.bg[0] - m.x, a.bg[1] - m.y, a.bg[2] - m.z);
#pragma unroll
    for (int i = 0; i < TY; i++) {
        auto behind = [&](float T, float g0, float g1, float g2) {
            return T < 0.0001f ? -(m.x * g0 + m.y * g1 + m.z * g2) : bg.x * g0 + bg.y * g1 + bg.z * g2;
        };
        px.RG[i] = pair(behind(lo_of(px.T[i]), lo_of(px.G[i][0]), lo_of(px.G[i][1]), lo_of(px.G[i][2])),
                        behind(hi_of(px.T[i]), hi_of(px.G[i][0]), hi_of(px.G[i][1]), hi_of(px.G[i][2])));
    }
    // where a lane's total goes: lane l has value (l >> 1) & 7 of the first
    // (l < 16) or second Gaussian; lanes 0 and 16 add the blue sums as well
    const int slot = (int)(lane >> 1) & 7;
    const bool first = lane < 16u;
    const float unit = slot < 6 ? 0.69314718055994531f : 1.0f;  // the ln 2 of d power
    while (feed.n > 0) {
        const int n = feed.n;
        __syncwarp();
        feed.store(R, lane);
        __syncwarp();
        feed.fetch(R, f, lane, bad);
        for (int k = 0; k < n; k += 2) {
            float v[16], b0, b1 = 0.0f;
            px.step(read_record(R, k), v, b0);
            if (k + 1 < n) {
                px.step(read_record(R, k + 1), v + 8, b1);
            } else {
#pragma unroll
                for (int q = 8; q < 16; q++) v[q] = 0.0f;
            }
            const float t16 = unit * warp_sum16_spread(v, lane);
            const float t2 = warp_sum2_spread(b0, b1, lane);
            const uint32_t gid = first ? R.gid[k] : (k + 1 < n ? R.gid[k + 1] : 0xFFFFFFFFu);
            if (gid != 0xFFFFFFFFu) {
                if (a.grad_rec) {
                    float* rec = a.grad_rec + 12 * (size_t)gid;
                    if ((lane & 1u) == 0u) atomicAdd(rec + slot, t16);
                    if ((lane & 15u) == 1u) atomicAdd(rec + 8, t2);
                } else {
                    float* dst = slot < 4   ? a.grad_con + 4 * (size_t)gid + slot
                                 : slot < 6 ? a.grad_xy + 2 * (size_t)gid + (slot - 4)
                                            : a.grad_rgb + 3 * (size_t)gid + (slot - 6);
                    if ((lane & 1u) == 0u) atomicAdd(dst, t16);
                    if ((lane & 15u) == 1u) atomicAdd(a.grad_rgb + 3 * (size_t)gid + 2, t2);
                }
            }
        }
    }
}

template <bool QUAD>
cudaError_t launch_train(const TrainRenderArgs& a, bool backward, int tiles, cudaStream_t stream)
{
    const dim3 block(kTrainWarps * 32);
    if (backward) {
        if (split_tiles(tiles)) k_render_backward<QUAD, kTrainWarps><<<tiles, block, 0, stream>>>(a);
        else k_render_backward<QUAD, 1><<<div_up(tiles, kTrainWarps), block, 0, stream>>>(a);
    } else {
        if (split_tiles(tiles)) k_render_train<QUAD, kTrainWarps><<<tiles, block, 0, stream>>>(a);
        else k_render_train<QUAD, 1><<<div_up(tiles, kTrainWarps), block, 0, stream>>>(a);
    }
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_render_train(const TrainRenderArgs& a, bool backward, cudaStream_t stream)
{
    const long long tiles = (long long)((a.W + 15) / 16) * ((a.H + 15) / 16) * max(a.n_views, 1);
    if (tiles <= 0) return cudaSuccess;
    if (tiles > INT32_MAX - kTrainWarps) return cudaErrorInvalidValue;
    return a.quad ? launch_train<true>(a, backward, (int)tiles, stream)
                  : launch_train<false>(a, backward, (int)tiles, stream);
}

cudaError_t launch_render(const RenderArgs& a, cudaStream_t stream)
{
    RenderParams p;
    p.n_host = a.num;
    p.d_num = a.d_num;
    p.cap = a.d_num ? a.cap : (long long)a.num;
    p.W = a.W;
    p.H = a.H;
    if (a.quad) {
        if (a.bx != 16 || a.by != 16) return cudaErrorInvalidValue;
        p.gx = quad_cols(div_up(a.W, 16));
        p.tiles = p.gx * quad_cols(div_up(a.H, 16));
        p.items = 4 * p.tiles;
    } else {
        p.gx = div_up(a.W, a.bx);
        p.tiles = p.gx * div_up(a.H, a.by);
        p.items = p.tiles;
    }
    p.P = a.P;
    p.xy = a.xy;
    p.rgbd = a.rgbd;
    p.con = a.con;
    p.keys = a.keys;
    p.vals = a.vals;
    p.ranges = a.ranges;
    p.bg = make_float3(a.bg[0], a.bg[1], a.bg[2]);
    p.out = reinterpret_cast<uchar3*>(a.out);
    p.queue = &a.ws->render_queue;
    p.status = &a.ws->status;
    p.views = nullptr;
    p.n_views = 0;
    return launch_prepared(a, p, stream);
}

cudaError_t launch_render_views(const RenderArgs& a, const RenderView* views_dev, int n_views, int total_tiles,
                                cudaStream_t stream)
{
    if (!views_dev || n_views <= 0) return cudaErrorInvalidValue;
    RenderParams p;
    p.n_host = a.num;
    p.d_num = a.d_num;
    p.cap = a.d_num ? a.cap : (long long)a.num;
    p.W = p.H = p.gx = 1;  // per view
    p.tiles = total_tiles;
    p.items = a.quad ? 4 * total_tiles : total_tiles;
    p.P = a.P;
    p.xy = a.xy;
    p.rgbd = a.rgbd;
    p.con = a.con;
    p.keys = a.keys;
    p.vals = a.vals;
    p.ranges = a.ranges;
    p.bg = make_float3(0.f, 0.f, 0.f);
    p.out = nullptr;
    p.queue = &a.ws->render_queue;
    p.status = &a.ws->status;
    p.views = views_dev;
    p.n_views = n_views;
    return launch_prepared(a, p, stream);
}

static cudaError_t launch_prepared(const RenderArgs& a, RenderParams& p, cudaStream_t stream)
{
    if (p.tiles <= 0) return cudaSuccess;
    cudaError_t e = a.queue_clear ? cudaSuccess : cudaMemsetAsync(p.queue, 0, sizeof(uint32_t), stream);
    if (e != cudaSuccess) return e;
    // TMA bulk copies, where asked for, need 16-byte aligned feature arrays
    const bool tma = use_render_tma() && ((reinterpret_cast<uintptr_t>(a.xy) | reinterpret_cast<uintptr_t>(a.rgbd) |
                                           reinterpret_cast<uintptr_t>(a.con)) & 15u) == 0;
    if (p.views) {
        if (!p.ranges || ((reinterpret_cast<uintptr_t>(a.xy) | reinterpret_cast<uintptr_t>(a.rgbd) |
                           reinterpret_cast<uintptr_t>(a.con)) & 15u) != 0)
            return cudaErrorInvalidValue;
        if (a.quad) return a.bx == 16 && a.by == 16 ? dispatch_quad<true>(a.variant, p, stream) : cudaErrorInvalidValue;
        if (a.bx == 16 && a.by == 16) return dispatch_batch<16, 16>(a.variant, p, stream);
        if (a.bx == 32 && a.by == 16) return dispatch_batch<32, 16>(a.variant, p, stream);
        if (a.bx == 32 && a.by == 32) return dispatch_batch<32, 32>(a.variant, p, stream);
        return cudaErrorInvalidValue;
    }
    if (a.quad) return a.bx == 16 && a.by == 16 ? dispatch_quad<false>(a.variant, p, stream) : cudaErrorInvalidValue;
    if (a.bx == 16 && a.by == 16) return dispatch_shape<16, 16>(a.variant, tma, p, stream);
    if (a.bx == 32 && a.by == 16) return dispatch_shape<32, 16>(a.variant, tma, p, stream);
    if (a.bx == 24 && a.by == 16) return dispatch_shape<24, 16>(a.variant, tma, p, stream);
    if (a.bx == 32 && a.by == 32) return dispatch_shape<32, 32>(a.variant, tma, p, stream);
    return cudaErrorInvalidValue;
}

}  // namespace gsr

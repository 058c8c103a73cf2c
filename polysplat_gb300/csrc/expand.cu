// Per-tile lists from sorted quad keys.  The fused 16x16 forward emits and
// sorts one key per 2x2 group of tiles and then writes out, for every tile, the
// keys of its quad whose mask names it: the same sorted per-tile arrays and
// ranges as sorting per-tile keys, while every digit pass moves a third to two
// thirds of the pairs.
//
// Number a quad's tiles 0..3 (kQuadShift's bits) and let P_b(i) be how many of
// the sorted keys before i name tile b of their quad.  Within a quad, key i's
// place in the list of tile b is P_b(i) - P_b(first key of the quad), and the
// list's length is the difference of P_b over the quad.  Each CTA takes one span
// of keys, so P is a count within the span plus the totals of the spans before.
//   1. k_quad_starts: the span-local P at both ends of every quad; span totals
//   2. k_quad_tiles:  list lengths, their prefix over the tiles = the ranges
//   3. k_quad_expand: every key to its places
// 9.5 M pairs of 3.7 M quad keys at 1080p: 11 + 7 + 33 us, for digit passes of 27
// us instead of 56 (five of them), no range pass (21) and 20 us less emission of
// large Gaussians.  26 M pairs of 21 M at 8K: 50 + 22 + 148 us, which the passes do
// not give back.  The expansion reads 12 bytes a key and writes 12 a pair at 4.5
// TB/s; spans of 4, 5 or 6 CTAs per SM and 4 keys a thread measure alike.
//
// Step 2 needs the lists before a CTA's own tiles.  Adding them up in every CTA
// saves a launch but is quadratic in the tiles, so above kDirectTiles a kernel of
// its own (k_quad_sums) leaves the CTAs' totals.  Frames with the totals / adding
// up: 8160 tiles 522 / 516 us, 14400 360 / 355, 32400 555 / 557, 129600 919 / 929,
// 291600 4856 / 4890, 518400 1916 / 1982 and 2758 / 2822.
#include <algorithm>
#include <cstdint>

#include "gsr_common.cuh"
#include "gsr_internal.h"

namespace gsr {

namespace {

constexpr int kExpThreads = 256;
constexpr int kExpWarps = kExpThreads / 32;
constexpr int kExpSteps = 8;  // keys a thread takes at a time
constexpr int kExpShare = 32 * kExpSteps;
constexpr int kExpChunk = kExpWarps * kExpShare;
constexpr int kExpCtas = 4;  // spans per SM
constexpr int kTileThreads = 1024;
constexpr int kMaxSpans = 1024;
constexpr int kDirectTiles = 32768;

// Arrays of one expansion, in the unsorted key buffer (the sort has read it).
struct QuadSeg {
    uint4* first;     // [quads] P within its span at the quad's first key ...
    uint4* last;      // [quads] ... and behind its last
    int* first_span;  // [quads]
    int* last_span;   // [quads]
    uint32_t* base;   // [quads][4] place of the tile's first key - P there
    uint32_t* tile;   // [quads] the quad's first tile
    uint4* totals;    // [spans]
    uint32_t* sums;   // [CTAs of k_quad_tiles] their tiles' list lengths, or nullptr
};

// K: 64-bit keys (quad << 32 | depth bits), or the depth-first pipeline's
// 32-bit quad ids.
template <typename K>
struct ExpandJob {
    const K* keys;
    const uint32_t* vals;
    const unsigned long long* count;
    long long cap;
    int gx, gy, quads, spans;
    QuadSeg seg;
    K* out_keys;
    uint32_t* out_vals;
    int2* ranges;
    int32_t* total;
};

__host__ __device__ inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

template <typename K>
__device__ __forceinline__ int key_count(const ExpandJob<K>& a)
{
    const long long n = (int)(uint32_t)*a.count;  // as the sort counts
    return (int)(n < 0 ? 0 : n > a.cap ? a.cap : n);
}

// Keys per span: whole warps' shares of a chunk.
__device__ __forceinline__ int span_length(int n, int spans)
{
    return ((n + spans - 1) / spans + kExpShare - 1) & ~(kExpShare - 1);
}

__device__ __forceinline__ uint4 add4(uint4 a, uint4 b)
{
    return make_uint4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

// The four tile bits of a value, one to a byte.
__device__ __forceinline__ uint32_t tile_bytes(uint32_t val)
{
    return (val >> kQuadShift) * 0x00204081u & 0x01010101u;
}

// Sum over the warp of one byte per tile and lane (32 kExpSteps at most each).
__device__ __forceinline__ uint2 warp_tiles(uint32_t bytes)
{
    return make_uint2(__reduce_add_sync(GSR_FULL_MASK, bytes & 0x00FF00FFu),
                      __reduce_add_sync(GSR_FULL_MASK, bytes >> 8 & 0x00FF00FFu));
}
__device__ __forceinline__ uint4 widen(uint2 s)
{
    return make_uint4(s.x & 0xFFFFu, s.y & 0xFFFFu, s.x >> 16, s.y >> 16);
}

// P where the warp's share of a chunk begins, and `run`, P where the chunk
// begins, moved past it.  Step k, lane l of warp w has key w * kExpShare +
// 32 k + l of the chunk.  The caller alternates s_sum, so one barrier is enough.
__device__ __forceinline__ uint4 warp_base(const uint32_t (&val)[kExpSteps], uint4& run, uint2 (&s_sum)[kExpWarps],
                                           unsigned lane, int warp)
{
    uint32_t bytes = 0;
#pragma unroll
    for (int k = 0; k < kExpSteps; k++) bytes += tile_bytes(val[k]);
    const uint2 mine = warp_tiles(bytes);
    if (lane == 0) s_sum[warp] = mine;
    __syncthreads();
    uint2 before = make_uint2(0, 0), all = make_uint2(0, 0);
#pragma unroll
    for (int w = 0; w < kExpWarps; w++) {
        const uint2 s = s_sum[w];
        if (w < warp) {
            before.x += s.x;
            before.y += s.y;
        }
        all.x += s.x;
        all.y += s.y;
    }
    const uint4 at = add4(run, widen(before));
    run = add4(run, widen(all));
    return at;
}

// P at this lane's key of the step that begins at `at`, which moves past it.
__device__ __forceinline__ uint4 step_counts(uint32_t val, uint4& at)
{
    const unsigned b0 = __ballot_sync(GSR_FULL_MASK, val & 1u << kQuadShift);
    const unsigned b1 = __ballot_sync(GSR_FULL_MASK, val & 2u << kQuadShift);
    const unsigned b2 = __ballot_sync(GSR_FULL_MASK, val & 4u << kQuadShift);
    const unsigned b3 = __ballot_sync(GSR_FULL_MASK, val & 8u << kQuadShift);
    const unsigned lt = lanemask_lt();
    const uint4 p = add4(at, make_uint4(__popc(b0 & lt), __popc(b1 & lt), __popc(b2 & lt), __popc(b3 & lt)));
    at = add4(at, make_uint4(__popc(b0), __popc(b1), __popc(b2), __popc(b3)));
    return p;
}

// Bound by the latency of its loads.  Counting every step instead of those with
// an end of a quad took 81 us for 50 (21 M keys): 1 step in 20 has one there.
template <typename K>
__global__ __launch_bounds__(kExpThreads, kExpCtas) void k_quad_starts(const __grid_constant__ ExpandJob<K> a)
{
    __shared__ uint2 s_sum[2][kExpWarps];
    const unsigned lane = threadIdx.x & 31u;
    const int warp = threadIdx.x >> 5;
    chain_wait();
    chain_ready();
    const int n = key_count(a);
    const int len = span_length(n, a.spans);
    const long long first = (long long)blockIdx.x * len;
    const int lo = (int)min((long long)n, first), end = (int)min((long long)n, first + len);
    constexpr int kWords = sizeof(K) / 4;  // the quad is a key's last word
    const uint32_t* hi = reinterpret_cast<const uint32_t*>(a.keys) + (kWords - 1);
    uint4 run = make_uint4(0, 0, 0, 0);
    int flip = 0;
    for (int c0 = lo; c0 < end; c0 += kExpChunk, flip ^= 1) {
        const int i0 = c0 + warp * kExpShare + (int)lane, left = end - i0;  // keys 32 k with 32 k < left
        const uint32_t* hp = hi + kWords * (size_t)i0;
        const uint32_t* vp = a.vals + i0;
        uint32_t quad[kExpSteps], val[kExpSteps];
#pragma unroll
        for (int k = 0; k < kExpSteps; k++) {
            quad[k] = 32 * k < left ? hp[32 * kWords * k] : 0u;
            val[k] = 32 * k < left ? vp[32 * k] : 0u;
        }
        uint32_t before = lane == 0 && i0 > 0 && left > 0 ? *(hp - kWords) : 0u;
        const uint4 at = warp_base(val, run, s_sum[flip], lane, warp);
        // counts are needed only in the steps in which a quad ends or begins
        uint32_t bytes = 0;  // this lane's tiles of the steps before
#pragma unroll
        for (int k = 0; k < kExpSteps; k++) {
            const int i = i0 + 32 * k;
            const uint32_t q = quad[k];
            uint32_t prev = __shfl_up_sync(GSR_FULL_MASK, q, 1);
            if (lane == 0) prev = before;
            before = __shfl_sync(GSR_FULL_MASK, q, 31);
            const bool begins = i < end && (i == 0 || prev != q), ends = i < end && i == n - 1;
            if (__any_sync(GSR_FULL_MASK, begins || ends)) {
                uint4 step = add4(at, widen(warp_tiles(bytes)));
                const uint4 p = step_counts(val[k], step);
                if (begins && q < (uint32_t)a.quads) {
                    a.seg.first[q] = p;
                    a.seg.first_span[q] = (int)blockIdx.x;
                }
                if (begins && i > 0 && prev < (uint32_t)a.quads) {
                    a.seg.last[prev] = p;
                    a.seg.last_span[prev] = (int)blockIdx.x;
                }
                if (ends && q < (uint32_t)a.quads) {
                    const uint32_t m = val[k] >> kQuadShift;
                    a.seg.last[q] = add4(p, make_uint4(m & 1u, m >> 1 & 1u, m >> 2 & 1u, m >> 3));
                    a.seg.last_span[q] = (int)blockIdx.x;
                }
            }
            bytes += tile_bytes(val[k]);
        }
    }
    if (threadIdx.x == 0) a.seg.totals[blockIdx.x] = run;
}

// Exclusive scan of one value per thread over the CTA; `sum` becomes the total.
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t (&s_warp)[kTileThreads / 32], uint32_t& sum)
{
    const unsigned lane = threadIdx.x & 31u;
    const int warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t u = __shfl_up_sync(GSR_FULL_MASK, incl, d);
        if (lane >= (unsigned)d) incl += u;
    }
    __syncthreads();  // the last call's sums have been read
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    const uint32_t w = s_warp[lane];
    sum = __reduce_add_sync(GSR_FULL_MASK, w);
    return incl - v + __reduce_add_sync(GSR_FULL_MASK, (int)lane < warp ? w : 0u);
}

__device__ __forceinline__ uint32_t comp(const uint4* p, uint32_t i, int b)
{
    return reinterpret_cast<const uint32_t*>(p + i)[b];
}

// P before each span, one of the four counts at a time, and the sum of the four.
struct SpanPrefix {
    uint32_t pre[4][kMaxSpans];
    uint32_t all[kMaxSpans];
};

template <typename K>
__device__ __forceinline__ void span_prefix(const ExpandJob<K>& a, SpanPrefix& s, uint32_t (&s_warp)[kTileThreads / 32])
{
    const int tid = threadIdx.x;
    const uint4 t = tid < a.spans ? a.seg.totals[tid] : make_uint4(0, 0, 0, 0);
    uint32_t sum;
    s.pre[0][tid] = block_scan(t.x, s_warp, sum);
    s.pre[1][tid] = block_scan(t.y, s_warp, sum);
    s.pre[2][tid] = block_scan(t.z, s_warp, sum);
    s.pre[3][tid] = block_scan(t.w, s_warp, sum);
    s.all[tid] = s.pre[0][tid] + s.pre[1][tid] + s.pre[2][tid] + s.pre[3][tid];
    __syncthreads();
}

// Length of tile t's list; q, b: its quad and number there, p: P at its start.
template <typename K>
__device__ __forceinline__ uint32_t list_length(const ExpandJob<K>& a, const SpanPrefix& s, int t, uint32_t& q, int& b,
                                                uint32_t& p)
{
    const int y = t / a.gx, x = t - y * a.gx;
    q = (uint32_t)((y >> 1) * quad_cols(a.gx) + (x >> 1));
    b = (x & 1) | (y & 1) << 1;
    p = s.pre[b][a.seg.first_span[q]] + comp(a.seg.first, q, b);
    return s.pre[b][a.seg.last_span[q]] + comp(a.seg.last, q, b) - p;
}

// Sum of the list lengths of each CTA's tiles, for grids in which adding up all
// earlier quads in every CTA of k_quad_tiles costs more than this launch.
template <typename K>
__global__ __launch_bounds__(kTileThreads) void k_quad_sums(const __grid_constant__ ExpandJob<K> a)
{
    __shared__ SpanPrefix s;
    __shared__ uint32_t s_warp[kTileThreads / 32];
    chain_wait();
    chain_ready();
    span_prefix(a, s, s_warp);
    const int t = blockIdx.x * kTileThreads + (int)threadIdx.x;
    uint32_t q, p, sum;
    int b;
    block_scan(t < a.gx * a.gy ? list_length(a, s, t, q, b, p) : 0u, s_warp, sum);
    if (threadIdx.x == 0) a.seg.sums[blockIdx.x] = sum;
}

// A thread per tile.  In grids of up to kDirectTiles every CTA sums the list
// lengths of the tiles before its own, quads at a time, instead of waiting for
// the CTAs that hold them (8 CTAs and 7 us at 1080p: latency); in larger ones it
// sums k_quad_sums' totals.
template <typename K>
__global__ __launch_bounds__(kTileThreads) void k_quad_tiles(const __grid_constant__ ExpandJob<K> a)
{
    __shared__ SpanPrefix s;
    __shared__ uint32_t s_warp[kTileThreads / 32];
    const int tid = threadIdx.x;
    chain_wait();
    chain_ready();
    span_prefix(a, s, s_warp);
    const int tiles = a.gx * a.gy, qgx = quad_cols(a.gx);
    const int t0 = blockIdx.x * kTileThreads;
    uint32_t q = 0, p = 0, before = 0, sum;
    int b = 0;
    if (a.seg.sums) {
        for (int k = tid; k < (int)blockIdx.x; k += kTileThreads) before += a.seg.sums[k];
    } else {
        // whole rows of quads before the CTA's first tile, then the tiles between
        const int rows = t0 / a.gx >> 1;
#pragma unroll 4
        for (int k = tid; k < rows * qgx; k += kTileThreads) {
            const uint4 f = a.seg.first[k], l = a.seg.last[k];
            const int fs = a.seg.first_span[k], ls = a.seg.last_span[k];
            before += (l.x - f.x) + (l.y - f.y) + (l.z - f.z) + (l.w - f.w) + s.all[ls] - s.all[fs];
        }
        for (int t = 2 * rows * a.gx + tid; t < t0; t += kTileThreads) before += list_length(a, s, t, q, b, p);
    }
    block_scan(before, s_warp, sum);
    const uint32_t earlier = sum;
    const int t = t0 + tid;
    const uint32_t n = t < tiles ? list_length(a, s, t, q, b, p) : 0u;
    const uint32_t start = earlier + block_scan(n, s_warp, sum);
    if (t < tiles) {
        const uint32_t cap = (uint32_t)a.cap;
        a.ranges[t] = make_int2((int)min(start, cap), (int)min(start + n, cap));
        a.seg.base[4 * q + b] = start - p;
        if (b == 0) a.seg.tile[q] = (uint32_t)t;
    }
    if (t == 0) *a.total = (int)(uint32_t)(*a.count >> 32);
}

template <typename K>
__global__ __launch_bounds__(kExpThreads, kExpCtas) void k_quad_expand(const __grid_constant__ ExpandJob<K> a)
{
    __shared__ uint2 s_sum[2][kExpWarps];
    __shared__ uint4 s_run[kExpWarps];
    const unsigned lane = threadIdx.x & 31u;
    const int warp = threadIdx.x >> 5;
    chain_wait();
    chain_ready();
    const int n = key_count(a);
    const int len = span_length(n, a.spans);
    const long long first = (long long)blockIdx.x * len;
    const int lo = (int)min((long long)n, first), end = (int)min((long long)n, first + len);
    if (lo >= end) return;
    uint4 run = make_uint4(0, 0, 0, 0);
    for (int s = threadIdx.x; s < (int)blockIdx.x; s += kExpThreads) run = add4(run, a.seg.totals[s]);
    run = make_uint4(__reduce_add_sync(GSR_FULL_MASK, run.x), __reduce_add_sync(GSR_FULL_MASK, run.y),
                     __reduce_add_sync(GSR_FULL_MASK, run.z), __reduce_add_sync(GSR_FULL_MASK, run.w));
    if (lane == 0) s_run[warp] = run;
    __syncthreads();
    run = s_run[0];
#pragma unroll
    for (int w = 1; w < kExpWarps; w++) run = add4(run, s_run[w]);
    const uint32_t cap = (uint32_t)a.cap;
    int flip = 0;
    for (int c0 = lo; c0 < end; c0 += kExpChunk, flip ^= 1) {
        const int i0 = c0 + warp * kExpShare + (int)lane, left = end - i0;
        const K* kp = a.keys + i0;
        const uint32_t* vp = a.vals + i0;
        K key[kExpSteps];
        uint32_t val[kExpSteps];
#pragma unroll
        for (int k = 0; k < kExpSteps; k++) {
            key[k] = 32 * k < left ? kp[32 * k] : K(0);
            val[k] = 32 * k < left ? vp[32 * k] : 0u;
        }
        uint4 at = warp_base(val, run, s_sum[flip], lane, warp);
#pragma unroll
        for (int k = 0; k < kExpSteps; k++) {
            const uint4 p = step_counts(val[k], at);
            const uint32_t m = val[k], gid = m & kQuadGidMask;
            const uint32_t q = (uint32_t)(key[k] >> 32 * (sizeof(K) / 4 - 1)), depth = (uint32_t)key[k];
            if (m >> kQuadShift != 0u && q < (uint32_t)a.quads) {
                const uint4 base = *reinterpret_cast<const uint4*>(a.seg.base + 4 * (size_t)q);
                const uint32_t t0 = a.seg.tile[q];
                auto put = [&](uint32_t tile, uint32_t pos) {
                    if (pos < cap) {
                        a.out_keys[pos] = sizeof(K) == 8 ? (K)((uint64_t)tile << 32 | depth) : (K)tile;
                        a.out_vals[pos] = gid;
                    }
                };
                if (m & 1u << kQuadShift) put(t0, base.x + p.x);
                if (m & 2u << kQuadShift) put(t0 + 1u, base.y + p.y);
                if (m & 4u << kQuadShift) put(t0 + (uint32_t)a.gx, base.z + p.z);
                if (m & 8u << kQuadShift) put(t0 + (uint32_t)a.gx + 1u, base.w + p.w);
            }
        }
    }
}

int expand_spans() { return std::min(kMaxSpans, device_sm_count() * kExpCtas); }

}  // namespace

size_t expand_scratch_bytes(int gx, int gy)
{
    const size_t quads = (size_t)quad_cols(gx) * quad_cols(gy);
    const size_t ctas = ((size_t)gx * gy + kTileThreads - 1) / kTileThreads;
    return 256 + 3 * align256(quads * 16) + 3 * align256(quads * 4) + (size_t)kMaxSpans * 16 + align256(ctas * 4);
}

template <typename K>
static cudaError_t expand(const ExpandArgs& e, cudaStream_t stream)
{
    ExpandJob<K> a;
    a.keys = static_cast<const K*>(e.keys);
    a.vals = e.vals;
    a.count = e.count;
    a.cap = e.cap;
    a.gx = e.gx;
    a.gy = e.gy;
    a.quads = quad_cols(e.gx) * quad_cols(e.gy);
    a.spans = expand_spans();
    char* p = reinterpret_cast<char*>(align256(reinterpret_cast<size_t>(e.scratch)));
    const size_t q16 = align256((size_t)a.quads * 16), q4 = align256((size_t)a.quads * 4);
    a.seg.first = reinterpret_cast<uint4*>(p);
    a.seg.last = reinterpret_cast<uint4*>(p + q16);
    a.seg.first_span = reinterpret_cast<int*>(p + 2 * q16);
    a.seg.last_span = reinterpret_cast<int*>(p + 2 * q16 + q4);
    const size_t cleared = 2 * q16 + 2 * q4;  // quads without keys: both ends alike
    a.seg.base = reinterpret_cast<uint32_t*>(p + cleared);
    a.seg.tile = reinterpret_cast<uint32_t*>(p + cleared + q16);
    a.seg.totals = reinterpret_cast<uint4*>(p + cleared + q16 + q4);
    const int tiles = e.gx * e.gy, ctas = div_up(tiles, kTileThreads);
    a.seg.sums = tiles > kDirectTiles ? reinterpret_cast<uint32_t*>(a.seg.totals + kMaxSpans) : nullptr;
    a.out_keys = static_cast<K*>(e.out_keys);
    a.out_vals = e.out_vals;
    a.ranges = e.ranges;
    a.total = e.total;
    cudaError_t err = cudaMemsetAsync(p, 0, cleared, stream);
    if (err != cudaSuccess) return err;
    if ((err = launch_chained(k_quad_starts<K>, a.spans, kExpThreads, 0, stream, a)) != cudaSuccess) return err;
    if (a.seg.sums && (err = launch_chained(k_quad_sums<K>, ctas, kTileThreads, 0, stream, a)) != cudaSuccess) return err;
    err = launch_chained(k_quad_tiles<K>, ctas, kTileThreads, 0, stream, a);
    if (err != cudaSuccess) return err;
    return launch_chained(k_quad_expand<K>, a.spans, kExpThreads, 0, stream, a);
}

cudaError_t launch_quad_expand(const ExpandArgs& e, cudaStream_t stream)
{
    if (e.scratch_bytes < expand_scratch_bytes(e.gx, e.gy) || e.cap >= (1LL << 30)) return cudaErrorInvalidValue;
    return e.key_bytes == 4 ? expand<uint32_t>(e, stream) : expand<uint64_t>(e, stream);
}

}  // namespace gsr

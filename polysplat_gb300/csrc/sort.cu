// Stable LSD radix sort of (key, u32 value) pairs for sm_103a, for 64-bit
// tile|depth keys and for 32-bit keys.
//
// Contract of the 64-bit sort (the reference's CUB call,
// csrc/cuda_rasterizer/sort.cu:107-125): ascending, stable, unsigned, over
// bits [0, end_bit); bits at or above end_bit ride along but do not take part
// in the order; the inputs are preserved.  The count may live on the device,
// so no host synchronisation is needed between the producer and the sort.
//
// Structure (one-sweep radix sort with decoupled look-back):
//   1. k_upsweep: one read of all keys builds the 256-bin histogram of the
//      first 8-bit digit, and clears the first look-back array.
//   2. k_pass (one launch per digit): persistent CTAs take 3584-key tiles in
//      order from an atomic counter, count the tile's digits and publish the
//      counts at once, rank the keys stably within each warp (match.any, lane
//      masks in shared memory, or bit ballots) straight to their places in
//      shared memory, look back over earlier tiles for the running per-digit
//      prefix (bounded, eight predecessors per round trip), and write the tile
//      out with coalesced stores.  While it holds a tile's keys it also counts
//      their next digit, so the next pass's histogram is complete when this
//      launch ends.
//
// Keys are mapped to an "ordering word" before digits are taken (OrderMap):
// the masked key, or -- for keys the preprocess emitted -- the depth bits
// minus the bits of 0.2f, whose width the preprocess recorded in the
// workspace header.  When fewer bits matter than the host planned for, the
// remaining pass launches return at once, and every pass picks its source and
// destination buffer on the device so that the last working pass lands in the
// output.
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>

#include "gsr_internal.h"

namespace gsr {
namespace {

constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagPrefix = 2u << 30;
constexpr uint32_t kValueMask = (1u << 30) - 1u;
constexpr int kWarpsPerCta = kSortThreads / 32;
constexpr int kWarpItems = kSortItems * 32;  // consecutive keys per warp
constexpr int kLook = 8;  // predecessors per look-back round trip

template <typename K>
struct SortJob {
    int num;
    const int32_t* d_num;
    long long cap;
    OrderMap order;
    const K* keys_in;
    const uint32_t* vals_in;
    K* keys_out;
    uint32_t* vals_out;
    SortScratch s;
    uint32_t spin_limit;  // look-back spin bound (sort_wait_limit() at launch)
};

template <typename K>
__device__ __forceinline__ int sort_count(const SortJob<K>& a)
{
    long long n = a.d_num ? (long long)*a.d_num : (long long)a.num;
    if (n < 0) n = 0;
    if (n > a.cap) n = a.cap;
    return (int)n;
}

__host__ __device__ inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// The ordering word of a key and how many of its bits matter.
struct KeyMap {
    int kind;
    int bits;
    int depth_bits;
    uint64_t mask;
    uint32_t tile_mask;
};

__device__ __forceinline__ int depth_width(const WorkspaceHeader* h)
{
    const uint32_t hi = h->depth_hi;
    return hi > kDepthBitsFloor ? bits_for(hi - kDepthBitsFloor) : 0;
}

__device__ __forceinline__ KeyMap key_map(const OrderMap& o, const WorkspaceHeader* h)
{
    KeyMap m;
    m.kind = o.kind;
    m.depth_bits = 0;
    m.tile_mask = 0;
    m.bits = o.end_bit;
    m.mask = o.end_bit >= 64 ? ~0ull : ((1ull << o.end_bit) - 1ull);
    if (o.kind == kOrderDepthCompressed64) {
        m.depth_bits = depth_width(h);
        m.tile_mask = (uint32_t)((1ull << (o.end_bit - 32)) - 1ull);
        m.bits = (o.end_bit - 32) + m.depth_bits;
    } else if (o.kind == kOrderDepth32) {
        m.bits = depth_width(h);
    }
    if (m.bits < 1) m.bits = 1;
    return m;
}

__device__ __forceinline__ uint64_t order_word(uint64_t k, const KeyMap& m)
{
    if (m.kind == kOrderDepthCompressed64) {
        const uint64_t tile = (uint64_t)((uint32_t)(k >> 32) & m.tile_mask);
        return (tile << m.depth_bits) | (uint64_t)((uint32_t)k - kDepthBitsFloor);
    }
    return k & m.mask;
}

__device__ __forceinline__ uint64_t order_word(uint32_t k, const KeyMap& m)
{
    if (m.kind == kOrderDepth32) return (uint64_t)(k - kDepthBitsFloor);
    return (uint64_t)k & m.mask;
}

__device__ __forceinline__ int passes_of(const KeyMap& m) { return (m.bits + 7) / 8; }

// Eight consecutive keys from position b (a multiple of 8): 16-byte loads
// for a full run of a 16-byte aligned buffer, single loads otherwise.
template <typename K>
__device__ __forceinline__ void load8(const K* src, long long b, int cnt, K (&k)[8])
{
    if (cnt == 8 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
        constexpr int kPer = 16 / sizeof(K);
        const uint4* v = reinterpret_cast<const uint4*>(src + b);
#pragma unroll
        for (int q = 0; q < 8 / kPer; q++) {
            const uint4 w = v[q];
            const K* e = reinterpret_cast<const K*>(&w);
#pragma unroll
            for (int j = 0; j < kPer; j++) k[q * kPer + j] = e[j];
        }
        return;
    }
#pragma unroll
    for (int j = 0; j < 8; j++) k[j] = j < cnt ? src[b + j] : K(0);
}

// ---------------------------------------------------------------------------
// Histogram of the first digit pass; every digit pass counts the next one's
// digits from the keys it holds anyway (one read of the keys instead of one
// per pass here: 27 against 44 us at 9.2 M keys).  Each thread takes runs of
// 8 consecutive keys and merges equal consecutive digits before touching
// shared memory: keys of one Gaussian are emitted together and share their
// depth digits, so this removes most same-address shared atomics.
template <typename K>
__global__ __launch_bounds__(256) void k_upsweep(SortJob<K> a)
{
    __shared__ uint32_t s_hist[256];
    s_hist[threadIdx.x] = 0u;
    __syncthreads();
    chain_wait();
    chain_ready();
    const int n = sort_count(a);
    const int tiles = (n + kSortTile - 1) / kSortTile;
    const KeyMap km = key_map(a.order, a.s.hdr);
    // clear the look-back state used by the first digit pass
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (long long)tiles * 256;
         i += (long long)gridDim.x * blockDim.x)
        a.s.look[0][i] = 0u;

    const long long runs = (n + 7) / 8;
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < runs;
         r += (long long)gridDim.x * blockDim.x) {
        const long long b = r * 8;
        K kk[8];
        const int cnt = (int)min(8LL, (long long)n - b);
        load8(a.keys_in, b, cnt, kk);
        uint32_t cur = (uint32_t)order_word(kk[0], km) & 0xFFu;
        uint32_t run = 1;
#pragma unroll
        for (int j = 1; j < 8; j++) {
            if (j >= cnt) break;
            const uint32_t d = (uint32_t)order_word(kk[j], km) & 0xFFu;
            if (d == cur) {
                run++;
            } else {
                atomicAdd(&s_hist[cur], run);
                cur = d;
                run = 1;
            }
        }
        atomicAdd(&s_hist[cur], run);
    }
    __syncthreads();
    if (s_hist[threadIdx.x]) atomicAdd(&a.s.hdr->hist[0][threadIdx.x], s_hist[threadIdx.x]);
}

// ---------------------------------------------------------------------------
template <typename K>
struct PassSmem {
    K keys[kSortTile];
    uint32_t vals[kSortTile];
    uint32_t whist[kWarpsPerCta][256];  // per-warp digit counts, then the warp's next position per digit
    int gofs[256];                      // global position of tile position 0 per digit
    uint32_t next_hist[256];            // this CTA's counts of the next pass's digit
    uint32_t lanes[kWarpsPerCta][256];  // lanes of the warp holding each digit (kRankOr)
    uint32_t warp_sums[kWarpsPerCta];
    int tile;
};

// Shifts that give 0 from 32 on, as PTX's do.
__device__ __forceinline__ uint32_t shl_clamp(uint32_t x, int n)
{
    uint32_t r;
    asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(n));
    return r;
}
__device__ __forceinline__ uint32_t shr_clamp(uint32_t x, int n)
{
    uint32_t r;
    asm("shr.u32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(n));
    return r;
}

// One digit of the ordering word, in 32-bit operations: the word is lo - floor
// in its low db bits and hi above them.
struct Digit {
    int lo_shift, hi_left, hi_right;
    uint32_t mask;
};

__device__ __forceinline__ Digit digit_at(const KeyMap& m, int db, int shift)
{
    Digit d;
    d.lo_shift = shift;
    d.hi_left = max(db - shift, 0);
    d.hi_right = max(shift - db, 0);
    d.mask = (1u << min(8, m.bits - shift)) - 1u;
    return d;
}

__device__ __forceinline__ uint32_t digit_of(uint64_t k, const Digit& d, uint32_t floor)
{
    const uint32_t lo = (uint32_t)k - floor, hi = (uint32_t)(k >> 32);
    return (shr_clamp(lo, d.lo_shift) | shr_clamp(shl_clamp(hi, d.hi_left), d.hi_right)) & d.mask;
}

__device__ __forceinline__ uint32_t digit_of(uint32_t k, const Digit& d, uint32_t floor)
{
    return shr_clamp(k - floor, d.lo_shift) & d.mask;
}

// Exclusive scan over the CTA of one value per thread (thread = digit).  The
// caller has a barrier before the next call.
__device__ __forceinline__ uint32_t digit_scan(uint32_t v, uint32_t* warp_sums, unsigned lane, int warp)
{
    uint32_t incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t n = __shfl_up_sync(GSR_FULL_MASK, incl, d);
        if (lane >= (unsigned)d) incl += n;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    uint32_t pre = incl - v;
#pragma unroll
    for (int w = 0; w < kWarpsPerCta; w++)
        if (w < warp) pre += warp_sums[w];
    return pre;
}

__device__ __forceinline__ unsigned lanemask_gt()
{
    unsigned m;
    asm("mov.u32 %0, %%lanemask_gt;" : "=r"(m));
    return m;
}

// What every tile of a pass shares.
template <typename K>
struct PassCtx {
    const K* kin;
    const uint32_t* vin;
    K* kout;
    uint32_t* vout;
    uint32_t* look;
    uint32_t* look_next;
    WorkspaceHeader* hdr;
    uint32_t* counter;  // next tile to claim
    Digit dg, dn;  // this pass's digit and the next one's
    uint32_t floor;
    uint32_t spin_limit;
    int n;
    bool more;  // a pass follows
};

// The digit by where it lies in the key: DLo within the low word, DHi within
// the high word, DMix across both.
enum : int { kDLo = 0, kDHi = 1, kDMix = 2 };

template <int WHERE>
__device__ __forceinline__ uint32_t digit_in(uint64_t k, const Digit& d, uint32_t floor)
{
    if (WHERE == kDLo) return ((uint32_t)k - floor) >> d.lo_shift & d.mask;
    if (WHERE == kDHi) return (uint32_t)(k >> 32) >> d.hi_right & d.mask;
    return digit_of(k, d, floor);
}
template <int WHERE>
__device__ __forceinline__ uint32_t digit_in(uint32_t k, const Digit& d, uint32_t floor)
{
    return digit_of(k, d, floor);
}

// How a warp finds the lanes with its digit.
enum : int { kRankBallot = 0, kRankMatch = 1, kRankOr = 2 };

// Sum of the counts of digit `tid` over the tiles before `tile`: walk back
// kLook predecessors per round trip; stop at the first inclusive prefix,
// re-reading any entry that is not published yet.  Whole windows of published
// counts, the usual case, are summed without looking at single entries.
template <typename K>
__device__ __forceinline__ uint32_t look_back(const PassCtx<K>& c, int tile, int tid)
{
    uint32_t excl = 0, spins = 0;
    int j = tile - 1;
    const uint32_t* at = c.look + (size_t)max(j, 0) * 256 + tid;
    while (j >= 0) {
        uint32_t v[kLook];
        uint32_t sum = 0, any = 0, all = 0xFFFFFFFFu;
        if (j >= kLook - 1) {
#pragma unroll
            for (int k = 0; k < kLook; k++) v[k] = ld_relaxed_u32(at - k * 256);
        } else {
#pragma unroll
            for (int k = 0; k < kLook; k++) v[k] = j - k >= 0 ? ld_relaxed_u32(at - k * 256) : kFlagPrefix;
        }
#pragma unroll
        for (int k = 0; k < kLook; k++) {
            sum += v[k];
            any |= v[k];
            all &= v[k];
        }
        if ((all & kFlagAgg) && !(any & kFlagPrefix)) {
            excl += sum;  // the flags wrap past bit 29 and are masked off below
            j -= kLook;
            at -= kLook * 256;
            continue;
        }
        bool stuck = false, done = false;
#pragma unroll
        for (int k = 0; k < kLook; k++) {
            const bool live = !done && !stuck;
            const bool pub = (v[k] & ~kValueMask) != 0u;
            stuck = stuck || (live && !pub);
            if (live && pub) {
                excl += v[k];
                j--;
                done = (v[k] & kFlagPrefix) != 0u;
            }
        }
        if (done) break;
        at = c.look + (size_t)max(j, 0) * 256 + tid;
        if (stuck && ++spins > c.spin_limit) {
            record_error(&c.hdr->status, kErrTimeout);
            break;
        }
    }
    return excl & kValueMask;
}

template <bool FULL, int RANK, int WHERE, typename K>
__device__ __forceinline__ void pass_tile(PassSmem<K>& S, const PassCtx<K>& c, int tile, int gstart, unsigned lane,
                                          int warp, int tid)
{
    const long long tbase = (long long)tile * kSortTile;
    const int tcount = FULL ? kSortTile : (int)((long long)c.n - tbase);
    const int first = warp * kWarpItems + (int)lane;
    uint32_t* wh = S.whist[warp];

    // ---- load the warp's chunk, count its digits ----
    K key[kSortItems];
    uint32_t val[kSortItems];
    {
        const K* kp = c.kin + tbase + first;
        const uint32_t* vp = c.vin + tbase + first;
#pragma unroll
        for (int i = 0; i < kSortItems; i++) key[i] = FULL || first + i * 32 < tcount ? kp[i * 32] : K(0);
#pragma unroll
        for (int i = 0; i < kSortItems; i++) val[i] = FULL || first + i * 32 < tcount ? vp[i * 32] : 0u;
    }
    if (c.more) c.look_next[(size_t)tile * 256 + tid] = 0u;
#pragma unroll
    for (int i = 0; i < kSortItems; i++)
        if (FULL || first + i * 32 < tcount) atomicAdd(&wh[digit_in<WHERE>(key[i], c.dg, c.floor)], 1u);
    if (c.more) {
#pragma unroll
        for (int i = 0; i < kSortItems; i++)
            if (FULL || first + i * 32 < tcount) atomicAdd(&S.next_hist[digit_of(key[i], c.dn, c.floor)], 1u);
    }
    __syncthreads();

    // ---- thread d: the tile's count of digit d, published before anything
    //      else so that later tiles can look back over it; then the first
    //      position of the digit in every warp ----
    uint32_t dtot = 0, cw[kWarpsPerCta];
    uint32_t* my = c.look + (size_t)tile * 256 + tid;
#pragma unroll
    for (int w = 0; w < kWarpsPerCta; w++) {
        cw[w] = S.whist[w][tid];
        dtot += cw[w];
    }
    st_relaxed_u32(my, (tile == 0 ? kFlagPrefix : kFlagAgg) | dtot);
    const uint32_t dstart = digit_scan(dtot, S.warp_sums, lane, warp);
    {
        uint32_t run = dstart;
#pragma unroll
        for (int w = 0; w < kWarpsPerCta; w++) {
            S.whist[w][tid] = run;
            run += cw[w];
        }
    }
    __syncthreads();

    // ---- stable ranks: wh[d] is the warp's next position of digit d in the
    //      tile's digit order; keys and values go straight to their places ----
    {
        const unsigned lt = lanemask_lt(), gt = lanemask_gt();
#pragma unroll
        for (int i = 0; i < kSortItems; i++) {
            const bool ok = FULL || first + i * 32 < tcount;
            const uint32_t d = digit_in<WHERE>(key[i], c.dg, c.floor);
            unsigned peers;
            if (RANK == kRankMatch) {
                peers = __match_any_sync(GSR_FULL_MASK, ok ? d : 0x100u);
            } else if (RANK == kRankOr) {
                uint32_t* m = S.lanes[warp];
                if (ok) atomicOr(&m[d], 1u << lane);
                __syncwarp();
                peers = ok ? m[d] : 0u;
            } else {
                peers = FULL ? GSR_FULL_MASK : __ballot_sync(GSR_FULL_MASK, ok);
#pragma unroll
                for (int b = 0; b < 8; b++) {
                    const bool bit = (d >> b) & 1u;
                    const unsigned bb = __ballot_sync(GSR_FULL_MASK, bit);
                    peers &= bit ? bb : ~bb;
                }
            }
            uint32_t pos = 0;
            if (ok) pos = wh[d] + __popc(peers & lt);
            __syncwarp();
            if (ok && (peers & gt) == 0u) {
                wh[d] = pos + 1u;
                if (RANK == kRankOr) S.lanes[warp][d] = 0u;
            }
            __syncwarp();
            if (ok) {
                S.keys[pos] = key[i];
                S.vals[pos] = val[i];
            }
        }
    }

    // ---- decoupled look-back: thread d owns digit d ----
    {
        const uint32_t excl = look_back(c, tile, tid);
        if (tile != 0) st_relaxed_u32(my, kFlagPrefix | ((excl + dtot) & kValueMask));
        S.gofs[tid] = gstart + (int)excl - (int)dstart;
    }
    __syncthreads();

    // ---- coalesced scatter of the digit runs; the claim of the next tile
    //      travels meanwhile ----
    if (tid == 0) S.tile = (int)atomicAdd(c.counter, 1u);
    bool oob = false;
#pragma unroll
    for (int i = 0; i < kSortItems; i++) {
        const int p = tid + i * kSortThreads;
        if (FULL || p < tcount) {
            const K k = S.keys[p];
            const uint32_t v = S.vals[p];
            const int g = S.gofs[digit_in<WHERE>(k, c.dg, c.floor)] + p;
            if ((unsigned)g < (unsigned)c.n) {
                c.kout[g] = k;
                c.vout[g] = v;
            } else {  // only after a look-back timeout: never write outside the buffer
                oob = true;
            }
        }
    }
    if (oob) record_error(&c.hdr->status, kErrTimeout);
}

template <int RANK, int WHERE, typename K>
__device__ __forceinline__ void pass_tiles(PassSmem<K>& S, const PassCtx<K>& c, int gstart, unsigned lane,
                                           int warp, int tid)
{
    const int tiles = (c.n + kSortTile - 1) / kSortTile;
    for (;;) {
        const int tile = S.tile;
        if (tile >= tiles) break;
        if ((long long)(tile + 1) * kSortTile <= (long long)c.n)
            pass_tile<true, RANK, WHERE>(S, c, tile, gstart, lane, warp, tid);
        else pass_tile<false, RANK, WHERE>(S, c, tile, gstart, lane, warp, tid);
#pragma unroll
        for (int k = 0; k < 8; k++) S.whist[warp][k * 32 + lane] = 0u;
        __syncthreads();
    }
}

// One digit pass.  Per 32 keys it issues about 85 warp instructions and 35 to
// 50 shared-memory wavefronts (ranking, the reorder and its bank conflicts);
// the shared-memory pipe (60-70% busy) and the latency of a tile's chain bound
// it, not DRAM: 60-65 us at 9.2 M 64-bit pairs (3.4-3.7 TB/s of the 24 bytes a
// pair), where a form with the counts published after the ranking, digits
// from 64-bit shifts and every access predicated took 78-102 us at 180-250
// instructions.
//
// RANK 2 picks the ranking per pass: match.any for depth digits, which a
// Gaussian's adjacent keys share (its time grows with the number of distinct
// digits among the lanes), lane masks in shared memory for digits holding
// tile ids (all passes of a 13-bit sort of 9.2 M 32-bit pairs: 126 us against
// 150 with ballots).  RANK 0 / 1 force ballots / match.any.
template <typename K, int RANK>
__global__ __launch_bounds__(kSortThreads, kSortCtas) void k_pass(SortJob<K> a, int pass)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PassSmem<K>& S = *reinterpret_cast<PassSmem<K>*>(smem_raw);
    static_assert(kSortThreads == 256, "thread d owns digit d");
    const unsigned lane = threadIdx.x & 31u;
    const int warp = threadIdx.x >> 5, tid = threadIdx.x;
    chain_wait();
    chain_ready();
    const KeyMap km = key_map(a.order, a.s.hdr);
    const int passes = passes_of(km);
    if (pass >= passes) return;  // nothing left to order in this digit
    const int shift = 8 * pass;
    const int bits = min(8, km.bits - shift);
    const int tile_from = a.order.kind == kOrderDepthCompressed64 ? km.depth_bits : a.order.tile_from_bit;
    const bool depth_digit = shift + bits <= tile_from;
    const int db = a.order.kind == kOrderDepthCompressed64 ? km.depth_bits : 32;
    PassCtx<K> c;
    c.n = sort_count(a);
    c.floor = a.order.kind == kOrderMasked ? 0u : kDepthBitsFloor;
    c.dg = digit_at(km, db, shift);
    // ping-pong so that the last working pass writes the output buffers
    const bool to_out = ((passes - 1 - pass) & 1) == 0;
    K* alt_k = reinterpret_cast<K*>(a.s.alt_keys);
    c.kin = a.keys_in;
    c.vin = a.vals_in;
    if (pass > 0) {
        const bool prev_out = ((passes - pass) & 1) == 0;
        c.kin = prev_out ? a.keys_out : alt_k;
        c.vin = prev_out ? a.vals_out : a.s.alt_vals;
    }
    c.kout = to_out ? a.keys_out : alt_k;
    c.vout = to_out ? a.vals_out : a.s.alt_vals;
    // selects rather than a dynamic index, so the parameter block stays out of local memory
    c.look = (pass & 1) ? a.s.look[1] : a.s.look[0];
    c.look_next = (pass & 1) ? a.s.look[0] : a.s.look[1];
    c.hdr = a.s.hdr;
    c.spin_limit = a.spin_limit;
    // the next pass's histogram is counted here, from the keys this pass holds
    c.more = pass + 1 < passes;
    c.dn = digit_at(km, db, c.more ? shift + 8 : shift);
    c.counter = &a.s.hdr->pass_counter[pass];

    S.next_hist[tid] = 0u;
    if (tid == 0) S.tile = (int)atomicAdd(c.counter, 1u);
#pragma unroll
    for (int k = 0; k < 8; k++) {
        S.whist[warp][k * 32 + lane] = 0u;
        S.lanes[warp][k * 32 + lane] = 0u;
    }
    // global start of digit tid
    const int gstart = (int)digit_scan(a.s.hdr->hist[pass][tid], S.warp_sums, lane, warp);
    __syncthreads();

    const int where = sizeof(K) == 4 || shift + bits <= db ? kDLo : shift >= db ? kDHi : kDMix;
    if (RANK == 1) {
        pass_tiles<kRankMatch, kDMix>(S, c, gstart, lane, warp, tid);
    } else if (RANK == 0) {
        pass_tiles<kRankBallot, kDMix>(S, c, gstart, lane, warp, tid);
    } else if (depth_digit) {
        pass_tiles<kRankMatch, kDLo>(S, c, gstart, lane, warp, tid);
    } else if (where == kDHi) {
        pass_tiles<kRankOr, kDHi>(S, c, gstart, lane, warp, tid);
    } else {
        pass_tiles<kRankOr, kDMix>(S, c, gstart, lane, warp, tid);
    }
    // every count of this CTA precedes the barrier that ended its last tile
    if (c.more && S.next_hist[tid]) atomicAdd(&a.s.hdr->hist[pass + 1][tid], S.next_hist[tid]);
}

// 2 (choose per sort and pass) unless GSR_SORT_RANK asks for "ballot" (0) or
// "match" (1) everywhere
int sort_rank_mode()
{
    static const int mode = [] {  // read once, thread-safe initialisation
        const char* e = getenv("GSR_SORT_RANK");
        return (e && strcmp(e, "ballot") == 0) ? 0 : (e && strcmp(e, "match") == 0) ? 1 : 2;
    }();
    return mode;
}

template <typename K>
cudaError_t run_sort(const SortJob<K>& job, int max_passes, cudaStream_t stream)
{
    if (job.cap >= (1LL << 30) || max_passes < 1 || max_passes > kMaxPasses) return cudaErrorInvalidValue;
    SortJob<K> a = job;
    a.spin_limit = sort_wait_limit();
    // clear the sort region of the header (pass counters and histograms)
    cudaError_t e = cudaSuccess;
    if (!a.s.header_clear)
        e = cudaMemsetAsync(reinterpret_cast<char*>(a.s.hdr) + kSortRegionOffset, 0,
                            sizeof(WorkspaceHeader) - kSortRegionOffset, stream);
    if (e != cudaSuccess) return e;
    // failure-detection hook: the first pass starts at tile 1, so tile 0 never
    // publishes and the look-back of the tiles after it runs out
    if (sort_stall_first_tile() && (e = cudaMemsetAsync(&a.s.hdr->pass_counter[0], 1, 1, stream)) != cudaSuccess)
        return e;
    const int sms = device_sm_count();
    int up_grid = (int)std::min<long long>((long long)sms * 4, std::max<long long>(1, (a.cap + 2047) / 2048));
    if ((e = launch_chained(k_upsweep<K>, up_grid, 256, 0, stream, a)) != cudaSuccess) return e;
    profile_mark(stream);

    const int mode = sort_rank_mode();
    auto kern = mode == 0 ? k_pass<K, 0> : mode == 1 ? k_pass<K, 1> : k_pass<K, 2>;
    // per device and ranking mode: the shared-memory attribute (a property of
    // the kernel on each device), then the occupancy; host threads may race
    // to fill these with the same values
    static std::atomic<int> per_sm_cache[kMaxDevices][3];
    const int dev = current_device();
    if (dev < 0) return cudaErrorInvalidDevice;
    const int smem = (int)sizeof(PassSmem<K>);
    int per_sm = per_sm_cache[dev][mode].load(std::memory_order_acquire);
    if (per_sm == 0) {
        if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess)
            return e;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kSortThreads, smem) != cudaSuccess ||
            per_sm < 1)
            per_sm = 1;
        per_sm_cache[dev][mode].store(per_sm, std::memory_order_release);
    }
    const int grid = (int)std::min<long long>((long long)sms * per_sm, std::max<long long>(1, a.s.tiles_cap));
    for (int p = 0; p < max_passes; p++) {
        if ((e = launch_chained(kern, grid, kSortThreads, smem, stream, a, p)) != cudaSuccess) return e;
        profile_mark(stream);
    }
    return cudaSuccess;
}

}  // namespace

// ---------------------------------------------------------------------------
// Workspace layout: [header+queue][alt keys 8*cap][alt vals 4*cap][look-back x2][tile ranges]

static size_t sort_area_bytes(long long cap)
{
    if (cap < 1) cap = 1;
    long long tiles = (cap + kSortTile - 1) / kSortTile;
    return kSmallWorkspaceBytes + align256((size_t)cap * 8) + align256((size_t)cap * 4) +
           2 * align256((size_t)tiles * 256 * 4);
}

size_t sort_workspace_bytes(long long cap) { return sort_area_bytes(cap) + (size_t)kWorkspaceRangeTiles * 8; }

int2* workspace_ranges(void* ws, long long cap)
{
    return reinterpret_cast<int2*>(reinterpret_cast<char*>(ws) + sort_area_bytes(cap));
}

SortScratch workspace_sort_scratch(void* ws, long long cap)
{
    SortScratch s;
    char* p = reinterpret_cast<char*>(ws);
    s.hdr = reinterpret_cast<WorkspaceHeader*>(p);
    size_t off = kSmallWorkspaceBytes;
    s.alt_keys = p + off;
    off += align256((size_t)(cap < 1 ? 1 : cap) * 8);
    s.alt_vals = reinterpret_cast<uint32_t*>(p + off);
    off += align256((size_t)(cap < 1 ? 1 : cap) * 4);
    s.tiles_cap = ((cap < 1 ? 1 : cap) + kSortTile - 1) / kSortTile;
    s.look[0] = reinterpret_cast<uint32_t*>(p + off);
    off += align256((size_t)s.tiles_cap * 256 * 4);
    s.look[1] = reinterpret_cast<uint32_t*>(p + off);
    return s;
}

size_t sort_scratch_bytes(long long cap, int key_bytes)
{
    if (cap < 1) cap = 1;
    long long tiles = (cap + kSortTile - 1) / kSortTile;
    return align256((size_t)cap * key_bytes) + align256((size_t)cap * 4) + 2 * align256((size_t)tiles * 256 * 4);
}

SortScratch carve_sort_scratch(WorkspaceHeader* hdr, void* mem, long long cap, int key_bytes)
{
    SortScratch s;
    char* p = reinterpret_cast<char*>(mem);
    s.hdr = hdr;
    if (cap < 1) cap = 1;
    s.alt_keys = p;
    size_t off = align256((size_t)cap * key_bytes);
    s.alt_vals = reinterpret_cast<uint32_t*>(p + off);
    off += align256((size_t)cap * 4);
    s.tiles_cap = (cap + kSortTile - 1) / kSortTile;
    s.look[0] = reinterpret_cast<uint32_t*>(p + off);
    off += align256((size_t)s.tiles_cap * 256 * 4);
    s.look[1] = reinterpret_cast<uint32_t*>(p + off);
    return s;
}

cudaError_t launch_sort(const SortArgs& a, cudaStream_t stream)
{
    if (a.end_bit < 1 || a.end_bit > 64) return cudaErrorInvalidValue;
    if (a.ws_bytes < sort_area_bytes(a.cap)) return cudaErrorInvalidValue;
    SortJob<uint64_t> j;
    j.num = a.num;
    j.d_num = a.d_num;
    j.cap = a.cap;
    j.order.kind = a.compress_depth && a.end_bit > 32 ? kOrderDepthCompressed64 : kOrderMasked;
    j.order.end_bit = a.end_bit;
    j.order.tile_from_bit = 32;  // tile << 32 | depth bits
    j.keys_in = a.keys_in;
    j.vals_in = a.vals_in;
    j.keys_out = a.keys_out;
    j.vals_out = a.vals_out;
    j.s = workspace_sort_scratch(a.ws, a.cap);
    j.s.header_clear = a.header_clear;
    j.spin_limit = kSpinLimit;
    return run_sort(j, (a.end_bit + 7) / 8, stream);
}

cudaError_t launch_sort32(int num, const int32_t* d_num, long long cap, OrderMap order, int max_passes,
                          const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out, uint32_t* vals_out,
                          const SortScratch& s, cudaStream_t stream)
{
    SortJob<uint32_t> j;
    j.num = num;
    j.d_num = d_num;
    j.cap = cap;
    j.order = order;
    j.keys_in = keys_in;
    j.vals_in = vals_in;
    j.keys_out = keys_out;
    j.vals_out = vals_out;
    j.s = s;
    j.spin_limit = kSpinLimit;
    return run_sort(j, max_passes, stream);
}

cudaError_t launch_sort64(int num, const int32_t* d_num, long long cap, OrderMap order, int max_passes,
                          const uint64_t* keys_in, const uint32_t* vals_in, uint64_t* keys_out, uint32_t* vals_out,
                          const SortScratch& s, cudaStream_t stream)
{
    SortJob<uint64_t> j;
    j.num = num;
    j.d_num = d_num;
    j.cap = cap;
    j.order = order;
    j.keys_in = keys_in;
    j.vals_in = vals_in;
    j.keys_out = keys_out;
    j.vals_out = vals_out;
    j.s = s;
    j.spin_limit = kSpinLimit;
    return run_sort(j, max_passes, stream);
}

}  // namespace gsr

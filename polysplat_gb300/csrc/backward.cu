// Differentiable forward and backward of the rasterizer (no counterpart in
// the reference, which renders only): the C ABI entries and the preprocess
// adjoint kernel.  The per-Gaussian adjoint is adjoint.h (checked in double
// against central differences); the render backward is in render.cu.
#include <algorithm>
#include <vector>

#include "adjoint.h"
#include "gsr_internal.h"

namespace gsr {
namespace {

// Views of one adjoint launch (more views take several launches, the later
// ones accumulating).
constexpr int kAdjViews = 16;
constexpr int kAdjThreads = 128;

struct PreBackArgs {
    int P, n_views;
    const float* means;
    const float* log_scales;
    const float* quats;
    const float* logits;
    const float* shs;  // [P,48] f32
    gsr_adj::Cam<float> cam[kAdjViews];
    // per-view gradient records of the screen-space features (conic and
    // opacity, xy, colour; 12 floats): view v's rows start at v * P (of the
    // launch's first view)
    const float4* grec;
    // or one view's gradients in three arrays
    const float* gxy;
    const float* gcon;
    const float* grgb;
    float* g_means;
    float* g_log_scales;
    float* g_quats;
    float* g_logits;
    float* g_shs;
    int accumulate;
};

// Gradients of Gaussian i's features in view v; false when all are zero (it
// reached no pixel of the view).
template <bool RECORDS>
__device__ __forceinline__ bool feature_grads(const PreBackArgs& a, int i, int v, float (&gxy)[2], float (&gcon)[4],
                                              float (&grgb)[3])
{
    if (RECORDS) {
        const size_t r = 3 * ((size_t)v * a.P + i);
        const float4 q0 = __ldg(a.grec + r), q1 = __ldg(a.grec + r + 1);
        const float blue = __ldg(reinterpret_cast<const float*>(a.grec + r + 2));
        gcon[0] = q0.x;
        gcon[1] = q0.y;
        gcon[2] = q0.z;
        gcon[3] = q0.w;
        gxy[0] = q1.x;
        gxy[1] = q1.y;
        grgb[0] = q1.z;
        grgb[1] = q1.w;
        grgb[2] = blue;
    } else {
        for (int k = 0; k < 4; k++) gcon[k] = __ldg(a.gcon + 4 * (size_t)i + k);
        for (int k = 0; k < 2; k++) gxy[k] = __ldg(a.gxy + 2 * (size_t)i + k);
        for (int k = 0; k < 3; k++) grgb[k] = __ldg(a.grgb + 3 * (size_t)i + k);
    }
    return gcon[0] != 0.f || gcon[1] != 0.f || gcon[2] != 0.f || gcon[3] != 0.f || gxy[0] != 0.f || gxy[1] != 0.f ||
           grgb[0] != 0.f || grgb[1] != 0.f || grgb[2] != 0.f;
}

// A CTA takes 128 Gaussians.  A view sees few of them (saturated tiles stop
// before most), so a thread per Gaussian that walks its views left 27 of 32
// lanes idle (603 us for 1 M Gaussians and 8 views).  Instead the CTA lists its
// (Gaussian, view) pairs with a gradient, and takes them a pair to a thread: the
// forward replayed and its adjoint, without the SH gradients, which are the
// product of 16 basis values and 3 colour gradients and are formed when each
// Gaussian's thread sums its pairs, in view order, and writes its 59
// gradients.  Rounds take up to 128 pairs and whole Gaussians.
template <bool RECORDS>
__global__ __launch_bounds__(kAdjThreads) void k_preprocess_backward(const __grid_constant__ PreBackArgs a)
{
    constexpr int kOut = 15;  // 11 gradients, 3 of the colour, and a stride without bank conflicts
    __shared__ uint16_t s_pair[kAdjThreads * kAdjViews];  // Gaussian | view << 8
    __shared__ float s_out[kAdjThreads][kOut];
    __shared__ int s_warp[kAdjThreads / 32];
    __shared__ int s_end;
    const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int i0 = (int)blockIdx.x * kAdjThreads, i = i0 + tid;
    // SH rows are 192 bytes: 16-byte accesses when both arrays start on 16 bytes
    const bool wide = ((reinterpret_cast<uintptr_t>(a.shs) | reinterpret_cast<uintptr_t>(a.g_shs)) & 15u) == 0;

    // ---- list the pairs ----
    uint32_t seen = 0u;
    if (i < a.P)
        for (int v = 0; v < a.n_views; v++) {
            float gxy[2], gcon[4], grgb[3];
            if (feature_grads<RECORDS>(a, i, v, gxy, gcon, grgb)) seen |= 1u << v;
        }
    const int n = __popc(seen);
    int incl = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(GSR_FULL_MASK, incl, d);
        if (lane >= d) incl += t;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    int first = incl - n, total = 0;
#pragma unroll
    for (int w = 0; w < kAdjThreads / 32; w++) {
        if (w < warp) first += s_warp[w];
        total += s_warp[w];
    }
    {
        int k = first;
        for (uint32_t m = seen; m; m &= m - 1) s_pair[k++] = (uint16_t)(tid | ((__ffs(m) - 1) << 8));
    }
    if (n == 0 && i < a.P && !a.accumulate) {  // never seen: zeros
        for (int k = 0; k < 3; k++) a.g_means[3 * (size_t)i + k] = a.g_log_scales[3 * (size_t)i + k] = 0.f;
        for (int k = 0; k < 4; k++) a.g_quats[4 * (size_t)i + k] = 0.f;
        a.g_logits[i] = 0.f;
        if (wide) {
            for (int k = 0; k < 12; k++)
                reinterpret_cast<float4*>(a.g_shs + 48 * (size_t)i)[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
            for (int k = 0; k < 48; k++) a.g_shs[48 * (size_t)i + k] = 0.f;
        }
    }

    for (int begin = 0; begin < total;) {
        // the round: the Gaussians whose pairs end within 128 of `begin`
        __syncthreads();  // s_pair is complete, s_out and s_end of the last round have been read
        if (tid == 0) s_end = begin;
        __syncthreads();
        const bool mine = n > 0 && first >= begin && first + n <= begin + kAdjThreads;
        if (mine) atomicMax(&s_end, first + n);
        __syncthreads();
        const int end = s_end;

        // ---- a pair to a thread ----
        if (begin + tid < end) {
            const int pr = s_pair[begin + tid], v = pr >> 8;
            const size_t j = (size_t)i0 + (pr & 0xFF);
            float gxy[2], gcon[4], grgb[3];
            feature_grads<RECORDS>(a, (int)j, v, gxy, gcon, grgb);
            float m[3], ls[3], q[4], gm[3], gls[3], gq[4], glogit, g[3];
            for (int k = 0; k < 3; k++) {
                m[k] = __ldg(a.means + 3 * j + k);
                ls[k] = __ldg(a.log_scales + 3 * j + k);
            }
            for (int k = 0; k < 4; k++) q[k] = __ldg(a.quats + 4 * j + k);
            gsr_adj::Fwd<float> f;
            gsr_adj::Tape<float> tp;
            gsr_adj::forward<float, false>(m, ls, q, __ldg(a.logits + j), nullptr, a.cam[v], f, tp);
            gsr_adj::backward<float, false>(m, nullptr, a.cam[v], tp, gxy, gcon, grgb, gm, gls, gq, glogit, nullptr);
            float sh[48];
            const float* row = a.shs + 48 * j;
            if (wide) {
#pragma unroll
                for (int k = 0; k < 12; k++) {
                    const float4 r = __ldg(reinterpret_cast<const float4*>(row) + k);
                    sh[4 * k] = r.x;
                    sh[4 * k + 1] = r.y;
                    sh[4 * k + 2] = r.z;
                    sh[4 * k + 3] = r.w;
                }
            } else {
#pragma unroll
                for (int k = 0; k < 48; k++) sh[k] = __ldg(row + k);
            }
            gsr_adj::color_adjoint(m, a.cam[v].campos, sh, grgb, gm, g);
            float* o = s_out[tid];
            for (int k = 0; k < 3; k++) {
                o[k] = gm[k];
                o[3 + k] = gls[k];
                o[11 + k] = g[k];
            }
            for (int k = 0; k < 4; k++) o[6 + k] = gq[k];
            o[10] = glogit;
        }
        __syncthreads();

        // ---- each Gaussian's sum over its views ----
        if (mine) {
            float sum[11], sh[48], m[3];
            for (int k = 0; k < 11; k++) sum[k] = 0.f;
            for (int k = 0; k < 48; k++) sh[k] = 0.f;
            for (int k = 0; k < 3; k++) m[k] = __ldg(a.means + 3 * (size_t)i + k);
            for (int k = first; k < first + n; k++) {
                const float* o = s_out[k - begin];
                for (int c = 0; c < 11; c++) sum[c] += o[c];
                gsr_adj::add_sh_gradient(m, a.cam[s_pair[k] >> 8].campos, o + 11, sh);
            }
            auto put = [&](float* dst, size_t off, float v) { dst[off] = a.accumulate ? dst[off] + v : v; };
            for (int k = 0; k < 3; k++) {
                put(a.g_means, 3 * (size_t)i + k, sum[k]);
                put(a.g_log_scales, 3 * (size_t)i + k, sum[3 + k]);
            }
            for (int k = 0; k < 4; k++) put(a.g_quats, 4 * (size_t)i + k, sum[6 + k]);
            put(a.g_logits, i, sum[10]);
            if (wide && !a.accumulate) {
                float4* row = reinterpret_cast<float4*>(a.g_shs + 48 * (size_t)i);
#pragma unroll
                for (int k = 0; k < 12; k++)
                    row[k] = make_float4(sh[4 * k], sh[4 * k + 1], sh[4 * k + 2], sh[4 * k + 3]);
            } else {
                for (int k = 0; k < 48; k++) put(a.g_shs, 48 * (size_t)i + k, sh[k]);
            }
        }
        begin = end;
    }
}

gsr_adj::Cam<float> adj_camera(int W, int H, const float* cam_pos, const float* cam_rot, float fx, float fy,
                               float zfar, float znear)
{
    gsr_adj::Cam<float> c;
    camera_matrices(W, H, cam_pos, cam_rot, fx, fy, zfar, znear, c.view, c.proj);
    for (int k = 0; k < 3; k++) c.campos[k] = cam_pos[k];
    c.fx = fx;
    c.fy = fy;
    c.tanx = W / (2.0f * fx);
    c.tany = H / (2.0f * fy);
    c.W = W;
    c.H = H;
    return c;
}

}  // namespace
}  // namespace gsr

using namespace gsr;

extern "C" {

gsr_status gsr_train_forward(int P, const float* means, const float* log_scales, const float* quats,
                             const float* logits, const float* shs, int width, int height, const float* cam_pos,
                             const float* cam_rot, float focal_x, float focal_y, float z_far, float z_near,
                             const float* bg_color, float* opacity, float* cov3d, int32_t* curr_offset,
                             void* workspace, size_t workspace_bytes, uint64_t* keys_unsorted,
                             uint32_t* values_unsorted, uint64_t* keys_sorted, uint32_t* values_sorted,
                             int64_t key_capacity, float* points_xy, float* rgb_depth, float* conic_opacity,
                             int32_t* ranges, int32_t* n_tile, float* T_final, float* image, gsr_stream_t stream)
{
    cudaStream_t s = (cudaStream_t)stream;
    if (P < 0 || width <= 0 || height <= 0 || !cam_pos || !cam_rot || !bg_color || !curr_offset || !workspace ||
        !ranges || !n_tile || !T_final || !image || !opacity || !cov3d)
        return GSR_INVALID_ARG;
    if (P > 0 && (!means || !log_scales || !quats || !logits || !shs)) return GSR_INVALID_ARG;
    if (workspace_bytes < sort_workspace_bytes(key_capacity) || key_capacity >= (1LL << 30)) return GSR_INVALID_ARG;
    const int tiles = div_up(width, 16) * div_up(height, 16);
    cudaError_t e = launch_scene_prepare(P, log_scales, quats, logits, opacity, cov3d, s);
    if (e == cudaSuccess) e = clear_header(workspace, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(curr_offset, 0, sizeof(int32_t), s);
    if (e != cudaSuccess) return GSR_CUDA_ERROR;
    PreprocessParams p;
    gsr_status st = preprocess_params(p, P, means, shs, opacity, cov3d, width, height, 16, 16, cam_pos, cam_rot, focal_x,
                                      focal_y, z_far, z_near, points_xy, rgb_depth, conic_opacity, keys_unsorted,
                                      values_unsorted, key_capacity, curr_offset, workspace, workspace_bytes);
    if (st != GSR_OK) return st;
    p.header_clear = 1;
    if (launch_preprocess(p, false, s) != cudaSuccess) return GSR_CUDA_ERROR;
    SortArgs sa;
    sa.num = 0;
    sa.d_num = curr_offset;
    sa.cap = key_capacity;
    sa.end_bit = 32 + bits_for((uint32_t)tiles);
    sa.compress_depth = true;
    sa.keys_in = keys_unsorted;
    sa.vals_in = values_unsorted;
    sa.keys_out = keys_sorted;
    sa.vals_out = values_sorted;
    sa.ws = workspace;
    sa.ws_bytes = workspace_bytes;
    sa.header_clear = true;
    if ((e = launch_sort(sa, s)) != cudaSuccess) return GSR_CUDA_ERROR;
    if ((e = launch_tile_ranges(0, curr_offset, key_capacity, tiles, keys_sorted, ranges, false, s)) != cudaSuccess)
        return GSR_CUDA_ERROR;
    TrainRenderArgs ra = {};
    ra.W = width;
    ra.H = height;
    ra.P = P;
    ra.d_num = curr_offset;
    ra.cap = key_capacity;
    ra.vals = values_sorted;
    ra.ranges = reinterpret_cast<const int2*>(ranges);
    ra.xy = reinterpret_cast<const float2*>(points_xy);
    ra.rgbd = reinterpret_cast<const float4*>(rgb_depth);
    ra.con = reinterpret_cast<const float4*>(conic_opacity);
    for (int k = 0; k < 3; k++) ra.bg[k] = bg_color[k];
    ra.image = image;
    ra.T_final = T_final;
    ra.n_tile = n_tile;
    e = launch_render_train(ra, false, s);
    return e == cudaSuccess ? GSR_OK : GSR_CUDA_ERROR;
}

gsr_status gsr_train_backward(int P, const float* means, const float* log_scales, const float* quats,
                              const float* logits, const float* shs, int width, int height, const float* cam_pos,
                              const float* cam_rot, float focal_x, float focal_y, float z_far, float z_near,
                              const float* bg_color, const int32_t* curr_offset, int64_t key_capacity,
                              const uint32_t* values_sorted, const int32_t* ranges, const int32_t* n_tile,
                              const float* T_final, const float* points_xy, const float* rgb_depth,
                              const float* conic_opacity, const float* grad_image, float* grad_xy, float* grad_con,
                              float* grad_rgb, float* g_means, float* g_log_scales, float* g_quats, float* g_logits,
                              float* g_shs, int accumulate, gsr_stream_t stream)
{
    cudaStream_t s = (cudaStream_t)stream;
    if (P < 0 || width <= 0 || height <= 0 || !cam_pos || !cam_rot || !bg_color || !curr_offset || !ranges ||
        !n_tile || !T_final || !grad_image || !grad_xy || !grad_con || !grad_rgb)
        return GSR_INVALID_ARG;
    if (P == 0) return GSR_OK;
    if (!means || !log_scales || !quats || !logits || !shs || !g_means || !g_log_scales || !g_quats || !g_logits ||
        !g_shs)
        return GSR_INVALID_ARG;
    cudaError_t e = cudaMemsetAsync(grad_xy, 0, sizeof(float) * 2 * (size_t)P, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(grad_con, 0, sizeof(float) * 4 * (size_t)P, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(grad_rgb, 0, sizeof(float) * 3 * (size_t)P, s);
    if (e != cudaSuccess) return GSR_CUDA_ERROR;
    TrainRenderArgs ra = {};
    ra.W = width;
    ra.H = height;
    ra.P = P;
    ra.d_num = curr_offset;
    ra.cap = key_capacity;
    ra.vals = values_sorted;
    ra.ranges = reinterpret_cast<const int2*>(ranges);
    ra.xy = reinterpret_cast<const float2*>(points_xy);
    ra.rgbd = reinterpret_cast<const float4*>(rgb_depth);
    ra.con = reinterpret_cast<const float4*>(conic_opacity);
    for (int k = 0; k < 3; k++) ra.bg[k] = bg_color[k];
    ra.T_final = const_cast<float*>(T_final);
    ra.n_tile = const_cast<int32_t*>(n_tile);
    ra.grad_image = grad_image;
    ra.grad_xy = grad_xy;
    ra.grad_con = grad_con;
    ra.grad_rgb = grad_rgb;
    if ((e = launch_render_train(ra, true, s)) != cudaSuccess) return GSR_CUDA_ERROR;
    PreBackArgs pa = {};
    pa.P = P;
    pa.n_views = 1;
    pa.means = means;
    pa.log_scales = log_scales;
    pa.quats = quats;
    pa.logits = logits;
    pa.shs = shs;
    pa.cam[0] = adj_camera(width, height, cam_pos, cam_rot, focal_x, focal_y, z_far, z_near);
    pa.gxy = grad_xy;
    pa.gcon = grad_con;
    pa.grgb = grad_rgb;
    pa.g_means = g_means;
    pa.g_log_scales = g_log_scales;
    pa.g_quats = g_quats;
    pa.g_logits = g_logits;
    pa.g_shs = g_shs;
    pa.accumulate = accumulate;
    k_preprocess_backward<false><<<div_up(P, kAdjThreads), kAdjThreads, 0, s>>>(pa);
    return cudaGetLastError() == cudaSuccess ? GSR_OK : GSR_CUDA_ERROR;
}

size_t gsr_train_views_scratch_bytes(int n_views)
{
    if (n_views <= 0 || n_views > 32767) return 0;
    return ((size_t)n_views * sizeof(PreprocessParams) + 255) & ~(size_t)255;
}

gsr_status gsr_train_forward_views(int P, const float* means, const float* log_scales, const float* quats,
                                   const float* logits, const float* shs, int n_views, int width, int height,
                                   const float* cam_pos, const float* cam_rot, const float* cam_intr,
                                   const float* bg_color, float* opacity, float* cov3d, void* view_scratch,
                                   size_t view_scratch_bytes, int32_t* curr_offset, void* workspace,
                                   size_t workspace_bytes, uint64_t* keys_unsorted, uint32_t* values_unsorted,
                                   uint64_t* keys_sorted, uint32_t* values_sorted, int64_t key_capacity,
                                   float* points_xy, float* rgb_depth, float* conic_opacity, int32_t* ranges,
                                   int32_t* n_tile, float* T_final, float* image, int flags, gsr_stream_t stream)
{
    cudaStream_t s = (cudaStream_t)stream;
    if (P < 0 || n_views <= 0 || width <= 0 || height <= 0 || !cam_pos || !cam_rot || !cam_intr || !bg_color ||
        !curr_offset || !workspace || !ranges || !n_tile || !T_final || !image || !opacity || !cov3d ||
        !view_scratch || (flags & ~GSR_QUAD_KEYS) != 0)
        return GSR_INVALID_ARG;
    const bool quad = (flags & GSR_QUAD_KEYS) != 0;
    if (quad && (long long)P * n_views > (long long)kQuadGidMask + 1) return GSR_INVALID_ARG;
    if (P > 0 && (!means || !log_scales || !quats || !logits || !shs || !points_xy || !rgb_depth || !conic_opacity))
        return GSR_INVALID_ARG;
    if (view_scratch_bytes < gsr_train_views_scratch_bytes(n_views)) return GSR_INVALID_ARG;
    if (workspace_bytes < sort_workspace_bytes(key_capacity) || key_capacity >= (1LL << 30)) return GSR_INVALID_ARG;
    const int tiles = div_up(width, 16) * div_up(height, 16);
    // values carry view * P + Gaussian; key tile ids view * kt + tile (or quad)
    if ((long long)P * n_views >= (1LL << 31) || (long long)tiles * n_views >= (1LL << 30)) return GSR_INVALID_ARG;
    const int kt = quad ? quad_cols(div_up(width, 16)) * quad_cols(div_up(height, 16)) : tiles;
    cudaError_t e = launch_scene_prepare(P, log_scales, quats, logits, opacity, cov3d, s);
    if (e == cudaSuccess) e = clear_header(workspace, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(curr_offset, 0, sizeof(int32_t), s);
    if (e != cudaSuccess) return GSR_CUDA_ERROR;
    // every view's parameter block, as the single-view preprocess fills it,
    // with its rows at view * P and its tiles at view * tiles
    PreprocessParams* d_params = reinterpret_cast<PreprocessParams*>(view_scratch);
    std::vector<PreprocessParams> hp((size_t)n_views);
    for (int v = 0; v < n_views; v++) {
        const float* in = cam_intr + 4 * (size_t)v;  // focal_x, focal_y, z_far, z_near
        const size_t r = (size_t)v * P;
        const gsr_status st = preprocess_params(hp[v], P, means, shs, opacity, cov3d, width, height, 16, 16,
                                                cam_pos + 3 * (size_t)v, cam_rot + 9 * (size_t)v, in[0], in[1], in[2],
                                                in[3], points_xy + 2 * r, rgb_depth + 4 * r, conic_opacity + 4 * r,
                                                keys_unsorted, values_unsorted, key_capacity, curr_offset, workspace,
                                                workspace_bytes);
        if (st != GSR_OK) return st;
        if (hp[v].mq.capacity <= 0) return GSR_INVALID_ARG;
        hp[v].gid_base = (int)r;
        hp[v].tile_base = v * kt;
        hp[v].views = d_params;
        hp[v].quad = quad ? 1 : 0;
    }
    if (P == 0) {
        // no Gaussian: no key, and every pixel is the background
        e = cudaMemsetAsync(ranges, 0, sizeof(int32_t) * 2 * (size_t)kt * n_views, s);
    } else {
        PreprocessParams base = hp[0];
        base.n_views = n_views;
        base.header_clear = 1;
        base.interleave = 1;  // every view has the scene's P
        // a pageable source is staged before the call returns
        e = cudaMemcpyAsync(d_params, hp.data(), sizeof(PreprocessParams) * (size_t)n_views, cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = launch_preprocess_views(base, n_views, n_views * div_up(P, 256), false, s);
        if (e != cudaSuccess) return GSR_CUDA_ERROR;
        SortArgs sa;
        sa.num = 0;
        sa.d_num = curr_offset;
        sa.cap = key_capacity;
        sa.end_bit = 32 + bits_for((uint32_t)(kt * n_views));
        sa.compress_depth = true;
        sa.keys_in = keys_unsorted;
        sa.vals_in = values_unsorted;
        sa.keys_out = keys_sorted;
        sa.vals_out = values_sorted;
        sa.ws = workspace;
        sa.ws_bytes = workspace_bytes;
        sa.header_clear = true;
        if ((e = launch_sort(sa, s)) != cudaSuccess) return GSR_CUDA_ERROR;
        e = launch_tile_ranges(0, curr_offset, key_capacity, kt * n_views, keys_sorted, ranges, false, s);
    }
    if (e != cudaSuccess) return GSR_CUDA_ERROR;
    TrainRenderArgs ra = {};
    ra.W = width;
    ra.H = height;
    ra.P = P * n_views;
    ra.n_views = n_views;
    ra.quad = quad ? 1 : 0;
    ra.d_num = curr_offset;
    ra.cap = key_capacity;
    ra.vals = values_sorted;
    ra.ranges = reinterpret_cast<const int2*>(ranges);
    ra.xy = reinterpret_cast<const float2*>(points_xy);
    ra.rgbd = reinterpret_cast<const float4*>(rgb_depth);
    ra.con = reinterpret_cast<const float4*>(conic_opacity);
    for (int k = 0; k < 3; k++) ra.bg[k] = bg_color[k];
    ra.image = image;
    ra.T_final = T_final;
    ra.n_tile = n_tile;
    e = launch_render_train(ra, false, s);
    return e == cudaSuccess ? GSR_OK : GSR_CUDA_ERROR;
}

gsr_status gsr_train_backward_views(int P, const float* means, const float* log_scales, const float* quats,
                                    const float* logits, const float* shs, int n_views, int width, int height,
                                    const float* cam_pos, const float* cam_rot, const float* cam_intr,
                                    const float* bg_color, const int32_t* curr_offset, int64_t key_capacity,
                                    const uint32_t* values_sorted, const int32_t* ranges, const int32_t* n_tile,
                                    const float* T_final, const float* points_xy, const float* rgb_depth,
                                    const float* conic_opacity, const float* grad_image, float* grad_feat,
                                    float* g_means, float* g_log_scales, float* g_quats, float* g_logits,
                                    float* g_shs, int accumulate, int flags, gsr_stream_t stream)
{
    cudaStream_t s = (cudaStream_t)stream;
    if (P < 0 || n_views <= 0 || width <= 0 || height <= 0 || !cam_pos || !cam_rot || !cam_intr || !bg_color ||
        !curr_offset || !ranges || !n_tile || !T_final || !grad_image || !grad_feat || (flags & ~GSR_QUAD_KEYS) != 0)
        return GSR_INVALID_ARG;
    const bool quad = (flags & GSR_QUAD_KEYS) != 0;
    if (quad && (long long)P * n_views > (long long)kQuadGidMask + 1) return GSR_INVALID_ARG;
    if ((reinterpret_cast<uintptr_t>(grad_feat) & 15u) != 0) return GSR_INVALID_ARG;  // read as 16-byte vectors
    const int tiles = div_up(width, 16) * div_up(height, 16);
    if ((long long)P * n_views >= (1LL << 31) || (long long)tiles * n_views >= (1LL << 30)) return GSR_INVALID_ARG;
    if (P == 0) return GSR_OK;
    if (!means || !log_scales || !quats || !logits || !shs || !g_means || !g_log_scales || !g_quats || !g_logits ||
        !g_shs || !values_sorted || !points_xy || !rgb_depth || !conic_opacity)
        return GSR_INVALID_ARG;
    const size_t rows = (size_t)P * n_views;
    cudaError_t e = cudaMemsetAsync(grad_feat, 0, sizeof(float) * 12 * rows, s);
    if (e != cudaSuccess) return GSR_CUDA_ERROR;
    TrainRenderArgs ra = {};
    ra.W = width;
    ra.H = height;
    ra.P = (int)rows;
    ra.n_views = n_views;
    ra.quad = quad ? 1 : 0;
    ra.d_num = curr_offset;
    ra.cap = key_capacity;
    ra.vals = values_sorted;
    ra.ranges = reinterpret_cast<const int2*>(ranges);
    ra.xy = reinterpret_cast<const float2*>(points_xy);
    ra.rgbd = reinterpret_cast<const float4*>(rgb_depth);
    ra.con = reinterpret_cast<const float4*>(conic_opacity);
    for (int k = 0; k < 3; k++) ra.bg[k] = bg_color[k];
    ra.T_final = const_cast<float*>(T_final);
    ra.n_tile = const_cast<int32_t*>(n_tile);
    ra.grad_image = grad_image;
    ra.grad_rec = grad_feat;
    if ((e = launch_render_train(ra, true, s)) != cudaSuccess) return GSR_CUDA_ERROR;
    for (int v0 = 0; v0 < n_views; v0 += kAdjViews) {
        PreBackArgs pa = {};
        pa.P = P;
        pa.n_views = std::min(kAdjViews, n_views - v0);
        pa.means = means;
        pa.log_scales = log_scales;
        pa.quats = quats;
        pa.logits = logits;
        pa.shs = shs;
        for (int k = 0; k < pa.n_views; k++) {
            const int v = v0 + k;
            const float* in = cam_intr + 4 * (size_t)v;
            pa.cam[k] = adj_camera(width, height, cam_pos + 3 * (size_t)v, cam_rot + 9 * (size_t)v, in[0], in[1],
                                   in[2], in[3]);
        }
        pa.grec = reinterpret_cast<const float4*>(grad_feat) + 3 * (size_t)v0 * P;
        pa.g_means = g_means;
        pa.g_log_scales = g_log_scales;
        pa.g_quats = g_quats;
        pa.g_logits = g_logits;
        pa.g_shs = g_shs;
        pa.accumulate = (accumulate || v0 > 0) ? 1 : 0;
        k_preprocess_backward<true><<<div_up(P, kAdjThreads), kAdjThreads, 0, s>>>(pa);
        if (cudaGetLastError() != cudaSuccess) return GSR_CUDA_ERROR;
    }
    return GSR_OK;
}

}  // extern "C"

// Backward pass of the one-pixel point rasterizer for sm_100a.
// Stands in for BlendPointCloudBackward and its kernels (darglein/ADOP src/lib/rendering/PointRenderer.cu:
// CombineAndFillBackward :851-900, RenderBackward :396-724, NormalizeGradient :1534-1547) and the gradient
// of the environment-map composite (RenderModule.cpp:121-125, grid_sample backward).
//
// Differences in how the same sums are formed (results agree within float-ordering tolerance):
//  * the forward pass lists, per 32 x 16 screen tile, the points that were accepted on some layer; the backward pass runs
//    one block per tile over that list, with the tile's region of every layer (weight, forward image, upstream gradient)
//    staged in shared memory, instead of one thread per point of the cloud reading scattered pixels (kernels with the
//    reference's structure stay behind it for calls without a usable list);
//  * a point's descriptor gradient is summed over its layers and leaves as one vector atomic; its image-space ghost
//    gradient is summed over its layers too (scaled by 0.5^layer), so the projection chain runs once per visible point;
//  * the point gradient and its counter leave as ONE 16-byte vector atomic (x, y, z, count);
//  * pose and intrinsics gradients, which the reference adds with 7 + 14 same-address atomics per splat,
//    are reduced warp -> block in shared memory and leave as one atomic per component and block;
//  * the all-points kernels read the ghost stencil from one interleaved record per pixel [I_0..I_C-1, G_0..G_C-1] that a
//    preparation pass builds (a neighbour then costs one or two 32-byte sectors instead of 2C).
#include <algorithm>

#include "common.cuh"
#include "per_device.h"

namespace adop {

// ------------------------------------------------------------------------------------------------------
// K4: preparation pass over the pyramid pixels of one view (all-points path only).
//  * writes the interleaved record [I_0..I_C-1 | G_0..G_C-1] (I = the forward image before the environment-map
//    composite: the background colour where nothing was blended, PointRenderer.cu:1523);
//  * sums the gradient of the background colour over uncovered pixels (CombineAndFillBackward, :851-900);
//  * with the fused composite, scatters the environment-map gradient (bilinear, 4 taps).
__host__ __device__ inline int backward_record_floats(int C) { return (2 * C + 3) & ~3; }

// Planes of view `view` of a launch that serves several views: the layer table points at the first of them, the planes of a
// batch follow each other.
__device__ __forceinline__ const float* view_weight(const LayerTable& lt, int l, int view) { return lt.weight[l] + (size_t)view * lt.w[l] * lt.h[l]; }
template <int C>
__device__ __forceinline__ const float* view_color(const LayerTable& lt, int l, int view) { return lt.color[l] + (size_t)view * C * lt.w[l] * lt.h[l]; }
template <int C>
__device__ __forceinline__ const float* view_grad(const LayerTable& lt, int l, int view) { return lt.grad[l] + (size_t)view * C * lt.w[l] * lt.h[l]; }
// The visible lists of the launch's views: the first one's, and the distance from list to list
struct ViewLists
{
    VisibleList first;
    size_t view_ints;
};

// The environment-map gradient of an uncovered pixel (bilinear scatter, 4 taps): as in the forward resolve kernel the
// uncovered pixels are scattered single-pixel holes, so each warp parks them and works them off 32 at a time.
template <int C>
__device__ __forceinline__ void scatter_environment_gradient(const LayerTable& lt, int view, const ViewCam& cam, const KernelParams& kp, unsigned r,
                                                             float* __restrict__ grad_env, int env_h, int env_w, bool interleaved)
{
    const int l = layer_of_record(lt, r);
    const unsigned pix = r - lt.rec_off[l];
    const int w = lt.w[l];
    const size_t plane = (size_t)w * lt.h[l];
    const int gy = pix / w, gx = pix - gy * w;
    float gup[C];
#pragma unroll
    for (int c = 0; c < C; ++c) gup[c] = __ldg(view_grad<C>(lt, l, view) + c * plane + pix);
    Intr5 crop_l = scale_intr(cam.crop, __int_as_float((127 - l) << 23));
    V2 uv = env_uv_for_pixel(gx, gy, cam.V, cam.K, cam.dist, crop_l);
    BilinearTap tp = bilinear_taps(uv, env_w, env_h);
    const float om = 1.0f - kp.mask_background_value;
    const float w00 = (1.0f - tp.wx) * (1.0f - tp.wy), w01 = tp.wx * (1.0f - tp.wy);
    const float w10 = (1.0f - tp.wx) * tp.wy, w11 = tp.wx * tp.wy;
    if (interleaved && C % 4 == 0)
    {
        // [eh,ew,C] scratch: one vector atomic per tap and four channels instead of one per channel
        float4* e = reinterpret_cast<float4*>(grad_env);
        const size_t t00 = ((size_t)tp.y0 * env_w + tp.x0) * (C / 4), t01 = ((size_t)tp.y0 * env_w + tp.x1) * (C / 4);
        const size_t t10 = ((size_t)tp.y1 * env_w + tp.x0) * (C / 4), t11 = ((size_t)tp.y1 * env_w + tp.x1) * (C / 4);
#pragma unroll
        for (int k = 0; k < C / 4; ++k)
        {
            const float a = om * gup[4 * k], b = om * gup[4 * k + 1], c2 = om * gup[4 * k + 2], d = om * gup[4 * k + 3];
            atomicAdd(e + t00 + k, make_float4(a * w00, b * w00, c2 * w00, d * w00));
            atomicAdd(e + t01 + k, make_float4(a * w01, b * w01, c2 * w01, d * w01));
            atomicAdd(e + t10 + k, make_float4(a * w10, b * w10, c2 * w10, d * w10));
            atomicAdd(e + t11 + k, make_float4(a * w11, b * w11, c2 * w11, d * w11));
        }
        return;
    }
#pragma unroll
    for (int c = 0; c < C; ++c)
    {
        float* e = grad_env + (size_t)c * env_h * env_w;
        float ge = om * gup[c];
        atomicAdd(e + (size_t)tp.y0 * env_w + tp.x0, ge * w00);
        atomicAdd(e + (size_t)tp.y0 * env_w + tp.x1, ge * w01);
        atomicAdd(e + (size_t)tp.y1 * env_w + tp.x0, ge * w10);
        atomicAdd(e + (size_t)tp.y1 * env_w + tp.x1, ge * w11);
    }
}

struct HoleArgs
{
    float* grad_background;
    float* grad_env;
    int env_h, env_w;
    bool env_interleaved;
};
template <int C>
__device__ __forceinline__ void prepare_backward_part(const LayerTable& lt, int view, const ViewCam& cam, const KernelParams& kp,
                                                      const float* __restrict__ background, float* __restrict__ records, const HoleArgs& ha)
{
    constexpr int RB = (2 * C + 3) & ~3;
    float* __restrict__ grad_background = ha.grad_background;
    float* __restrict__ grad_env = ha.grad_env;
    const int env_h = ha.env_h, env_w = ha.env_w;
    const bool env_interleaved = ha.env_interleaved;
    __shared__ float s_bg[C];
    __shared__ unsigned s_parked[kBlock / 32][64];
    unsigned* parked = s_parked[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    int n_parked = 0;  // the same in every lane of the warp
    if (threadIdx.x < C) s_bg[threadIdx.x] = 0.f;
    __syncthreads();
    const unsigned total = lt.rec_off[kMaxLayers];
    const unsigned stride = gridDim.x * blockDim.x;
    float g[C], bgc[C];
#pragma unroll
    for (int c = 0; c < C; ++c) { g[c] = 0.f; bgc[c] = __ldg(background + c); }
    // warp-uniform trip count: the parking uses full-warp votes
    for (unsigned base = blockIdx.x * blockDim.x; base < total; base += stride)
    {
        const unsigned r = base + threadIdx.x;
        bool hole = false;
        if (r < total)
        {
            const int l = layer_of_record(lt, r);
            const unsigned pix = r - lt.rec_off[l];
            const size_t plane = (size_t)lt.w[l] * lt.h[l];
            // every load of the pixel is requested before the coverage is known
            const float wgt = __ldg(view_weight(lt, l, view) + pix);
            float rec[RB];
#pragma unroll
            for (int c = 0; c < C; ++c)
            {
                rec[C + c] = __ldcs(view_grad<C>(lt, l, view) + c * plane + pix);
                rec[c] = __ldg(view_color<C>(lt, l, view) + c * plane + pix);
            }
            const bool covered = wgt != 0.f;
            if (!covered)
            {
                // the image before the environment map was added (PointRenderer.cu:1523)
#pragma unroll
                for (int c = 0; c < C; ++c) rec[c] = bgc[c];
            }
#pragma unroll
            for (int k = 2 * C; k < RB; ++k) rec[k] = 0.f;
            float4* dst = reinterpret_cast<float4*>(records + (size_t)r * RB);
#pragma unroll
            for (int k = 0; k < RB / 4; ++k) dst[k] = make_float4(rec[4 * k], rec[4 * k + 1], rec[4 * k + 2], rec[4 * k + 3]);
            if (!covered)
            {
#pragma unroll
                for (int c = 0; c < C; ++c) g[c] += rec[C + c];
                hole = grad_env != nullptr;
            }
        }
        const unsigned vote = __ballot_sync(0xffffffffu, hole);
        if (vote)
        {
            if (hole) parked[n_parked + __popc(vote & ((1u << lane) - 1u))] = r;
            n_parked += __popc(vote);
            __syncwarp();
            if (n_parked >= 32)
            {
                n_parked -= 32;
                scatter_environment_gradient<C>(lt, view, cam, kp, parked[n_parked + lane], grad_env, env_h, env_w, env_interleaved);
            }
            __syncwarp();
        }
    }
    if (lane < n_parked) scatter_environment_gradient<C>(lt, view, cam, kp, parked[lane], grad_env, env_h, env_w, env_interleaved);
    if (grad_background)
    {
#pragma unroll
        for (int c = 0; c < C; ++c)
        {
            float v = warp_sum(g[c]);
            if ((threadIdx.x & 31) == 0 && v != 0.f) atomicAdd(&s_bg[c], v);
        }
        __syncthreads();
        if (threadIdx.x < C && s_bg[threadIdx.x] != 0.f) atomicAdd(grad_background + threadIdx.x, s_bg[threadIdx.x]);
    }
}
template <int C>
__global__ void __launch_bounds__(kBlock) k_prepare_backward(LayerTable lt, const ViewCam* __restrict__ camp, KernelParams kp,
                                                              const float* __restrict__ background, float* __restrict__ records, HoleArgs ha)
{
    prepare_backward_part<C>(lt, 0, *camp, kp, background, records, ha);
}

// ------------------------------------------------------------------------------------------------------
// K5: gradients of the splats.
struct BackwardTargets
{
    const float* texture;
    const float* texture_interleaved;  // optional [T,C]
    int num_texels;
    const float* background;
    float* grad_texture;
    float* grad_texture_interleaved;   // optional [T,C]; when set the descriptor gradient goes there
    float4* grad_points;
    // the tensors' first rows; a view's rows come from the table behind the camera records (ViewRows)
    double* grad_pose;        // 6 doubles per image
    float* count_pose;
    float* grad_intrinsics;   // one row per camera
    float* count_intrinsics;
};

// interleaved [I | G] of a pyramid pixel, written by the preparation pass
template <int C>
__device__ __forceinline__ void load_record(const float* __restrict__ records, size_t r, float* out)
{
    constexpr int RB = (2 * C + 3) & ~3;
    const float4* src = reinterpret_cast<const float4*>(records + r * RB);
#pragma unroll
    for (int k = 0; k < RB / 4; ++k)
    {
        float4 a = __ldg(src + k);
        out[4 * k] = a.x; out[4 * k + 1] = a.y; out[4 * k + 2] = a.z; out[4 * k + 3] = a.w;
    }
}

// per-thread partial sums of the view's pose / intrinsics gradient
template <int MODEL>
struct GeoAccum
{
    static constexpr int NI = MODEL == kPinholeDistortion ? 13 : 5;
    float pose[6];
    float intr[NI];
    float cnt;
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int k = 0; k < 6; ++k) pose[k] = 0.f;
#pragma unroll
        for (int k = 0; k < NI; ++k) intr[k] = 0.f;
        cnt = 0.f;
    }
};

// The ghost-geometry image gradient of one splat (PointRenderer.cu:522-611): central differences over the four
// neighbours of (T_p - I_x) * G_x, averaged over the channels. rn[k] = record of neighbour k (left, right, up, down).
template <int C>
__device__ __forceinline__ V2 stencil_gradient(const KernelParams& kp, const float* T_p, const float (*rn)[(2 * C + 3) & ~3],
                                               float z, const float* __restrict__ W, const float* __restrict__ D, const size_t* nb)
{
    float dR[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
    {
        float acc = 0.f;
        if (kp.test_backward_mode == 4)  // PointRenderer.cu:543-566
        {
            const float W_x = __ldg(W + nb[k]), D_x = __ldg(D + nb[k]);
#pragma unroll
            for (int c = 0; c < C; ++c)
            {
                float dI;
                if (W_x == 0.f || z * kp.depth_accept_plus_one < D_x) dI = T_p[c] - rn[k][c];
                else if (z > D_x * kp.depth_accept_plus_one) dI = 0.f;
                else dI = (W_x / (W_x + 1.f) * rn[k][c] + 1.f / (W_x + 1.f) * T_p[c] - rn[k][c]);
                acc += dI * rn[k][C + c];
            }
        }
        else
        {
#pragma unroll
            for (int c = 0; c < C; ++c) acc += (T_p[c] - rn[k][c]) * rn[k][C + c];
        }
        dR[k] = acc;
    }
    V2 g;
    g.x = 0.5f * (-dR[0] + dR[1]) / (float)C;
    g.y = 0.5f * (-dR[2] + dR[3]) / (float)C;
    return g;
}

// Chain the image gradient through the projection (PointRenderer.cu:613-720) and add to the partial sums.
// Returns false when the chain rejects the point; gp = (x, y, z, count) partial sum of the point gradient.
template <int MODEL>
__device__ __forceinline__ bool chain_gradient(const ViewCam& cam, const KernelParams& kp, const FetchedPoint& f, V2 g,
                                               float scale, float* gp, GeoAccum<MODEL>& acc)
{
    Intr5 crop_l = scale_intr(cam.crop, scale);
    if (MODEL == kPinholeDistortion)
    {
        GradPinhole o;
        if (!project_pinhole_backward(f.p, f.n, f.has_normal, g, cam.V, cam.K, crop_l, cam.dist, kp.check_normal != 0,
                                      kp.dist_cutoff, &o))
            return false;
        gp[0] += o.g_point[0]; gp[1] += o.g_point[1]; gp[2] += o.g_point[2]; gp[3] += 1.f;
#pragma unroll
        for (int k = 0; k < 6; ++k) acc.pose[k] += o.g_pose[k];
        // damping of PointRenderer.cu:647-678 (skew gets no gradient)
        const float kf = kp.K_gradient_factor, df = kp.distortion_gradient_factor;
        acc.intr[0] += kf * o.g_k[0]; acc.intr[1] += kf * o.g_k[1]; acc.intr[2] += kf * o.g_k[2]; acc.intr[3] += kf * o.g_k[3];
        acc.intr[5] += df * o.g_dis[0]; acc.intr[6] += df * o.g_dis[1];
        acc.intr[7] += df * (o.g_dis[2] * 0.25f);
        acc.intr[8] += df * (o.g_dis[3] * 0.1f); acc.intr[9] += df * (o.g_dis[4] * 0.1f); acc.intr[10] += df * (o.g_dis[5] * 0.1f);
        acc.intr[11] += df * (o.g_dis[6] * 0.1f); acc.intr[12] += df * (o.g_dis[7] * 0.1f);
    }
    else
    {
        GradOcam o;
        if (!project_ocam_backward(f.p, f.n, f.has_normal, g, cam.V, crop_l, cam.ocam, kp.check_normal != 0, kp.dist_cutoff, &o))
            return false;
        gp[0] += o.g_point[0]; gp[1] += o.g_point[1]; gp[2] += o.g_point[2]; gp[3] += 1.f;
#pragma unroll
        for (int k = 0; k < 6; ++k) acc.pose[k] += o.g_pose[k];
#pragma unroll
        for (int k = 0; k < 5; ++k) acc.intr[k] += o.g_affine[k];
    }
    acc.cnt += 1.f;
    return true;
}

// Block reduction of the per-view pose / intrinsics sums: warp shuffle, shared memory (double for the pose, which the
// reference accumulates in double, :1113), then one global atomic per component and block.
template <int MODEL>
struct GeoShared
{
    double pose[6];
    float intr[GeoAccum<MODEL>::NI];
    float cnt;
    int any;
};
template <int MODEL>
__device__ __forceinline__ void geo_shared_init(GeoShared<MODEL>* s)
{
    if (threadIdx.x < 6) s->pose[threadIdx.x] = 0.0;
    if (threadIdx.x < GeoAccum<MODEL>::NI) s->intr[threadIdx.x] = 0.f;
    if (threadIdx.x == 0) { s->cnt = 0.f; s->any = 0; }
}
// every thread of the block must call this; image, camera: the view's rows of the tensors, counted from bt's pointers
template <int MODEL>
__device__ __forceinline__ void geo_block_reduce(GeoShared<MODEL>* s, const GeoAccum<MODEL>& acc, const BackwardTargets& bt, int image = 0, int camera = 0,
                                                 int intrinsics_cols = 0)
{
    constexpr int NI = GeoAccum<MODEL>::NI;
    if (!(bt.grad_pose || bt.grad_intrinsics)) return;
    const unsigned any = __ballot_sync(0xffffffffu, acc.cnt > 0.f);
    if (any)
    {
        const bool lane0 = (threadIdx.x & 31) == 0;
        if (bt.grad_pose)
        {
#pragma unroll
            for (int k = 0; k < 6; ++k)
            {
                float v = warp_sum(acc.pose[k]);
                if (lane0) atomicAdd(&s->pose[k], (double)v);
            }
        }
        if (bt.grad_intrinsics)
        {
#pragma unroll
            for (int k = 0; k < NI; ++k)
            {
                float v = warp_sum(acc.intr[k]);
                if (lane0) atomicAdd(&s->intr[k], v);
            }
        }
        float c = warp_sum(acc.cnt);
        if (lane0) { atomicAdd(&s->cnt, c); s->any = 1; }
    }
    __syncthreads();
    if (!s->any) return;
    if (bt.grad_pose)
    {
        if (threadIdx.x < 6) atomicAdd(bt.grad_pose + (size_t)image * 6 + threadIdx.x, s->pose[threadIdx.x]);
        if (threadIdx.x == 6) atomicAdd(bt.count_pose + image, s->cnt);
    }
    if (bt.grad_intrinsics)
    {
        if (threadIdx.x >= 32 && threadIdx.x < 32 + NI) atomicAdd(bt.grad_intrinsics + (size_t)camera * intrinsics_cols + (threadIdx.x - 32), s->intr[threadIdx.x - 32]);
        // the reference counts 1/1024 per pinhole contribution and 1 per OCam contribution (:680-681, :718)
        if (threadIdx.x == 64) atomicAdd(bt.count_intrinsics + camera, MODEL == kPinholeDistortion ? s->cnt * (1.f / 1024.f) : s->cnt);
    }
}

// K5 (all points): the reference's structure, one thread per point walking its layers (RenderBackward, :396-724). Used
// when the forward pass recorded no visible list (or a tile's bucket overflowed, or the list was used before).
// records: [I | G] of every pixel from a launch of the preparation pass; null: the same values from the planes.
template <int C, int MODEL, bool RECORDS>
__device__ __forceinline__ void splat_backward_part(const PointStreams& pts, const ViewCam& cam, const KernelParams& kp, const LayerTable& lt, int view,
                                                    const BackwardTargets& bt, const float* records, int image, int camera, int intrinsics_cols)
{
    constexpr int RB = (2 * C + 3) & ~3;
    __shared__ GeoShared<MODEL> s_geo;
    geo_shared_init(&s_geo);
    __syncthreads();
    const bool want_geo = bt.grad_points || bt.grad_pose || bt.grad_intrinsics;
    GeoAccum<MODEL> acc;
    acc.clear();
    const int stride = gridDim.x * blockDim.x;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < pts.n; i += stride)
    {
        const bool drop_out = point_dropped(kp, view, pts.n, i);
        FetchedPoint f = fetch_point(pts, i);
        RasterPoint q;
        if (!project_for_raster(cam, f.p, f.r, f.n, f.has_normal, kp.check_normal != 0, kp.dist_cutoff, &q,
                                kp.drop_out_points_by_radius != 0)) continue;
        float x = q.x, y = q.y, rad = q.radius_px, scale = 1.f;
        const bool point_grad = want_geo && ((kp.ghost_gradients && drop_out) || (!kp.ghost_gradients && !drop_out));
        int ti = -1;
        float T_p[C], dg[C];
        bool have_t = false, have_dg = false;
        float gp[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < C; ++c) dg[c] = 0.f;
#pragma unroll 1
        for (int l = 0; l < lt.L; ++l, scale *= 0.5f, rad *= 0.5f, x *= 0.5f, y *= 0.5f)
        {
            if (kp.drop_out_points_by_radius && rad < kp.drop_out_radius_threshold) continue;
            const int px = round_half_even_bounded(x), py = round_half_even_bounded(y);
            const int w = lt.w[l], h = lt.h[l];
            if ((unsigned)px >= (unsigned)w || (unsigned)py >= (unsigned)h) continue;
            const size_t pix = (size_t)py * w + px;
            const float* D = lt.depth[l] + (size_t)view * w * h;
            const float* W = view_weight(lt, l, view);
            if (q.z > __ldg(D + pix) * kp.depth_accept_plus_one) break;
            const float wgt = __ldg(W + pix);
            const size_t rbase = (size_t)lt.rec_off[l] + pix;
            if (!drop_out)
            {
                if (wgt == 0.f) continue;
                if (bt.grad_texture)
                {
                    float rc[RB];
                    if (RECORDS) load_record<C>(records, rbase, rc);
                    else
                    {
#pragma unroll
                        for (int c = 0; c < C; ++c) rc[C + c] = __ldg(view_grad<C>(lt, l, view) + (size_t)c * w * h + pix);
                    }
                    const float iw = 1.f / wgt;
#pragma unroll
                    for (int c = 0; c < C; ++c) dg[c] += iw * rc[C + c];
                    have_dg = true;
                }
            }
            const int edge = min(min(px, py), min(w - 1 - px, h - 1 - py));
            if (!(point_grad && edge > 2)) continue;
            if (!have_t)
            {
                ti = pts.index ? __ldg(pts.index + i) : i;
                load_descriptor<C>(bt.texture, bt.texture_interleaved, bt.num_texels, ti, T_p);
                have_t = true;
            }
            const size_t nb[4] = {pix - 1, pix + 1, pix - (size_t)w, pix + (size_t)w};
            float rn[4][RB];
#pragma unroll
            for (int k = 0; k < 4; ++k)
            {
                if (RECORDS) load_record<C>(records, (size_t)lt.rec_off[l] + nb[k], rn[k]);
                else
                {
                    const bool covered = __ldg(W + nb[k]) != 0.f;
#pragma unroll
                    for (int c = 0; c < C; ++c)
                    {
                        rn[k][c] = covered ? __ldg(view_color<C>(lt, l, view) + (size_t)c * w * h + nb[k]) : __ldg(bt.background + c);
                        rn[k][C + c] = __ldg(view_grad<C>(lt, l, view) + (size_t)c * w * h + nb[k]);
                    }
                }
            }
            V2 g = stencil_gradient<C>(kp, T_p, rn, q.z, W, D, nb);
            chain_gradient<MODEL>(cam, kp, f, g, scale, gp, acc);
        }
        if (have_dg)
        {
            if (ti < 0) ti = pts.index ? __ldg(pts.index + i) : i;
            add_descriptor_gradient<C>(bt.grad_texture, bt.grad_texture_interleaved, bt.num_texels, ti, dg);
        }
        if (gp[3] > 0.f && bt.grad_points) atomicAdd(bt.grad_points + i, make_float4(gp[0], gp[1], gp[2], gp[3]));
    }
    geo_block_reduce<MODEL>(&s_geo, acc, bt, image, camera, intrinsics_cols);
}
template <int C, int MODEL>
__global__ void __launch_bounds__(kBlock) k_splat_backward_all(PointStreams pts, const ViewCam* __restrict__ camp, const ViewRows* __restrict__ rows,
                                                                KernelParams kp, LayerTable lt, BackwardTargets bt, const float* records, int intrinsics_cols)
{
    splat_backward_part<C, MODEL, true>(pts, *camp, kp, lt, 0, bt, records, rows->image, rows->camera, intrinsics_cols);
}

// ------------------------------------------------------------------------------------------------------
// K5 (visible list): the backward pass over the points that the forward pass listed, grouped by screen tile.
//   k_backward_tiles  one block per screen tile at a time. The tile's region of every layer - weight, forward image and
//                   upstream gradient, with a one-pixel halo (plus one pixel for the rounding of the halved coordinates
//                   on the coarser layers) - is copied from the NCHW planes into shared memory with asynchronous
//                   16-byte copies of whole rows; every listed point of the tile then takes its pixel and its four
//                   stencil neighbours, layer by layer, from there (a point whose pixel falls outside the staged region
//                   reads the planes directly). Per point: ONE descriptor-gradient atomic (summed over its layers) and
//                   ONE work item for the chain kernel: the point's image-space ghost gradient summed over its layers,
//                   each scaled by 0.5^layer (the projection chain is linear in that gradient, and a layer's crop
//                   transform is the full-resolution one times 0.5^layer, PointRenderer.cu:616).
//   k_chain_and_holes  one launch whose blocks split 5 : 3 between two independent parts: per work item, the summed
//                   image-space gradient chained through the projection to the point, pose and intrinsics gradients
//                   (block-reduced); and the background-colour and environment-map gradient of the uncovered pixels.
// Nothing here waits on another block. These kernels are bound by memory latency, not by bandwidth or arithmetic: each
// keeps several independent loads per thread in flight and as many blocks resident as registers and shared memory allow.
constexpr int kTileThreads = 256;
constexpr int kTilePass = 2 * kTileThreads;  // points of a tile that are staged and sorted in shared memory at a time
constexpr int kSortBins = kMaxLayers * kTileH;  // sort key of a point: (layers it visits, image row)
// staged region of layer l: rows [ (y0 >> l) - 1, + rows ), columns [ start, + pitch ), start = x0 - 4 on layer 0 and
// ((x0 >> l) - 1) & ~3 on the others (a multiple of four, so that rows can be copied as aligned 16-byte pieces)
__host__ __device__ constexpr int region_pitch(int l) { return l == 0 ? kTileW + 8 : (l == 1 ? 24 : (l == 2 ? 16 : 12)); }
__host__ __device__ constexpr int region_rows(int l) { return l == 0 ? kTileH + 2 : (l == 1 ? 11 : (l == 2 ? 7 : (l == 3 ? 5 : 4))); }
__host__ __device__ constexpr int region_offset(int l)
{
    int n = 0;
    for (int k = 0; k < l; ++k) n += region_pitch(k) * region_rows(k);
    return n;
}
// floats per plane: the regions of the first four layers, or of all eight (two kernel variants, so that every offset
// into the staged planes is a compile-time constant)
template <bool DEEP>
struct PlaneStride { static constexpr int value = DEEP ? region_offset(kMaxLayers) : region_offset(4); };
inline size_t tile_smem_bytes(int C, int L)
{
    const int stride = L > 4 ? region_offset(kMaxLayers) : region_offset(4);
    return sizeof(float) * (size_t)stride * (2 * C + 1) + sizeof(int4) * kTilePass + sizeof(unsigned short) * kTilePass;
}

__device__ __forceinline__ void async_copy_16(void* smem, const void* gmem)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void async_copy_4(void* smem, const void* gmem)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void async_copy_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Copies layer LAYER's region of the 2C + 1 planes into shared memory (asynchronously; the caller waits). A thread takes a place
// of the region and walks the planes: the place's row, column and bounds are worked out once for all 2C + 1 copies (spread
// over the threads plane by plane, every copy cost a handful of divisions and pointer selections, a fifth of the
// kernel's instructions). The layers start at different threads, so that the small regions do not all fall to the first warps.
template <int C, int LAYER, int STRIDE>
__device__ __forceinline__ void stage_region(const LayerTable& lt, int view, float* s_tile, int x0, int y0)
{
    constexpr int pitch = region_pitch(LAYER), rows = region_rows(LAYER), threads = kTileThreads;
    const int w = lt.w[LAYER], h = lt.h[LAYER];
    const size_t plane = (size_t)w * h;
    const float* weight = view_weight(lt, LAYER, view);
    const float* color = view_color<C>(lt, LAYER, view);
    const float* grad = view_grad<C>(lt, LAYER, view);
    const int sx = LAYER == 0 ? x0 - 4 : (((x0 >> LAYER) - 1) & ~3), sy = (y0 >> LAYER) - 1;
    float* dst = s_tile + region_offset(LAYER);
    const bool vec = (w & 3) == 0 && ((reinterpret_cast<uintptr_t>(weight) | reinterpret_cast<uintptr_t>(color) | reinterpret_cast<uintptr_t>(grad)) & 15) == 0;
    if (vec)
    {
        constexpr int p4 = pitch / 4, places = rows * p4, first = (region_offset(LAYER) / 4) % threads;
        for (int q = ((int)threadIdx.x + threads - first) % threads; q < places; q += threads)
        {
            const int row = q / p4, c4 = q - row * p4;
            const int gy = sy + row, gx = sx + 4 * c4;
            if ((unsigned)gy >= (unsigned)h || (unsigned)gx >= (unsigned)w) continue;
            const size_t at = (size_t)gy * w + gx;
            float* d = dst + row * pitch + 4 * c4;
            async_copy_16(d, weight + at);
            const float* src = color + at;
#pragma unroll
            for (int c = 0; c < C; ++c, src += plane) async_copy_16(d + (1 + c) * STRIDE, src);
            src = grad + at;
#pragma unroll
            for (int c = 0; c < C; ++c, src += plane) async_copy_16(d + (1 + C + c) * STRIDE, src);
        }
    }
    else
    {
        constexpr int places = rows * pitch, first = region_offset(LAYER) % threads;
        for (int q = ((int)threadIdx.x + threads - first) % threads; q < places; q += threads)
        {
            const int row = q / pitch, col = q - row * pitch;
            const int gy = sy + row, gx = sx + col;
            if ((unsigned)gy >= (unsigned)h || (unsigned)gx >= (unsigned)w) continue;
            const size_t at = (size_t)gy * w + gx;
            float* d = dst + q;
            async_copy_4(d, weight + at);
            const float* src = color + at;
#pragma unroll
            for (int c = 0; c < C; ++c, src += plane) async_copy_4(d + (1 + c) * STRIDE, src);
            src = grad + at;
#pragma unroll
            for (int c = 0; c < C; ++c, src += plane) async_copy_4(d + (1 + C + c) * STRIDE, src);
        }
    }
}
template <int C, int LAYER, int STRIDE, int LMAX>
__device__ __forceinline__ void stage_regions(const LayerTable& lt, int view, float* s_tile, int x0, int y0)
{
    if (LAYER < lt.L) stage_region<C, LAYER, STRIDE>(lt, view, s_tile, x0, y0);
    if constexpr (LAYER + 1 < LMAX) stage_regions<C, LAYER + 1, STRIDE, LMAX>(lt, view, s_tile, x0, y0);
}

// One (point, layer) visit of the backward pass: descriptor gradient and ghost-geometry image gradient of the point's pixel
// on a layer. at(p, dx, dy) reads a value of plane p (0 = weight, 1.. = image, 1 + C.. = upstream gradient) at an offset
// from the pixel; with p, dx, dy constants after unrolling the staged form is one shared-memory load with an immediate
// offset each.
template <int C, class PIX>
__device__ __forceinline__ void visit_layer(PIX at, bool drop_out, bool want_dg, bool stencil, const float* T_p, const float* bgc, float scale,
                                            float* dg, bool* have_dg, float* gx, float* gy, float* cnt)
{
    const float wgt = at(0, 0, 0);
    if (!drop_out)
    {
        if (wgt == 0.f) return;  // :473
        if (want_dg)
        {
            const float iw = reciprocal(wgt);
#pragma unroll
            for (int c = 0; c < C; ++c) dg[c] += iw * at(1 + C + c, 0, 0);
            *have_dg = true;
        }
    }
    if (!stencil) return;
    // ghost-geometry gradient (PointRenderer.cu:522-611): central differences of (T_p - I_x) * G_x over the four neighbours,
    // averaged over the channels; I = the image before the environment-map composite (:1523)
    float dR[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
    {
        const int dx = k == 0 ? -1 : (k == 1 ? 1 : 0), dy = k == 2 ? -1 : (k == 3 ? 1 : 0);
        const bool covered = at(0, dx, dy) != 0.f;
        float acc = 0.f;
#pragma unroll
        for (int c = 0; c < C; ++c)
        {
            const float I = covered ? at(1 + c, dx, dy) : bgc[c];
            acc += (T_p[c] - I) * at(1 + C + c, dx, dy);
        }
        dR[k] = acc;
    }
    *gx += (0.5f * (-dR[0] + dR[1]) / (float)C) * scale;
    *gy += (0.5f * (-dR[2] + dR[3]) / (float)C) * scale;
    *cnt += 1.f;
}

// per-point state of the tile kernel while it walks the point's layers
template <int C>
struct PointVisit
{
    float T_p[C], dg[C], bgc[C];
    bool drop_out, point_grad, want_dg, have_dg;
    float gx, gy, cnt;
    unsigned bmask;
};
// the visit of layer LAYER (and, recursively, of the coarser ones); x, y = the position on this layer, scale = 0.5^LAYER
template <int C, int LAYER, int STRIDE, int LMAX>
__device__ __forceinline__ void visit_layers(const LayerTable& lt, int view, const float* s_tile, int x0, int y0, float x, float y, float scale, PointVisit<C>& pv)
{
    if (LAYER < lt.L && (pv.bmask >> LAYER) != 0)  // no coarser layer to visit either: stop
    {
        if (pv.bmask & (1u << LAYER))
        {
            constexpr int pitch = region_pitch(LAYER), rows = region_rows(LAYER);
            const int px = round_half_even_bounded(x), py = round_half_even_bounded(y);
            const int w = lt.w[LAYER], h = lt.h[LAYER];
            const int sx = LAYER == 0 ? x0 - 4 : (((x0 >> LAYER) - 1) & ~3), sy = (y0 >> LAYER) - 1;
            const int cx = px - sx, cy = py - sy;
            const int edge = min(min(px, py), min(w - 1 - px, h - 1 - py));
            const bool stencil = pv.point_grad && edge > 2;
            // the pixel and its four neighbours lie in the staged region (else, rarely: read the planes)
            if (cx >= 1 && cx <= pitch - 2 && cy >= 1 && cy <= rows - 2)
            {
                const float* sp = s_tile + region_offset(LAYER) + cy * pitch + cx;
                visit_layer<C>([&](int p, int dx, int dy) { return sp[p * STRIDE + dy * pitch + dx]; },
                               pv.drop_out, pv.want_dg, stencil, pv.T_p, pv.bgc, scale, pv.dg, &pv.have_dg, &pv.gx, &pv.gy, &pv.cnt);
            }
            else
            {
                const size_t plane = (size_t)w * h;
                const size_t pix = (size_t)py * w + px;
                const float* W = view_weight(lt, LAYER, view);
                const float* I = view_color<C>(lt, LAYER, view);
                const float* G = view_grad<C>(lt, LAYER, view);
                visit_layer<C>([&](int p, int dx, int dy) {
                                   const size_t a = pix + dy * w + dx;
                                   return p == 0 ? __ldg(W + a) : (p <= C ? __ldg(I + (size_t)(p - 1) * plane + a) : __ldg(G + (size_t)(p - 1 - C) * plane + a));
                               },
                               pv.drop_out, pv.want_dg, stencil, pv.T_p, pv.bgc, scale, pv.dg, &pv.have_dg, &pv.gx, &pv.gy, &pv.cnt);
            }
        }
        if constexpr (LAYER + 1 < LMAX) visit_layers<C, LAYER + 1, STRIDE, LMAX>(lt, view, s_tile, x0, y0, x * 0.5f, y * 0.5f, scale * 0.5f, pv);
    }
}

template <int C, bool DEEP>
__global__ void __launch_bounds__(kTileThreads, C <= 4 ? (DEEP ? 3 : 4) : (C <= 8 ? 2 : 1))
    k_backward_tiles(PointStreams pts, KernelParams kp, LayerTable lt, TileTable tt, BackwardTargets bt, ViewLists lists, int want_geo)
{
    // blockIdx.y = view. First kernel of the pass: decides whether the view runs on its list and leaves the decision for
    // the kernels behind it
    const int view = (int)blockIdx.y;
    const VisibleList vl = list_of_view(lists.first, lists.view_ints, view);
    const bool go = (__ldg(vl.header + kListUnusable) | __ldg(vl.header + kListConsumed)) == 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) vl.header[kListGo] = go ? 1 : 0;
    if (!go) return;  // the all-points kernels take over
    constexpr int STRIDE = PlaneStride<DEEP>::value;
    constexpr int LMAX = DEEP ? kMaxLayers : 4;
    extern __shared__ __align__(16) float s_tile[];
    __shared__ int s_hist[kSortBins];
    // plane p of layer l: s_tile[p * STRIDE + region_offset(l) + row * pitch + col]
    int4* sE = reinterpret_cast<int4*>(s_tile + (size_t)STRIDE * (2 * C + 1));
    unsigned short* sOrder = reinterpret_cast<unsigned short*>(sE + kTilePass);
    PointVisit<C> pv;
#pragma unroll
    for (int c = 0; c < C; ++c) pv.bgc[c] = __ldg(bt.background + c);
    // The entry count of the next tile is fetched while this one is worked on.
    int tile = (int)blockIdx.x;
    int n_pts = tile < tt.n_tiles ? min(__ldg(vl.tile_cur + tile), tt.cap) : 0;
    for (; tile < tt.n_tiles; tile += (int)gridDim.x)
    {
        const int next = tile + (int)gridDim.x;
        const int next_n = next < tt.n_tiles ? min(__ldg(vl.tile_cur + next), tt.cap) : 0;
        const int ty = tile / tt.tiles_x, tx = tile - ty * tt.tiles_x;
        const int x0 = tx << kTileShiftX, y0 = ty << kTileShiftY;
        int4* ent = vl.entries + (size_t)tile * tt.cap;
        for (int pass0 = 0; pass0 < n_pts; pass0 += kTilePass)  // block-uniform
        {
            const int n_pass = min(n_pts - pass0, kTilePass);
            __syncthreads();  // the previous readers of the staged data are done
            if (pass0 == 0) stage_regions<C, 0, STRIDE, LMAX>(lt, view, s_tile, x0, y0);
            for (int q = threadIdx.x; q < n_pass; q += kTileThreads) async_copy_16(sE + q, ent + pass0 + q);
            if (threadIdx.x < kSortBins) s_hist[threadIdx.x] = 0;
            async_copy_wait_all();
            __syncthreads();
            // ---- order the points: by their coarsest layer, most layers first (the warps then walk the same layers in all
            // lanes), and within that by image row (the lanes of a warp then read mostly one row of the staged planes, in
            // different columns: few shared-memory bank conflicts)
            int key[kTilePass / kTileThreads], rank[kTilePass / kTileThreads];
#pragma unroll
            for (int j = 0; j < kTilePass / kTileThreads; ++j)
            {
                const int q = j * kTileThreads + threadIdx.x;
                key[j] = -1;
                if (q < n_pass)
                {
                    const int4 e = sE[q];
                    const unsigned bmask = ((unsigned)e.y >> 8) & 0xffu;
                    const int cls = 32 - __clz(bmask);  // 1 .. kMaxLayers (the backward mask of a listed point is not 0)
                    const int row = min(max(round_half_even_bounded(__int_as_float(e.w)) - y0, 0), kTileH - 1);
                    key[j] = (kMaxLayers - cls) * kTileH + row;
                    rank[j] = atomicAdd(&s_hist[key[j]], 1);
                }
            }
            __syncthreads();
            if (threadIdx.x < 32)
            {
                // exclusive prefix sums of the kSortBins counts: four bins per lane
                constexpr int per = kSortBins / 32;
                int v[per], sum = 0;
#pragma unroll
                for (int k = 0; k < per; ++k) { v[k] = s_hist[threadIdx.x * per + k]; sum += v[k]; }
                int incl = sum;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1)
                {
                    int t = __shfl_up_sync(0xffffffffu, incl, o);
                    if ((int)threadIdx.x >= o) incl += t;
                }
                int run = incl - sum;
#pragma unroll
                for (int k = 0; k < per; ++k) { s_hist[threadIdx.x * per + k] = run; run += v[k]; }
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < kTilePass / kTileThreads; ++j)
                if (key[j] >= 0) sOrder[s_hist[key[j]] + rank[j]] = (unsigned short)(j * kTileThreads + threadIdx.x);
            __syncthreads();
            // ---- the points
            for (int sidx = threadIdx.x; sidx < n_pass; sidx += kTileThreads)
            {
                const int4 e = sE[sOrder[sidx]];
                pv.bmask = ((unsigned)e.y >> 8) & 0xffu;
                const int i = (int)((unsigned)e.x & ~kEntryDropped);
                pv.drop_out = ((unsigned)e.x & kEntryDropped) != 0;
                pv.point_grad = want_geo && ((kp.ghost_gradients && pv.drop_out) || (!kp.ghost_gradients && !pv.drop_out));
                pv.want_dg = !pv.drop_out && bt.grad_texture != nullptr;
                const int ti = pts.index ? __ldg(pts.index + i) : i;
                if (pv.point_grad) load_descriptor<C>(bt.texture, bt.texture_interleaved, bt.num_texels, ti, pv.T_p);
                else
                {
#pragma unroll
                    for (int c = 0; c < C; ++c) pv.T_p[c] = 0.f;
                }
#pragma unroll
                for (int c = 0; c < C; ++c) pv.dg[c] = 0.f;
                pv.have_dg = false;
                pv.gx = pv.gy = pv.cnt = 0.f;
                visit_layers<C, 0, STRIDE, LMAX>(lt, view, s_tile, x0, y0, __int_as_float(e.z), __int_as_float(e.w), 1.f, pv);
                if (pv.have_dg) add_descriptor_gradient<C>(bt.grad_texture, bt.grad_texture_interleaved, bt.num_texels, ti, pv.dg);
                // the entry becomes the chain kernel's work item (every entry of this pass has been read into shared memory)
                if (want_geo)
                    reinterpret_cast<float4*>(ent)[pass0 + sidx] = pv.cnt > 0.f ? make_float4(__int_as_float(i), pv.gx, pv.gy, pv.cnt) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        n_pts = next_n;
    }
}

// Background-colour gradient (CombineAndFillBackward, PointRenderer.cu:851-900) and environment-map gradient (the
// composite's backward, RenderModule.cpp:121-125, grid_sample backward) of the uncovered pixels of one view: one thread
// per four pyramid pixels reads the weights; the holes, scattered single pixels, are parked per warp and worked off 32
// at a time (gradient of each channel; for the environment map the ray through the inverse camera model and the bilinear
// scatter).
// part of k_chain_and_holes: `block` of `blocks` thread blocks
template <int C>
__device__ __forceinline__ void hole_gradients_part(const LayerTable& lt, int view, const ViewCam* __restrict__ camp, const KernelParams& kp, const HoleArgs& ha,
                                                    int block, int blocks)
{
    float* __restrict__ grad_background = ha.grad_background;
    float* __restrict__ grad_env = ha.grad_env;
    const int env_h = ha.env_h, env_w = ha.env_w;
    const bool env_interleaved = ha.env_interleaved;
    const ViewCam& cam = *camp;
    __shared__ float s_bg[C];
    __shared__ unsigned s_parked[kBlock / 32][160];
    unsigned* parked = s_parked[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    int n_parked = 0;  // the same in every lane of the warp
    if (threadIdx.x < C) s_bg[threadIdx.x] = 0.f;
    __syncthreads();
    float g[C];
#pragma unroll
    for (int c = 0; c < C; ++c) g[c] = 0.f;
    auto work_off = [&](unsigned r)
    {
        const int l = layer_of_record(lt, r);
        const unsigned pix = r - lt.rec_off[l];
        const size_t plane = (size_t)lt.w[l] * lt.h[l];
        if (grad_background)
        {
#pragma unroll
            for (int c = 0; c < C; ++c) g[c] += __ldg(view_grad<C>(lt, l, view) + c * plane + pix);
        }
        if (grad_env) scatter_environment_gradient<C>(lt, view, cam, kp, r, grad_env, env_h, env_w, env_interleaved);
    };
    const unsigned total = lt.rec_off[kMaxLayers];
    const unsigned groups = (total + 3) / 4;
    const unsigned stride = (unsigned)blocks * blockDim.x;
    for (unsigned base = (unsigned)block * blockDim.x; base < groups; base += stride)  // warp-uniform trip count
    {
        // four consecutive pyramid pixels per thread (they may straddle a layer boundary: the weights are read one by one)
        const unsigned r0 = (base + threadIdx.x) * 4;
        bool hole[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            hole[k] = false;
            const unsigned r = r0 + k;
            if (r < total)
            {
                const int l = layer_of_record(lt, r);
                hole[k] = __ldg(view_weight(lt, l, view) + (r - lt.rec_off[l])) == 0.f;
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            const unsigned vote = __ballot_sync(0xffffffffu, hole[k]);
            if (hole[k]) parked[n_parked + __popc(vote & ((1u << lane) - 1u))] = r0 + k;
            n_parked += __popc(vote);
        }
        __syncwarp();
        while (n_parked >= 32)
        {
            n_parked -= 32;
            work_off(parked[n_parked + lane]);
        }
        __syncwarp();
    }
    if (lane < n_parked) work_off(parked[lane]);
    if (grad_background)
    {
#pragma unroll
        for (int c = 0; c < C; ++c)
        {
            float v = warp_sum(g[c]);
            if (lane == 0 && v != 0.f) atomicAdd(&s_bg[c], v);
        }
        __syncthreads();
        if (threadIdx.x < C && s_bg[threadIdx.x] != 0.f) atomicAdd(grad_background + threadIdx.x, s_bg[threadIdx.x]);
    }
}

// ---- per-point chain ---------------------------------------------------------------------------------------------------
// A visible point with its summed image-space gradient, as parked in shared memory by point_chain_part.
struct ChainItem
{
    int id;
    float gx, gy, count;
    float px, py, pz;
    int normal;
};

// Pinhole chain in a short form (same mathematics as project_pinhole_backward, PointRendererHelper.h:109-170, summed
// straight into the per-thread partial sums). With q = x g1x + y g1y (m = (x, y) the normalised point, g1 the gradient
// behind K) the sixteen entries of the distortion Jacobian and the four of J_m collapse:
//   d/dk1..k3 = {r2, r4, r6} q / den,  d/dk4..k6 = -rad {r2, r4, r6} q / den,  d/dp1 = 2xy g1x + (r2 + 2y2) g1y,  d/dp2 = (r2 + 2x2) g1x + 2xy g1y,
//   gm = rad g1 + 2 m drad q + tangential terms,   drad = (dnum - rad dden) / den.
// The partial sums are undamped; the damping factors of PointRenderer.cu:647-678 are applied once per block.
struct PinholeSums
{
    float pose[6];
    float k[4];
    float d[8];
    float cnt;
};
__device__ __forceinline__ void chain_pinhole_fast(const ViewCam& cam, bool check_normal, const ChainItem& it, float4* __restrict__ grad_points,
                                                   PinholeSums& a)
{
    const Rigid32& V = cam.V;
    V3 view;
    view.x = fmaf(V.r[0], it.px, fmaf(V.r[1], it.py, fmaf(V.r[2], it.pz, V.t[0])));
    view.y = fmaf(V.r[3], it.px, fmaf(V.r[4], it.py, fmaf(V.r[5], it.pz, V.t[1])));
    view.z = fmaf(V.r[6], it.px, fmaf(V.r[7], it.py, fmaf(V.r[8], it.pz, V.t[2])));
    if (!(view.z > 0.f)) return;
    if (check_normal)
    {
        V3 vn = rotate(V, unpack_normal_10bit(it.normal));
        if (fmaf(view.z, vn.z, fmaf(view.y, vn.y, view.x * vn.x)) > 0.f) return;
    }
    const float iz = reciprocal(view.z);
    const float x = view.x * iz, y = view.y * iz;
    const float x2 = x * x, y2 = y * y, r2 = x2 + y2, r4 = r2 * r2, r6 = r4 * r2, xy2 = 2.f * x * y;
    const Dist8& d = cam.dist;
    const float num = fmaf(fmaf(fmaf(d.k3, r2, d.k2), r2, d.k1), r2, 1.0f);
    const float den = fmaf(fmaf(fmaf(d.k6, r2, d.k5), r2, d.k4), r2, 1.0f);
    const float iden = reciprocal(den);
    const float rad = num * iden;
    const float dnum = fmaf(fmaf(3.f * d.k3, r2, 2.f * d.k2), r2, d.k1);
    const float dden = fmaf(fmaf(3.f * d.k6, r2, 2.f * d.k5), r2, d.k4);
    const float drad = fmaf(-rad, dden, dnum) * iden;
    const float dpx = fmaf(x, rad, fmaf(d.p1, xy2, d.p2 * fmaf(2.f, x2, r2)));
    const float dpy = fmaf(y, rad, fmaf(d.p2, xy2, d.p1 * fmaf(2.f, y2, r2)));
    // crop^T, K
    const float g2x = cam.crop.fx * it.gx;
    const float g2y = fmaf(cam.crop.s, it.gx, cam.crop.fy * it.gy);
    a.k[0] = fmaf(dpx, g2x, a.k[0]); a.k[1] = fmaf(dpy, g2y, a.k[1]); a.k[2] += g2x; a.k[3] += g2y;
    const float g1x = cam.K.fx * g2x;
    const float g1y = fmaf(cam.K.s, g2x, cam.K.fy * g2y);
    const float q = fmaf(x, g1x, y * g1y);
    const float qd = q * iden, qr = -rad * qd;
    a.d[0] = fmaf(r2, qd, a.d[0]); a.d[1] = fmaf(r4, qd, a.d[1]); a.d[2] = fmaf(r6, qd, a.d[2]);
    a.d[3] = fmaf(r2, qr, a.d[3]); a.d[4] = fmaf(r4, qr, a.d[4]); a.d[5] = fmaf(r6, qr, a.d[5]);
    const float ry = fmaf(2.f, y2, r2), rx = fmaf(2.f, x2, r2);
    a.d[6] += fmaf(xy2, g1x, ry * g1y);
    a.d[7] += fmaf(rx, g1x, xy2 * g1y);
    // J_m^T g1
    const float wq = 2.f * drad * q;
    const float j01 = 2.f * fmaf(d.p1, x, d.p2 * y);  // the off-diagonal tangential term
    const float gmx = fmaf(rad + fmaf(2.f * d.p1, y, 6.f * d.p2 * x), g1x, fmaf(j01, g1y, x * wq));
    const float gmy = fmaf(rad + fmaf(6.f * d.p1, y, 2.f * d.p2 * x), g1y, fmaf(j01, g1x, y * wq));
    // divide by z, rigid transform
    V3 gv;
    gv.x = iz * gmx;
    gv.y = iz * gmy;
    gv.z = -fmaf(x, gv.x, y * gv.y);
    const V3 gp = rotate_inv(V, gv);
    a.pose[0] += gv.x; a.pose[1] += gv.y; a.pose[2] += gv.z;
    a.pose[3] += fmaf(view.y, gv.z, -view.z * gv.y);
    a.pose[4] += fmaf(view.z, gv.x, -view.x * gv.z);
    a.pose[5] += fmaf(view.x, gv.y, -view.y * gv.x);
    a.cnt += it.count;
    if (grad_points) atomicAdd(grad_points + it.id, make_float4(gp.x, gp.y, gp.z, it.count));
}

// General form (used for the omnidirectional model): chain of one point's summed image-space gradient (already scaled
// to full resolution) with `count` contributions, through the Jacobian functions of the arithmetic header.
template <int MODEL>
__device__ __forceinline__ bool chain_gradient_sum(const ViewCam& cam, const KernelParams& kp, const FetchedPoint& f, V2 g, float count,
                                                   float* gp, GeoAccum<MODEL>& acc)
{
    static_assert(MODEL == kOcam, "the pinhole model takes chain_pinhole_fast");
    GradOcam o;
    if (!project_ocam_backward(f.p, f.n, f.has_normal, g, cam.V, cam.crop, cam.ocam, kp.check_normal != 0, kp.dist_cutoff, &o))
        return false;
    gp[0] = o.g_point[0]; gp[1] = o.g_point[1]; gp[2] = o.g_point[2]; gp[3] = count;
#pragma unroll
    for (int k = 0; k < 6; ++k) acc.pose[k] += o.g_pose[k];
#pragma unroll
    for (int k = 0; k < 5; ++k) acc.intr[k] += o.g_affine[k];
    acc.cnt += count;
    return true;
}

// part of k_chain_and_holes: `block` of `blocks` thread blocks
// The reference adds the pose gradient in double (PointRenderer.cu:1113). Here a lane adds kPoseRun items in float32 before the warp's sum
// goes to the block's doubles, however many items fall to a block: with the views of a batch in one launch a lane can meet
// hundreds (350 equal terms added in float32 were 4.5e-6 off). It costs nothing measurable: chain and holes of the 16-view
// 1080p step 848 us with the sums kept to the end, 818 us so.
constexpr int kPoseRun = 16;
template <int MODEL>
__device__ __forceinline__ void point_chain_part(const PointStreams& pts, const ViewCam* __restrict__ camp, const ViewRows* __restrict__ rows,
                                                 int intrinsics_cols, const KernelParams& kp, const BackwardTargets& bt,
                                                 const VisibleList& vl, const TileTable& tt, int block, int blocks)
{
    __shared__ ViewCam s_cam;
    __shared__ GeoShared<MODEL> s_geo;
    // points with a gradient are parked per warp, with their position, and chained 32 at a time with every lane busy
    __shared__ ChainItem s_park[kBlock / 32][96];
    ChainItem* park = s_park[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    int n_parked = 0;
    for (int k = threadIdx.x; k < (int)(sizeof(ViewCam) / 4); k += kBlock) reinterpret_cast<int*>(&s_cam)[k] = __ldg(reinterpret_cast<const int*>(camp) + k);
    geo_shared_init(&s_geo);
    __syncthreads();
    const ViewCam& cam = s_cam;
    const bool check_normal = kp.check_normal != 0 && pts.normal != nullptr;
    GeoAccum<MODEL> acc;
    acc.clear();
    PinholeSums ps;
#pragma unroll
    for (int k = 0; k < 6; ++k) ps.pose[k] = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) ps.k[k] = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) ps.d[k] = 0.f;
    ps.cnt = 0.f;
    auto chain_one = [&](const ChainItem& it)
    {
        if (MODEL == kPinholeDistortion)
            chain_pinhole_fast(cam, check_normal, it, bt.grad_points, ps);
        else
        {
            FetchedPoint f;
            f.p.x = it.px; f.p.y = it.py; f.p.z = it.pz; f.r = 0.f;
            f.has_normal = pts.normal != nullptr;
            f.n = unpack_normal_10bit(it.normal);
            V2 g; g.x = it.gx; g.y = it.gy;
            float gp[4];
            if (chain_gradient_sum<kOcam>(cam, kp, f, g, it.count, gp, reinterpret_cast<GeoAccum<kOcam>&>(acc)) && bt.grad_points)
                atomicAdd(bt.grad_points + it.id, make_float4(gp[0], gp[1], gp[2], gp[3]));
        }
    };
    int run = 0;  // the same in every lane of the warp
    auto move_pose_sums = [&]()
    {
        if (!bt.grad_pose) return;
        float* pose = MODEL == kPinholeDistortion ? ps.pose : acc.pose;
#pragma unroll
        for (int k = 0; k < 6; ++k)
        {
            const float v = warp_sum(pose[k]);
            if (lane == 0) atomicAdd(&s_geo.pose[k], (double)v);
            pose[k] = 0.f;
        }
    };
    constexpr int U = 2;  // items per thread and round: their dependent loads (item -> position) are in flight together
    for (int tile = block; tile < tt.n_tiles; tile += blocks)
    {
        const int total = min(__ldg(vl.tile_cur + tile), tt.cap);
        const float4* work = reinterpret_cast<const float4*>(vl.entries + (size_t)tile * tt.cap);  // the tile kernel's work items
        for (int k0 = 0; k0 < total; k0 += kBlock * U)  // warp-uniform trip count
        {
            float4 v[U], p[U];
            int nrm[U];
#pragma unroll
            for (int j = 0; j < U; ++j)
            {
                const int k = k0 + j * kBlock + threadIdx.x;
                v[j] = k < total ? __ldcs(work + k) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int j = 0; j < U; ++j)
            {
                p[j] = make_float4(0.f, 0.f, 0.f, 0.f); nrm[j] = 0;
                if (v[j].w > 0.f)
                {
                    const int id = __float_as_int(v[j].x);
                    p[j] = __ldg(pts.position + id);
                    if (pts.normal) nrm[j] = __ldg(pts.normal + id);
                }
            }
#pragma unroll
            for (int j = 0; j < U; ++j)
            {
                const bool has = v[j].w > 0.f;
                const unsigned vote = __ballot_sync(0xffffffffu, has);
                if (has)
                {
                    ChainItem& it = park[n_parked + __popc(vote & ((1u << lane) - 1u))];
                    it.id = __float_as_int(v[j].x); it.gx = v[j].y; it.gy = v[j].z; it.count = v[j].w;
                    it.px = p[j].x; it.py = p[j].y; it.pz = p[j].z; it.normal = nrm[j];
                }
                n_parked += __popc(vote);
            }
            __syncwarp();
            while (n_parked >= 32)
            {
                n_parked -= 32;
                chain_one(park[n_parked + lane]);
                if (++run == kPoseRun) { move_pose_sums(); run = 0; }
            }
            __syncwarp();
        }
    }
    if (lane < n_parked) chain_one(park[lane]);
    if (MODEL == kPinholeDistortion)
    {
        // into the common form, with the damping of PointRenderer.cu:647-678 (skew gets no gradient)
        const float kf = kp.K_gradient_factor, df = kp.distortion_gradient_factor;
#pragma unroll
        for (int k = 0; k < 6; ++k) acc.pose[k] = ps.pose[k];
        acc.intr[0] = kf * ps.k[0]; acc.intr[1] = kf * ps.k[1]; acc.intr[2] = kf * ps.k[2]; acc.intr[3] = kf * ps.k[3];
        acc.intr[5] = df * ps.d[0]; acc.intr[6] = df * ps.d[1]; acc.intr[7] = df * (ps.d[2] * 0.25f);
        acc.intr[8] = df * (ps.d[3] * 0.1f); acc.intr[9] = df * (ps.d[4] * 0.1f); acc.intr[10] = df * (ps.d[5] * 0.1f);
        acc.intr[11] = df * (ps.d[6] * 0.1f); acc.intr[12] = df * (ps.d[7] * 0.1f);
        acc.cnt = ps.cnt;
    }
    geo_block_reduce<MODEL>(&s_geo, acc, bt, __ldg(&rows->image), __ldg(&rows->camera), intrinsics_cols);
}

// The chain kernel and the hole kernel of the launch's views: they are independent, the first waits on memory most of
// the time and the second on arithmetic, so side by side they take little more than the longer of the two.
// blockIdx.y = view; blocks x of [0, chain_blocks) chain the tile kernel's work items, the others walk the uncovered pixels.
// The views of a launch share the camera model; each view's rows of the pose and intrinsics gradients come from the row
// table that k_build_cams left behind the camera records.
template <int C, int MODEL>
__global__ void __launch_bounds__(kBlock, MODEL == kPinholeDistortion ? 4 : 3)
    k_chain_and_holes(PointStreams pts, const ViewCam* __restrict__ cams, const ViewRows* __restrict__ rows, KernelParams kp, LayerTable lt, BackwardTargets bt,
                      int intrinsics_cols, ViewLists lists, TileTable tt, HoleArgs ha, int chain_blocks)
{
    const int view = (int)blockIdx.y;
    const VisibleList vl = list_of_view(lists.first, lists.view_ints, view);
    if (__ldg(vl.header + kListGo) == 0) return;  // the all-points kernels do this work
    if ((int)blockIdx.x < chain_blocks)
        point_chain_part<MODEL>(pts, cams + view, rows + view, intrinsics_cols, kp, bt, vl, tt, (int)blockIdx.x, chain_blocks);
    else
        hole_gradients_part<C>(lt, view, cams + view, kp, ha, (int)blockIdx.x - chain_blocks, (int)gridDim.x - chain_blocks);
}

// Behind the visible lists: the end of the pass. A view that ran on its list only has the list marked as consumed when its
// entries were turned into work items; for a view whose list was not usable the whole launch walks all points. Nearly always
// there is nothing to do, and a launch per view and step for nothing was 32 of the 130 launches of a 16-view training step; but
// no block may wait for another one either (a launch whose blocks do has to fit the GPU at once, which a part of it, an MPS
// share or a green context, refuses). So
//  * up to four channels (kBehindFromPlanes) everything is one launch for all views, which takes pixels and holes straight
//    from the planes: they fit L2, and 16 views of 10 M points at 1080p take 13.3 ms (15.3 ms from records);
//  * with more channels they do not fit, and a visit would fetch 54 sectors instead of 10 (two views of 3 M points at 1080p,
//    16 channels: 2.8 ms, from records 1.9 ms). There a launch that prepares the records goes before, and as many views share
//    the two as the workspace has room for records.
template <int C> constexpr bool kBehindFromPlanes = C <= 4;
struct RecordSpace
{
    float* first;        // records of the launch's first view
    size_t view_floats;  // distance from view to view
};
template <int C>
__global__ void __launch_bounds__(kBlock) k_prepare_behind_lists(LayerTable lt, const ViewCam* __restrict__ cams, KernelParams kp, const float* __restrict__ background,
                                                                  ViewLists lists, RecordSpace records, HoleArgs ha)
{
    const int view = (int)blockIdx.y;
    if (__ldg(list_of_view(lists.first, lists.view_ints, view).header + kListGo) != 0) return;
    prepare_backward_part<C>(lt, view, cams[view], kp, background, records.first + view * records.view_floats, ha);
}
template <int C, int MODEL>
__global__ void __launch_bounds__(kBlock) k_behind_lists(PointStreams pts, const ViewCam* __restrict__ cams, const ViewRows* __restrict__ rows, KernelParams kp,
                                                          LayerTable lt, BackwardTargets bt, int intrinsics_cols, ViewLists lists, RecordSpace records, HoleArgs ha,
                                                          int views, int mark_consumed)
{
    for (int view = 0; view < views; ++view)
    {
        int* header = list_of_view(lists.first, lists.view_ints, view).header;
        if (__ldg(header + kListGo) != 0)  // the same in every block: written by an earlier kernel
        {
            if (mark_consumed && blockIdx.x == 0 && threadIdx.x == 0) header[kListConsumed] = 1;
            continue;
        }
        if (kBehindFromPlanes<C> && (ha.grad_background || ha.grad_env))
            hole_gradients_part<C>(lt, view, cams + view, kp, ha, (int)blockIdx.x, (int)gridDim.x);
        splat_backward_part<C, MODEL, !kBehindFromPlanes<C>>(pts, cams[view], kp, lt, view, bt, records.first + view * records.view_floats, rows[view].image,
                                                             rows[view].camera, intrinsics_cols);
        __syncthreads();  // the next view starts its block sums anew
    }
}

// ------------------------------------------------------------------------------------------------------
// NormalizeGradient, PointRenderer.cu:1534-1547
__global__ void k_normalize_points(float4* g, int n)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    // a point without contributions (w = 0) stays as it is: on a large cloud most points, and then whole sectors, are not
    // written back
    float4 v = g[i];
    if (v.w == 0.f) return;
    if (v.w > 0.f) { v.x = v.x / v.w; v.y = v.y / v.w; v.z = v.z / v.w; }
    v.w = 0.f;
    g[i] = v;
}
__global__ void k_normalize_pose(double* g, const float* cnt, int n)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * 6) return;
    float c = cnt[i / 6];
    if (c > 0.f) g[i] = g[i] / (double)c;
}
__global__ void k_normalize_intrinsics(float* g, const float* cnt, int n, int cols)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * cols) return;
    float c = cnt[i / cols];
    if (c > 0.f) g[i] = g[i] / c;
}

// ------------------------------------------------------------------------------------------------------
constexpr int kTileWaves = 2;
static int blocks_per_view(int resident, int waves, int views, int most)
{
    int n = (resident * waves + views - 1) / views;
    if (n > most) n = most;
    return n < 1 ? 1 : n;
}

// The list kernels of `views` consecutive views of one camera model. lt, kp, cams, rows and lists are those of the first;
// bt's pose and intrinsics rows are the tensors' first rows; records: room for record_views views.
template <int C, int MODEL>
static adop_status launch_list_backward(const PointStreams& pts, const ViewCam* cams, const ViewRows* rows, const KernelParams& kp, const LayerTable& lt,
                                        const TileTable& tt, const BackwardTargets& bt, float* records, int record_views, int intrinsics_cols,
                                        const HoleArgs& ha, cudaStream_t st, const ViewLists& lists, int views)
{
    const int want_geo = (bt.grad_points || bt.grad_pose || bt.grad_intrinsics) ? 1 : 0;
    const size_t smem = tile_smem_bytes(C, lt.L);
    const bool deep = lt.L > 4;
    static OncePerDevice smem_set[2];  // (the kernel decides the size: one value for each)
    int device = 0;
    ADOP_CUDA_TRY(cudaGetDevice(&device));
    ADOP_CUDA_TRY(smem_set[deep].run(device, [&] {
        return deep ? cudaFuncSetAttribute(k_backward_tiles<C, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
                    : cudaFuncSetAttribute(k_backward_tiles<C, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    }));
    int per_sm = 0;
    cudaError_t oe = deep ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_backward_tiles<C, true>, kTileThreads, smem)
                          : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_backward_tiles<C, false>, kTileThreads, smem);
    if (oe != cudaSuccess || per_sm < 1) per_sm = 1;
    // blocks per view: about kTileWaves times as many blocks as are resident, so that the GPU's own block scheduler evens
    // out crowded and empty tiles, but never more than a view has tiles
    const dim3 grid_tiles((unsigned)blocks_per_view(per_sm * sm_count(), kTileWaves, views, tt.n_tiles), (unsigned)views);
    if (deep) ADOP_LAUNCH("k_backward_tiles", st, (k_backward_tiles<C, true><<<grid_tiles, kTileThreads, smem, st>>>(pts, kp, lt, tt, bt, lists, want_geo)));
    else ADOP_LAUNCH("k_backward_tiles", st, (k_backward_tiles<C, false><<<grid_tiles, kTileThreads, smem, st>>>(pts, kp, lt, tt, bt, lists, want_geo)));
    static const int g = resident_grid(k_chain_and_holes<C, MODEL>, 1ll << 40);
    const unsigned groups = (lt.rec_off[kMaxLayers] + 3) / 4;
    const int hole_need = (ha.grad_env || ha.grad_background) ? (int)((groups + kBlock - 1) / kBlock) : 0;
    if (hole_need || want_geo)
    {
        // The resident blocks are shared out over the views, rounded down: a handful of blocks over that (three views, 198 x 3
        // blocks in 592 places) run alone at the end, at twice the time (1080p, six million points: 336 us, rounded down 185). The chain
        // blocks get five eighths of a view's blocks when both parts have work (between a half and three quarters the kernel's
        // time is flat, beyond it rises quickly). Where a chain block would walk many tiles, which differ in their points, four times
        // as many blocks even that out. One row of blocks : four, by tiles per chain block: 44 (1080p, four views) 254 : 277 us, 66 (six) 339 : 371,
        // 78 (1280 x 720, sixteen) 372 : 371, 88 (1080p, eight; eight channels) 665 : 599, 177 (sixteen, four channels) 936 : 850, 176 (four at
        // 4K, eight channels) 2134 : 1466.
        // Below that, two to four views keep two rows: crops of a training batch differ in their points, and blocks that are done early leave
        // room for the next view's (four 512 x 512 crops, whole step with one row 428 us, with two 409 us), though views that are alike lose by it
        // (1080p, two views 136 : 160 us, four 254 : 268).
        const auto chain_share = [&](int blocks) { return want_geo ? (hole_need ? blocks * 5 / 8 : blocks) : 0; };
        const int one_row = std::max(1, g / views);
        const int rows_of_blocks = tt.n_tiles > 80 * std::max(1, chain_share(one_row)) ? 4 : (views >= 2 && views <= 4 ? 2 : 1);
        const int per_view = std::max(1, g * rows_of_blocks / views);
        int chain_blocks = chain_share(per_view);
        if (want_geo && chain_blocks < 1) chain_blocks = 1;
        if (chain_blocks > tt.n_tiles) chain_blocks = tt.n_tiles;
        int hole_blocks = per_view - chain_blocks < hole_need ? per_view - chain_blocks : hole_need;
        if (hole_need && hole_blocks < 1) hole_blocks = 1;
        ADOP_LAUNCH("k_chain_and_holes", st, (k_chain_and_holes<C, MODEL><<<dim3((unsigned)(chain_blocks + hole_blocks), (unsigned)views), kBlock, 0, st>>>(
                                                 pts, cams, rows, kp, lt, bt, intrinsics_cols, lists, tt, ha, chain_blocks)));
    }
    static const int g_behind = resident_grid(k_behind_lists<C, MODEL>, 1ll << 40);
    const int together = kBehindFromPlanes<C> ? views : record_views;
    for (int v = 0; v < views; v += together)
    {
        const int n = views - v < together ? views - v : together;
        const LayerTable ltv = layer_table_of_view(lt, C, v);
        KernelParams kv = kp;
        kv.batch_slot += v;
        if (kv.dropout_mask) kv.dropout_mask += (size_t)v * pts.n;
        ViewLists lv = lists;
        lv.first = list_of_view(lists.first, lists.view_ints, v);
        const RecordSpace rs = {records, (size_t)lt.rec_off[kMaxLayers] * backward_record_floats(C)};
        if (!kBehindFromPlanes<C>)
        {
            static const int g_prepare = resident_grid(k_prepare_behind_lists<C>, 1ll << 40);
            const dim3 grid((unsigned)blocks_per_view(g_prepare, 1, n, (int)((lt.rec_off[kMaxLayers] + kBlock - 1) / kBlock)), (unsigned)n);
            ADOP_LAUNCH("k_prepare_behind_lists", st, (k_prepare_behind_lists<C><<<grid, kBlock, 0, st>>>(ltv, cams + v, kv, bt.background, lv, rs, ha)));
        }
        ADOP_LAUNCH("k_behind_lists", st, (k_behind_lists<C, MODEL><<<g_behind, kBlock, 0, st>>>(pts, cams + v, rows + v, kv, ltv, bt, intrinsics_cols, lv, rs, ha, n, want_geo)));
    }
    ADOP_CUDA_TRY(cudaGetLastError());
    return ADOP_OK;
}

// The backward pass of one view without a list.
template <int C, int MODEL>
static adop_status launch_all_points_backward(const PointStreams& pts, const ViewCam* cam, const ViewRows* rows, const KernelParams& kp, const LayerTable& lt,
                                              const BackwardTargets& bt, float* records, int intrinsics_cols, const HoleArgs& ha, cudaStream_t st)
{
    static const int g_prepare = resident_grid(k_prepare_backward<C>, 1ll << 40);
    static const int g_splat = resident_grid(k_splat_backward_all<C, MODEL>, 1ll << 40);
    const int need = (pts.n + kBlock - 1) / kBlock, need_px = (int)((lt.rec_off[kMaxLayers] + kBlock - 1) / kBlock);
    ADOP_LAUNCH("k_prepare_backward", st, (k_prepare_backward<C><<<need_px < g_prepare ? need_px : g_prepare, kBlock, 0, st>>>(lt, cam, kp, bt.background, records, ha)));
    ADOP_LAUNCH("k_splat_backward_all", st, (k_splat_backward_all<C, MODEL><<<need < g_splat ? (need < 1 ? 1 : need) : g_splat, kBlock, 0, st>>>(
                                                pts, cam, rows, kp, lt, bt, records, intrinsics_cols)));
    ADOP_CUDA_TRY(cudaGetLastError());
    return ADOP_OK;
}

// `views` consecutive views of one camera model, with lists or without; the pointers are the first view's.
template <int C, int MODEL>
static adop_status launch_views_backward(const PointStreams& pts, const ViewCam* cams, const ViewRows* rows, const KernelParams& kp, const LayerTable& lt,
                                         const TileTable& tt, const BackwardTargets& bt, float* records, int record_views, int intrinsics_cols,
                                         const HoleArgs& ha, cudaStream_t st, const ViewLists& lists, int views)
{
    if (lists.first.header) return launch_list_backward<C, MODEL>(pts, cams, rows, kp, lt, tt, bt, records, record_views, intrinsics_cols, ha, st, lists, views);
    for (int v = 0; v < views; ++v)
    {
        KernelParams kv = kp;
        kv.batch_slot += v;
        if (kv.dropout_mask) kv.dropout_mask += (size_t)v * pts.n;
        const adop_status r = launch_all_points_backward<C, MODEL>(pts, cams + v, rows + v, kv, layer_table_of_view(lt, C, v), bt, records, intrinsics_cols, ha, st);
        if (r != ADOP_OK) return r;
    }
    return ADOP_OK;
}

}  // namespace adop

using namespace adop;

extern "C" adop_status adop_raster_normalize_gradients(float* grad_points, int32_t num_points, double* grad_pose,
                                                       const float* count_pose, int32_t num_images, float* grad_intrinsics,
                                                       const float* count_intrinsics, int32_t num_cameras,
                                                       int32_t intrinsics_cols, void* stream)
{
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (grad_pose)
    {
        if (!count_pose || num_images <= 0) return ADOP_ERR_INVALID_ARGUMENT;
        int n = num_images * 6;
        ADOP_LAUNCH("k_normalize", st, (k_normalize_pose<<<(n + 127) / 128, 128, 0, st>>>(grad_pose, count_pose, num_images)));
    }
    if (grad_points && num_points > 0)
        ADOP_LAUNCH("k_normalize", st, (k_normalize_points<<<(num_points + 255) / 256, 256, 0, st>>>(reinterpret_cast<float4*>(grad_points), num_points)));
    if (grad_intrinsics)
    {
        if (!count_intrinsics || num_cameras <= 0 || intrinsics_cols <= 0) return ADOP_ERR_INVALID_ARGUMENT;
        int n = num_cameras * intrinsics_cols;
        ADOP_LAUNCH("k_normalize", st, (k_normalize_intrinsics<<<(n + 127) / 128, 128, 0, st>>>(grad_intrinsics, count_intrinsics, num_cameras, intrinsics_cols)));
    }
    ADOP_CUDA_TRY(cudaGetLastError());
    return ADOP_OK;
}

extern "C" adop_status adop_raster_backward(const adop_scene* s, const adop_view* views, int32_t B,
                                            const adop_render_params* rp, int32_t L, adop_backward_io* io, void* stream)
{
    adop_status vs = validate_common(s, views, B, rp, L);
    if (vs != ADOP_OK) return vs;
    if (!io) return ADOP_ERR_INVALID_ARGUMENT;
    const int C = s->channels, N = s->num_points, T = s->num_texels, cols = s->intrinsics_cols;
    for (int l = 0; l < L; ++l)
        if (!io->layers[l].color || !io->layers[l].depth || !io->layers[l].weight || !io->grad_color[l])
            return ADOP_ERR_INVALID_ARGUMENT;
    if ((io->grad_pose && !io->count_pose) || (io->grad_intrinsics && !io->count_intrinsics)) return ADOP_ERR_INVALID_ARGUMENT;
    if (reinterpret_cast<uintptr_t>(io->grad_points) & 15) return ADOP_ERR_INVALID_ARGUMENT;
    if (!io->workspace || (reinterpret_cast<uintptr_t>(io->workspace) & 15)) return ADOP_ERR_INVALID_ARGUMENT;
    if (io->workspace_bytes < adop_raster_workspace_bytes(views[0].w, views[0].h, L, C)) return ADOP_ERR_WORKSPACE_TOO_SMALL;
    const bool env = rp->composite_environment_map && s->env_map && io->grad_env_map;
    if (env)
        for (int b = 0; b < B; ++b)
            if (views[b].camera_model != ADOP_CAMERA_PINHOLE_DISTORTION) return ADOP_ERR_UNSUPPORTED;

    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // environment-map gradient: summed in an [eh,ew,C] scratch with vector atomics when the caller gave one
    const bool env_inter = env && io->grad_env_map_interleaved && C % 4 == 0 &&
                           (reinterpret_cast<uintptr_t>(io->grad_env_map_interleaved) & 15) == 0;
    // descriptor gradients stay in the [T,C] buffer when there is no [C,T] tensor to move them into
    const bool interleaved_only = !io->grad_texture && io->grad_texture_interleaved;
    FillTable fills;
    if (!io->accumulate)
    {
        if (!io->grad_texture_interleaved) fills.add(io->grad_texture, (size_t)C * T, 0u);
        fills.add(io->grad_background, (size_t)C, 0u);
        fills.add(io->grad_points, (size_t)N * 4, 0u);
        fills.add(io->grad_pose, (size_t)s->num_images * 12, 0u);
        fills.add(io->count_pose, (size_t)s->num_images, 0u);
        fills.add(io->grad_intrinsics, (size_t)s->num_cameras * cols, 0u);
        fills.add(io->count_intrinsics, (size_t)s->num_cameras, 0u);
        if (s->env_h > 0 && s->env_w > 0 && !env_inter) fills.add(io->grad_env_map, (size_t)C * s->env_h * s->env_w, 0u);
    }
    if (env_inter) fills.add(io->grad_env_map_interleaved, (size_t)C * s->env_h * s->env_w, 0u);
    if (io->grad_texture || !io->accumulate) fills.add(io->grad_texture_interleaved, (size_t)C * T, 0u);
    const adop_status fs = launch_fills(fills, st);
    if (fs != ADOP_OK) return fs;
    LayerTable base;
    fill_layer_dims(views[0].w, views[0].h, L, &base);
    const TileTable tiles = make_tile_table(views[0].w, views[0].h, N);
    ViewCam* cams = static_cast<ViewCam*>(io->workspace);
    PointStreams pts;
    pts.position = reinterpret_cast<const float4*>(s->position);
    pts.normal = s->normal;
    pts.index = s->index;
    pts.n = N;
    // The debug stencil rule (test_backward_mode 4) needs the point's depth next to its neighbours' and always takes the
    // all-points kernels.
    const bool use_list = io->visible_list && rp->test_backward_mode != 4;
    float* ge = env ? (env_inter ? io->grad_env_map_interleaved : io->grad_env_map) : nullptr;
    BackwardTargets bt;
    bt.texture = s->texture;
    bt.texture_interleaved = s->texture_interleaved;
    bt.grad_texture_interleaved = io->grad_texture_interleaved;
    bt.num_texels = T;
    bt.background = s->background;
    // the kernels take a non-null grad_texture as "descriptor gradients wanted" and write the [T,C] buffer if there is one
    bt.grad_texture = interleaved_only ? io->grad_texture_interleaved : io->grad_texture;
    bt.grad_points = reinterpret_cast<float4*>(io->grad_points);
    bt.grad_pose = io->grad_pose;
    bt.count_pose = io->grad_pose ? io->count_pose : nullptr;
    bt.grad_intrinsics = io->grad_intrinsics;
    bt.count_intrinsics = io->grad_intrinsics ? io->count_intrinsics : nullptr;
    // the workspace holds the records of one view at least
    float* records = reinterpret_cast<float*>(static_cast<char*>(io->workspace) + kCamRegionBytes);
    const size_t record_bytes = (size_t)base.rec_off[kMaxLayers] * backward_record_floats(C) * sizeof(float);
    const size_t record_room = (io->workspace_bytes - kCamRegionBytes) / record_bytes;
    const int record_views = (int)(record_room < kCamChunk ? record_room : kCamChunk);
    for (int l = 0; l < L; ++l)
    {
        base.depth[l] = io->layers[l].depth;
        base.weight[l] = io->layers[l].weight;
        base.color[l] = io->layers[l].color;
        base.grad[l] = io->grad_color[l];
    }
    const ViewRows* rows = view_rows(cams);
    for (int b0 = 0; b0 < B; b0 += kCamChunk)
    {
        const int chunk = B - b0 < kCamChunk ? B - b0 : kCamChunk;
        CamChunkSource src;
        fill_cam_chunk(&src, s, views + b0, chunk);
        ADOP_LAUNCH("k_build_cams", st, (k_build_cams<<<1, kCamChunk, 0, st>>>(src, cams)));
        HoleArgs ha;
        ha.grad_background = io->grad_background; ha.grad_env = ge; ha.env_h = s->env_h; ha.env_w = s->env_w; ha.env_interleaved = env_inter;
        // runs of consecutive views with the same camera model
        for (int b = b0, e; b < b0 + chunk; b = e)
        {
            for (e = b + 1; e < b0 + chunk && views[e].camera_model == views[b].camera_model; ++e) {}
            ViewLists lists;
            // the list's layout (tiles, bucket size) follows from the view size and the point count, as in the forward pass
            lists.first = make_visible_list(use_list ? const_cast<int32_t*>(io->visible_list) : nullptr, N, views[0].w, views[0].h, b);
            lists.view_ints = visible_list_ints(N, views[0].w, views[0].h);
            const LayerTable lt = layer_table_of_view(base, C, b);
            const KernelParams kp = make_kernel_params(rp, io->dropout_mask, N, b);
            const bool pinhole = views[b].camera_model == kPinholeDistortion;
            const ViewCam* cam = cams + (b - b0);
            const ViewRows* row = rows + (b - b0);
            adop_status r;
#define ADOP_VIEWS_BACKWARD(CC)                                                                                                                      \
    r = pinhole ? launch_views_backward<CC, kPinholeDistortion>(pts, cam, row, kp, lt, tiles, bt, records, record_views, cols, ha, st, lists, e - b)               \
                : launch_views_backward<CC, kOcam>(pts, cam, row, kp, lt, tiles, bt, records, record_views, cols, ha, st, lists, e - b)
            switch (C)
            {
                case 3: ADOP_VIEWS_BACKWARD(3); break;
                case 4: ADOP_VIEWS_BACKWARD(4); break;
                case 8: ADOP_VIEWS_BACKWARD(8); break;
                case 16: ADOP_VIEWS_BACKWARD(16); break;
                default:
                    snprintf(last_error_buffer(), 512, "%d descriptor channels: the kernels are built for 3, 4, 8 and 16", C);
                    return ADOP_ERR_UNSUPPORTED;
            }
#undef ADOP_VIEWS_BACKWARD
            if (r != ADOP_OK) return r;
        }
    }
    if (io->grad_texture && io->grad_texture_interleaved)
    {
        adop_status ds = adop_texture_deinterleave(io->grad_texture_interleaved, io->grad_texture, C, T, io->accumulate ? 1 : 0, stream);
        if (ds != ADOP_OK) return ds;
    }
    if (env_inter)
    {
        // [eh,ew,C] -> [C,eh,ew]
        adop_status ds = adop_texture_deinterleave(io->grad_env_map_interleaved, io->grad_env_map, C, s->env_h * s->env_w, io->accumulate ? 1 : 0, stream);
        if (ds != ADOP_OK) return ds;
    }
    if (io->normalize)
        return adop_raster_normalize_gradients(io->grad_points, N, io->grad_pose, io->count_pose, s->num_images,
                                               io->grad_intrinsics, io->count_intrinsics, s->num_cameras, cols, stream);
    return ADOP_OK;
}

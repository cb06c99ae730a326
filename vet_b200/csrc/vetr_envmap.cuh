// Texture environment map kernels: EnvironmentMapImpl::Sample2 / forward_mps5 (rendering/EnvironmentMap.cu:378-485,
// 692-758) as one forward and one backward kernel over all views, levels and pixels.
//
// The reference builds a ray list (BuildSphericalRayList, :201-287), writes sample coordinates for every sphere
// (CreateSampleUVMapAllSpheres, :587-684), calls grid_sample twice on [S * rays] coordinates, and then runs about ten
// element-wise libtorch operators per sphere; autograd replays all of it backwards.  Here a thread owns a pixel: ray,
// sphere hits, the trilinear fetches of grid_sample (bilinear, zero padding, align_corners) and the front-to-back
// chain stay in registers; per pixel the forward kernel reads 4 bytes (the transmittance) and writes 4 C bytes, and the
// textures (S R^2 (C + 1) floats) are shared by all pixels through L2.
//
// The arithmetic is written operation for operation like the CPU restatement the tests compare with (the build uses
// -fmad=false, so nothing is contracted); asinf, atan2f and expf are the device's own.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>

#include "vetr_math.cuh"

namespace vetr
{
constexpr int kEnvMaxSpheres = 8;  // MAX_NUM_SPHERES, EnvironmentMap.cu:91
constexpr int kEnvThreads    = 256, kEnvBackThreads = 128;

struct EnvView
{
    int image_index, camera_index;
    float crop[5];
    float rot[4];
};

struct EnvArgs  // kernel parameter block
{
    int n_views, L, S, R, C, up_axis, non_subzero, flags;
    int lw[VETR_MAX_LAYERS], lh[VETR_MAX_LAYERS];
    float inv_lw[VETR_MAX_LAYERS];
    int lend[VETR_MAX_LAYERS];        // pixels of levels 0..l over all views (running total; below 2^30)
    float scale[VETR_MAX_LAYERS];     // 0.5^l
    float radii[kEnvMaxSpheres];
    EnvView views[VETR_MAX_VIEWS];
    const double* poses;
    const float* intr;
    const float* density;  // [S,R,R]
    const float* color;    // [C,S,R,R]
    const float* weight[VETR_MAX_LAYERS];  // [n_views,1,h_l,w_l]
    float* out[VETR_MAX_LAYERS];           // [n_views,C,h_l,w_l]
    const float* grad[VETR_MAX_LAYERS];    // incoming gradient of out (backward)
    float* g_density;
    float* g_color;
};

struct EnvCam  // what a pixel needs of its view: camera -> world, intrinsics, inverse crop rotation
{
    Pose Vi;  // Sophus SE3::inverse: (q^-1, q^-1 * (-t))
    float K[5], crop[5], rinv[4];
};

__device__ __forceinline__ float3 rotate_vector(const Pose& P, float3 v)  // Eigen quaternion * vector
{
    float3 qv = make_float3(P.qx, P.qy, P.qz);
    float3 uv = cross3(qv, v);
    uv        = make_float3(uv.x + uv.x, uv.y + uv.y, uv.z + uv.z);
    float3 c  = cross3(qv, uv);
    return make_float3(v.x + P.qw * uv.x + c.x, v.y + P.qw * uv.y + c.y, v.z + P.qw * uv.z + c.z);
}

__device__ __forceinline__ EnvCam load_env_cam(const EnvArgs& a, int b)
{
    EnvCam c;
    const EnvView& v = a.views[b];
    const double* p  = a.poses + 8 * (long long)v.image_index;
    Pose V;
    V.qx = (float)p[0], V.qy = (float)p[1], V.qz = (float)p[2], V.qw = (float)p[3];
    V.tx = (float)p[4], V.ty = (float)p[5], V.tz = (float)p[6];
    c.Vi.qx = -V.qx, c.Vi.qy = -V.qy, c.Vi.qz = -V.qz, c.Vi.qw = V.qw;
    c.Vi.tx = c.Vi.ty = c.Vi.tz = 0.f;
    float3 ti = rotate_vector(c.Vi, make_float3(-V.tx, -V.ty, -V.tz));
    c.Vi.tx = ti.x, c.Vi.ty = ti.y, c.Vi.tz = ti.z;
    const float* k = a.intr + 13 * (long long)v.camera_index;
    for (int i = 0; i < 5; ++i) c.K[i] = k[i], c.crop[i] = v.crop[i];
    // Eigen's 2x2 inverse of crop_rotation
    const float det = v.rot[0] * v.rot[3] - v.rot[2] * v.rot[1];
    const float inv = 1.f / det;
    c.rinv[0] = v.rot[3] * inv, c.rinv[1] = -v.rot[1] * inv, c.rinv[2] = -v.rot[2] * inv, c.rinv[3] = v.rot[0] * inv;
    return c;
}

__device__ __forceinline__ float2 env_unproject2(const float* K, float2 ip)  // IntrinsicsPinhole::unproject2
{
    float y = (ip.y - K[3]) / K[1];
    float x = (ip.x - K[2] - K[4] * y) / K[0];
    return make_float2(x, y);
}

struct EnvRay
{
    float3 o, d;
    float q2a, qb, f;  // coefficients of the sphere intersection, EnvironmentMap.cu:616-618
};

// BuildSphericalRayList, pinhole branch (EnvironmentMap.cu:201-241): the origin is the pixel's point on the camera's
// z = 1 plane in world space, the direction points away from the eye.
__device__ __forceinline__ EnvRay env_ray(const EnvCam& c, int lw, int lh, float scale, int gx, int gy)
{
    const float cx = (float)(lw / 2), cy = (float)(lh / 2);
    const float dx = (float)gx - cx, dy = (float)gy - cy;
    float2 ip = make_float2(c.rinv[0] * dx + c.rinv[1] * dy, c.rinv[2] * dx + c.rinv[3] * dy);
    ip        = make_float2(ip.x + cx, ip.y + cy);
    float crop[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) crop[k] = c.crop[k] * scale;
    const float2 np = env_unproject2(c.K, env_unproject2(crop, ip));
    const float3 r  = rotate_vector(c.Vi, make_float3(np.x, np.y, 1.f));
    EnvRay ray;
    ray.o = make_float3(r.x + c.Vi.tx, r.y + c.Vi.ty, r.z + c.Vi.tz);
    float3 d = make_float3(ray.o.x - c.Vi.tx, ray.o.y - c.Vi.ty, ray.o.z - c.Vi.tz);
    const float n2 = d.x * d.x + d.y * d.y + d.z * d.z;
    if (n2 > 0.f)
    {
        const float n = sqrtf(n2);
        d = make_float3(d.x / n, d.y / n, d.z / n);
    }
    ray.d   = d;
    ray.q2a = 2.f * (d.x * d.x) + 2.f * (d.y * d.y) + 2.f * (d.z * d.z);
    ray.qb  = 2.f * (ray.o.x * d.x) + 2.f * (ray.o.y * d.y) + 2.f * (ray.o.z * d.z);
    ray.f   = ray.qb * ray.qb - 2.f * ray.q2a * (ray.o.x * ray.o.x + ray.o.y * ray.o.y + ray.o.z * ray.o.z);
    return ray;
}

__device__ __forceinline__ float env_unnormalize(float c, int size) { return ((c + 1.f) / 2.f) * (float)(size - 1); }

// CreateSampleUVMapAllSpheres for one sphere (EnvironmentMap.cu:620-682): texel coordinates of the ray's sample, false if
// the ray misses the sphere.
__device__ __forceinline__ bool env_coordinates(const EnvArgs& a, const EnvRay& ray, int s, float& ix, float& iy)
{
    float3 sv = ray.d;
    if (s != a.S - 1)
    {
        const float r   = a.radii[s];
        const float det = ray.f + 2.f * ray.q2a * (r * r);
        if (!(det >= 0.f)) return false;
        const float res = (-ray.qb + sqrtf(det)) / ray.q2a;
        const float3 p  = make_float3(ray.o.x + res * ray.d.x, ray.o.y + res * ray.d.y, ray.o.z + res * ray.d.z);
        const float len = sqrtf(p.x * p.x + p.y * p.y + p.z * p.z);
        sv = make_float3(p.x / len, p.y / len, p.z / len);
    }
    const float pi = 3.14159265358979323846f;
    float la, lb, lc;  // lat = asin(la), lon = atan2(lb, lc)
    if (a.up_axis == 0) la = sv.x, lb = sv.y, lc = sv.z;
    else if (a.up_axis == 1) la = sv.y, lb = sv.x, lc = sv.z;
    else la = sv.z, lb = sv.x, lc = sv.y;
    la = fminf(fmaxf(la, -1.f), 1.f);
    const float lat = asinf(la), lon = atan2f(lb, lc);
    const float u = 2.f * (lon / 2.f / pi);
    const float v = 2.f * (lat / pi);
    ix = env_unnormalize(u, a.R), iy = env_unnormalize(v, a.R);
    return true;
}

// Up to kEnvFlatSpheres spheres, grid_sample's third coordinate of sphere s, formed in fp32 as unnormalize(2 s / (S - 1) - 1),
// is s exactly: a sample lies on its slice, has four corners instead of eight, and offsets are taken inside the slice.  With
// six and more some come out beside the slice (0.99999994 for s = 1 of 6), and the neighbouring slice gets its share.
constexpr int kEnvFlatSpheres = 5;

// The corners of sphere s's sample: texel offset inside the slice (flat) or inside one [S,R,R] plane, and weight; outside the
// texture -1 and 0.  Corners of weight 0 read nothing, whatever the texel holds.
template <bool kFlat>
struct EnvCorners
{
    static constexpr int N = kFlat ? 4 : 8;
    int off[N];
    float w[N];
};

// Fills the corners and returns the base texel's index, which samples with the same corners share (`alone`, an index of the
// caller's, where the base texel lies outside the texture).
template <bool kFlat>
__device__ __forceinline__ int env_corners(const EnvArgs& a, float ix, float iy, int s, EnvCorners<kFlat>& c, int alone = -1)
{
    const float fx = floorf(ix), fy = floorf(iy);
    // the base texel, kept inside [-2, size] so that the int conversion and the + 1 of the far corners are defined for
    // every float (anything out there is outside the texture and reads zero either way)
    const int x0 = (int)fminf(fmaxf(fx, -2.f), (float)a.R), y0 = (int)fminf(fmaxf(fy, -2.f), (float)a.R);
    const float wx[2] = {(fx + 1.f) - ix, ix - fx}, wy[2] = {(fy + 1.f) - iy, iy - fy};
    int z0      = 0;
    float wz[2] = {1.f, 0.f};
    if (!kFlat)
    {
        const float iz = env_unnormalize((float)s / (float)(a.S - 1) * 2.f - 1.f, a.S);  // more than one sphere
        const float fz = floorf(iz);
        z0    = (int)fminf(fmaxf(fz, -2.f), (float)a.S);
        wz[0] = (fz + 1.f) - iz, wz[1] = iz - fz;
    }
    const int base = (z0 * a.R + y0) * a.R + x0;
    const bool inx[2] = {(unsigned)x0 < (unsigned)a.R, (unsigned)(x0 + 1) < (unsigned)a.R};
    const bool iny[2] = {(unsigned)y0 < (unsigned)a.R, (unsigned)(y0 + 1) < (unsigned)a.R};
#pragma unroll
    for (int q = 0; q < EnvCorners<kFlat>::N; ++q)
    {
        const int i = q & 1, j = q >> 1 & 1, k = q >> 2;
        const float w = kFlat ? wx[i] * wy[j] : wx[i] * wy[j] * wz[k];
        const bool in = inx[i] && iny[j] && (kFlat || (unsigned)(z0 + k) < (unsigned)a.S);
        c.off[q] = in ? base + (k * a.R + j) * a.R + i : -1;
        c.w[q]   = in ? w : 0.f;
    }
    return c.off[0] >= 0 ? base : alone;
}

template <bool kFlat>
__device__ __forceinline__ float env_fetch(const float* plane, const EnvCorners<kFlat>& c)
{
    float v[EnvCorners<kFlat>::N];
#pragma unroll
    for (int q = 0; q < EnvCorners<kFlat>::N; ++q) v[q] = c.w[q] != 0.f ? __ldg(plane + c.off[q]) : 0.f;
    float acc = 0.f;
#pragma unroll
    for (int q = 0; q < EnvCorners<kFlat>::N; ++q) acc += v[q] * c.w[q];
    return acc;
}

// Decodes a thread's pixel: level, view, x, y.  Pixels are numbered level by level, and inside a level view by view in
// row-major order, so that a warp covers 32 consecutive pixels of a row.
struct EnvPixelId
{
    int l, b, x, y;
    int pix;  // index inside the level's [n_views, h, w] plane
};

__device__ __forceinline__ bool env_locate(const EnvArgs& a, int idx, EnvPixelId& p)
{
    if (idx >= a.lend[a.L - 1]) return false;
    int l = 0;
    while (idx >= a.lend[l]) ++l;
    p.l   = l;
    p.pix = idx - (l == 0 ? 0 : a.lend[l - 1]);
    const int lw = a.lw[l], per_view = lw * a.lh[l];
    int b = 0, r = p.pix;
    for (; r >= per_view; r -= per_view) ++b;  // at most VETR_MAX_VIEWS - 1 steps
    // row: float estimate, then correction steps either way (the estimate is off by at most one up to 2^23 rows)
    int y = __float2int_rz((float)r * a.inv_lw[l]), x = r - y * lw;
    while (x < 0) x += lw, --y;
    while (x >= lw) x -= lw, ++y;
    p.b = b, p.x = x, p.y = y;
    return true;
}

__device__ __forceinline__ float env_start_T(float weight, int flags)
{
    return (flags & VETR_ENV_DEPTH_TEST_WEIGHT) ? (weight > 0.5f ? 0.f : 1.f) : weight;
}

// Bound by instruction issue (74 % of the slots, 2300 instructions per pixel and four spheres; 3400 with eight corners per sample, a
// test and a branch per corner and plane, and 64-bit divisions for the pixel).  1920x1080, four levels, four spheres of 1024 x 1024:
// 335 -> 231 us; five of 512 x 512 397 -> 266, eight of 1024 x 1024 661 -> 584.
template <bool kFlat>
__global__ void __launch_bounds__(kEnvThreads) envmap_forward_kernel(const __grid_constant__ EnvArgs a)
{
    __shared__ EnvCam s_cam[VETR_MAX_VIEWS];
    if (threadIdx.x < a.n_views) s_cam[threadIdx.x] = load_env_cam(a, threadIdx.x);
    __syncthreads();
    const long long plane = (long long)a.S * a.R * a.R, slice = kFlat ? (long long)a.R * a.R : 0;
    for (int idx = blockIdx.x * kEnvThreads + threadIdx.x; idx < a.lend[a.L - 1]; idx += gridDim.x * kEnvThreads)
    {
        EnvPixelId p;
        env_locate(a, idx, p);
        const int lw = a.lw[p.l], lh = a.lh[p.l];
        const float wgt   = a.weight[p.l][p.pix];
        const bool masked = (a.flags & VETR_ENV_NOT_AT_POINTS) && wgt > 0.001f;
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        float T      = env_start_T(wgt, a.flags);
        if (!masked)
        {
            const EnvRay ray = env_ray(s_cam[p.b], lw, lh, a.scale[p.l], p.x, p.y);
            for (int s = 0; s < a.S; ++s)
            {
                float ix, iy;
                if (!env_coordinates(a, ray, s, ix, iy)) continue;  // alpha = 0: nothing added, T unchanged
                EnvCorners<kFlat> c;
                env_corners<kFlat>(a, ix, iy, s, c);
                float alpha = 1.f;
                if (s != a.S - 1) alpha = 1.f / (1.f + expf(-env_fetch<kFlat>(a.density + s * slice, c)));
#pragma unroll
                for (int ch = 0; ch < 4; ++ch)
                    if (ch < a.C)
                    {
                        float col = env_fetch<kFlat>(a.color + ch * plane + s * slice, c);
                        if (a.non_subzero) col = fabsf(col);
                        acc[ch] = T * alpha * col + acc[ch];
                    }
                T = (1.f - alpha) * T;
            }
        }
        const long long per_view = (long long)lw * lh;
        float* o = a.out[p.l] + ((long long)p.b * a.C) * per_view + (p.y * lw + p.x);
#pragma unroll
        for (int ch = 0; ch < 4; ++ch)
            if (ch < a.C)
            {
                float v = acc[ch];
                if (a.flags & VETR_ENV_ADD)
                {
                    float base = o[ch * per_view];
                    if ((a.flags & VETR_ENV_DEPTH_TEST_WEIGHT) && !(wgt > 0.5f)) base = 0.f;
                    v = base + acc[ch];
                }
                o[ch * per_view] = v;
            }
    }
}

// Backward.  Per pixel, with D_s = colour_s . G and the transmittance T_s in front of sphere s:
//   d env / d colour_s = T_s alpha_s G,    d env / d alpha_s = T_s (D_s - rest_s),
//   rest_s = sum over the spheres behind s of their contribution per unit of transmittance behind s
//          = alpha_{s+1} D_{s+1} + (1 - alpha_{s+1}) rest_{s+1}
// (no division by 1 - alpha, which a saturated sigmoid makes zero).  First sweep, front to back: sample, keep alpha, D, T
// and the colours' signs.  Second sweep, back to front: the gradients of the sphere's samples,
// scattered to its corners.  Neighbouring pixels of a row fall into the same texel (a level-0 row of 1920
// pixels crosses a few hundred texels), so before the atomics the lanes of a warp that share a base texel, in runs of
// consecutive lanes, are summed with a segmented shuffle reduction and the run's first lane issues one atomic per corner and
// value.  Five steps, or three where no run of the warp is longer than eight lanes.  More such forms lose: with all of 0 to 5, or
// 5, 3 and 2, the loop's instructions are too many (1280 x 720 x 2, three spheres of 200 x 200: five 322 us, 5 and 3 337, 5, 3 and 2
// 344, all 377; 1920 x 1080, four of 1024 x 1024: 574, 533, 538, 572).
//
// What the first sweep keeps per sphere lies in shared memory, so that both loops over spheres stay loops: unrolled, with the
// state in registers, the kernel was several times the size, with three blocks of 256 per SM, and with eight spheres formed the
// texel coordinates twice.  Blocks of 128 threads, nine per SM (55 registers): with four blocks of 256 a medium-sized
// image leaves a last wave nearly empty (480 x 270 x 2, three spheres: 125 us, unrolled 112, now 110); ten per SM spill.
// kMaxSpheres is kEnvFlatSpheres or eight.  1920x1080, four levels, one view: four spheres of 1024 x 1024 707 -> 538 us, two
// of them 347 -> 272, five of 512 x 512 1072 -> 629, eight of 1024 x 1024 2160 -> 1457.
#ifndef VETR_ENV_BACK_CTAS
#    define VETR_ENV_BACK_CTAS 9
#endif
template <int kMaxSpheres>
__global__ void __launch_bounds__(kEnvBackThreads, VETR_ENV_BACK_CTAS) envmap_backward_kernel(const __grid_constant__ EnvArgs a)
{
    __shared__ EnvCam s_cam[VETR_MAX_VIEWS];
    __shared__ float kept[kMaxSpheres][5][kEnvBackThreads];  // a thread's own: alpha, D, T, texel coordinates
    if (threadIdx.x < a.n_views) s_cam[threadIdx.x] = load_env_cam(a, threadIdx.x);
    __syncthreads();
    constexpr bool kFlat  = kMaxSpheres <= kEnvFlatSpheres;
    constexpr int kN      = EnvCorners<kFlat>::N;
    const int plane = a.S * a.R * a.R, slice = kFlat ? a.R * a.R : 0;  // below 2^31; all channels' planes need not be
    const int lane = threadIdx.x & 31;
    const int span = (a.lend[a.L - 1] + 31) / 32 * 32;  // whole warps stay in the loop together
    for (int idx = blockIdx.x * kEnvBackThreads + threadIdx.x; idx < span; idx += gridDim.x * kEnvBackThreads)
    {
        EnvPixelId p;
        bool active = env_locate(a, idx, p);
        float G[4]  = {0.f, 0.f, 0.f, 0.f};
        float wgt   = 0.f;
        EnvRay ray;
        if (active)
        {
            wgt = a.weight[p.l][p.pix];
            if ((a.flags & VETR_ENV_NOT_AT_POINTS) && wgt > 0.001f) active = false;
        }
        if (active)
        {
            const long long per_view = (long long)a.lw[p.l] * a.lh[p.l];
            const float* g = a.grad[p.l] + ((long long)p.b * a.C) * per_view + (p.y * a.lw[p.l] + p.x);
#pragma unroll
            for (int ch = 0; ch < 4; ++ch)
                if (ch < a.C) G[ch] = g[ch * per_view];
            ray = env_ray(s_cam[p.b], a.lw[p.l], a.lh[p.l], a.scale[p.l], p.x, p.y);
        }
        unsigned hits     = 0;  // bit s: the ray hits sphere s
        unsigned negative = 0;  // bit 4 s + ch: the raw colour sample is negative (S <= 8, C <= 4)
        unsigned zero     = 0;  // the raw colour sample is exactly zero (abs has no gradient there)
        float T = env_start_T(wgt, a.flags);
        if (active)
        {
#pragma unroll 1
            for (int s = 0; s < a.S; ++s)
            {
                float x, y;
                if (env_coordinates(a, ray, s, x, y))
                {
                    hits |= 1u << s;
                    EnvCorners<kFlat> c;
                    env_corners<kFlat>(a, x, y, s, c);
                    float alpha = 1.f;
                    if (s != a.S - 1) alpha = 1.f / (1.f + expf(-env_fetch<kFlat>(a.density + s * slice, c)));
                    float d = 0.f;
#pragma unroll
                    for (int ch = 0; ch < 4; ++ch)
                        if (ch < a.C)
                        {
                            float col = env_fetch<kFlat>(a.color + ((long long)ch * plane + s * slice), c);
                            if (a.non_subzero)
                            {
                                if (col < 0.f) negative |= 1u << (4 * s + ch);
                                if (col == 0.f) zero |= 1u << (4 * s + ch);
                                col = fabsf(col);
                            }
                            d += col * G[ch];
                        }
                    kept[s][0][threadIdx.x] = alpha, kept[s][1][threadIdx.x] = d, kept[s][2][threadIdx.x] = T;
                    kept[s][3][threadIdx.x] = x, kept[s][4][threadIdx.x] = y;
                    T = (1.f - alpha) * T;
                }
            }
        }
        float rest = 0.f;
#pragma unroll 1
        for (int s = a.S - 1; s >= 0; --s)
        {
            const bool live = hits >> s & 1;
            EnvCorners<kFlat> c;
            float gv[5] = {0.f, 0.f, 0.f, 0.f, 0.f};  // gradient of the density sample, then of the colour samples
            int key = -1 - lane;                      // never equal between lanes
            if (live)
            {
                const float alpha = kept[s][0][threadIdx.x], dot = kept[s][1][threadIdx.x], Tin = kept[s][2][threadIdx.x];
                const float g_alpha = Tin * (dot - rest);
                rest                = alpha * dot + (1.f - alpha) * rest;
                key   = env_corners<kFlat>(a, kept[s][3][threadIdx.x], kept[s][4][threadIdx.x], s, c, key);
                gv[0] = s == a.S - 1 ? 0.f : g_alpha * (alpha * (1.f - alpha));  // alpha is the sigmoid
#pragma unroll
                for (int ch = 0; ch < 4; ++ch)
                    if (ch < a.C)
                    {
                        float v = Tin * alpha * G[ch];
                        if (negative >> (4 * s + ch) & 1) v = -v;
                        if (zero >> (4 * s + ch) & 1) v = 0.f;
                        gv[1 + ch] = v;
                    }
            }
            else
            {
#pragma unroll
                for (int q = 0; q < kN; ++q) c.off[q] = -1, c.w[q] = 0.f;
            }
            // runs of consecutive lanes with the same base texel (the corner offsets of such lanes are the same)
            const int prev       = __shfl_up_sync(0xffffffffu, key, 1);
            const bool head      = lane == 0 || key != prev;
            const unsigned heads = __ballot_sync(0xffffffffu, head);
            const unsigned later = heads >> lane >> 1;  // lanes behind this one that begin a run
            const int behind     = later ? __ffs(later) - 1 : 31 - lane;  // lanes behind this one in its run
            const auto scatter   = [&](auto steps)
            {
#pragma unroll
                for (int q = 0; q < kN; ++q)
                {
                    // a corner no lane of the warp uses (the empty z slice of a sample that sits on a slice)
                    if (!kFlat && !__any_sync(0xffffffffu, c.w[q] != 0.f)) continue;
#pragma unroll
                    for (int v = 0; v < 5; ++v)
                    {
                        if (v > a.C) continue;
                        if (v == 0 && s == a.S - 1) continue;  // the last sphere's alpha is a constant
                        float x = c.off[q] >= 0 ? c.w[q] * gv[v] : 0.f;
#pragma unroll
                        for (int k = 0; k < decltype(steps)::value; ++k)
                        {
                            const float y = __shfl_down_sync(0xffffffffu, x, 1 << k);
                            if (behind >= 1 << k) x += y;
                        }
                        if (head && c.off[q] >= 0 && x != 0.f)
                            atomicAdd((v == 0 ? a.g_density : a.g_color + (long long)(v - 1) * plane) + (s * slice + c.off[q]), x);
                    }
                }
            };
            if (__any_sync(0xffffffffu, behind >= 8))
                scatter(std::integral_constant<int, 5>{});
            else
                scatter(std::integral_constant<int, 3>{});
        }
    }
}

}  // namespace vetr

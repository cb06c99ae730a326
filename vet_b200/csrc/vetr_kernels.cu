// B200 (sm_100a) kernels and C ABI of the blending point rasterizer.  See include/vetr.h for the interface and the
// reference functions each entry point replaces.
//
// Data layout in HBM
//   pixel space : all views and all pyramid levels of a call form ONE array of PT = n_views * P pixels
//                 (view-major, then level, then bands of VETR_PIXEL_BAND rows, column by column inside a band; see
//                 pixel_offset).  counts[PT], ends[PT] (int32).
//   records     : one 32-byte record per fragment = one DRAM sector: 64-bit key (depth bits << 32 | point index),
//                 alpha, descriptor index, descriptor.  The list of pixel g is recs[ends[g] - counts[g] .. ends[g]).
//                 Lists of consecutive pixels are contiguous, so a CTA that owns a run of pixels streams its fragments
//                 with coalesced loads.
//   work items  : the pixel space is cut into runs of ~kQuantum units of work (1 per fragment, kPixelWork per pixel)
//                 by the scan itself (item_start[]), so the persistent item kernels are balanced by fragments, not
//                 by pixels, and no host round trip is needed to size anything.
//   backward    : level_mask[n_views * n] (which levels hold a fragment of a point), point_grad[(view, level, point)]
//                 (image-space gradient parked per fragment), img4 / grad4[PT] (channel-interleaved image copies).
//
// Kernels (nothing here is a contraction, so no tensor cores)
//   project_kernel<count>    stream positions, strict-fp32 projection, per-level pixel, one reduction per fragment
//   scan_*                   exclusive scan of counts -> ends, total F, longest list, work-item table, in two kernels (the last block
//                            of the first scans the sums of the tiles)
//   project_kernel<collect>  re-project, request the payload, reserve all slots of a thread's points, store the 32-byte records
//   sort_blend_kernel        per work item: stage records in shared memory, rank-sort each list by (depth, index),
//                            write every record to its sorted place, blend front to back, write all outputs (+ _long variant)
//   pack_images_kernel       channel-interleaved copies of the forward image and its gradient
//   backward_kernel          per work item: stream sorted records, image-space gradient of each fragment (parked for
//                            the per-point pass), O(n) transmittance / suffix sweeps per pixel, vector reductions of
//                            descriptor / confidence gradients (+ _long variants; mode 3 parks the alpha gradient)
//   point_backward_kernel    one thread per point over all views: projection Jacobians per fragment, position gradient
//                            written once, camera gradients reduced per CTA and view (mode 3: confidence gradient too)
//   fuzzy_dt_*               mode 0 (no lists): depth pre-pass, splat, combine, per-point backward
//   exchange_finalize_kernel multi-GPU: sum over ranks + epilogue over NVLink peer memory (plain or multicast)
//   grid_row_sums / grid_loss (cells, chunks)   error-grid rasterisation (a lane prepares a cell, then lanes own pixel rows)
//   zero_buffers / finalize / apply_tangent   zero fill, epilogue, pose update
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <limits>
#include <new>
#include <vector>

#include "../../include/vetr.h"
#include "vetr_math.cuh"

namespace vetr
{
// First statement of the kernels that launch() starts (but those that wait at their end, below), and of those in between: the next kernel on the stream
// may be set up on SMs that have room as soon as all blocks of this one run, and this one goes on when the kernel before it has ended and its writes
// are to be seen.  Nothing is read or written before; because every kernel waits, the end of one is the end of all before it.
__device__ __forceinline__ void begin_kernel()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// First statement of a kernel that has nothing to do with what the kernel before it does, only with what was there when that one started (it
// was launched in the plain way, or is such a kernel itself): it starts on the SMs that the other one's blocks have left, and ends
// after it, so that a kernel behind it may take the end of both for granted.  For that one block has to wait, the first; the others give their room back,
// to blocks of either kernel that want it.  The next kernel may be set up when the first block has waited: earlier, its blocks come to lie next to
// each other on the SMs that are free first (mode 3, 35 k points x 4 views 385x385 184 -> 201 us), unless it starts beside the same kernel.
// All blocks waiting / like this, us: 3 M points in a 1920x1080 frame and in it one list of 3000 780 / 745, 50 of 2000 630 / 597, 600 of 1000 786 / 756
// (three quarters of sort_blend_kernel<true>'s blocks came after the longest list); training, mode 2, 1 M points and 300 lists of 600
// 901 / 840, 60 k points x 8 views 200x150 415 / 352 (the second of the two kernels for long lists came after the first); no long lists the same.
template <bool kMoreBeside = false>  // the next kernel starts beside the previous one as well
struct BesidePrevious
{
    __device__ __forceinline__ BesidePrevious()
    {
        if (kMoreBeside) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    __device__ __forceinline__ ~BesidePrevious()
    {
        if (blockIdx.x != 0) return;
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (!kMoreBeside) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
};
struct BeginKernel
{
    __device__ __forceinline__ BeginKernel() { begin_kernel(); }
};

#ifndef VETR_ITEM_THREADS
#    define VETR_ITEM_THREADS 128
#endif
#ifndef VETR_QUANTUM
#    define VETR_QUANTUM 512
#endif
#ifndef VETR_LONG_LIST
#    define VETR_LONG_LIST 256
#endif
#ifndef VETR_BLEND_CTAS
#    define VETR_BLEND_CTAS 8
#endif
#ifndef VETR_BACK_CTAS
#    define VETR_BACK_CTAS 9
#endif
constexpr int kThreads    = VETR_ITEM_THREADS;  // CTA size of the item kernels
constexpr int kQuantum    = VETR_QUANTUM;       // units of work per item
#ifndef VETR_PIXEL_WORK
#    define VETR_PIXEL_WORK 4
#endif
constexpr int kPixelWork  = VETR_PIXEL_WORK;     // work units charged per pixel -> at most kQuantum / kPixelWork pixels per item
constexpr int kMaxPixels  = kQuantum / kPixelWork;
constexpr int kLongList   = VETR_LONG_LIST;         // lists longer than this take the slow path
constexpr int kCap        = kQuantum + kLongList;   // fragments staged per item (an item holds < kQuantum + its first list)
constexpr int kBlendCtas  = VETR_BLEND_CTAS;        // resident CTAs per SM the item kernels are compiled for; 8 is also what
constexpr int kBackCtas   = VETR_BACK_CTAS;         // fits the shared memory of sort_blend_kernel
constexpr int kProjThreads     = 256;
static_assert(kQuantum % kPixelWork == 0, "an item of kQuantum work units holds at most kQuantum / kPixelWork pixels");
static_assert(kMaxPixels <= kThreads, "one thread per pixel of an item");
static_assert(kMaxPixels <= 256, "seg_of is a byte");
constexpr int kScanTile   = 4096;  // elements per CTA in the scan (256 threads x 16)
constexpr float kMaxDepth = 100000.f;  // MAX_DEPTH_CONST, RenderConstants.h:30

struct ViewDev
{
    int image_index, camera_index;
    float crop[5];
    float rot[4];
};

struct Frame  // kernel parameter block (travels by value; no global or __constant__ state)
{
    int n_views, L, C, n, n_tex, w, h;
    int mode, drop_by_radius, use_env, viewer_only, dbg_max_len, need_point_grad, bg_alpha_to_point0, keep_sorted;
    float radius_threshold, dist_cutoff, stability_cutoff, k_grad_factor, dist_grad_factor, mask_value, accept_blend;
    float depth_accept;
    int ghost;
    int lw[VETR_MAX_LAYERS], lh[VETR_MAX_LAYERS];
    float inv_lw[VETR_MAX_LAYERS], inv_band[VETR_MAX_LAYERS];  // 1 / w and 1 / (kBand w) of a level
    long long lbase[VETR_MAX_LAYERS];  // first pixel of a level in the pixel space of one view (banded order, see pixel_offset)
    long long rbase[VETR_MAX_LAYERS];  // the same in plain row-major order (the interleaved image copies)
    long long P, PT;                   // pixels of one view / of all views in the pixel space (levels padded to whole bands)
    long long Prm;                     // row-major pixels of one view (sum of w * h)
    ViewDev views[VETR_MAX_VIEWS];
    const float4* position;
    const int* index;
    const float* texture;
    const float* confidence;
    const float* background;
    const double* poses;
    const float* intr;
    const float* dropout;
    int* counts;
    int* ends;
    uint4* recs;  // 32-byte fragment records: [2i] = {point index, depth bits, alpha bits, descriptor index}, [2i+1] = descriptor
    long long capacity;
    int* status;      // {F, overflow, longest, number of work items}
    int* item_start;  // [n_items + 1]
    int* next_item;   // counts the items handed out; the last entry of the caller's table, which is never one of the above
    unsigned char* level_mask;  // [n_views * n]: levels of the view on which the point has a fragment (written by collect)
    float2* point_grad;         // [(view * L + level) * n + point]: image-space gradient of that fragment (backward scratch)
    float4* img4;               // [PT] forward image, channels interleaved, indexed like counts[] (backward scratch)
    float4* grad4;              // [PT] its incoming gradient
};

// Order of the pixels of a level in the pixel space: bands of kBand = 4 rows, column by column inside a band,
//     offset(x, y) = (y / 4) * 4 w + 4 x + y % 4,
// so that 4-row x k-column patches of the image are contiguous.  Points arrive in Morton order: the
// fragments of neighbouring points then land in a few nearby runs of the fragment buffer instead of one run per image
// row, and a work item (a run of consecutive pixels) covers a compact patch.  The last band of a level is padded to
// full height; padded pixels have no fragments and are skipped wherever pixels are visited.
constexpr int kBand = VETR_PIXEL_BAND;  // rows per band (a power of two); 4 measured best among 1, 2, 4, 8, 16
constexpr int kBandShift = kBand == 1 ? 0 : kBand == 2 ? 1 : kBand == 4 ? 2 : kBand == 8 ? 3 : 4;
static_assert((1 << kBandShift) == kBand, "VETR_PIXEL_BAND must be 1, 2, 4, 8 or 16");
__device__ __forceinline__ int pixel_offset(int w, int x, int y) { return (y >> kBandShift) * (w << kBandShift) + (x << kBandShift) + (y & (kBand - 1)); }

// Mode 3 keeps the bilinear corner of a fragment in the two top bits of the record's descriptor index.
constexpr int kCornerShift = 30;
constexpr int kTexMask     = (1 << kCornerShift) - 1;

// 32 bytes = one sector in one request (addresses are multiples of 32).  Not ordered with the compiler's own accesses to the
// same bytes: a kernel that reads what it wrote has a barrier in between.  Two 16-byte halves cost twice the requests, and scattered
// ones twice the partial sectors.  8 M points x 4 views: collection 745 -> 679 us, sort + blend 1093 -> 1032 us; mode 3, 3 M x 2 views:
// 586 -> 515 and 1179 -> 1108 us.
__device__ __forceinline__ void load_sector(const uint4* p, uint4& a, uint4& b)
{
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
                 : "l"(p));
}
__device__ __forceinline__ void store_sector(uint4* p, uint4 a, uint4 b)
{
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w),
                 "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}

// One fragment record = one 32-byte sector.
__device__ __forceinline__ void store_record(const Frame& f, int slot, unsigned long long key, float alpha, int tex, float4 d)
{
    store_sector(f.recs + 2 * (size_t)slot, make_uint4((unsigned)key, (unsigned)(key >> 32), __float_as_uint(alpha), (unsigned)tex),
                 make_uint4(__float_as_uint(d.x), __float_as_uint(d.y), __float_as_uint(d.z), __float_as_uint(d.w)));
}
__device__ __forceinline__ void load_record(const Frame& f, int slot, uint4& h, uint4& d) { load_sector(f.recs + 2 * (size_t)slot, h, d); }
__device__ __forceinline__ unsigned long long record_key(uint4 h) { return ((unsigned long long)h.y << 32) | h.x; }
// A key as a positive fp64 number, which orders as the key does (depths are finite, so none is a NaN): one comparison instead of two.
// Ranking with 8 M points x 4 views: sort_blend_kernel 918 -> 901 us; mode 3, 3 M x 2 views 1023 -> 995.
__device__ __forceinline__ double ordered(unsigned long long key) { return __longlong_as_double((long long)key); }
__device__ __forceinline__ float4 as_float4(uint4 v)
{
    return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}

__device__ __forceinline__ Camera load_camera(const Frame& f, int b)
{
    Camera c;
    const ViewDev& v = f.views[b];
    const double* p  = f.poses + 8 * (long long)v.image_index;
    c.V.qx = (float)p[0], c.V.qy = (float)p[1], c.V.qz = (float)p[2], c.V.qw = (float)p[3];
    c.V.tx = (float)p[4], c.V.ty = (float)p[5], c.V.tz = (float)p[6];
    const float* k = f.intr + 13 * (long long)v.camera_index;
#pragma unroll
    for (int i = 0; i < 5; ++i) c.K[i] = k[i];
    bool hd = false;
#pragma unroll
    for (int i = 0; i < 8; ++i)
    {
        c.dist[i] = k[5 + i];
        hd |= c.dist[i] != 0.f;
    }
    c.has_dist = hd;
#pragma unroll
    for (int i = 0; i < 5; ++i) c.crop[i] = v.crop[i];
#pragma unroll
    for (int i = 0; i < 4; ++i) c.rot[i] = v.rot[i];
    c.cx = (float)(f.w / 2);
    c.cy = (float)(f.h / 2);
    rotation_matrix(c.V, c.R);
    return c;
}

// ---------------------------------------------------------------------------------------------------------
// Pass 1 and 3: projection + counting / collection.  kPts points per thread.  Modes 1 and 2 run in three sweeps over
// the thread's points so that independent memory operations are in flight together: (1) project and find the pixel of
// every (point, level), (2) load the payload and issue ALL count reductions / slot reservations, (3) store the records.
// (The slot reservation is an atomic with a return value: with one in flight per thread the kernel waits on it.)

__device__ __forceinline__ bool point_is_live(const Frame& f, int b, int pid)
{
    if (f.dropout && f.dropout[(size_t)b * f.n + pid] == 1.f) return false;
    if (f.viewer_only && f.confidence[f.index[pid]] < f.stability_cutoff) return false;
    return true;
}

// Few points: one point per thread, because a pass that does not fill the chip lasts as long as one thread's chain of points.  Many:
// several, which share the block's camera and keep more memory operations in flight per warp.  Mode 3 has kernels of its own; its
// loop over levels and corners shared the registers of modes 1 and 2 (and theirs its).  us, modes 1 and 2 / mode 3, on a planar
// cloud and (in brackets) a cube's surface at 1920 x 1080:
//                        several per thread             one per thread
//   count    100 k       7.3 (7.5)  / 10.8 (11.5)       4.4 (4.8)  /  8.4 (10.3)
//            2 M         26.6 (26.4) / 63.5 (51.1)      26.9 (26.1) / 57.7 (42.9)
//            2 M x 4     89.4 (87.3) / 222 (184)        96.0 (93.3)
//   collect  100 k       15.4 (18.4) / 45.5 (50.8)      10.8 (12.5) / 25.0 (30.4)
//            1 M x 4     133 (91)   / 512 (283)         133 (89)   / 508 (291)
//            2 M x 4     247 (158)  / 914 (417)         250 (147)  / 919 (448)
//            4 M x 4     448 (232)  / 1534 (550)        452 (252)  / 1545 (631)
// The collection waits for its atomics (55 % of the issue slots), so it wants warps, blocks of 128 threads, and the payload asked
// for ahead of the atomics instead of after them.  8 M points x 4 views, modes 1 and 2, two points per thread: twelve blocks per SM
// (40 registers) 614 us, ten 621, nine 621; the payload after the slots 647 (eight to fourteen blocks, or blocks of 64 and 256:
// 653 to 725).  One point per thread at 1 M points: sixteen blocks (32 registers) 80 us, thirteen 83, seven of 256 threads 85,
// two points 85.
// The count pass is bound by instruction issue (89 %) and stays at 256 threads: 320 us, six blocks 319, twelve of 128 341.  Mode 3
// counts two points per thread with six blocks: 4 M x 4 of the cube 232 us, four points 268, with four blocks 287.
constexpr int kCollectThreads = 128;
constexpr long long kCollectPairs = 1 << 23;          // points times views from which on a thread collects two points, modes 1, 2
constexpr long long kCollectPairsBilinear = 1 << 21;  // and mode 3
constexpr long long kCountSeveral = 1 << 21;          // and from which on it counts several
constexpr int count_points(bool bilinear) { return bilinear ? 2 : 4; }
constexpr int project_ctas(bool collect, int points, bool bilinear)
{
    return collect ? (points > 1 ? 12 : bilinear ? 10 : 16) : bilinear ? 6 : 5;
}
template <bool kCollect, int kPts, bool kBilinear>
__global__ void __launch_bounds__(kCollect ? kCollectThreads : kProjThreads, project_ctas(kCollect, kPts, kBilinear)) project_kernel(const __grid_constant__ Frame f)
{
    begin_kernel();
    constexpr int kThreadsHere = kCollect ? kCollectThreads : kProjThreads;
    __shared__ Camera s_cam;
    const int b     = blockIdx.y;
    const int first = blockIdx.x * (kThreadsHere * kPts) + threadIdx.x;

    float4 pos[kPts];  // requested before the camera, which the block waits for
#pragma unroll
    for (int it = 0; it < kPts; ++it)
    {
        const int pid = first + it * kThreadsHere;
        pos[it]       = pid < f.n ? __ldg(f.position + pid) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    int tex[kPts];
    if (kCollect)
#pragma unroll
        for (int it = 0; it < kPts; ++it) tex[it] = first + it * kThreadsHere < f.n ? __ldg(f.index + first + it * kThreadsHere) : 0;
    if (threadIdx.x == 0) s_cam = load_camera(f, b);
    __syncthreads();
    const Camera& cam   = s_cam;
    const int vbase     = b * (int)f.P;

    if constexpr (!kBilinear)
    {
        int g[kPts][VETR_MAX_LAYERS];  // pixel of (point, level) in the global pixel space, then its record slot; -1 = none
        unsigned zbits[kPts];
#pragma unroll
        for (int it = 0; it < kPts; ++it)
        {
            const int pid = first + it * kThreadsHere;
#pragma unroll
            for (int l = 0; l < VETR_MAX_LAYERS; ++l) g[it][l] = -1;
            zbits[it] = 0;
            if (pid >= f.n || !point_is_live(f, b, pid)) continue;
            const Projected pr = project_point(pos[it], cam, f.dist_cutoff);
            if (pr.z == 0.f) continue;
            zbits[it]    = __float_as_uint(pr.z);
            float2 ip    = pr.ip;
            float radius = pr.radius_px;
            bool alive   = true;
#pragma unroll
            for (int l = 0; l < VETR_MAX_LAYERS; ++l)
            {
                if (l >= f.L || (f.drop_by_radius && radius < f.radius_threshold)) alive = false;
                if (alive)
                {
                    const int lw = f.lw[l], lh = f.lh[l];
                    const int x = round_half_even(ip.x), y = round_half_even(ip.y);
                    if ((unsigned)x < (unsigned)lw && (unsigned)y < (unsigned)lh) g[it][l] = vbase + (int)f.lbase[l] + pixel_offset(lw, x, y);
                }
                radius *= 0.5f, ip.x *= 0.5f, ip.y *= 0.5f;
            }
        }
        if constexpr (!kCollect)
        {
#pragma unroll
            for (int it = 0; it < kPts; ++it)
#pragma unroll
                for (int l = 0; l < VETR_MAX_LAYERS; ++l)
                    if (g[it][l] >= 0) atomicAdd(f.counts + g[it][l], 1);
        }
        else
        {
        // what the blend needs of the point travels next to every key (coalesced loads here, one per point, instead of
        // a dependent gather per fragment later); asked for ahead of the slots, so that the two waits overlap
        float conf[kPts];
        float4 desc[kPts];
#pragma unroll
        for (int it = 0; it < kPts; ++it)
        {
            bool any = false;
#pragma unroll
            for (int l = 0; l < VETR_MAX_LAYERS; ++l) any |= g[it][l] >= 0;
            if (!any) continue;
            conf[it]   = __ldg(f.confidence + tex[it]);
            desc[it].x = __ldg(f.texture + tex[it]);
            desc[it].y = __ldg(f.texture + (size_t)f.n_tex + tex[it]);
            desc[it].z = __ldg(f.texture + 2 * (size_t)f.n_tex + tex[it]);
            desc[it].w = f.C > 3 ? __ldg(f.texture + 3 * (size_t)f.n_tex + tex[it]) : 0.f;
        }
#pragma unroll
        for (int it = 0; it < kPts; ++it)
#pragma unroll
            for (int l = 0; l < VETR_MAX_LAYERS; ++l)
                if (g[it][l] >= 0) g[it][l] = atomicAdd(f.ends + g[it][l], 1);
#pragma unroll
        for (int it = 0; it < kPts; ++it)
        {
            const int pid = first + it * kThreadsHere;
            if (pid >= f.n) break;
            unsigned bits = 0;
#pragma unroll
            for (int l = 0; l < VETR_MAX_LAYERS; ++l) bits |= g[it][l] >= 0 ? 1u << l : 0u;
            if (f.level_mask) f.level_mask[(size_t)b * f.n + pid] = (unsigned char)bits;
            if (!bits) continue;
            const unsigned long long key = ((unsigned long long)zbits[it] << 32) | (unsigned)pid;
#pragma unroll
            for (int l = 0; l < VETR_MAX_LAYERS; ++l)
                if (g[it][l] >= 0 && (long long)g[it][l] < f.capacity) store_record(f, g[it][l], key, conf[it], tex[it], desc[it]);
        }
        }
    }
    else
    // mode 3: every (point, level) touches the four pixels around its position.  The record's descriptor index carries
    // the corner (0..3) in its two top bits: the backward pass files a fragment's result under (point, level, corner).
#pragma unroll
    for (int it = 0; it < kPts; ++it)
    {
        const int pid = first + it * kThreadsHere;
        if (pid >= f.n) break;
        unsigned level_bits = 0;
        Projected pr;
        pr.z = 0.f;
        if (point_is_live(f, b, pid)) pr = project_point(pos[it], cam, f.dist_cutoff);
        if (pr.z == 0.f)
        {
            if (kCollect && f.level_mask) f.level_mask[(size_t)b * f.n + pid] = 0;
            continue;
        }
        float2 ip     = pr.ip;
        float radius  = pr.radius_px;
        const unsigned long long key = ((unsigned long long)__float_as_uint(pr.z) << 32) | (unsigned)pid;
        float conf   = 0.f;
        float4 desc  = make_float4(0.f, 0.f, 0.f, 0.f);
        if (kCollect && !(f.drop_by_radius && radius < f.radius_threshold))
        {
            conf   = __ldg(f.confidence + tex[it]);
            desc.x = __ldg(f.texture + tex[it]);
            desc.y = __ldg(f.texture + (size_t)f.n_tex + tex[it]);
            desc.z = __ldg(f.texture + 2 * (size_t)f.n_tex + tex[it]);
            desc.w = f.C > 3 ? __ldg(f.texture + 3 * (size_t)f.n_tex + tex[it]) : 0.f;
        }
#pragma unroll 1
        for (int l = 0; l < f.L; ++l, radius *= 0.5f, ip.x *= 0.5f, ip.y *= 0.5f)
        {
            if (f.drop_by_radius && radius < f.radius_threshold) break;
            const int lw = f.lw[l], lh = f.lh[l];
            const int gbase = vbase + (int)f.lbase[l];
            const int bx = round_down(ip.x), by = round_down(ip.y);
            if (bx == INT32_MIN || by == INT32_MIN) continue;  // unrepresentable position
            int slot[4];
#pragma unroll
            for (int cidx = 0; cidx < 4; ++cidx)
            {
                const int x = bx + (cidx & 1), y = by + (cidx >> 1);
                slot[cidx]  = -1;
                if ((unsigned)x >= (unsigned)lw || (unsigned)y >= (unsigned)lh) continue;
                const int g = gbase + pixel_offset(lw, x, y);
                if (!kCollect)
                    atomicAdd(f.counts + g, 1);
                else
                    slot[cidx] = atomicAdd(f.ends + g, 1);
            }
            if (kCollect)
            {
#pragma unroll
                for (int cidx = 0; cidx < 4; ++cidx)
                {
                    if (slot[cidx] < 0) continue;
                    level_bits |= 1u << l;
                    if ((long long)slot[cidx] < f.capacity)
                        store_record(f, slot[cidx], key, blending_fac(ip, cidx, nullptr, nullptr) * conf,  // RenderForward.cu:1619
                                     tex[it] | (cidx << kCornerShift), desc);
                }
            }
        }
        if (kCollect && f.level_mask) f.level_mask[(size_t)b * f.n + pid] = (unsigned char)level_bits;
    }
}

// ---------------------------------------------------------------------------------------------------------
// Pass 2: exclusive scan of counts -> ends (start offsets until the collection pass has advanced them to the
// list ends), total fragment count, longest list, and the work-item table.

// A tile's 4096 elements are four rows of 256 threads x 4: a thread takes four consecutive elements of every row with one 16-byte
// access, a warp 512 consecutive bytes.  (16 consecutive elements per thread, as before, are 64 bytes apart between lanes.)
// kVec: the arrays are 16-byte aligned.
template <bool kVec>
__device__ __forceinline__ int4 scan_load(const int* p, long long i, long long n)
{
    if (kVec && i + 4 <= n) return *reinterpret_cast<const int4*>(p + i);
    return make_int4(i < n ? p[i] : 0, i + 1 < n ? p[i + 1] : 0, i + 2 < n ? p[i + 2] : 0, i + 3 < n ? p[i + 3] : 0);
}
template <bool kVec>
__device__ __forceinline__ void scan_store(int* p, long long i, long long n, int4 v)
{
    if (kVec && i + 4 <= n)
        *reinterpret_cast<int4*>(p + i) = v;
    else
    {
        if (i < n) p[i] = v.x;
        if (i + 1 < n) p[i + 1] = v.y;
        if (i + 2 < n) p[i + 2] = v.z;
        if (i + 3 < n) p[i + 3] = v.w;
    }
}
// Loads the thread's 16 elements of a tile that starts at `base` and forms before[r], the sum of the tile's elements in front of
// the four of row r.  s_warp: 32 words.
template <bool kVec>
__device__ __forceinline__ void scan_tile(const int* in, long long base, long long n, int* s_warp, int4 (&c)[4], int (&before)[4])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int r = 0; r < 4; ++r) c[r] = scan_load<kVec>(in, base + r * 1024 + threadIdx.x * 4, n);
#pragma unroll
    for (int r = 0; r < 4; ++r)
    {
        const int own = c[r].x + c[r].y + c[r].z + c[r].w;
        int inc       = own;
        for (int o = 1; o < 32; o <<= 1)
        {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) s_warp[r * 8 + warp] = inc;
        before[r] = inc - own;
    }
    __syncthreads();
    if (warp == 0)
    {
        const int own = s_warp[lane];
        int inc       = own;
        for (int o = 1; o < 32; o <<= 1)
        {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        s_warp[lane] = inc - own;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r) before[r] += s_warp[r * 8 + warp];
}

// True in the last block of a grid to come here (in all its threads): what the blocks before it wrote is then visible to it.
// *ticket is 0 before.
__device__ __forceinline__ bool last_block(unsigned* ticket)
{
    __shared__ bool s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (s_last) __threadfence();
    return s_last;
}

// One block: exclusive scan of the tile sums in place; writes F, the overflow flag and the number of work items.
__device__ void scan_spine(long long* tile_sums, int n_tiles, long long n_pixels, long long capacity, int* status, int* item_start, int* next_item)
{
    constexpr int kEach = 8;  // consecutive tiles per thread
    __shared__ long long s_warp[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long carry = 0;
    for (int base = 0; base < n_tiles; base += 256 * kEach)
    {
        const int first = base + threadIdx.x * kEach;
        long long v[kEach], own = 0;
#pragma unroll
        for (int k = 0; k < kEach; ++k)
        {
            v[k] = first + k < n_tiles ? __ldcg(tile_sums + first + k) : 0;
            own += v[k];
        }
        long long inc = own;
        for (int o = 1; o < 32; o <<= 1)
        {
            const long long t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        __syncthreads();  // the previous round's sums have been read
        if (lane == 31) s_warp[warp] = inc;
        __syncthreads();
        long long run = carry + inc - own;
        for (int w = 0; w < 8; ++w)
        {
            if (w < warp) run += s_warp[w];
            carry += s_warp[w];
        }
#pragma unroll
        for (int k = 0; k < kEach; ++k)
        {
            if (first + k < n_tiles) tile_sums[first + k] = run;
            run += v[k];
        }
    }
    if (threadIdx.x == 0)
    {
        const long long F   = carry;
        const bool overflow = F > capacity || F > 0x7fffffffLL;
        status[0]           = (int)(F > 0x7fffffffLL ? 0x7fffffffLL : F);
        status[1]           = overflow ? 1 : 0;
        const long long work = F + (long long)kPixelWork * n_pixels;
        const int items      = overflow ? 0 : (int)((work + kQuantum - 1) / kQuantum);
        status[3]            = items;
        item_start[items]    = (int)n_pixels;  // sentinel
        *next_item           = 0;
    }
}

// Sums of the tiles; the last block to finish scans them (a launch of its own for that cost a small scene as much as the tiles).
template <bool kVec>
__global__ void __launch_bounds__(256) scan_tile_sums_kernel(const int* __restrict__ counts, long long n, long long* tile_sums, int* status,
                                                             long long capacity, int* item_start, int* next_item, unsigned* ticket)
{
    begin_kernel();
    __shared__ long long s_sum[8];
    __shared__ int s_max[8];
    const long long base = (long long)blockIdx.x * kScanTile;
    long long sum = 0;
    int mx        = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r)
    {
        const int4 c = scan_load<kVec>(counts, base + r * 1024 + threadIdx.x * 4, n);
        sum += (long long)c.x + c.y + c.z + c.w;
        mx = max(max(mx, max(c.x, c.y)), max(c.z, c.w));
    }
    for (int o = 16; o > 0; o >>= 1)
    {
        sum += __shfl_down_sync(0xffffffffu, sum, o);
        mx = max(mx, __shfl_down_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = sum, s_max[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        for (int i = 1; i < 8; ++i) sum += s_sum[i], mx = max(mx, s_max[i]);
        tile_sums[blockIdx.x] = sum;
        if (mx > 0) atomicMax(status + 2, mx);
    }
    if (last_block(ticket)) scan_spine(tile_sums, (int)gridDim.x, n, capacity, status, item_start, next_item);
}

// Writes the exclusive offsets and cuts the pixel space into work items: with work(p) = end(p) + kPixelWork*(p+1)
// (strictly increasing), item k owns the pixels with k*Q < work(p) <= (k+1)*Q; pixel p opens every item k with
// work(p-1) <= k*Q < work(p).  Inside a tile work is counted from the tile's own first item, in 32 bits.  One 1920x1080 view:
// 21 -> 7 us (before: 16 consecutive elements per thread, items in 64-bit divisions).
template <bool kVec>
__global__ void __launch_bounds__(256) scan_apply_kernel(const int* __restrict__ counts, long long n,
                                                         const long long* __restrict__ tile_offsets,
                                                         int* __restrict__ ends, const int* __restrict__ status,
                                                         int* __restrict__ item_start)
{
    begin_kernel();
    __shared__ int s_warp[32];
    const long long base = (long long)blockIdx.x * kScanTile;
    int4 c[4];
    int before[4];
    scan_tile<kVec>(counts, base, n, s_warp, c, before);
    const long long offset = tile_offsets[blockIdx.x], work = offset + kPixelWork * base;
    const int first_item   = (int)(work / kQuantum);
    const unsigned work0   = (unsigned)(work % kQuantum);
    const bool overflow    = status[1] != 0;  // the offsets are then not meant to be used
#pragma unroll
    for (int r = 0; r < 4; ++r)
    {
        const int e    = r * 1024 + threadIdx.x * 4;  // element in the tile
        const int v[4] = {c[r].x, c[r].y, c[r].z, c[r].w};
        int run        = before[r];
        int start[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            start[i] = (int)(offset + run);
            if (!overflow && base + e + i < n)
            {
                const unsigned w_prev = work0 + (unsigned)run + kPixelWork * (e + i);  // work(g-1), work(g) from the tile's first item on
                const unsigned w_here = w_prev + (unsigned)v[i] + kPixelWork;
                for (unsigned k = (w_prev + kQuantum - 1) / kQuantum; k * kQuantum < w_here; ++k) item_start[first_item + k] = (int)base + e + i;
            }
            run += v[i];
        }
        scan_store<kVec>(ends, base + e, n, make_int4(start[0], start[1], start[2], start[3]));
    }
}

// ---------------------------------------------------------------------------------------------------------
// Shared pieces of the item kernels.

struct PixInfo  // decoded pixel of the global pixel space, 8 bytes
{
    short x, y;
    unsigned char level, view;
    unsigned char interior;  // ImageView::distanceFromEdge > 2: the pixel takes part in the position gradient
    unsigned char valid;     // 0: padding row of the level's last band
};

// View, level and offset inside the level of pixel g, without divisions (a run of comparisons each).
__device__ __forceinline__ void locate_pixel(const Frame& f, unsigned g, int& view, int& level, unsigned& offset)
{
    const unsigned P = (unsigned)f.P;
    int v = 0;
#pragma unroll
    for (int i = 1; i < VETR_MAX_VIEWS; ++i)
        if (i < f.n_views && g >= i * P) v = i;
    unsigned q = g - v * P;
    int l      = 0;
#pragma unroll
    for (int i = 1; i < VETR_MAX_LAYERS; ++i)
        if (i < f.L && q >= (unsigned)f.lbase[i]) l = i;
    view = v, level = l, offset = q - (unsigned)f.lbase[l];
}

__device__ __forceinline__ PixInfo decode_pixel(const Frame& f, unsigned g)
{
    PixInfo r;
    int view, l;
    unsigned q;
    locate_pixel(f, g, view, l, q);
    const int w = f.lw[l], h = f.lh[l], bw = w << kBandShift;
    // band = q / (kBand w): float estimate, then one correction step either way (exact: the estimate is off by at most one)
    int band = __float2int_rz(__fmul_rn((float)q, f.inv_band[l]));
    int rem  = (int)q - band * bw;
    if (rem < 0) rem += bw, --band;
    if (rem >= bw) rem -= bw, ++band;
    const int x = rem >> kBandShift, y = (band << kBandShift) + (rem & (kBand - 1));
    r.x = (short)x, r.y = (short)y, r.level = (unsigned char)l, r.view = (unsigned char)view;
    r.valid    = y < h;
    r.interior = min(min(x, w - 1 - x), min(y, h - 1 - y)) > 2;
    return r;
}

// Index of a pixel in the row-major image copies (img4 / grad4).
__device__ __forceinline__ int row_major_index(const Frame& f, const PixInfo& px)
{
    return px.view * (int)f.Prm + (int)f.rbase[px.level] + px.y * f.lw[px.level] + px.x;
}

__device__ __forceinline__ int list_end(const Frame& f, int g) { return g < 0 ? 0 : f.ends[g]; }

// Which list a staged fragment belongs to.  The thread that owns a pixel writes its index over the pixel's slots when
// the list is short; the few long lists of an item are recorded separately and matched by range.  (A binary search
// per fragment costs more instructions than everything else the sort does for it.)
constexpr int kFillMax  = 128;
constexpr int kMaxLong  = kCap / kFillMax + 1;
struct SegTable
{
    unsigned char seg_of[kCap];
    unsigned char long_pix[kMaxLong];
    int n_long[2];  // alternating between consecutive items, so that the reset never races with a fill
};
__device__ __forceinline__ void seg_fill(SegTable& t, int parity, int pixel, int ss, int se)
{
    if (se - ss <= kFillMax)
        for (int k = ss; k < se; ++k) t.seg_of[k] = (unsigned char)pixel;
    else
        t.long_pix[atomicAdd(&t.n_long[parity], 1)] = (unsigned char)pixel;
}
__device__ __forceinline__ int seg_lookup(const SegTable& t, int parity, const int* seg_end, int i)
{
    int a = t.seg_of[i];
    const int nl = t.n_long[parity];
    for (int k = 0; k < nl; ++k)
    {
        const int p = t.long_pix[k];
        if (i >= seg_end[p] && i < seg_end[p + 1]) a = p;
    }
    return a;
}

__device__ __forceinline__ float4 load_descriptor(const Frame& f, int tex)
{
    float4 d;
    d.x = __ldg(f.texture + tex);
    d.y = __ldg(f.texture + (size_t)f.n_tex + tex);
    d.z = __ldg(f.texture + 2 * (size_t)f.n_tex + tex);
    d.w = f.C > 3 ? __ldg(f.texture + 3 * (size_t)f.n_tex + tex) : 0.f;
    return d;
}

// First pixel of an item that the item kernels leave to the long-list kernels (0 or 1 pixels).
__device__ __forceinline__ int long_prefix(const Frame& f, int lo)
{
    return (f.ends[lo] - list_end(f, lo - 1)) > kLongList ? 1 : 0;
}

// The pixels and fragments of a CTA's work items, read ahead of their use: the table entries two items ahead, the list ends
// that they lead to one item ahead, so that an item starts with its records instead of two round trips to the tables.  (8 M
// points x 4 views: sort_blend_kernel 1126 -> 1093 us, backward_kernel 1123 -> 1113 us; 100 k points: 15.4 -> 14.1, 17.8 -> 16.6 us.)
struct ItemStream
{
    int item, n_items;
    int next_lo, next_hi;           // range of the item after the one whose ends are in flight
    int lo, hi, before, first, last;  // item in flight: pixels [lo, hi), list ends of lo - 1, lo and hi - 1
    __device__ __forceinline__ void range(const Frame& f, int i)
    {
        next_lo = next_hi = 0;
        if (i < n_items) next_lo = f.item_start[i], next_hi = f.item_start[i + 1];
    }
    __device__ __forceinline__ void ends(const Frame& f)
    {
        lo = next_lo, hi = next_hi;
        before = first = last = 0;
        if (lo < hi) before = list_end(f, lo - 1), first = f.ends[lo], last = f.ends[hi - 1];
    }
    __device__ __forceinline__ ItemStream(const Frame& f) : item(blockIdx.x), n_items(f.status[3])
    {
        range(f, item);
        ends(f);
        range(f, item + gridDim.x);
    }
    // The next item: np pixels from p0 on (without one that is left to the long-list kernels), their nf fragments from f0 on.
    // False behind the last item; np may be 0.
    __device__ __forceinline__ bool next(const Frame& f, int& p0, int& np, int& f0, int& nf)
    {
        if (item >= n_items) return false;
        const int skip = lo < hi && first - before > kLongList ? 1 : 0;
        p0 = lo + skip, np = hi - p0;
        f0 = skip ? first : before, nf = last - f0;
        ends(f);
        range(f, item + 2 * (int)gridDim.x);
        item += gridDim.x;
        return true;
    }
};

// The same for items from a counter behind every CTA's first three: thread 0 asks for an item before the one in front of it is looked up in the
// table.  A CTA that has come late, or has items of much work, takes fewer of those.
struct ItemQueue
{
    struct Smem
    {
        int id[2];  // item whose table entry is read next; in turn, because nobody waits for those who read it
    };
    Smem& s;
    int item, n_items, turn;          // item: in thread 0, the next but one
    int next_lo, next_hi;             // range of the item after the one whose ends are in flight; behind the last item 0, -1
    int lo, hi, before, first, last;  // item in flight: pixels [lo, hi), list ends of lo - 1, lo and hi - 1
    __device__ __forceinline__ void range(const Frame& f, int i)
    {
        next_lo = 0, next_hi = -1;
        if (i < n_items) next_lo = f.item_start[i], next_hi = f.item_start[i + 1];
    }
    __device__ __forceinline__ void ends(const Frame& f)
    {
        lo = next_lo, hi = next_hi;
        before = first = last = 0;
        if (lo < hi) before = list_end(f, lo - 1), first = f.ends[lo], last = f.ends[hi - 1];
    }
    __device__ __forceinline__ ItemQueue(const Frame& f, Smem& smem) : s(smem), item(blockIdx.x + 2 * (int)gridDim.x), n_items(f.status[3]), turn(0)
    {
        range(f, blockIdx.x);
        ends(f);
        range(f, blockIdx.x + gridDim.x);
    }
    // As ItemStream's, but all threads call it together, and every warp has left the previous item when it returns.
    __device__ __forceinline__ bool next(const Frame& f, int& p0, int& np, int& f0, int& nf)
    {
        if (threadIdx.x == 0) s.id[turn] = item;
        __syncthreads();
        if (hi < 0) return false;
        const int skip = lo < hi && first - before > kLongList ? 1 : 0;
        p0 = lo + skip, np = hi - p0;
        f0 = skip ? first : before, nf = last - f0;
        ends(f);
        range(f, s.id[turn]);
        turn ^= 1;
        if (threadIdx.x == 0) item = atomicAdd(f.next_item, 1) + 3 * (int)gridDim.x;
        return true;
    }
};

// Work items whose first pixel holds a long list, for the kernels that take one such list per CTA.  Testing an item costs
// four dependent loads (two table entries, two list ends), and only a few items in a thousand qualify, so the threads of
// a CTA test one item each and the CTA then works through the hits: next() is called by all threads and returns the same
// pixel to all of them.  CTA b owns the items b, b + gridDim.x, ... (long lists cluster at the coarse levels, i.e. in
// consecutive items: the stride spreads them over the CTAs).
struct LongItemScan
{
    int base, k, n;  // base: index of the next batch among the CTA's own items
    __device__ __forceinline__ LongItemScan() : base(0), k(0), n(0) {}
    __device__ bool next(const Frame& f, int n_items, int* s_hits, int* s_count, int& lo)
    {
        for (;;)
        {
            if (k < n)
            {
                lo = s_hits[k++];
                return true;
            }
            __syncthreads();  // every thread has taken the last hit of the previous batch
            if ((long long)blockIdx.x + (long long)base * gridDim.x >= n_items) return false;
            if (threadIdx.x == 0) *s_count = 0;
            __syncthreads();
            const long long item = (long long)blockIdx.x + (long long)(base + threadIdx.x) * gridDim.x;
            if (item < n_items)
            {
                const int first = f.item_start[item], last = f.item_start[item + 1];
                if (first < last && long_prefix(f, first)) s_hits[atomicAdd(s_count, 1)] = first;
            }
            __syncthreads();
            n = *s_count, k = 0;
            base += blockDim.x;
        }
    }
};

struct OutPtrs
{
    float* color[VETR_MAX_LAYERS];
    float* weight[VETR_MAX_LAYERS];
    float* mask[VETR_MAX_LAYERS];
    float* depth[VETR_MAX_LAYERS];
};

// Outputs of pixel g of the global pixel space (planar [view, channel, y, x] tensors per level).
__device__ __forceinline__ void write_pixel(const Frame& f, const OutPtrs& out, unsigned g, const float c[4], float T, float depth)
{
    const PixInfo px = decode_pixel(f, g);
    if (!px.valid) return;
    const int level = px.level, view = px.view;
    const int w = f.lw[level], hw = w * f.lh[level], o = px.y * w + px.x;
    float* col = out.color[level] + (size_t)(view * f.C) * hw + o;
    col[0] = c[0], col[hw] = c[1], col[2 * hw] = c[2];
    if (f.C > 3) col[3 * hw] = c[3];
    const size_t po = (size_t)view * hw + o;
    if (out.weight[0]) out.weight[level][po] = T;
    if (out.mask[0]) out.mask[level][po] = (T == 0.f) ? f.mask_value : 1.f;
    if (out.depth[0]) out.depth[level][po] = depth;
}

// Front-to-back fold of one list (BlendMulti / BlendMultiBilinear, RenderForward.cu:1320-1356, 1597-1639).
struct Fold
{
    float T;
    float c[4];
    __device__ __forceinline__ void init()
    {
        T    = 1.f;
        c[0] = c[1] = c[2] = c[3] = 0.f;
    }
    __device__ __forceinline__ void add(float a, float4 d)
    {
        c[0] = vetr_blend(T, a, d.x, c[0]);
        c[1] = vetr_blend(T, a, d.y, c[1]);
        c[2] = vetr_blend(T, a, d.z, c[2]);
        c[3] = vetr_blend(T, a, d.w, c[3]);
        T    = vetr_new_T(T, a);
    }
    __device__ __forceinline__ void background(const Frame& f, const float bg[4])
    {
        const bool bilinear = f.mode == VETR_MODE_BILINEAR_BLEND;
        if (!f.use_env && !(bilinear && !(T >= 0.001f)))
        {
            c[0] = vetr_blend(T, 1.f, bg[0], c[0]), c[1] = vetr_blend(T, 1.f, bg[1], c[1]), c[2] = vetr_blend(T, 1.f, bg[2], c[2]);
            if (f.C > 3) c[3] = vetr_blend(T, 1.f, bg[3], c[3]);
        }
    }
};

// Mode 2 (BlendMultiFuzzy, RenderForward.cu:1412-1492): fragments within depth_accept_blend of the list's FIRST depth
// are averaged and blended as one; the reference then resets its reference depth to -100000, so every later fragment
// is a group of its own.  Transcribed literally.
struct FuzzyFold
{
    Fold fold;
    float last_min_d, acc_conf, acc_desc[4];
    int n_acc;
    __device__ __forceinline__ void init()
    {
        fold.init();
        last_min_d = acc_conf = 0.f;
        acc_desc[0] = acc_desc[1] = acc_desc[2] = acc_desc[3] = 0.f;
        n_acc       = 0;
    }
    __device__ __forceinline__ void flush()
    {
        const float n    = (float)n_acc;
        const float conf = acc_conf / n;
        fold.add(conf, make_float4(acc_desc[0] / n, acc_desc[1] / n, acc_desc[2] / n, acc_desc[3] / n));
    }
    __device__ __forceinline__ void add(float depth, float conf, float4 d, float accept)
    {
        if (last_min_d == 0.f) last_min_d = depth;
        if (!(depth - last_min_d < accept))
        {
            flush();
            last_min_d = -100000.f;
            acc_conf   = 0.f;
            n_acc      = 0;
            acc_desc[0] = acc_desc[1] = acc_desc[2] = acc_desc[3] = 0.f;
        }
        acc_conf += conf;
        acc_desc[0] += d.x, acc_desc[1] += d.y, acc_desc[2] += d.z, acc_desc[3] += d.w;
        ++n_acc;
    }
    __device__ __forceinline__ void finish()
    {
        if (n_acc > 0) flush();
    }
    // Once the first group is closed, every later fragment is a group of its own (depths are positive, so none lies within
    // `accept` of -100000 unless `accept` is larger than that): what follows is the plain fold, without the averages.
    __device__ __forceinline__ bool plain_from_here(float accept) const { return last_min_d == -100000.f && accept <= 100000.f; }
};

// ---------------------------------------------------------------------------------------------------------
// Pass 4: sort + blend.

struct BlendSmem
{
    unsigned long long key[kCap];  // arrival order
    float4 desc[kCap];
    float alpha[kCap];
    int tex[kCap];
    unsigned short perm[kCap];     // sorted position -> arrival slot
    int seg_end[kMaxPixels + 1];
    SegTable seg;
};

// What leaving a phase out saved, 8 M points x 4 views: ranking 290 us of 1020, fold 230, records back 130, pixels 30; one 1920x1080 view
// of 3 M points forward only 44, 47, 13, 12 of 182.  Records go back from the slot that they arrived in, by the thread that has just ranked
// them, which reads shared memory without conflicts and spares a phase, and the fold asks for its operands one fragment ahead (slot, then
// contents: two dependent reads): 1017 -> 916 us, 183 -> 166; mode 3, 3 M points x 2 views 1083 -> 989.
//
// kQueue: beside sort_blend_long_kernel, which has started before it, with the items from a counter, because blocks come to run as those of the other
// kernel leave room (see kQueueFragments).
template <bool kQueue>
__global__ void __launch_bounds__(kThreads, kBlendCtas) sort_blend_kernel(const __grid_constant__ Frame f,
                                                                          const __grid_constant__ OutPtrs out)
{
    const std::conditional_t<kQueue, BesidePrevious<>, BeginKernel> begin;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BlendSmem& s = *reinterpret_cast<BlendSmem*>(smem_raw);
    const int tid     = threadIdx.x;
    const bool bilinear = f.mode == VETR_MODE_BILINEAR_BLEND;
    const float bg[4]   = {f.background[0], f.background[1], f.background[2], f.C > 3 ? f.background[3] : 0.f};
    if (tid == 0) s.seg.n_long[0] = s.seg.n_long[1] = 0;
    int parity = 0;

    __shared__ ItemQueue::Smem s_items;
    auto items = [&]
    {
        if constexpr (kQueue)
            return ItemQueue(f, s_items);
        else
            return ItemStream(f);
    }();
    int lo, np, f0, nf;
    while (items.next(f, lo, np, f0, nf))
    {
        if (np <= 0) continue;
        if (!kQueue) __syncthreads();  // every warp has left the previous item
        parity ^= 1;
        if (tid == 0) s.seg.n_long[parity ^ 1] = 0;
        // the thread's first record is requested before the per-pixel set-up, each further one before the previous is stored
        uint4 h_next = make_uint4(0, 0, 0, 0), d_next = h_next;
        if (tid < nf) load_record(f, f0 + tid, h_next, d_next);
        if (tid < np)
        {
            const int ss = list_end(f, lo + tid - 1) - f0, se = f.ends[lo + tid] - f0;
            s.seg_end[tid + 1] = se;
            seg_fill(s.seg, parity, tid, ss, se);
        }
        if (tid == 0) s.seg_end[0] = 0;
        // stream keys and payload of the item (contiguous, coalesced)
        for (int i = tid; i < nf; i += kThreads)
        {
            const uint4 h = h_next, d = d_next;
            if (i + kThreads < nf) load_record(f, f0 + i + kThreads, h_next, d_next);
            s.desc[i]     = as_float4(d);
            s.key[i]      = record_key(h);
            s.alpha[i]    = __uint_as_float(h.z);
            s.tex[i]      = (int)h.w;
        }
        __syncthreads();
        // rank sort inside each list; keys are unique (distinct point indices), so ranks are a permutation
        for (int i = tid; i < nf; i += kThreads)
        {
            const int a  = seg_lookup(s.seg, parity, s.seg_end, i);
            const int ss = s.seg_end[a], se = s.seg_end[a + 1];
            const unsigned long long key = s.key[i];
            int rank = 0;
            for (int k = ss; k < se; ++k) rank += ordered(s.key[k]) < ordered(key);
            s.perm[ss + rank] = (unsigned short)i;
            // the sorted lists go back for the backward pass (all of the item's records are in shared memory by now)
            if (f.keep_sorted) store_record(f, f0 + ss + rank, key, s.alpha[i], s.tex[i], s.desc[i]);
        }
        __syncthreads();
        // fold: one thread per pixel
        if (tid < np)
        {
            const int ss = s.seg_end[tid], se = s.seg_end[tid + 1];
            int cnt = se - ss;
            if (f.dbg_max_len > 0) cnt = min(cnt, f.dbg_max_len);
            Fold fold;
            fold.init();
            int r = ss;
            if (f.mode == VETR_MODE_FUZZY_BLEND)
            {
                FuzzyFold ff;
                ff.init();
                while (r < ss + cnt && !ff.plain_from_here(f.accept_blend))
                {
                    const int u = s.perm[r++];
                    ff.add(__uint_as_float((unsigned)(s.key[u] >> 32)), s.alpha[u], s.desc[u], f.accept_blend);
                }
                ff.finish();
                fold = ff.fold;
            }
            if (const int last = ss + cnt - 1; r <= last)
            {
                const int u = s.perm[r];
                int next    = s.perm[min(r + 1, last)];
                float a     = s.alpha[u];
                float4 d    = s.desc[u];
                for (; r <= last; ++r)
                {
                    const float a0  = a;  // this fragment's; the next one's are requested, and the slot of the one behind it
                    const float4 d0 = d;
                    a = s.alpha[next], d = s.desc[next];
                    next = s.perm[min(r + 2, last)];
                    fold.add(a0, d0);
                    if (bilinear && fold.T < 0.001f) break;
                }
            }
            fold.background(f, bg);
            float depth = se > ss ? __uint_as_float((unsigned)(s.key[s.perm[ss]] >> 32)) : kMaxDepth;
            write_pixel(f, out, (unsigned)(lo + tid), fold.c, fold.T, depth);
        }
    }
}

// Lists longer than kLongList: one CTA per list, beside the end of sort_blend_kernel, whose CTAs take the same share of the items but not the same
// time (the two together: 3 M points, one 1920x1080 view, 190 -> 171 us; mode 3, 3 M x 2 views, 1230 -> 1130).  Up to kLongSortMax fragments the keys are merge-sorted in shared memory
// and the records follow, half a record at a time (the reference's <= 4096 bucket is a CTA-wide shared-memory sort as well,
// AlphaListSort.cu:601-703); runs of that many of a longer list are merged in global memory.  The fold runs in blocks of kFoldCap fragments.
//
// Bound by latency: the fold of a list is one chain.  So as much as possible is taken out of it - a lane forms the
// transmittances (one multiplication per fragment), four more the channels (one fused multiply-add per fragment), both on
// 16-byte loads - and lists are small in shared memory, so that five are in flight per SM instead of two.  The sort costs
// 32 comparisons and log2(n / 32) binary searches per fragment instead of n comparisons.  3 M points x 2 views, mode 3:
// 812 -> 228 us; 8 M x 4 views, mode 1: 126 -> 47 us; one 1280x720 view of 1 M points, mode 3: 203 -> 57 us (before: the whole
// fold in one thread, records and keys of 2048 fragments in shared memory, 128 threads, n comparisons per fragment).
constexpr int kLongThreads = 256;
constexpr int kLongSortMax = 2048;
constexpr int kFoldCap     = 1024;
static_assert(kFoldCap % 4 == 0 && kCap % 4 == 0, "chains read four fragments at a time");
struct LongBlendSmem
{
    union
    {
        unsigned long long key[2][kLongSortMax];  // merge sort: two buffers in turn
        uint4 half[kLongSortMax];                 // half a record of every fragment, while the records are put in order
        struct                                    // fold
        {
            float alpha[kFoldCap], trans[kFoldCap];  // trans: transmittance in front of the fragment
            float desc[4][kFoldCap];                 // by channel
            float depth[kFoldCap];                   // mode 2
        } fold;
    };
    unsigned short idx[2][kLongSortMax];  // arrival slot of a key
};

// Sorts the n <= kLongSortMax records that start at `first` by key.
__device__ void sort_long_list_shared(const Frame& f, LongBlendSmem& ls, int first, int n)
{
    uint4* recs = f.recs + 2 * (size_t)first;
    for (int i = threadIdx.x; i < n; i += blockDim.x) ls.key[0][i] = record_key(recs[2 * i]);
    __syncthreads();
    // runs of 32: rank by comparison with the run
    for (int i = threadIdx.x; i < n; i += blockDim.x)
    {
        const int r0 = i & ~31, m = min(32, n - r0);
        const unsigned long long key = ls.key[0][i];
        int rank = 0;
        for (int k = 0; k < m; ++k) rank += ordered(ls.key[0][r0 + k]) < ordered(key);
        ls.key[1][r0 + rank] = key;
        ls.idx[1][r0 + rank] = (unsigned short)i;
    }
    __syncthreads();
    // pairs of runs: a key moves by the number of smaller keys in the other run (keys of a list are distinct)
    int cur = 1;
    for (int width = 32; width < n; width *= 2, cur ^= 1)
    {
        for (int i = threadIdx.x; i < n; i += blockDim.x)
        {
            const unsigned long long key = ls.key[cur][i];
            const int run = i & -width, other = min(run ^ width, n);
            int lo = other, hi = min(other + width, n);
            while (lo < hi)
            {
                const int mid = (lo + hi) >> 1;
                if (ls.key[cur][mid] < key)
                    lo = mid + 1;
                else
                    hi = mid;
            }
            const int to = (run & ~width) + (i - run) + (lo - other);
            ls.key[cur ^ 1][to] = key;
            ls.idx[cur ^ 1][to] = ls.idx[cur][i];
        }
        __syncthreads();
    }
    for (int part = 0; part < 2; ++part)
    {
        for (int i = threadIdx.x; i < n; i += blockDim.x) ls.half[i] = recs[2 * i + part];
        __syncthreads();
        for (int r = threadIdx.x; r < n; r += blockDim.x) recs[2 * r + part] = ls.half[ls.idx[cur][r]];
        __syncthreads();  // the next half, or the fold, reuses this shared memory and reads the records back
    }
}

// Any list: runs of kLongSortMax like that, then in global memory by the whole CTA.  Sorting network with all comparators pointing the same
// way, so that positions >= n behave as +infinity without padding.  One list of 20 000 among 300 k points, one 1920x1080 frame: the network alone 4.99 ms,
// started beside sort_blend_kernel 5.25 (of 200 000: 64.2, 68.5; most likely the L1 that the kernel before leaves it is smaller), with runs 2.71 (44.2); of
// 3000 700 -> 280 us; 100 lists of 3000 among 3 M points 2695 -> 892 us.
__device__ void sort_long_list(const Frame& f, LongBlendSmem& ls, int first, int n)
{
    for (int run = 0; run < n; run += kLongSortMax) sort_long_list_shared(f, ls, first + run, min(kLongSortMax, n - run));
    uint4* recs = f.recs + 2 * (size_t)first;
    int n2 = 1;
    while (n2 < n) n2 <<= 1;
    for (int k = 2 * kLongSortMax; k <= n2; k <<= 1)
    {
        for (int j = k >> 1; j > 0; j >>= 1)
        {
            for (int i = threadIdx.x; i < n2; i += blockDim.x)
            {
                int partner = (j == (k >> 1)) ? (i ^ (k - 1)) : (i ^ j);
                if (partner > i && partner < n)
                {
                    uint4 a = recs[2 * i], b = recs[2 * partner];
                    if (record_key(a) > record_key(b))
                    {
                        recs[2 * i] = b, recs[2 * partner] = a;
                        uint4 da = recs[2 * i + 1], db = recs[2 * partner + 1];
                        recs[2 * i + 1] = db, recs[2 * partner + 1] = da;
                    }
                }
            }
            __syncthreads();
        }
    }
}

// Transmittances of m fragments of one list by one thread: trans[i] in front of fragment i, returns the one behind the last.
// alpha[m .. next multiple of four) is 0, which leaves the product as it is.  kStop: `m` becomes the number of fragments up
// to the one that takes the transmittance below 0.001 (mode 3 ends a list there).
template <bool kStop>
__device__ __forceinline__ float transmittance_chain(const float* alpha, float* trans, int& m, float T)
{
    for (int i = 0; i < m; i += 4)
    {
        const float4 a = *reinterpret_cast<const float4*>(alpha + i);
        const float t1 = vetr_new_T(T, a.x), t2 = vetr_new_T(t1, a.y), t3 = vetr_new_T(t2, a.z), t4 = vetr_new_T(t3, a.w);
        *reinterpret_cast<float4*>(trans + i) = make_float4(T, t1, t2, t3);
        if (kStop)
        {
            const int k = t1 < 0.001f ? 1 : t2 < 0.001f ? 2 : t3 < 0.001f ? 3 : t4 < 0.001f ? 4 : 0;
            if (k)  // a padding fragment repeats the value of the last one, so i + k <= m
            {
                m = i + k;
                return k == 1 ? t1 : k == 2 ? t2 : k == 3 ? t3 : t4;
            }
        }
        T = t4;
    }
    return T;
}

template <bool kFirst>  // started before sort_blend_kernel, or beside its end
__global__ void __launch_bounds__(kLongThreads) sort_blend_long_kernel(const __grid_constant__ Frame f,
                                                                       const __grid_constant__ OutPtrs out)
{
    const std::conditional_t<kFirst, BeginKernel, BesidePrevious<>> begin;
    if (f.status[2] <= kLongList) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    LongBlendSmem& s = *reinterpret_cast<LongBlendSmem*>(smem_raw);
    __shared__ FuzzyFold s_fuzzy;  // carried between blocks (mode 2, until its first group is closed)
    __shared__ float s_T, s_color[4];
    __shared__ int s_used, s_stop, s_grouped;
    const int tid       = threadIdx.x;
    const int n_items   = f.status[3];
    const bool bilinear = f.mode == VETR_MODE_BILINEAR_BLEND, fuzzy = f.mode == VETR_MODE_FUZZY_BLEND;
    __shared__ int s_long_hits[kLongThreads], s_long_count;
    LongItemScan scan;
    int lo;
    while (scan.next(f, n_items, s_long_hits, &s_long_count, lo))
    {
        const int e0 = list_end(f, lo - 1);
        const int n  = f.ends[lo] - e0;
        __syncthreads();
        sort_long_list(f, s, e0, n);
        int cnt = n;
        if (f.dbg_max_len > 0) cnt = min(cnt, f.dbg_max_len);
        if (tid == 0)
        {
            s_fuzzy.init();
            s_T       = 1.f;
            s_stop    = 0;
            s_grouped = fuzzy;
        }
        if (tid < 4) s_color[tid] = 0.f;
        __syncthreads();
        for (int blk = 0; blk < cnt && !s_stop; blk += kFoldCap)
        {
            const int m = min(kFoldCap, cnt - blk);
            for (int i = tid; i < m; i += kLongThreads)
            {
                const uint4 h  = f.recs[2 * (size_t)(e0 + blk + i)];
                const float4 d = as_float4(f.recs[2 * (size_t)(e0 + blk + i) + 1]);
                s.fold.alpha[i]   = __uint_as_float(h.z);
                s.fold.depth[i]   = __uint_as_float(h.y);
                s.fold.desc[0][i] = d.x, s.fold.desc[1][i] = d.y, s.fold.desc[2][i] = d.z, s.fold.desc[3][i] = d.w;
            }
            if (m + tid < ((m + 3) & ~3)) s.fold.alpha[m + tid] = 0.f;
            __syncthreads();
            bool chain = true;
            if (s_grouped)
            {
                // mode 2: one thread forms the first group; what it took is left behind as fragments that change nothing
                __syncthreads();  // all threads have read s_grouped
                if (tid == 0)
                {
                    FuzzyFold ff = s_fuzzy;
                    int i        = 0;
                    while (i < m && !ff.plain_from_here(f.accept_blend))
                    {
                        ff.add(s.fold.depth[i], s.fold.alpha[i],
                               make_float4(s.fold.desc[0][i], s.fold.desc[1][i], s.fold.desc[2][i], s.fold.desc[3][i]), f.accept_blend);
                        ++i;
                    }
                    if (ff.plain_from_here(f.accept_blend))
                    {
                        ff.finish();
                        s_T = ff.fold.T;
                        for (int k = 0; k < 4; ++k) s_color[k] = ff.fold.c[k];
                        s_grouped = 0;
                    }
                    s_fuzzy = ff;
                    s_used  = i;
                }
                __syncthreads();
                const int taken = s_used;
                chain           = !s_grouped;
                for (int i = tid; chain && i < taken; i += kLongThreads)
                    s.fold.alpha[i] = s.fold.desc[0][i] = s.fold.desc[1][i] = s.fold.desc[2][i] = s.fold.desc[3][i] = 0.f;
                __syncthreads();
            }
            if (chain)
            {
                if (tid == 0)
                {
                    int used = m;
                    const float T = bilinear ? transmittance_chain<true>(s.fold.alpha, s.fold.trans, used, s_T)
                                             : transmittance_chain<false>(s.fold.alpha, s.fold.trans, used, s_T);
                    s_T = T, s_used = used, s_stop = bilinear && T < 0.001f;
                }
                __syncthreads();
                if (tid < 4)  // vetr_blend, one channel per lane
                {
                    const int used  = s_used;
                    const float* d4 = s.fold.desc[tid];
                    float c = s_color[tid];
                    int i   = 0;
                    for (; i + 4 <= used; i += 4)
                    {
                        const float4 T = *reinterpret_cast<const float4*>(s.fold.trans + i);
                        const float4 a = *reinterpret_cast<const float4*>(s.fold.alpha + i);
                        const float4 d = *reinterpret_cast<const float4*>(d4 + i);
                        c = vetr_blend(T.x, a.x, d.x, c), c = vetr_blend(T.y, a.y, d.y, c);
                        c = vetr_blend(T.z, a.z, d.z, c), c = vetr_blend(T.w, a.w, d.w, c);
                    }
                    for (; i < used; ++i) c = vetr_blend(s.fold.trans[i], s.fold.alpha[i], d4[i], c);
                    s_color[tid] = c;
                }
            }
            __syncthreads();
        }
        if (tid == 0)
        {
            Fold fold;
            if (s_grouped)
            {
                FuzzyFold ff = s_fuzzy;
                ff.finish();
                fold = ff.fold;
            }
            else
            {
                fold.T = s_T;
                for (int k = 0; k < 4; ++k) fold.c[k] = s_color[k];
            }
            const float bg[4] = {f.background[0], f.background[1], f.background[2], f.C > 3 ? f.background[3] : 0.f};
            fold.background(f, bg);
            write_pixel(f, out, (unsigned)lo, fold.c, fold.T, __uint_as_float(f.recs[2 * (size_t)e0].y));
        }
    }
}

// ---------------------------------------------------------------------------------------------------------
// Backward.

struct BackPtrs
{
    const float* out_color[VETR_MAX_LAYERS];
    const float* grad_color[VETR_MAX_LAYERS];
    float4* g_desc;
    float* g_conf;
    float4* g_points;
    float* g_background;
    double* g_pose;
    float* g_pose_count;
    float* g_intr;
    float* g_intr_count;
};

struct BackSmem
{
    int pid[kCap];
    int tex[kCap];
    float alpha[kCap];
    float dot[kCap];     // d_i . G (mode 2: replaced by the gradient of the group's confidence)
    float trans[kCap];   // T_i ; NaN = fragment not blended (early termination / list truncation)
    float4 grad[kMaxPixels];  // incoming gradient of the pixel
    int seg_end[kMaxPixels + 1];
    PixInfo pix[kMaxPixels];
    SegTable seg;
    double red[kThreads / 32][8];  // cross-warp reduction scratch
};

// Modes 1 and 3: suffix sum S behind every fragment (mode 1 does not need the point index after stage A: same memory).
struct BackSmemSuffix : BackSmem
{
    float after[kCap];
};
template <bool kBilinear>
__device__ __forceinline__ float* suffix_of(BackSmem& s)
{
    if constexpr (kBilinear)
        return static_cast<BackSmemSuffix&>(s).after;
    else
        return reinterpret_cast<float*>(s.pid);
}

// Mode 2 additionally needs every fragment's depth; the suffix sums take the memory of the point indices as in mode 1.
struct BackSmemFuzzy : BackSmem
{
    float depth[kCap];
};

// Gradient accumulation with fire-and-forget reductions.  The gradient buffers are never read by these kernels, so
// the compiler may move other memory operations across them (no memory clobber).
__device__ __forceinline__ void red_add_v4(float4* addr, float4 v)
{
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w));
}
__device__ __forceinline__ void red_add(float* addr, float v)
{
    asm volatile("red.global.add.f32 [%0], %1;" ::"l"(addr), "f"(v));
}

// Camera-gradient accumulators of one thread for the pixels of a single view: pose in double like the reference's
// atomics (RenderBackward.cu:1423), the rest in float.
template <bool kIntr>
struct CamAcc
{
    double pose[6];
    float pose_count;
    float intr[kIntr ? 14 : 1];  // 13 gradients + count
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int k = 0; k < 6; ++k) pose[k] = 0.0;
        pose_count = 0.f;
#pragma unroll
        for (int k = 0; k < (kIntr ? 14 : 1); ++k) intr[k] = 0.f;
    }
};

// Sum over the lanes of a warp of N values per lane, N a power of two: at every step a lane hands the half of its values
// that the other half-warp is going to own to its partner, so N = 8 takes 9 shuffles instead of 40.  Afterwards v[0] of
// lane l is the total of value warp_sum_slot<N>(l).
template <int N>
__device__ __forceinline__ void warp_sum(double (&v)[N])
{
    const int lane = threadIdx.x & 31;
    int bit = 16;
#pragma unroll
    for (int h = N / 2; h >= 1; h /= 2, bit /= 2)
    {
        const bool up = lane & bit;
#pragma unroll
        for (int i = 0; i < h; ++i)
        {
            const double send = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
        }
    }
    for (; bit >= 1; bit /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], bit);
}
template <int N>
__device__ __forceinline__ int warp_sum_slot(int lane)
{
    int slot = 0, bit = 16;
#pragma unroll
    for (int h = N / 2; h >= 1; h /= 2, bit /= 2) slot += lane & bit ? h : 0;
    return slot;
}

// Sums the accumulators over the CTA and adds the totals to the outputs of `view`: one atomic per value and
// (CTA, view) instead of one per fragment.  `red`: one row per warp.
constexpr int kCamValues = 24;  // 8 (pose, its count, one unused) + 16 (intrinsics, their count, two unused)
template <bool kIntr>
__device__ void reduce_cam(const Frame& f, const BackPtrs& bp, CamAcc<kIntr>& acc, int view, double (*red)[kCamValues])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const ViewDev& vw = f.views[view];
    __syncthreads();  // the previous view's totals have been read
    {
        double v[8] = {acc.pose[0], acc.pose[1], acc.pose[2], acc.pose[3], acc.pose[4], acc.pose[5], (double)acc.pose_count, 0.0};
        warp_sum<8>(v);
        if ((lane & 3) == 0) red[warp][warp_sum_slot<8>(lane)] = v[0];
    }
    if constexpr (kIntr)
    {
        double v[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = k < 14 ? (double)acc.intr[k < 14 ? k : 0] : 0.0;
        warp_sum<16>(v);
        if ((lane & 1) == 0) red[warp][8 + warp_sum_slot<16>(lane)] = v[0];
    }
    __syncthreads();
    const int k = threadIdx.x;
    if (k < (kIntr ? 22 : 7) && k != 7)
    {
        double x = 0.0;
        for (int w = 0; w < (int)blockDim.x / 32; ++w) x += red[w][k];
        if (x != 0.0)
        {
            if (k < 6)
            {
                if (bp.g_pose) atomicAdd(bp.g_pose + 6 * vw.image_index + k, x);
            }
            else if (k == 6)
            {
                if (bp.g_pose) atomicAdd(bp.g_pose_count + vw.image_index, (float)x);
            }
            else if (k < 21)
                atomicAdd(bp.g_intr + 13 * vw.camera_index + (k - 8), (float)x);
            else
                atomicAdd(bp.g_intr_count + vw.camera_index, (float)x);
        }
    }
    acc.clear();
}

// Image-space gradient of all fragments of a point in one view, brought to level 0.  The chain of Jacobians behind it is
// linear and differs between the levels only by the factor 0.5^level of the crop matrix (a power of two: exact), so the
// camera gradients, sums over many points, take it once per point and view instead of once per fragment.  Summed in fp64: the
// terms of a point cancel (the Jacobians of a bilinear point's four corners add up to zero).  They stay fp64 through the
// camera's matrices, so that the sum is rounded to fp32 no more often than a single fragment's gradient is.
struct PointGrad
{
    double x, y;
    int hits;
    __device__ __forceinline__ void clear() { x = y = 0.0, hits = 0; }
    __device__ __forceinline__ void add(float2 g, int level)
    {
        const float scale = level_scale(level);
        x += (double)(g.x * scale), y += (double)(g.y * scale), ++hits;
    }
    static __device__ __forceinline__ float level_scale(int level) { return __int_as_float((127 - level) << 23); }
};

// Point gradient of one fragment (RenderBackward.cu:1380-1400): gp.xyz += J^T dR.
__device__ __forceinline__ void point_terms(const Camera& cam, const PointJac& jac, float2 dR, int level, float4& gp)
{
    const float scale = PointGrad::level_scale(level);
    const float crop2[5] = {cam.crop[0] * scale, cam.crop[1] * scale, 0.f, 0.f, cam.crop[4] * scale};  // IntrinsicsPinhole::scale
    float g[3];
    project_backward_point(cam, project_backward_view(jac, dR.x, dR.y, cam, crop2), g);
    gp.x += g[0], gp.y += g[1], gp.z += g[2], gp.w += 1.f;
}

// Pose and intrinsics gradients of one point in one view (RenderBackward.cu:1400-1460 and :3130-3180).
template <bool kIntr>
__device__ __forceinline__ void camera_terms(const Frame& f, const Camera& cam, const PointJac& jac, const PointGrad& g,
                                             CamAcc<kIntr>& acc)
{
    const ViewGrad v = project_backward_view(jac, g.x, g.y, cam, cam.crop);
    float g_pose[6];
    project_backward_pose(jac, v, g_pose);
#pragma unroll
    for (int k = 0; k < 6; ++k) acc.pose[k] += (double)g_pose[k];
    // RenderBackward.cu:379 (mode 0) and :3144 (mode 3) count 1 per hit, :993 and :1425 (modes 2, 1) count 1/1024
    acc.pose_count += (f.mode == VETR_MODE_BILINEAR_BLEND || f.mode == VETR_MODE_FUZZY_DT) ? (float)g.hits : (float)g.hits * (1.f / 1024.f);
    if (kIntr)
    {
        float g_k[5], g_dis[8];
        project_backward_intrinsics(jac, v, cam, f.dist_cutoff, g_k, g_dis);
        g_k[4] *= 0.f;
#pragma unroll
        for (int k = 0; k < 5; ++k) acc.intr[k] += f.k_grad_factor * g_k[k];
        g_dis[2] *= 0.25f;
#pragma unroll
        for (int k = 3; k < 8; ++k) g_dis[k] *= 0.1f;
#pragma unroll
        for (int k = 0; k < 8; ++k) acc.intr[5 + k] += f.dist_grad_factor * g_dis[k];
        acc.intr[kIntr ? 13 : 0] += (float)g.hits * (1.f / 1024.f);
    }
}

// Modes 1 and 2: approximate image-space gradient of a fragment from the neighbouring pixels
// (RenderBackward.cu:1347-1374).  `g` is the pixel in the global pixel space; the images are the channel-interleaved
// copies pack_images_kernel makes, so the eight neighbour values of all channels are eight 16-byte loads.
struct Neighbours
{
    float4 il, ir, iu, id, gl, gr, gu, gd;  // forward image and its gradient left / right / above / below the pixel
    __device__ __forceinline__ void load(const Frame& f, int g, int w)
    {
        const float4* I  = f.img4 + g;
        const float4* Gp = f.grad4 + g;
        il = __ldg(I - 1), ir = __ldg(I + 1), iu = __ldg(I - w), id = __ldg(I + w);
        gl = __ldg(Gp - 1), gr = __ldg(Gp + 1), gu = __ldg(Gp - w), gd = __ldg(Gp + w);
    }
    __device__ __forceinline__ float2 gradient(const Frame& f, float4 d) const
    {
        const float dv[4] = {d.x, d.y, d.z, d.w};
        const float Il[4] = {il.x, il.y, il.z, il.w}, Ir[4] = {ir.x, ir.y, ir.z, ir.w};
        const float Iu[4] = {iu.x, iu.y, iu.z, iu.w}, Id[4] = {id.x, id.y, id.z, id.w};
        const float Gl[4] = {gl.x, gl.y, gl.z, gl.w}, Gr[4] = {gr.x, gr.y, gr.z, gr.w};
        const float Gu[4] = {gu.x, gu.y, gu.z, gu.w}, Gd[4] = {gd.x, gd.y, gd.z, gd.w};
        float dx = 0.f, dy = 0.f;
#pragma unroll
        for (int ci = 0; ci < 4; ++ci)
        {
            if (ci < f.C)
            {
                float Tp = dv[ci];
                float a0 = -(Tp - Il[ci]) * Gl[ci];
                float a1 = (Tp - Ir[ci]) * Gr[ci];
                float b0 = -(Tp - Iu[ci]) * Gu[ci];
                float b1 = (Tp - Id[ci]) * Gd[ci];
                dx += 0.5f * (a0 + a1);
                dy += 0.5f * (b0 + b1);
            }
        }
        // x / 4 and x * 0.25 round alike
        return f.C == 4 ? make_float2(dx * 0.25f, dy * 0.25f) : make_float2(dx / (float)f.C, dy / (float)f.C);
    }
};

__device__ __forceinline__ float2 neighbour_gradient(const Frame& f, int g, int w, float4 d)
{
    Neighbours nb;
    nb.load(f, g, w);
    return nb.gradient(f, d);
}

__device__ __forceinline__ float4 load_grad(const Frame& f, int g) { return __ldg(f.grad4 + g); }

// Channel-interleaved copies of the forward image and of its gradient over the global pixel space (the caller's
// tensors are planar [view, channel, y, x] per level).
__device__ __forceinline__ float4 pack_pixel(const Frame& f, const BackPtrs& bp, long long r, int& view, int& l, int& o)
{
    // pixels in plain row-major order (view, level, y, x): coalesced reads of the planar tensors
    const int Prm = (int)f.Prm;
    view = 0, l = 0;
#pragma unroll
    for (int i = 1; i < VETR_MAX_VIEWS; ++i)
        if (i < f.n_views && r >= (long long)i * Prm) view = i;
    const int q = (int)(r - (long long)view * Prm);
#pragma unroll
    for (int i = 1; i < VETR_MAX_LAYERS; ++i)
        if (i < f.L && q >= (int)f.rbase[i]) l = i;
    o = q - (int)f.rbase[l];  // y * w + x
    const int hw   = f.lw[l] * f.lh[l];
    const float* I = bp.out_color[l] + (size_t)(view * f.C) * hw + o;
    const float* G = bp.grad_color[l] + (size_t)(view * f.C) * hw + o;
    const float4 g = make_float4(__ldg(G), __ldg(G + hw), __ldg(G + 2 * hw), f.C > 3 ? __ldg(G + 3 * hw) : 0.f);
    f.img4[r]  = make_float4(__ldg(I), __ldg(I + hw), __ldg(I + 2 * hw), f.C > 3 ? __ldg(I + 3 * hw) : 0.f);
    f.grad4[r] = g;
    return g;
}
__global__ void __launch_bounds__(256) pack_images_kernel(const __grid_constant__ Frame f, const __grid_constant__ BackPtrs bp)
{
    begin_kernel();
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int view, l, o;
    if (r < f.Prm * f.n_views) pack_pixel(f, bp, r, view, l, o);
}

__device__ __forceinline__ float dot4(float4 a, float4 b, int C)
{
    // same order as the reference's loop over channels (RenderBackward.cu:1146-1155)
    float r = 0.f;
    r += a.x * b.x;
    r += a.y * b.y;
    r += a.z * b.z;
    if (C > 3) r += a.w * b.w;
    return r;
}

// Image-space gradient of a fragment that takes no part in the position gradient (border pixel, cut-off list).
constexpr int kNoGradientBits = 0x7fffffff;

// Stage A of a fragment (needs nothing from the sweeps): streams the fragment's key and payload, computes d.G, and
// in modes 1 and 2 its image-space gradient (which depends on the descriptor and the neighbouring pixels only).  That
// gradient is parked under (view, level, point); point_backward_kernel turns it into position / camera gradients with
// coalesced position loads and without atomics, instead of a position gather per fragment here.
template <bool kBilinear>
__device__ __forceinline__ void fragment_stage_a(const Frame& f, BackSmem& s, int g, const PixInfo& px, float4 G, int slot,
                                                 uint4 h, uint4 payload, bool blended, float* depth_out = nullptr)
{
    const float4 d = as_float4(payload);
    const int pid  = (int)h.x;
    if (depth_out) depth_out[slot] = __uint_as_float(h.y);
    s.pid[slot]    = pid;
    s.tex[slot]    = (int)h.w;
    s.alpha[slot]  = __uint_as_float(h.z);
    s.dot[slot]    = dot4(d, G, f.C);
    if (!kBilinear && f.need_point_grad)
    {
        float2 dR = make_float2(__int_as_float(kNoGradientBits), 0.f);
        if (blended && px.interior) dR = neighbour_gradient(f, row_major_index(f, px), f.lw[px.level], d);
        f.point_grad[((size_t)px.view * f.L + px.level) * f.n + pid] = dR;
    }
}

// Stage B of a fragment (after the sweeps): the descriptor gradient, and the confidence gradient - directly in modes 1
// and 2; in mode 3 it is weighted by the bilinear weight of the fragment's corner, which needs the point's projection, so
// the fragment's alpha gradient is parked under (view, level, point, corner) for point_backward_kernel (the reference
// writes it for interior pixels only, RenderBackward.cu:3053).  `blended` = false: the list ended before this fragment.
template <bool kBilinear>
__device__ __forceinline__ void fragment_stage_b(const Frame& f, const BackPtrs& bp, const PixInfo& px, float4 G, int pid,
                                                 int tex_word, float Ta, float galpha, bool blended)
{
    if (kBilinear)
    {
        const int corner  = (unsigned)tex_word >> kCornerShift;
        float* parked     = reinterpret_cast<float*>(f.point_grad);
        const size_t slot = ((((size_t)px.view * f.L + px.level) * f.n + pid) << 2) + corner;
        parked[slot]      = blended && px.interior ? galpha : __int_as_float(kNoGradientBits);
        if (!blended) return;
    }
    const int tex = kBilinear ? tex_word & kTexMask : tex_word;
    // descriptor gradient: T * alpha * G  (RenderBackward.cu:1149-1152)
    red_add_v4(bp.g_desc + tex, make_float4(Ta * G.x, Ta * G.y, Ta * G.z, f.C > 3 ? Ta * G.w : 0.f));
    if (!kBilinear) red_add(bp.g_conf + tex, galpha);
}

// Transmittance forward and suffix sum backward over one list held in shared memory: the O(n) form of the
// reference's double loop (RenderBackward.cu:1118-1181).  Leaves T_i in trans[] and the suffix sum behind fragment i in
// suffix[]; what hangs on them (alpha_gradient: a division) is left to the fragment-parallel stage B.  The lists of a warp
// are swept side by side while the rest of the CTA waits, so what counts is the latency of a step: the chains are one
// multiplication and one addition, and the operands of four steps are requested together.  8 M points x 4 views, mode 1:
// backward_kernel 1591 -> 1123 us; mode 3, 3 M x 2: 741 -> 637 us (before: one step at a time, with its division).
template <bool kBilinear>
__device__ __forceinline__ void sweep_list(const Frame& f, BackSmem& s, int ss, int se, float4 G, float4 bgc,
                                           float bg_acc[4], float& p0_acc)
{
    const float* alpha = s.alpha + ss;
    const float* dot   = s.dot + ss;
    float* trans       = s.trans + ss;
    float* suffix      = suffix_of<kBilinear>(s) + ss;
    int cnt = se - ss;
    if (f.dbg_max_len > 0) cnt = min(cnt, f.dbg_max_len);
    float T = 1.f;
    int eff = cnt;
    int i   = 0;
    for (; i + 4 <= cnt; i += 4)
    {
        const float a0 = alpha[i], a1 = alpha[i + 1], a2 = alpha[i + 2], a3 = alpha[i + 3];
        const float t1 = vetr_new_T(T, a0), t2 = vetr_new_T(t1, a1), t3 = vetr_new_T(t2, a2), t4 = vetr_new_T(t3, a3);
        trans[i] = T, trans[i + 1] = t1, trans[i + 2] = t2, trans[i + 3] = t3;
        T = t4;
        if (kBilinear)
        {
            const int k = t1 < 0.001f ? 1 : t2 < 0.001f ? 2 : t3 < 0.001f ? 3 : t4 < 0.001f ? 4 : 0;
            if (k)
            {
                eff = i + k;
                T   = k == 1 ? t1 : k == 2 ? t2 : k == 3 ? t3 : t4;
                i   = cnt;
                break;
            }
        }
    }
    for (; i < cnt; ++i)
    {
        trans[i] = T;
        T        = vetr_new_T(T, alpha[i]);
        if (kBilinear && T < 0.001f)
        {
            eff = i + 1;
            break;
        }
    }
    for (int k = eff; k < se - ss; ++k) trans[k] = __int_as_float(0x7fffffff);  // NaN: not blended, no gradient
    const bool bg_term = !f.use_env && !(kBilinear && !(T >= 0.001f));
    float S = 0.f;
    if (bg_term)
    {
        float dotb = dot4(bgc, G, f.C);
        bg_acc[0] += T * 1.f * G.x, bg_acc[1] += T * 1.f * G.y, bg_acc[2] += T * 1.f * G.z;
        if (f.C > 3) bg_acc[3] += T * 1.f * G.w;
        if (!kBilinear && f.bg_alpha_to_point0) p0_acc += dotb * T;
        S = T * 1.f * dotb;
    }
    i = eff;
    for (; i >= 4; i -= 4)
    {
        const float T3 = trans[i - 1], T2 = trans[i - 2], T1 = trans[i - 3], T0 = trans[i - 4];
        const float a3 = alpha[i - 1], a2 = alpha[i - 2], a1 = alpha[i - 3], a0 = alpha[i - 4];
        const float d3 = dot[i - 1], d2 = dot[i - 2], d1 = dot[i - 3], d0 = dot[i - 4];
        const float S2 = S + T3 * a3 * d3, S1 = S2 + T2 * a2 * d2, S0 = S1 + T1 * a1 * d1;
        suffix[i - 1] = S, suffix[i - 2] = S2, suffix[i - 3] = S1, suffix[i - 4] = S0;
        S = S0 + T0 * a0 * d0;
    }
    for (; i > 0; --i)
    {
        suffix[i - 1] = S;
        S += trans[i - 1] * alpha[i - 1] * dot[i - 1];
    }
}

// d(loss)/d(alpha) of a fragment from what the sweeps left.
__device__ __forceinline__ float alpha_gradient(float T, float a, float dot, float suffix) { return T * dot - suffix / (1 - a + 1e-9f); }

// Mode 2 sweeps over one list (BlendBackwardsFuzzy, RenderBackward.cu:603-749) in O(n): groups are formed against the
// first depth of every group, the background is an entry of depth 100000 (confidence 1, colour = background), a
// group's descriptor / confidence gradients are shared equally by its fragments, and the term a later group passes to
// the confidence of an earlier fragment uses that fragment's GROUP confidence and is not divided by the group size.
//
// Three steps, with a barrier between them: fuzzy_groups (one thread per list) cuts the list into groups and runs the chain of
// transmittances, fuzzy_group_terms (a thread per fragment) forms what hangs on a group's mean colour, fuzzy_suffix (one
// thread per list) sums from the back; fuzzy_alpha_gradient puts a fragment's confidence gradient together.  Bound by the latency
// of the two chains, which are down to a comparison and a multiplication, and an addition, per fragment; four groups of one
// fragment each go through a step together.  1 M points, 801x603, one view: backward_kernel 295 -> 169 us, lists of more than 256
// fragments 105 -> 61 us (before: everything in the list's own thread, descriptors in shared memory, half as many CTAs per SM).
//
// fuzzy_groups: n fragments of one list.  Leaves the transmittance in front of its group in trans[] (NaN = not blended), the
// group's confidence in alpha[], and in group[], which takes the memory of depth[], its number of members at the first of
// them (negative if the background belongs to the group too; it is not counted) and 0 at the others.  Returns the suffix sum
// behind the last fragment.
__device__ __forceinline__ float fuzzy_groups(const Frame& f, float* alpha, float* trans, float* depth, int n, float4 G, float4 bgc,
                                              float bg_acc[4])
{
    int* group = reinterpret_cast<int*>(depth);
    int cnt    = n;
    if (f.dbg_max_len > 0) cnt = min(cnt, f.dbg_max_len);
    const float accept = f.accept_blend;
    bool background    = !f.use_env;  // still to come
    float T            = 1.f;
    int i              = 0;
    while (i < cnt)
    {
        const float d0 = depth[i];
        if (i > 0 && i + 4 < cnt)
        {
            const float d1 = depth[i + 1], d2 = depth[i + 2], d3 = depth[i + 3], d4 = depth[i + 4];
            if (!(d1 - d0 < accept) && !(d2 - d1 < accept) && !(d3 - d2 < accept) && !(d4 - d3 < accept))
            {
                const float t1 = vetr_new_T(T, alpha[i]), t2 = vetr_new_T(t1, alpha[i + 1]), t3 = vetr_new_T(t2, alpha[i + 2]);
                trans[i] = T, trans[i + 1] = t1, trans[i + 2] = t2, trans[i + 3] = t3;
                T        = vetr_new_T(t3, alpha[i + 3]);
                group[i] = group[i + 1] = group[i + 2] = group[i + 3] = 1;
                i += 4;
                continue;
            }
        }
        // one group: fragments within `accept` of its first depth (the first group of a list may also be measured from 0)
        const float ref = i == 0 && d0 < accept ? 0.f : d0;
        float conf      = alpha[i];
        int j           = i + 1;
        for (; j < cnt && depth[j] - ref < accept; ++j) conf += alpha[j];
        const bool joined = background && j == cnt && kMaxDepth - ref < accept;
        const int members = j - i;
        float inv_w       = 1.f;
        if (joined) conf += 1.f;
        if (members + joined > 1) inv_w = 1.f / (float)(members + joined), conf *= inv_w;
        for (int t = i; t < j; ++t) trans[t] = T, alpha[t] = conf, group[t] = 0;
        group[i] = joined ? -members : members;
        if (joined)
        {
            bg_acc[0] += T * conf * G.x * inv_w, bg_acc[1] += T * conf * G.y * inv_w, bg_acc[2] += T * conf * G.z * inv_w;
            if (f.C > 3) bg_acc[3] += T * conf * G.w * inv_w;
            background = false;
        }
        T = vetr_new_T(T, conf);
        i = j;
    }
    for (i = cnt; i < n; ++i) trans[i] = __int_as_float(0x7fffffff), group[i] = 0;
    if (!background) return 0.f;
    bg_acc[0] += T * G.x, bg_acc[1] += T * G.y, bg_acc[2] += T * G.z;
    if (f.C > 3) bg_acc[3] += T * G.w;
    float v = G.x * bgc.x * T + G.y * bgc.y * T + G.z * bgc.z * T;
    if (f.C > 3) v += G.w * bgc.w * T;
    return v;
}

// The thread of a group's first fragment i, for all members: the factor of G of the descriptor gradient in trans[], the group's
// own part of the confidence gradient in dot[] (d . G on entry), and in suffix[] what the group passes to the ones before it
// (the other members hold a zero).  The mean colour of several members is summed in list order.  recs: the list's records.
__device__ __forceinline__ void fuzzy_group_terms(const Frame& f, const float* alpha, float* dot, float* trans, float* suffix,
                                                  int group, const uint4* recs, int i, float4 G, float4 bgc)
{
    const int members = abs(group);
    const float T = trans[i], conf = alpha[i];
    float4 col    = as_float4(recs[2 * i + 1]);
    float inv_w = 1.f, q = dot[i];
    if (group != 1)
    {
        for (int t = 1; t < members; ++t)
        {
            const float4 d = as_float4(recs[2 * (i + t) + 1]);
            col.x += d.x, col.y += d.y, col.z += d.z, col.w += d.w;
        }
        if (group < 0) col.x += bgc.x, col.y += bgc.y, col.z += bgc.z, col.w += bgc.w;
        inv_w = 1.f / (float)(members + (group < 0));
        col.x *= inv_w, col.y *= inv_w, col.z *= inv_w, col.w *= inv_w;
        q = dot4(col, G, f.C);
    }
    const float g_alpha = q * T;
    float v = 0.f;
    v += G.x * col.x * T * conf;
    v += G.y * col.y * T * conf;
    v += G.z * col.z * T * conf;
    if (f.C > 3) v += G.w * col.w * T * conf;
    for (int t = i; t < i + members; ++t)
    {
        trans[t]  = T * conf * inv_w;
        dot[t]    = g_alpha * inv_w;
        suffix[t] = t == i ? v : 0.f;
    }
}

// Sums what the groups behind a fragment's group pass to it; S: what comes from behind the list.
__device__ __forceinline__ void fuzzy_suffix(const Frame& f, float* suffix, int n, float S)
{
    int i = n;
    if (f.dbg_max_len > 0) i = min(i, f.dbg_max_len);
    for (; i >= 4; i -= 4)
    {
        const float v3 = suffix[i - 1], v2 = suffix[i - 2], v1 = suffix[i - 3], v0 = suffix[i - 4];
        const float S2 = S + v3, S1 = S2 + v2, S0 = S1 + v1;
        suffix[i - 1] = S, suffix[i - 2] = S2, suffix[i - 3] = S1, suffix[i - 4] = S0;
        S = S0 + v0;
    }
    for (; i > 0; --i)
    {
        const float v = suffix[i - 1];
        suffix[i - 1] = S;
        S += v;
    }
}

__device__ __forceinline__ float fuzzy_alpha_gradient(float conf, float dot, float suffix) { return dot - suffix / (1 - conf + 1e-9f); }

// Background gradient and the confidence term the reference routes to descriptor 0: CTA reduction, one atomic each.
__device__ __forceinline__ void reduce_background(const Frame& f, const BackPtrs& bp, BackSmem& s, const float bg_acc[4],
                                                  float p0_acc)
{
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float v[5] = {bg_acc[0], bg_acc[1], bg_acc[2], bg_acc[3], p0_acc};
    for (int k = 0; k < 5; ++k)
    {
        float x = v[k];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) s.red[warp][k] = (double)x;
    }
    __syncthreads();
    if (threadIdx.x < 5)
    {
        float x = 0.f;
        for (int w = 0; w < kThreads / 32; ++w) x += (float)s.red[w][threadIdx.x];
        if (x != 0.f)
        {
            if (threadIdx.x < 4)
            {
                if ((int)threadIdx.x < f.C) atomicAdd(bp.g_background + threadIdx.x, x);
            }
            else
                atomicAdd(bp.g_conf + 0, x);
        }
    }
}


template <bool kFuzzy, bool kBilinear>
struct BackSmemOf
{
    using type = BackSmem;
};
template <>
struct BackSmemOf<true, false>
{
    using type = BackSmemFuzzy;
};
template <>
struct BackSmemOf<false, true>
{
    using type = BackSmemSuffix;
};

// Position / camera gradients are left to point_backward_kernel in every mode.
template <bool kFuzzy, bool kBilinear>
__global__ void __launch_bounds__(kThreads, kBackCtas) backward_kernel(const __grid_constant__ Frame f,
                                                                       const __grid_constant__ BackPtrs bp)
{
    begin_kernel();
    static_assert(!(kFuzzy && kBilinear), "mode 2 and mode 3 exclude each other");
    using Smem = typename BackSmemOf<kFuzzy, kBilinear>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem& s = *reinterpret_cast<Smem*>(smem_raw);
    const int tid     = threadIdx.x;
    const float4 bgc  = make_float4(f.background[0], f.background[1], f.background[2], f.C > 3 ? f.background[3] : 0.f);
    float bg_acc[4] = {0.f, 0.f, 0.f, 0.f};
    float p0_acc    = 0.f;
    if (tid == 0) s.seg.n_long[0] = s.seg.n_long[1] = 0;
    int parity = 0;

    ItemStream items(f);
    int lo, np, f0, nf;
    while (items.next(f, lo, np, f0, nf))
    {
        if (np <= 0) continue;
        {
            __syncthreads();  // every warp has left the previous item
            parity ^= 1;
            if (tid == 0) s.seg.n_long[parity ^ 1] = 0;
            if (tid < np)
            {
                const int ss = list_end(f, lo + tid - 1) - f0, se = f.ends[lo + tid] - f0;
                s.seg_end[tid + 1] = se;
                const PixInfo px   = decode_pixel(f, (unsigned)(lo + tid));
                s.pix[tid]         = px;
                s.grad[tid]        = px.valid ? load_grad(f, row_major_index(f, px)) : make_float4(0.f, 0.f, 0.f, 0.f);
                seg_fill(s.seg, parity, tid, ss, se);
            }
            if (tid == 0) s.seg_end[0] = 0;
            __syncthreads();
            for (int i = tid; i < nf; i += kThreads)
            {
                // Measured slower, both times through registers (spills, or one resident CTA less): requesting the next
                // record before working on this one; requesting the eight neighbour values together with the record.
                uint4 h, d;
                load_record(f, f0 + i, h, d);
                const int a = seg_lookup(s.seg, parity, s.seg_end, i);
                const bool blended = f.dbg_max_len <= 0 || i - s.seg_end[a] < f.dbg_max_len;  // list truncation
                if constexpr (kFuzzy)
                    fragment_stage_a<false>(f, s, lo + a, s.pix[a], s.grad[a], i, h, d, blended, s.depth);
                else
                    fragment_stage_a<kBilinear>(f, s, lo + a, s.pix[a], s.grad[a], i, h, d, blended);
            }
            __syncthreads();
            [[maybe_unused]] float S_behind = 0.f;
            if (tid < np && s.pix[tid].valid)
            {
                if constexpr (kFuzzy)
                {
                    const int ss = s.seg_end[tid];
                    S_behind     = fuzzy_groups(f, s.alpha + ss, s.trans + ss, s.depth + ss, s.seg_end[tid + 1] - ss, s.grad[tid], bgc, bg_acc);
                }
                else
                    sweep_list<kBilinear>(f, s, s.seg_end[tid], s.seg_end[tid + 1], s.grad[tid], bgc, bg_acc, p0_acc);
            }
            __syncthreads();
            if constexpr (kFuzzy)
            {
                for (int i = tid; i < nf; i += kThreads)
                    if (const int group = __float_as_int(s.depth[i]))
                        fuzzy_group_terms(f, s.alpha, s.dot, s.trans, suffix_of<false>(s), group, f.recs + 2 * (size_t)f0, i,
                                          s.grad[seg_lookup(s.seg, parity, s.seg_end, i)], bgc);
                __syncthreads();
                if (tid < np) fuzzy_suffix(f, suffix_of<false>(s) + s.seg_end[tid], s.seg_end[tid + 1] - s.seg_end[tid], S_behind);
                __syncthreads();
            }
            for (int i = tid; i < nf; i += kThreads)
            {
                const float Ti     = s.trans[i];
                const bool blended = Ti == Ti;  // NaN: the list ended before this fragment
                if (!kBilinear && !blended) continue;
                const int a = seg_lookup(s.seg, parity, s.seg_end, i);
                const float al = s.alpha[i], suffix = suffix_of<kBilinear>(s)[i];
                const float galpha = kFuzzy ? fuzzy_alpha_gradient(al, s.dot[i], suffix) : alpha_gradient(Ti, al, s.dot[i], suffix);
                const float Ta     = kFuzzy ? Ti : Ti * al;
                fragment_stage_b<kBilinear>(f, bp, s.pix[a], s.grad[a], kBilinear ? s.pid[i] : 0, s.tex[i], Ta, galpha, blended);
            }
        }
    }
    reduce_background(f, bp, s, bg_acc, p0_acc);
}

// Lists longer than kLongList, beside the end of backward_kernel: one CTA per list, blocks of kCap fragments, a forward sweep that records the
// transmittance at every block start and a backward sweep over the blocks that carries the suffix sum.  One thread runs the
// two chains of a list (transmittance: a multiplication per fragment; suffix sum: an addition); the division and the
// products that hang on them are left to all threads.  Bound by those chains, hence as many lists in flight as fit an SM:
// 8 M points x 4 views, mode 1: 559 -> 40 us; 3 M x 2 views, mode 3: 535 -> 74 us (before: one CTA per SM, both sweeps with
// their divisions in one thread).
template <bool kBilinear>
__global__ void __launch_bounds__(kThreads) backward_long_kernel(const __grid_constant__ Frame f,
                                                                 const __grid_constant__ BackPtrs bp)
{
    const BesidePrevious<> beside;
    if (f.status[2] <= kLongList) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BackSmemSuffix& s = *reinterpret_cast<BackSmemSuffix*>(smem_raw);
    __shared__ float s_T, s_S;
    __shared__ int s_stop;
    __shared__ float s_block_T[256];  // transmittance at block starts; lists beyond 256 * kCap fragments are cut there
    const int tid       = threadIdx.x;
    const int n_items   = f.status[3];
    constexpr bool bilinear = kBilinear;
    const float4 bgc    = make_float4(f.background[0], f.background[1], f.background[2], f.C > 3 ? f.background[3] : 0.f);
    float bg_acc[4] = {0.f, 0.f, 0.f, 0.f};
    float p0_acc    = 0.f;

    __shared__ int s_long_hits[kThreads], s_long_count;
    LongItemScan scan;
    int lo;
    while (scan.next(f, n_items, s_long_hits, &s_long_count, lo))
    {
        const int e0 = list_end(f, lo - 1);
        const int n  = f.ends[lo] - e0;
        const PixInfo px = decode_pixel(f, (unsigned)lo);
        const float4 G = load_grad(f, row_major_index(f, px));
        int cnt = n;
        if (f.dbg_max_len > 0) cnt = min(cnt, f.dbg_max_len);
        cnt = min(cnt, 256 * kCap);
        if (tid == 0) s_T = 1.f, s_stop = cnt;
        __syncthreads();
        // sweep 1: transmittances, those at block starts, and the position where a mode-3 list stops
        for (int blk = 0; blk * kCap < s_stop; ++blk)
        {
            const int m = min(kCap, cnt - blk * kCap);
            for (int i = tid; i < m; i += kThreads) s.alpha[i] = __uint_as_float(f.recs[2 * (size_t)(e0 + blk * kCap + i)].z);
            if (m + tid < ((m + 3) & ~3)) s.alpha[m + tid] = 0.f;
            __syncthreads();
            if (tid == 0)
            {
                const float T  = s_T;
                s_block_T[blk] = T;
                int used       = m;
                const float T_end = transmittance_chain<kBilinear>(s.alpha, s.trans, used, T);
                s_T = T_end;
                if (bilinear && T_end < 0.001f) s_stop = blk * kCap + used;
            }
            __syncthreads();
        }
        const int eff_cnt = s_stop;
        if (tid == 0)
        {
            const float T_end  = s_T;
            const bool bg_term = !f.use_env && !(bilinear && !(T_end >= 0.001f));
            float S = 0.f;
            if (bg_term)
            {
                float dotb = dot4(bgc, G, f.C);
                bg_acc[0] += T_end * 1.f * G.x, bg_acc[1] += T_end * 1.f * G.y, bg_acc[2] += T_end * 1.f * G.z;
                if (f.C > 3) bg_acc[3] += T_end * 1.f * G.w;
                if (!bilinear && f.bg_alpha_to_point0) p0_acc += dotb * T_end;
                S = T_end * 1.f * dotb;
            }
            s_S = S;
        }
        // sweep 2: blocks back to front
        const int last = (eff_cnt + kCap - 1) / kCap - 1;
        for (int blk = last; blk >= 0; --blk)
        {
            const int m = min(kCap, eff_cnt - blk * kCap);
            for (int i = tid; i < m; i += kThreads)
                fragment_stage_a<kBilinear>(f, s, lo, px, G, i, f.recs[2 * (size_t)(e0 + blk * kCap + i)],
                                            f.recs[2 * (size_t)(e0 + blk * kCap + i) + 1], true);
            __syncthreads();
            if (tid == 0)
            {
                if (blk != last)  // sweep 1 left the last block's transmittances in place
                {
                    int used = m;
                    transmittance_chain<false>(s.alpha, s.trans, used, s_block_T[blk]);
                }
                float S = s_S;
                int i   = m;
                for (; i & 3; --i)
                {
                    s.after[i - 1] = S;
                    S += s.trans[i - 1] * s.alpha[i - 1] * s.dot[i - 1];
                }
                for (; i > 0; i -= 4)
                {
                    const float4 T = *reinterpret_cast<const float4*>(s.trans + i - 4);
                    const float4 a = *reinterpret_cast<const float4*>(s.alpha + i - 4);
                    const float4 d = *reinterpret_cast<const float4*>(s.dot + i - 4);
                    const float S1 = S + T.w * a.w * d.w, S2 = S1 + T.z * a.z * d.z, S3 = S2 + T.y * a.y * d.y;
                    *reinterpret_cast<float4*>(s.after + i - 4) = make_float4(S3, S2, S1, S);
                    S = S3 + T.x * a.x * d.x;
                }
                s_S = S;
            }
            __syncthreads();
            for (int i = tid; i < m; i += kThreads)
            {
                const float a = s.alpha[i], Ti = s.trans[i];
                fragment_stage_b<kBilinear>(f, bp, px, G, s.pid[i], s.tex[i], Ti * a, alpha_gradient(Ti, a, s.dot[i], s.after[i]), true);
            }
            __syncthreads();
        }
        // fragments behind the cut take no part in the position gradient (mode 3: nor in the confidence gradient)
        if (kBilinear || f.need_point_grad)
            for (int i = eff_cnt + tid; i < n; i += kThreads)
            {
                const uint4 h = f.recs[2 * (size_t)(e0 + i)];
                if (kBilinear)
                    fragment_stage_b<kBilinear>(f, bp, px, G, (int)h.x, (int)h.w, 0.f, 0.f, false);
                else
                    f.point_grad[((size_t)px.view * f.L + px.level) * f.n + (int)h.x] = make_float2(__int_as_float(kNoGradientBits), 0.f);
            }
    }
    reduce_background(f, bp, s, bg_acc, p0_acc);
}

// Mode 2, lists longer than kLongList: one CTA per list with the whole list staged (the group structure does not split
// into blocks), beside the end of backward_kernel (mode 2, 1 M points, 801x603: the whole call 431 -> 373 us).  Lists beyond kFuzzyLongMax are skipped and flagged in the status word (the reference itself sorts only
// the first 4096 fragments of a list, AlphaListSort.cu:289-290, so its result for longer lists is not defined either).
//
// Launched twice, beside backward_kernel and each other: lists of up to kFuzzyMidMax fragments, eight of which fit an SM, and the longer ones, one per
// SM.  Two steps of a list are one thread's chain each (fuzzy_groups, fuzzy_suffix), so a launch with few lists takes as long as the longest of them.
// A training step without a drop-out radius, us, line at 512 / 1024 / 2048 / 4095: 60 k points, 8 views 200x150 (longest list 578) 364 / 353 / 430 /
// 440; 200 k, one view (1256) 448 / 410 / 397 / 447; 400 k, 4 views 400x300 (1110) 948 / 833 / 986 / 1091; 1 M, 8 views 801x603 (1545) 3250 / 2853 /
// 3010 / 3397; with the radius, 1 M, one view (179), no difference.
constexpr int kFuzzyLongMax = 4096;  // what the reference sorts of a list (AlphaListSort.cu:289-290)
constexpr int kFuzzyMidMax  = 1024;
template <int kMax>
struct FuzzyLongSmem
{
    int tex[kMax];
    float alpha[kMax];
    float dot[kMax];
    float trans[kMax];
    float depth[kMax];
    float suffix[kMax];
};

// Lists of more than kMin and up to kMax fragments.
template <int kMin, int kMax>
__global__ void __launch_bounds__(kThreads) backward_fuzzy_long_kernel(const __grid_constant__ Frame f,
                                                                       const __grid_constant__ BackPtrs bp)
{
    const BesidePrevious<kMin == kLongList> beside;
    if (f.status[2] <= kMin) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FuzzyLongSmem<kMax>& s = *reinterpret_cast<FuzzyLongSmem<kMax>*>(smem_raw);
    const int tid     = threadIdx.x;
    const int n_items = f.status[3];
    const float4 bgc  = make_float4(f.background[0], f.background[1], f.background[2], f.C > 3 ? f.background[3] : 0.f);
    float bg_acc[4] = {0.f, 0.f, 0.f, 0.f};
    __shared__ int s_long_hits[kThreads], s_long_count;
    LongItemScan scan;
    int lo;
    while (scan.next(f, n_items, s_long_hits, &s_long_count, lo))
    {
        const int e0 = list_end(f, lo - 1);
        const int n  = f.ends[lo] - e0;
        if (n > kMax || n <= kMin)
        {
            if (n > kFuzzyLongMax && kMax == kFuzzyLongMax && tid == 0) atomicOr(f.status + 1, 2);
            continue;
        }
        const PixInfo px = decode_pixel(f, (unsigned)lo);
        const float4 G = load_grad(f, row_major_index(f, px));
        __syncthreads();  // every warp has left the previous list
        const bool spatial = px.interior;
        for (int i = tid; i < n; i += kThreads)
        {
            const uint4 h  = f.recs[2 * (size_t)(e0 + i)];
            const float4 d = as_float4(f.recs[2 * (size_t)(e0 + i) + 1]);
            s.tex[i] = (int)h.w, s.alpha[i] = __uint_as_float(h.z), s.depth[i] = __uint_as_float(h.y);
            s.dot[i] = dot4(d, G, f.C);
            const bool blended = f.dbg_max_len <= 0 || i < f.dbg_max_len;
            if (f.need_point_grad)
                f.point_grad[((size_t)px.view * f.L + px.level) * f.n + (int)h.x] =
                    spatial && blended ? neighbour_gradient(f, row_major_index(f, px), f.lw[px.level], d)
                                       : make_float2(__int_as_float(kNoGradientBits), 0.f);
        }
        __syncthreads();
        float S_behind = 0.f;
        if (tid == 0) S_behind = fuzzy_groups(f, s.alpha, s.trans, s.depth, n, G, bgc, bg_acc);
        __syncthreads();
        for (int i = tid; i < n; i += kThreads)
            if (const int group = __float_as_int(s.depth[i]))
                fuzzy_group_terms(f, s.alpha, s.dot, s.trans, s.suffix, group, f.recs + 2 * (size_t)e0, i, G, bgc);
        __syncthreads();
        if (tid == 0) fuzzy_suffix(f, s.suffix, n, S_behind);
        __syncthreads();
        for (int i = tid; i < n; i += kThreads)
        {
            const float coef = s.trans[i];
            if (coef != coef) continue;
            red_add_v4(bp.g_desc + s.tex[i], make_float4(coef * G.x, coef * G.y, coef * G.z, f.C > 3 ? coef * G.w : 0.f));
            red_add(bp.g_conf + s.tex[i], fuzzy_alpha_gradient(s.alpha[i], s.dot[i], s.suffix[i]));
        }
    }
    if (tid == 0)
        for (int ci = 0; ci < f.C; ++ci)
            if (bg_acc[ci] != 0.f) atomicAdd(bp.g_background + ci, bg_acc[ci]);
}

// ---------------------------------------------------------------------------------------------------------
// Position, pose and intrinsics gradients (and the confidence gradient of mode 3), one pass over the points.
//
// Modes 1 and 2: ProjectPointPinholeBackward of the image-space gradients that stage A parked for the point's fragments.
// Mode 3: the fragments' alpha gradients were parked under (view, level, point, corner); here the point is projected once
// per view exactly as the forward pass did (same bits), which gives the corner weights and their Jacobians
// (compute_blending_fac) of all its fragments: confidence gradient += w * g_alpha, image-space gradient =
// J_uv * confidence * g_alpha (RenderBackward.cu:3076-3180).  Every fragment's position term is formed on its own and has the
// bits of the per-fragment form; the camera gradients take the image-space gradient of a point and view summed over levels
// and corners (PointGrad).  Positions, masks and parked values are read coalesced; a point's gradient is added to g_points
// by the one thread that owns the point.
//
// Bound by instruction issue.  A CTA owns `tiles` runs of 256 points and takes them view by view, so that the camera
// sums - 21 doubles over the CTA - are formed once per (CTA, view); the points' sums stay in shared memory meanwhile.
// 8 M points x 4 views with pose and intrinsics gradients: 1638 us with one reduction per 512 points and the camera chain per
// fragment, 600 us like this; mode 3, 3 M points x 2 views: 1587 -> 326 us.
constexpr int kPointTilesMax = 8;

// kCam: 0 = no camera gradients (their sums are not kept: a step of 20 M points and 8 views 1.5 % slower with them than before they were
// fp64, 1.4 % faster without), 1 = pose, 2 = intrinsics (and the pose where it is wanted).
template <int kCam, bool kBilinear>
__global__ void __launch_bounds__(kProjThreads, kCam == 2 || kBilinear ? 3 : 4)
    point_backward_kernel(const __grid_constant__ Frame f, const __grid_constant__ BackPtrs bp, int tiles)
{
    begin_kernel();
    extern __shared__ __align__(16) float4 s_gp[];  // [tiles][kProjThreads], every thread its own column
    __shared__ Camera s_cam[VETR_MAX_VIEWS];
    __shared__ double s_red[kProjThreads / 32][kCamValues];
    if (f.status[1] != 0) return;  // overflow / skipped list: some fragments never parked a value
    if (threadIdx.x < f.n_views) s_cam[threadIdx.x] = load_camera(f, threadIdx.x);
    __syncthreads();
    const int first      = blockIdx.x * (kProjThreads * tiles) + threadIdx.x;
    constexpr bool kIntr = kCam == 2;
    const bool spatial   = f.need_point_grad != 0;
    for (int it = 0; it < tiles; ++it) s_gp[it * kProjThreads + threadIdx.x] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int b = 0; b < f.n_views; ++b)
    {
        CamAcc<kIntr> acc;
        acc.clear();
        bool any = false;
        const unsigned char* masks = f.level_mask + (size_t)b * f.n;
        unsigned next_mask         = first < f.n ? masks[first] : 0u;  // requested one tile ahead
        for (int it = 0; it < tiles; ++it)
        {
            const int pid       = first + it * kProjThreads;
            const unsigned mask = next_mask;
            next_mask           = it + 1 < tiles && pid + kProjThreads < f.n ? masks[pid + kProjThreads] : 0u;
            if (!mask) continue;
            const float4 pos = __ldg(f.position + pid);
            float4 gp        = s_gp[it * kProjThreads + threadIdx.x];
            PointGrad g;
            g.clear();
            PointJac jac;
            if constexpr (!kBilinear)
            {
                float2 dR[VETR_MAX_LAYERS];
#pragma unroll
                for (int l = 0; l < VETR_MAX_LAYERS; ++l)
                    if (mask >> l & 1u) dR[l] = f.point_grad[((size_t)b * f.L + l) * f.n + pid];
                if (!project_backward_prepare(pos, s_cam[b], f.dist_cutoff, jac)) continue;
#pragma unroll
                for (int l = 0; l < VETR_MAX_LAYERS; ++l)
                    if ((mask >> l & 1u) && __float_as_int(dR[l].x) != kNoGradientBits)
                    {
                        if (kCam) g.add(dR[l], l);
                        point_terms(s_cam[b], jac, dR[l], l, gp);
                    }
            }
            else
            {
                const float* parked = reinterpret_cast<const float*>(f.point_grad);
                float4 ga[VETR_MAX_LAYERS];  // the four corners' alpha gradients of every level
#pragma unroll
                for (int l = 0; l < VETR_MAX_LAYERS; ++l)
                    if (mask >> l & 1u) ga[l] = *reinterpret_cast<const float4*>(parked + ((((size_t)b * f.L + l) * f.n + pid) << 2));
                const int tex      = __ldg(f.index + pid);
                const float conf   = __ldg(f.confidence + tex);
                const Projected pr = project_point(pos, s_cam[b], f.dist_cutoff);
                const bool jac_ok  = spatial && project_backward_prepare(pos, s_cam[b], f.dist_cutoff, jac);
                float2 ip   = pr.ip;
                float gconf = 0.f;
#pragma unroll
                for (int l = 0; l < VETR_MAX_LAYERS; ++l, ip.x *= 0.5f, ip.y *= 0.5f)
                {
                    if (!(mask >> l & 1u)) continue;
                    const int bx = round_down(ip.x), by = round_down(ip.y);
                    const float gl[4] = {ga[l].x, ga[l].y, ga[l].z, ga[l].w};
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                    {
                        // the same in-image test as the collection pass: corners outside never became fragments
                        const int x = bx + (c & 1), y = by + (c >> 1);
                        if ((unsigned)x >= (unsigned)f.lw[l] || (unsigned)y >= (unsigned)f.lh[l]) continue;
                        if (__float_as_int(gl[c]) == kNoGradientBits) continue;
                        float jx, jy;
                        const float w = blending_fac(ip, c, &jx, &jy);
                        gconf += w * gl[c];  // RenderBackward.cu:3076-3079
                        if (!jac_ok) continue;
                        const float single = conf * gl[c];
                        const float2 dR    = make_float2(jx * single, jy * single);
                        if (kCam) g.add(dR, l);
                        point_terms(s_cam[b], jac, dR, l, gp);
                    }
                }
                if (gconf != 0.f) red_add(bp.g_conf + tex, gconf);
            }
            s_gp[it * kProjThreads + threadIdx.x] = gp;
            if (kCam && g.hits)
            {
                camera_terms<kIntr>(f, s_cam[b], jac, g, acc);
                any = true;
            }
        }
        if (kCam && __syncthreads_or(any)) reduce_cam<kIntr>(f, bp, acc, b, s_red);
    }
    if (bp.g_points)
        for (int it = 0; it < tiles; ++it)
        {
            const int pid   = first + it * kProjThreads;
            const float4 gp = s_gp[it * kProjThreads + threadIdx.x];
            if (pid < f.n && gp.w != 0.f)
            {
                float4 cur = bp.g_points[pid];
                cur.x += gp.x, cur.y += gp.y, cur.z += gp.z, cur.w += gp.w;
                bp.g_points[pid] = cur;
            }
        }
}

// ---------------------------------------------------------------------------------------------------------
// Mode 0 (FUZZY_DT): no lists.  Per pixel: nearest depth (int bits, in `ends`), accumulators in the fragment buffer
// (record g: float4 descriptor sum, then the number of accepted points as a float), count of accepted points (`counts`).

// Mode 0 without interleaved copies (no pixel scratch, or fewer points than pixels) reads the caller's planar images: one
// 4-byte load per channel.
__device__ __forceinline__ float2 neighbour_gradient_planar(const Frame& f, const BackPtrs& bp, const PixInfo& px, float4 d)
{
    const int w = f.lw[px.level], h = f.lh[px.level];
    const int hw = w * h;
    const int o  = (px.view * f.C) * hw + px.y * w + px.x;
    const float* I  = bp.out_color[px.level] + o;
    const float* Gp = bp.grad_color[px.level] + o;
    float dx = 0.f, dy = 0.f;
    const float dv[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
    for (int ci = 0; ci < 4; ++ci)
    {
        if (ci < f.C)
        {
            const float* Ic = I + ci * hw;
            const float* Gc = Gp + ci * hw;
            float Tp = dv[ci];
            float a0 = -(Tp - __ldg(Ic - 1)) * __ldg(Gc - 1);
            float a1 = (Tp - __ldg(Ic + 1)) * __ldg(Gc + 1);
            float b0 = -(Tp - __ldg(Ic - w)) * __ldg(Gc - w);
            float b1 = (Tp - __ldg(Ic + w)) * __ldg(Gc + w);
            dx += 0.5f * (a0 + a1);
            dy += 0.5f * (b0 + b1);
        }
    }
    return make_float2(dx / (float)f.C, dy / (float)f.C);
}

__device__ __forceinline__ float4 load_grad_planar(const Frame& f, const BackPtrs& bp, const PixInfo& px)
{
    const int w = f.lw[px.level], h = f.lh[px.level];
    const int hw = w * h;
    const float* G = bp.grad_color[px.level] + (px.view * f.C) * hw + px.y * w + px.x;
    float4 g;
    g.x = __ldg(G);
    g.y = __ldg(G + hw);
    g.z = __ldg(G + 2 * hw);
    g.w = f.C > 3 ? __ldg(G + 3 * hw) : 0.f;
    return g;
}

// Start of a call: no depth, empty accumulators, status.
__global__ void __launch_bounds__(256) fuzzy_dt_clear_kernel(const __grid_constant__ Frame f)
{
    begin_kernel();
    const long long g = (long long)blockIdx.x * 256 + threadIdx.x;
    if (g < f.PT)
    {
        f.ends[g]      = __float_as_int(kMaxDepth);
        const uint4 no = make_uint4(0u, 0u, 0u, 0u);
        store_sector(f.recs + 2 * (size_t)g, no, no);
    }
    if (g < 4) f.status[g] = 0;
}

// kPass 0: DepthPrepassMulti (RenderForward.cu:180-308; no drop-out test).  kPass 1: RenderForwardMulti (:312-406).
template <int kPass>
__global__ void __launch_bounds__(kProjThreads) fuzzy_dt_point_kernel(const __grid_constant__ Frame f)
{
    begin_kernel();
    __shared__ Camera s_cam;
    const int b = blockIdx.y;
    if (threadIdx.x == 0) s_cam = load_camera(f, b);
    __syncthreads();
    const Camera& cam = s_cam;
    const int vbase   = b * (int)f.P;
    const int pid     = blockIdx.x * kProjThreads + threadIdx.x;
    if (pid >= f.n) return;
    const int tex = __ldg(f.index + pid);
    if (f.viewer_only && f.confidence[tex] < f.stability_cutoff) return;
    if (kPass == 1 && f.dropout && f.dropout[(size_t)b * f.n + pid] == 1.f) return;
    const Projected pr = project_point(__ldg(f.position + pid), cam, f.dist_cutoff);
    if (pr.z == 0.f) return;
    float2 ip    = pr.ip;
    float radius = pr.radius_px;
    float4 desc  = make_float4(0.f, 0.f, 0.f, 0.f);
    if (kPass == 1)
    {
        desc.x = __ldg(f.texture + tex);
        desc.y = __ldg(f.texture + (size_t)f.n_tex + tex);
        desc.z = __ldg(f.texture + 2 * (size_t)f.n_tex + tex);
        desc.w = f.C > 3 ? __ldg(f.texture + 3 * (size_t)f.n_tex + tex) : 0.f;
    }
    for (int l = 0; l < f.L; ++l, radius *= 0.5f, ip.x *= 0.5f, ip.y *= 0.5f)
    {
        if (f.drop_by_radius && radius < f.radius_threshold) break;
        const int lw = f.lw[l], lh = f.lh[l];
        const int x = round_half_even(ip.x), y = round_half_even(ip.y);
        if ((unsigned)x >= (unsigned)lw || (unsigned)y >= (unsigned)lh) continue;
        const int g = vbase + (int)f.lbase[l] + pixel_offset(lw, x, y);
        if (kPass == 0)
            atomicMin(f.ends + g, __float_as_int(pr.z));  // z > 0: integer order = float order
        else
        {
            const float image_depth = __int_as_float(f.ends[g]);
            if (pr.z > image_depth * (f.depth_accept + 1)) continue;
            red_add_v4(reinterpret_cast<float4*>(f.recs + 2 * (size_t)g), desc);
            red_add(reinterpret_cast<float*>(f.recs + 2 * (size_t)g + 1), 1.f);
        }
    }
}

// CombineAndFill (PointRenderer.cu:24-52) + CreateMask + depth output, one thread per pixel of the pixel space.
__global__ void __launch_bounds__(256) fuzzy_dt_combine_kernel(const __grid_constant__ Frame f, const __grid_constant__ OutPtrs out)
{
    begin_kernel();
    __shared__ int s_sum[8], s_max[8];
    const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int n_acc = 0;
    if (g < f.PT)
    {
        const float4 acc = as_float4(f.recs[2 * (size_t)g]);
        const float w    = __uint_as_float(f.recs[2 * (size_t)g + 1].x);
        n_acc            = (int)w;
        f.counts[g]      = n_acc;
        float c[4];
        if (w == 0.f)
            c[0] = f.background[0], c[1] = f.background[1], c[2] = f.background[2], c[3] = f.C > 3 ? f.background[3] : 0.f;
        else
            c[0] = acc.x / w, c[1] = acc.y / w, c[2] = acc.z / w, c[3] = acc.w / w;
        write_pixel(f, out, (unsigned)g, c, w, __int_as_float(f.ends[g]));
    }
    int sum = n_acc, mx = n_acc;
    for (int o = 16; o > 0; o >>= 1)
    {
        sum += __shfl_down_sync(0xffffffffu, sum, o);
        mx = max(mx, __shfl_down_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = sum, s_max[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        for (int i = 1; i < 8; ++i) sum += s_sum[i], mx = max(mx, s_max[i]);
        if (sum) atomicAdd(f.status + 0, sum);
        if (mx) atomicMax(f.status + 2, mx);
    }
}

// CombineAndFillBackward (RenderBackward.cu:27-76): the background colour receives the gradient of every empty pixel.  With
// interleaved copies the kernel that makes them has every pixel's gradient at hand and sums these as well (2 views 1280x720:
// 39 us for both, before 27 + 27 us in two launches); without them the empty pixels are visited by themselves.
__device__ __forceinline__ void fuzzy_dt_background_sum(const Frame& f, const BackPtrs& bp, const float (&v)[4])
{
    __shared__ float s_red[8][4];
    for (int k = 0; k < 4; ++k)
    {
        float x = v[k];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5][k] = x;
    }
    __syncthreads();
    if ((int)threadIdx.x < f.C)
    {
        float x = 0.f;
        for (int w = 0; w < 8; ++w) x += s_red[w][threadIdx.x];
        if (x != 0.f) atomicAdd(bp.g_background + threadIdx.x, x);
    }
}
__global__ void __launch_bounds__(256) fuzzy_dt_background_kernel(const __grid_constant__ Frame f,
                                                                   const __grid_constant__ BackPtrs bp)
{
    begin_kernel();
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < f.PT; g += (long long)gridDim.x * blockDim.x)
        if (f.counts[g] == 0)
        {
            const PixInfo px = decode_pixel(f, (unsigned)g);
            if (!px.valid) continue;
            const float4 G = load_grad_planar(f, bp, px);
            v[0] += G.x, v[1] += G.y, v[2] += G.z, v[3] += G.w;
        }
    fuzzy_dt_background_sum(f, bp, v);
}
__global__ void __launch_bounds__(256) fuzzy_dt_pack_kernel(const __grid_constant__ Frame f, const __grid_constant__ BackPtrs bp)
{
    begin_kernel();
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    const long long total = f.Prm * f.n_views;
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < total; r += (long long)gridDim.x * blockDim.x)
    {
        int view, l, o;
        const float4 G = pack_pixel(f, bp, r, view, l, o);
        const int w    = f.lw[l];
        // row: float estimate, then one correction step either way (the estimate is off by at most one)
        int y = __float2int_rz((float)o * f.inv_lw[l]), x = o - y * w;
        if (x < 0) x += w, --y;
        if (x >= w) x -= w, ++y;
        if (f.counts[view * (int)f.P + (int)f.lbase[l] + pixel_offset(w, x, y)] == 0) v[0] += G.x, v[1] += G.y, v[2] += G.z, v[3] += G.w;
    }
    fuzzy_dt_background_sum(f, bp, v);
}

// RenderBackward (RenderBackward.cu:131-474): one thread per point and view.  Pixel positions come from the backward's own
// copy of the projection, which leaves out the crop rotation (RenderBackward.cu:78-116).
template <int kCam>  // as in point_backward_kernel
__global__ void __launch_bounds__(kProjThreads, 4) fuzzy_dt_backward_kernel(const __grid_constant__ Frame f,
                                                                         const __grid_constant__ BackPtrs bp)
{
    begin_kernel();
    constexpr bool kIntr = kCam == 2;
    __shared__ Camera s_cam;
    __shared__ double s_red[kProjThreads / 32][kCamValues];
    const int b = blockIdx.y;
    if (threadIdx.x == 0) s_cam = load_camera(f, b);
    __syncthreads();
    const Camera& cam = s_cam;
    const int vbase   = b * (int)f.P;
    const int pid     = blockIdx.x * kProjThreads + threadIdx.x;
    CamAcc<kIntr> acc;
    acc.clear();
    PointGrad grad;
    grad.clear();
    float4 gp = make_float4(0.f, 0.f, 0.f, 0.f);
    if (pid < f.n)
    {
        const bool drop_out = f.dropout && f.dropout[(size_t)b * f.n + pid] == 1.f;
        const float4 pos    = __ldg(f.position + pid);
        const Projected pr  = project_point(pos, cam, f.dist_cutoff, false);
        PointJac jac;
        if (pr.z != 0.f && project_backward_prepare(pos, cam, f.dist_cutoff, jac))  // (z > 0: never declines)
        {
            const int tex = __ldg(f.index + pid);
            float2 ip     = pr.ip;
            float radius  = pr.radius_px;
            // Without camera gradients there are registers to request count and depth of the point's pixel on all levels together;
            // with them that costs spills.  Bound by the latency of the gathers (62 % of the issue slots, 23 of 32 lanes): 2 M points, 2 views
            // 1280x720, the whole pass: 214 -> 196 us; in this form with pose and intrinsics gradients 269 -> 275.
            constexpr bool kTogether = kCam == 0;
            int hits[VETR_MAX_LAYERS], nearest[VETR_MAX_LAYERS];
            if constexpr (kTogether)
            {
#pragma unroll
                for (int l = 0; l < VETR_MAX_LAYERS; ++l, radius *= 0.5f, ip.x *= 0.5f, ip.y *= 0.5f)
                {
                    hits[l] = nearest[l] = 0;
                    if (l >= f.L || (f.drop_by_radius && radius < f.radius_threshold)) continue;
                    const int lw = f.lw[l];
                    const int x = round_half_even(ip.x), y = round_half_even(ip.y);
                    if ((unsigned)x >= (unsigned)lw || (unsigned)y >= (unsigned)f.lh[l]) continue;
                    const int g = vbase + (int)f.lbase[l] + pixel_offset(lw, x, y);
                    hits[l] = f.counts[g], nearest[l] = f.ends[g];
                }
                ip = pr.ip, radius = pr.radius_px;
            }
#pragma unroll 1
            for (int l = 0; l < f.L; ++l, radius *= 0.5f, ip.x *= 0.5f, ip.y *= 0.5f)
            {
                if (f.drop_by_radius && radius < f.radius_threshold) continue;
                const int lw = f.lw[l], lh = f.lh[l];
                const int x = round_half_even(ip.x), y = round_half_even(ip.y);
                if ((unsigned)x >= (unsigned)lw || (unsigned)y >= (unsigned)lh) continue;
                const int g = vbase + (int)f.lbase[l] + pixel_offset(lw, x, y);
                int hit = 0, depth = 0;
                if constexpr (kTogether)
                {
#pragma unroll
                    for (int k = 0; k < VETR_MAX_LAYERS; ++k) hit = l == k ? hits[k] : hit, depth = l == k ? nearest[k] : depth;
                }
                const float w = (float)(kTogether ? hit : f.counts[g]);
                if (w == 0.f) continue;
                if (pr.z > __int_as_float(kTogether ? depth : f.ends[g]) * (f.depth_accept + 1)) continue;
                PixInfo px;
                px.x = (short)x, px.y = (short)y, px.level = (unsigned char)l, px.view = (unsigned char)b, px.valid = 1;
                px.interior = min(min(x, f.lw[l] - 1 - x), min(y, f.lh[l] - 1 - y)) > 2;
                if (!drop_out)
                {
                    const float iw = 1.f / w;
                    const float4 G = f.img4 ? load_grad(f, row_major_index(f, px)) : load_grad_planar(f, bp, px);
                    red_add_v4(bp.g_desc + tex, make_float4(iw * G.x, iw * G.y, iw * G.z, f.C > 3 ? iw * G.w : 0.f));
                }
                const bool point_grad = (f.ghost && drop_out) | (!f.ghost && !drop_out);
                if (!(point_grad && px.interior)) continue;
                const float4 d  = load_descriptor(f, tex);
                const float2 dR = f.img4 ? neighbour_gradient(f, row_major_index(f, px), lw, d) : neighbour_gradient_planar(f, bp, px, d);
                if (kCam) grad.add(dR, l);
                point_terms(cam, jac, dR, l, gp);
            }
            if (gp.w != 0.f)
            {
                if (kCam) camera_terms<kIntr>(f, cam, jac, grad, acc);
                if (bp.g_points) red_add_v4(bp.g_points + pid, gp);
            }
        }
    }
    if (kCam) reduce_cam<kIntr>(f, bp, acc, b, s_red);
}

// ---------------------------------------------------------------------------------------------------------
// Epilogues.

// Epilogue of the gradients in one launch: descriptor gradient to the planar layout, point gradients divided by the hit
// count (NormalizeGradient, PointRenderer.cu:1273-1280), rows of camera gradients divided by theirs
// (NormalizeGradientDevTensor, :1092-1109).  Block ranges in this order; a part without blocks is not wanted.  Four launches
// of this took 11 us for a scene of 5000 points, most of it start-up.
struct FinalizeArgs
{
    const float4* g_desc;
    float* g_texture;
    float4* g_points;
    float* g_points_count;
    double* g_pose;
    const float* g_pose_count;
    float* g_intr;
    const float* g_intr_count;
    int C, n_tex, n, n_img, n_cam;
    unsigned desc_end, points_end, pose_end;  // first block behind each part
};

template <typename T, int N>
__device__ __forceinline__ void normalize_row(T* g, const float* count, int i, int n)
{
    if (i >= n) return;
    const float c = count[i];
    if (c > 0)
        for (int k = 0; k < N; ++k) g[(long long)i * N + k] = g[(long long)i * N + k] / c;
}

__global__ void __launch_bounds__(256) finalize_kernel(const __grid_constant__ FinalizeArgs a)
{
    begin_kernel();
    const unsigned b = blockIdx.x;
    if (b < a.desc_end)
    {
        const long long i = (long long)b * 256 + threadIdx.x;
        if (i >= a.n_tex) return;
        const float4 v = a.g_desc[i];
        a.g_texture[i] = v.x;
        a.g_texture[(long long)a.n_tex + i] = v.y;
        a.g_texture[2LL * a.n_tex + i] = v.z;
        if (a.C > 3) a.g_texture[3LL * a.n_tex + i] = v.w;
    }
    else if (b < a.points_end)
    {
        const long long i = (long long)(b - a.desc_end) * 256 + threadIdx.x;
        if (i >= a.n) return;
        float4 v = a.g_points[i];
        const float c = v.w;
        if (a.g_points_count) a.g_points_count[i] = c;
        if (c > 0) v.x = v.x / c, v.y = v.y / c, v.z = v.z / c;
        v.w           = 0.f;
        a.g_points[i] = v;
    }
    else if (b < a.pose_end)
        normalize_row<double, 6>(a.g_pose, a.g_pose_count, (int)((b - a.points_end) * 256 + threadIdx.x), a.n_img);
    else
        normalize_row<float, 13>(a.g_intr, a.g_intr_count, (int)((b - a.pose_end) * 256 + threadIdx.x), a.n_cam);
}

// Fills up to VETR_MAX_ZERO buffers with zeros in one launch: 16 bytes per thread and step where a buffer starts on such a
// boundary.
struct ZeroArgs
{
    unsigned* ptr[VETR_MAX_ZERO];
    long long end[VETR_MAX_ZERO];  // running total of 16-byte units (the last one of a buffer may be partial)
    int words[VETR_MAX_ZERO];      // 4-byte words in the last unit (1 to 4)
    int n;
};

__global__ void __launch_bounds__(256) zero_buffers_kernel(const __grid_constant__ ZeroArgs a)
{
    begin_kernel();
    const long long total = a.end[a.n - 1];
    for (long long u = (long long)blockIdx.x * 256 + threadIdx.x; u < total; u += (long long)gridDim.x * 256)
    {
        int k = 0;
        while (u >= a.end[k]) ++k;
        const long long at = u - (k ? a.end[k - 1] : 0);
        unsigned* to       = a.ptr[k] + 4 * at;
        const int words    = u == a.end[k] - 1 ? a.words[k] : 4;
        if (words == 4 && ((uintptr_t)to & 15) == 0)
            *reinterpret_cast<uint4*>(to) = make_uint4(0u, 0u, 0u, 0u);
        else
            for (int i = 0; i < words; ++i) to[i] = 0u;
    }
}

// ApplyTangent (PointRenderer.cu:1325-1341): pose <- exp_se3(t) * pose in double; tangent = (translation, rotation).
__global__ void apply_tangent_kernel(double* tangent, double* poses, int n)
{
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n) return;
    double* t = tangent + 6 * idx;
    double* p = poses + 8 * idx;
    double ux = t[0], uy = t[1], uz = t[2], wx = t[3], wy = t[4], wz = t[5];
    double th2 = wx * wx + wy * wy + wz * wz, th = sqrt(th2);
    double imag, real, a, bb;
    if (th < 1e-10)
    {
        double th4 = th2 * th2;
        imag = 0.5 - th2 / 48.0 + th4 / 3840.0;
        real = 1.0 - th2 / 8.0 + th4 / 384.0;
        a    = 0.5;
        bb   = 1.0 / 6.0;
    }
    else
    {
        imag = sin(0.5 * th) / th;
        real = cos(0.5 * th);
        a    = (1 - cos(th)) / th2;
        bb   = (th - sin(th)) / (th2 * th);
    }
    double x1 = imag * wx, y1 = imag * wy, z1 = imag * wz, w1 = real;
    double O[9] = {0, -wz, wy, wz, 0, -wx, -wy, wx, 0};
    double u[3] = {ux, uy, uz}, te[3];
    for (int r = 0; r < 3; ++r)
    {
        te[r] = u[r];
        for (int c = 0; c < 3; ++c)
        {
            double o2 = O[3 * r] * O[c] + O[3 * r + 1] * O[3 + c] + O[3 * r + 2] * O[6 + c];
            te[r] += (a * O[3 * r + c] + bb * o2) * u[c];
        }
    }
    double x2 = p[0], y2 = p[1], z2 = p[2], w2 = p[3];
    double q[4] = {w1 * x2 + x1 * w2 + y1 * z2 - z1 * y2, w1 * y2 - x1 * z2 + y1 * w2 + z1 * x2,
                   w1 * z2 + x1 * y2 - y1 * x2 + z1 * w2, w1 * w2 - x1 * x2 - y1 * y2 - z1 * z2};
    double nrm = sqrt(q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3]);
    double tp[3] = {p[4], p[5], p[6]};
    double cx = y1 * tp[2] - z1 * tp[1], cy = z1 * tp[0] - x1 * tp[2], cz = x1 * tp[1] - y1 * tp[0];
    cx *= 2, cy *= 2, cz *= 2;
    double rx = tp[0] + w1 * cx + (y1 * cz - z1 * cy);
    double ry = tp[1] + w1 * cy + (z1 * cx - x1 * cz);
    double rz = tp[2] + w1 * cz + (x1 * cy - y1 * cx);
    for (int k = 0; k < 4; ++k) p[k] = q[k] / nrm;
    p[4] = rx + te[0], p[5] = ry + te[1], p[6] = rz + te[2];
    for (int k = 0; k < 6; ++k) t[k] = 0.0;
}

// ---------------------------------------------------------------------------------------------------------
// Multi-GPU epilogue: sum of the raw gradient buffers of all ranks + the count normalisation + the channel-major
// transpose, in one kernel over peer memory.  Every rank owns one contiguous slice of each of the three segments
// (descriptor, position, confidence gradients): it reads that slice from every rank's raw buffer (peer loads over
// NVLink, summed in rank order, so every rank ends up with the same bits), finalises it and stores the result into
// every rank's output buffer (peer stores).  The kernel waits on nothing: the caller orders it after the backward
// kernels of ALL ranks and orders the consumers after the exchange kernels of ALL ranks (a collective on the same
// stream before and after, e.g. the all-reduce of the pose gradients and of their counts).

struct ExchangeArgs
{
    int rank, world, C, n_tex, n;
    long long out_points, out_conf;  // float offsets of the position / confidence segments in the output buffers
    const float* raw[VETR_MAX_RANKS];
    float* out[VETR_MAX_RANKS];
    const float* raw_mc;  // multicast address of the raw buffers (NVLink SHARP), or nullptr
    float* out_mc;        // multicast address of the output buffers
    int segments;         // VETR_SEG_* bits: which of the three segments this launch handles
};

__device__ __forceinline__ void slice_of(long long count, int rank, int world, long long& lo, long long& hi)
{
    lo = count * rank / world;
    hi = count * (rank + 1) / world;
}

// Every access is 16 bytes per lane and contiguous across a warp: few large requests cross a link (and the switch)
// faster than many small ones.  kMulticast: the accesses go through the NVSwitch multicast object that spans all
// ranks' buffers - multimem.ld_reduce returns the sum over the ranks of one address (the switch fetches and adds),
// multimem.st stores to all ranks at once - so the SM issues 1/world of the loads and stores.

__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// sum over the ranks of the float4 at float offset `at` of the raw buffers (rank order 0, 1, ... in the plain form)
template <bool kMulticast>
__device__ __forceinline__ float4 rank_sum4(const ExchangeArgs& a, long long at)
{
    if constexpr (kMulticast)
    {
        float4 v;
        asm volatile("multimem.ld_reduce.relaxed.sys.global.add.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                     : "l"(a.raw_mc + at)
                     : "memory");
        return v;
    }
    else
    {
        float4 v = __ldcg(reinterpret_cast<const float4*>(a.raw[0] + at));
        for (int k = 1; k < a.world; ++k) v = add4(v, __ldcg(reinterpret_cast<const float4*>(a.raw[k] + at)));
        return v;
    }
}

// store one float4 at float offset `at` of every rank's output buffer
template <bool kMulticast>
__device__ __forceinline__ void rank_store4(const ExchangeArgs& a, long long at, float4 v)
{
    if constexpr (kMulticast)
        asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(a.out_mc + at), "f"(v.x), "f"(v.y),
                     "f"(v.z), "f"(v.w)
                     : "memory");
    else
        for (int k = 0; k < a.world; ++k) *reinterpret_cast<float4*>(a.out[k] + at) = v;
}

// scalar forms for the few elements that do not fill a 16-byte group (plain peer accesses in both variants)
__device__ __forceinline__ float rank_sum1(const ExchangeArgs& a, long long at)
{
    float v = __ldcg(a.raw[0] + at);
    for (int k = 1; k < a.world; ++k) v += __ldcg(a.raw[k] + at);
    return v;
}
__device__ __forceinline__ void rank_store1(const ExchangeArgs& a, long long at, float v)
{
    for (int k = 0; k < a.world; ++k) a.out[k][at] = v;
}

constexpr int kExchangeWarps = 8;

template <bool kMulticast>
__global__ void __launch_bounds__(32 * kExchangeWarps) exchange_finalize_kernel(const __grid_constant__ ExchangeArgs a)
{
    __shared__ float4 s_tile[kExchangeWarps][2][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long gtid    = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long stride  = (long long)gridDim.x * blockDim.x;
    const long long gwarp   = (long long)blockIdx.x * kExchangeWarps + warp;
    const long long n_warps = (long long)gridDim.x * kExchangeWarps;
    const long long n_tex   = a.n_tex;
    const long long raw_points = 4 * n_tex, raw_conf = 4 * n_tex + 4LL * a.n;
    long long lo, hi;

    // descriptor gradient [n_tex] float4 -> texture gradient [C, n_tex].  A warp takes 32 texels (one coalesced float4
    // load per lane), turns them by 90 degrees in shared memory and stores 4 texels x 1 channel per lane, i.e. a
    // 128-byte run in each channel row.  Rows start at c * n_tex floats: 16-byte aligned only if n_tex % 4 == 0.
    const long long tiles = (n_tex & 3) == 0 ? n_tex / 32 : 0;
    slice_of(tiles, a.rank, a.world, lo, hi);
    if (!(a.segments & VETR_SEG_DESC)) hi = lo;
    const int c = lane >> 3, q = lane & 7;
    for (long long tile = lo + gwarp; tile < hi; tile += 2 * n_warps)
    {
        const bool second = tile + n_warps < hi;
        const float4 v0 = rank_sum4<kMulticast>(a, 4 * (tile * 32 + lane));
        float4 v1       = make_float4(0.f, 0.f, 0.f, 0.f);
        if (second) v1 = rank_sum4<kMulticast>(a, 4 * ((tile + n_warps) * 32 + lane));
        s_tile[warp][0][lane] = v0;
        s_tile[warp][1][lane] = v1;
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 2; ++u)
        {
            if (u == 1 && !second) break;
            const float* tf = reinterpret_cast<const float*>(s_tile[warp][u]);
            const float4 o  = make_float4(tf[(4 * q) * 4 + c], tf[(4 * q + 1) * 4 + c], tf[(4 * q + 2) * 4 + c], tf[(4 * q + 3) * 4 + c]);
            if (c < a.C) rank_store4<kMulticast>(a, c * n_tex + (tile + u * n_warps) * 32 + 4 * q, o);
        }
        __syncwarp();
    }
    // texels that do not fill a tile (all of them if the rows are not 16-byte aligned), one by one
    {
        const long long first = tiles * 32;
        slice_of(n_tex - first, a.rank, a.world, lo, hi);
        if (!(a.segments & VETR_SEG_DESC)) hi = lo;
        for (long long t = first + lo + gtid; t < first + hi; t += stride)
        {
            const float4 v = rank_sum4<false>(a, 4 * t);
            rank_store1(a, t, v.x), rank_store1(a, n_tex + t, v.y), rank_store1(a, 2 * n_tex + t, v.z);
            if (a.C > 3) rank_store1(a, 3 * n_tex + t, v.w);
        }
    }

    // position gradient sums with the hit count in .w -> average (NormalizeGradient, PointRenderer.cu:1273-1280)
    slice_of(a.n, a.rank, a.world, lo, hi);
    if (!(a.segments & VETR_SEG_POINTS)) hi = lo;
    for (long long base = lo + gtid; base < hi; base += stride * 4)
    {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (base + u * stride < hi) v[u] = rank_sum4<kMulticast>(a, raw_points + 4 * (base + u * stride));
#pragma unroll
        for (int u = 0; u < 4; ++u)
        {
            if (base + u * stride >= hi) continue;
            float4 r = v[u];
            if (r.w > 0) r.x = r.x / r.w, r.y = r.y / r.w, r.z = r.z / r.w;
            r.w = 0.f;
            rank_store4<kMulticast>(a, a.out_points + 4 * (base + u * stride), r);
        }
    }

    // confidence gradient, four texels per access (every segment offset is a multiple of 4 floats); the last rank also
    // takes the n_tex % 4 texels that are left over
    const long long groups = n_tex / 4;
    slice_of(groups, a.rank, a.world, lo, hi);
    if (!(a.segments & VETR_SEG_CONF)) hi = lo;
    for (long long base = lo + gtid; base < hi; base += stride * 4)
    {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (base + u * stride < hi) v[u] = rank_sum4<kMulticast>(a, raw_conf + 4 * (base + u * stride));
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (base + u * stride < hi) rank_store4<kMulticast>(a, a.out_conf + 4 * (base + u * stride), v[u]);
    }
    if (a.rank == a.world - 1 && (a.segments & VETR_SEG_CONF))
        for (long long t = 4 * groups + gtid; t < n_tex; t += stride) rank_store1(a, a.out_conf + t, rank_sum1(a, raw_conf + t));
    __threadfence_system();  // the peer stores are performed before the kernel counts as finished
}

// ---------------------------------------------------------------------------------------------------------
// L1 loss of the whole output pyramid against a target pyramid and its gradient, in one launch (what a training step
// does between the forward and the backward pass; with library element-wise kernels it is seven launches per level).

struct L1Args
{
    const float* image[VETR_MAX_LAYERS];
    const float* target[VETR_MAX_LAYERS];
    float* grad[VETR_MAX_LAYERS];
    long long end[VETR_MAX_LAYERS];  // running element count: level l covers [end[l-1], end[l])
    float inv_numel[VETR_MAX_LAYERS];
    int levels;
    float* loss;
};

__global__ void __launch_bounds__(256) l1_loss_grad_kernel(const __grid_constant__ L1Args a)
{
    begin_kernel();
    __shared__ float s_part[8];
    const long long total  = a.end[a.levels - 1];
    const long long stride = (long long)gridDim.x * blockDim.x * 4;
    float sum = 0.f;
    // four consecutive elements per thread where they lie in one level and are 16-byte aligned, else one by one
    for (long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4; i < total; i += stride)
    {
        int l = 0;
#pragma unroll
        for (int k = 1; k < VETR_MAX_LAYERS; ++k)
            if (k < a.levels && i >= a.end[k - 1]) l = k;
        const long long base = l ? a.end[l - 1] : 0, j = i - base, n = a.end[l] - base;
        const float w = a.inv_numel[l];
        if (j + 4 <= n && ((j & 3) == 0))
        {
            const float4 x = __ldg(reinterpret_cast<const float4*>(a.image[l] + j));
            const float4 t = __ldg(reinterpret_cast<const float4*>(a.target[l] + j));
            const float d[4] = {x.x - t.x, x.y - t.y, x.z - t.z, x.w - t.w};
            float g[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) g[k] = d[k] > 0.f ? w : (d[k] < 0.f ? -w : 0.f), sum += fabsf(d[k]) * w;
            *reinterpret_cast<float4*>(a.grad[l] + j) = make_float4(g[0], g[1], g[2], g[3]);
        }
        else
        {
            for (long long e = i; e < min(i + 4, total); ++e)
            {
                int le = 0;
#pragma unroll
                for (int k = 1; k < VETR_MAX_LAYERS; ++k)
                    if (k < a.levels && e >= a.end[k - 1]) le = k;
                const long long je = e - (le ? a.end[le - 1] : 0);
                const float d = a.image[le][je] - a.target[le][je], we = a.inv_numel[le];
                a.grad[le][je] = d > 0.f ? we : (d < 0.f ? -we : 0.f);
                sum += fabsf(d) * we;
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        float t = 0.f;
        for (int k = 0; k < 8; ++k) t += s_part[k];
        atomicAdd(a.loss, t);
    }
}

}  // namespace vetr

#include "vetr_envmap.cuh"
#include "vetr_grid.cuh"
#include "vetr_knn.cuh"
#include "vetr_points.cuh"

// =========================================================================================================
// C ABI

using namespace vetr;

struct vetr_ctx
{
    int device           = 0;
    cudaStream_t stream  = nullptr;
    int last_cuda        = 0;
    int sm_count         = 148;
    long long* tile_sums = nullptr;  // scan scratch
    long long tile_cap   = 0;
    int2* grid_queue     = nullptr;  // (cell, chunk) queue of vetr_grid_loss, allocated by its first call
    unsigned long long* grid_queue_count = nullptr;  // {queue length, no cell by rows, pixels of vast cells}
    // running sums of the loss image's rows: the last one is in use, the ones before it were outgrown and stay until the context
    // goes, because a recorded graph may still write to them (each at least twice the one before: together no more than the last)
    double* grid_prefix[32] = {};
    int grid_prefix_n         = 0;
    long long grid_prefix_cap = 0;
    // scratch of vetr_knn_radius, grown on demand: per point (sorted copy, cell, queue) and per cell (first slot)
    float4* knn_sorted   = nullptr;
    int* knn_point_cell  = nullptr;
    int* knn_queue       = nullptr;
    long long knn_cap_points = 0;
    int* knn_cells       = nullptr;
    long long knn_cap_cells = 0;
    int* knn_tile_sums   = nullptr;  // 16384 tile sums, then 16 words: bounds[6], occupied (64 bit), queue count, 2 of the point removal
    int* points_flags    = nullptr;  // keep flags of vetr_remove_points_plan
    long long points_cap = 0;
    // resident CTAs per SM of the item kernels, and of the kernels for lists longer than kLongList
    int blend_ctas_per_sm = 1, back_ctas_per_sm = 1, fuzzy_ctas_per_sm = 1, bilinear_ctas_per_sm = 1;
    int blend_long_ctas_per_sm = 1, back_long_ctas_per_sm = 1, bilinear_long_ctas_per_sm = 1, fuzzy_mid_ctas_per_sm = 1;
    long long launches   = 0;
    bool timing          = false;
    cudaEvent_t ev[VETR_T_N][2] = {};
    bool ev_used[VETR_T_N]      = {};
};

// Brackets the launches of one pass with events when timing is on, and counts kernels.
struct PassScope
{
    vetr_ctx* c;
    int id;
    PassScope(vetr_ctx* ctx, int pass, int kernels) : c(ctx), id(pass)
    {
        c->launches += kernels;
        if (c->timing) cudaEventRecord(c->ev[id][0], c->stream);
    }
    ~PassScope()
    {
        if (c->timing)
        {
            cudaEventRecord(c->ev[id][1], c->stream);
            c->ev_used[id] = true;
        }
    }
};

// Launches a kernel that waits for the one before it on the stream: begin_kernel() at the start or, where it has nothing to do with what that one does,
// BesidePrevious at the end (always with overlap).  overlap: its blocks may be set up while the kernel before it ends, which hides
// the way from one kernel to the next.  Waiting at the start, 100 k points at 512x512 101 -> 85 us, a smallest batch 85 -> 82, 3 M points at 1920x1080
// forward only 344 -> 335, mode 2 with 1 M points 459 -> 440, mode 0 with 2 M points and two views 388 -> 374, mode 3 with 3 M points and two views
// the same.  Not where
// - the kernel is an item kernel (sort + blend, backward, the long lists that go first) and waits at its start: its blocks take every n-th item, and set
//   up early they come to lie next to each other on the SMs that are free first, and so do the items of much work (mode 3 at 1280x720 428 -> 450 us);
// - there is much to do (20 M points, eight views 18120 -> 18440 us, 8 M points and four views the same): nothing to be gained.
constexpr long long kOverlapPoints = 1 << 24;            // points times views, elements
constexpr long long kOverlapUnits  = 3 * kOverlapPoints;  // 16-byte units of zeros: a point's gradients are 2.25 of them
template <typename... Parameters, typename... Arguments>
static void launch(bool overlap, void (*kernel)(Parameters...), dim3 grid, int block, size_t smem, cudaStream_t stream, const Arguments&... arguments)
{
    cudaLaunchConfig_t config = {};
    cudaLaunchAttribute attribute;
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    config.gridDim = grid, config.blockDim = dim3(block), config.dynamicSmemBytes = smem, config.stream = stream;
    config.attrs = &attribute, config.numAttrs = overlap ? 1 : 0;
    cudaLaunchKernelEx(&config, kernel, arguments...);
}

#define VETR_CUDA(ctx, call)                      \
    do                                            \
    {                                             \
        cudaError_t e_ = (call);                  \
        if (e_ != cudaSuccess)                    \
        {                                         \
            (ctx)->last_cuda = (int)e_;           \
            return VETR_E_CUDA;                   \
        }                                         \
    } while (0)

// Pixel space of one view: every level's height is padded to a multiple of kBand rows (the banded order of pixel_offset).
// rbase / *row_major: the same levels in plain row-major order without padding.
static int64_t pyramid(int w, int h, int L, int* lw, int* lh, long long* lbase, long long* rbase = nullptr,
                       long long* row_major = nullptr)
{
    long long base = 0, rm = 0;
    for (int l = 0; l < L; ++l)
    {
        if (lw) lw[l] = w, lh[l] = h, lbase[l] = base;
        if (rbase) rbase[l] = rm;
        base += (long long)w * ((h + kBand - 1) / kBand * kBand);
        rm += (long long)w * h;
        w /= 2;
        h /= 2;
    }
    if (row_major) *row_major = rm;
    return base;
}

extern "C" int64_t vetr_pyramid_pixels(int w, int h, int num_layers)
{
    if (w <= 0 || h <= 0 || num_layers < 1 || num_layers > VETR_MAX_LAYERS) return -1;
    return pyramid(w, h, num_layers, nullptr, nullptr, nullptr);
}

extern "C" int64_t vetr_item_table_entries(int64_t capacity, int64_t n_pixels_total)
{
    if (capacity < 0 || n_pixels_total < 0) return -1;
    int64_t cap = capacity < 0x7fffffffLL ? capacity : 0x7fffffffLL;
    return (cap + (int64_t)kPixelWork * n_pixels_total + kQuantum - 1) / kQuantum + 2;
}

extern "C" int64_t vetr_max_fragments(int n_points, int n_views, const vetr_params* p)
{
    if (!p) return -1;
    int64_t f = (int64_t)n_points * p->num_layers * n_views;
    if (p->render_mode == VETR_MODE_BILINEAR_BLEND) f *= 4;
    return f;
}

extern "C" int64_t vetr_list_capacity(int n_points, int n_views, int w, int h, const vetr_params* p)
{
    if (!p) return -1;
    int64_t f = vetr_max_fragments(n_points, n_views, p);
    if (p->render_mode == VETR_MODE_FUZZY_DT)
    {
        // mode 0 keeps no lists: the buffer holds one accumulator record per pixel of the pixel space instead
        const int64_t px = vetr_pyramid_pixels(w, h, p->num_layers);
        if (px < 0) return -1;
        f = px * n_views;
    }
    return f;
}

extern "C" const char* vetr_strerror(int status)
{
    switch (status)
    {
        case VETR_OK: return "ok";
        case VETR_E_INVALID_ARG: return "invalid argument";
        case VETR_E_CUDA: return "CUDA runtime error";
        case VETR_E_UNSUPPORTED: return "unsupported camera model or option";
        case VETR_E_LIST_OVERFLOW: return "fragment buffer too small";
        case VETR_E_TOO_LARGE: return "size exceeds a fixed limit";
        default: return "unknown status";
    }
}

extern "C" int vetr_last_cuda_error(const vetr_ctx* ctx) { return ctx ? ctx->last_cuda : 0; }

static int ensure_scratch(vetr_ctx* ctx, long long n_tiles)
{
    if (n_tiles > ctx->tile_cap)
    {
        if (ctx->tile_sums) cudaFree(ctx->tile_sums);
        ctx->tile_sums = nullptr;
        long long cap  = n_tiles + n_tiles / 4 + 16;
        VETR_CUDA(ctx, cudaMalloc(&ctx->tile_sums, (cap + 1) * sizeof(long long)));  // and the ticket
        ctx->tile_cap = cap;
    }
    return VETR_OK;
}

extern "C" int vetr_create(vetr_ctx** out, int device, void* cuda_stream)
{
    if (!out) return VETR_E_INVALID_ARG;
    vetr_ctx* ctx = new (std::nothrow) vetr_ctx();
    if (!ctx) return VETR_E_INVALID_ARG;
    ctx->device = device;
    ctx->stream = (cudaStream_t)cuda_stream;
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&ctx->sm_count, cudaDevAttrMultiProcessorCount, device);
    const auto prepare = [&e](auto kernel, int threads, size_t smem, int* ctas_per_sm)
    {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess && ctas_per_sm) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, kernel, threads, smem);
        if (ctas_per_sm && *ctas_per_sm < 1) *ctas_per_sm = 1;
    };
    prepare(sort_blend_kernel<false>, kThreads, sizeof(BlendSmem), &ctx->blend_ctas_per_sm);
    prepare(sort_blend_kernel<true>, kThreads, sizeof(BlendSmem), nullptr);
    prepare(sort_blend_long_kernel<false>, kLongThreads, sizeof(LongBlendSmem), &ctx->blend_long_ctas_per_sm);
    prepare(sort_blend_long_kernel<true>, kLongThreads, sizeof(LongBlendSmem), nullptr);
    prepare(backward_kernel<false, false>, kThreads, sizeof(BackSmem), &ctx->back_ctas_per_sm);
    prepare(backward_kernel<false, true>, kThreads, sizeof(BackSmemSuffix), &ctx->bilinear_ctas_per_sm);
    prepare(backward_kernel<true, false>, kThreads, sizeof(BackSmemFuzzy), &ctx->fuzzy_ctas_per_sm);
    prepare(backward_long_kernel<false>, kThreads, sizeof(BackSmemSuffix), &ctx->back_long_ctas_per_sm);
    prepare(backward_long_kernel<true>, kThreads, sizeof(BackSmemSuffix), &ctx->bilinear_long_ctas_per_sm);
    prepare(backward_fuzzy_long_kernel<kLongList, kFuzzyMidMax>, kThreads, sizeof(FuzzyLongSmem<kFuzzyMidMax>), &ctx->fuzzy_mid_ctas_per_sm);
    prepare(backward_fuzzy_long_kernel<kFuzzyMidMax, kFuzzyLongMax>, kThreads, sizeof(FuzzyLongSmem<kFuzzyLongMax>), nullptr);
    if (e != cudaSuccess)
    {
        delete ctx;
        *out = nullptr;
        return VETR_E_CUDA;
    }
    *out = ctx;
    return VETR_OK;
}

extern "C" void vetr_destroy(vetr_ctx* ctx)
{
    if (!ctx) return;
    cudaSetDevice(ctx->device);
    if (ctx->tile_sums) cudaFree(ctx->tile_sums);
    if (ctx->grid_queue) cudaFree(ctx->grid_queue);
    for (int i = 0; i < ctx->grid_prefix_n; ++i) cudaFree(ctx->grid_prefix[i]);
    cudaFree(ctx->knn_sorted), cudaFree(ctx->knn_point_cell), cudaFree(ctx->knn_queue);
    cudaFree(ctx->knn_cells), cudaFree(ctx->knn_tile_sums), cudaFree(ctx->points_flags);
    for (int i = 0; i < VETR_T_N; ++i)
        for (int k = 0; k < 2; ++k)
            if (ctx->ev[i][k]) cudaEventDestroy(ctx->ev[i][k]);
    delete ctx;
}

extern "C" int vetr_set_timing(vetr_ctx* ctx, int enable)
{
    if (!ctx) return VETR_E_INVALID_ARG;
    VETR_CUDA(ctx, cudaSetDevice(ctx->device));
    if (enable && !ctx->ev[0][0])
        for (int i = 0; i < VETR_T_N; ++i)
            for (int k = 0; k < 2; ++k) VETR_CUDA(ctx, cudaEventCreate(&ctx->ev[i][k]));
    ctx->timing = enable != 0;
    for (int i = 0; i < VETR_T_N; ++i) ctx->ev_used[i] = false;
    return VETR_OK;
}

extern "C" int vetr_get_timings(vetr_ctx* ctx, float* out_ms)
{
    if (!ctx || !out_ms) return VETR_E_INVALID_ARG;
    VETR_CUDA(ctx, cudaSetDevice(ctx->device));
    VETR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (int i = 0; i < VETR_T_N; ++i)
    {
        out_ms[i] = 0.f;
        if (ctx->ev_used[i]) VETR_CUDA(ctx, cudaEventElapsedTime(&out_ms[i], ctx->ev[i][0], ctx->ev[i][1]));
    }
    return VETR_OK;
}

extern "C" int64_t vetr_launch_count(const vetr_ctx* ctx) { return ctx ? ctx->launches : 0; }

extern "C" int vetr_set_stream(vetr_ctx* ctx, void* cuda_stream)
{
    if (!ctx) return VETR_E_INVALID_ARG;
    ctx->stream = (cudaStream_t)cuda_stream;
    return VETR_OK;
}

static int fill_frame(vetr_ctx* ctx, Frame& f, const vetr_params* p, const vetr_cloud* cloud, const vetr_texture* tex,
                      const vetr_cameras* cams, const vetr_view* views, int n_views, const vetr_lists* lists)
{
    if (!ctx || !p || !cloud || !tex || !cams || !views || !lists) return VETR_E_INVALID_ARG;
    if (n_views < 1 || n_views > VETR_MAX_VIEWS) return VETR_E_INVALID_ARG;
    if (p->num_layers < 1 || p->num_layers > VETR_MAX_LAYERS) return VETR_E_INVALID_ARG;
    if (p->num_channels != 3 && p->num_channels != 4) return VETR_E_INVALID_ARG;
    if (p->render_mode < VETR_MODE_FUZZY_DT || p->render_mode > VETR_MODE_BILINEAR_BLEND) return VETR_E_UNSUPPORTED;
    if (cloud->n < 0 || tex->n_tex < 1 || !cloud->position || !cloud->index || !tex->texture || !tex->confidence ||
        !tex->background || !cams->poses_se3 || !cams->intrinsics)
        return VETR_E_INVALID_ARG;
    if (((uintptr_t)cloud->position & 15) != 0) return VETR_E_INVALID_ARG;
    if (!lists->counts || !lists->ends || !lists->frags || !lists->status || lists->capacity < 0 ||
        ((uintptr_t)lists->frags & 31) != 0)
        return VETR_E_INVALID_ARG;
    memset(&f, 0, sizeof(f));
    f.n_views = n_views, f.L = p->num_layers, f.C = p->num_channels, f.n = cloud->n, f.n_tex = tex->n_tex;
    f.w = views[0].w, f.h = views[0].h;
    if (f.w <= 0 || f.h <= 0) return VETR_E_INVALID_ARG;
    for (int b = 0; b < n_views; ++b)
    {
        const vetr_view& v = views[b];
        if (v.w != f.w || v.h != f.h) return VETR_E_INVALID_ARG;
        if (v.camera_model != 0) return VETR_E_UNSUPPORTED;
        if (v.image_index < 0 || v.image_index >= cams->n_img || v.camera_index < 0 || v.camera_index >= cams->n_cam)
            return VETR_E_INVALID_ARG;
        f.views[b].image_index = v.image_index, f.views[b].camera_index = v.camera_index;
        memcpy(f.views[b].crop, v.crop, sizeof(v.crop));
        memcpy(f.views[b].rot, v.rot, sizeof(v.rot));
    }
    f.mode = p->render_mode, f.drop_by_radius = p->drop_out_points_by_radius, f.use_env = p->use_environment_map;
    f.viewer_only = p->viewer_only, f.dbg_max_len = p->debug_max_list_length, f.need_point_grad = p->need_point_gradient;
    f.bg_alpha_to_point0 = p->background_alpha_to_point0, f.keep_sorted = p->keep_sorted_lists;
    f.radius_threshold = p->drop_out_radius_threshold, f.dist_cutoff = p->dist_cutoff;
    f.stability_cutoff = p->stability_cutoff_value, f.k_grad_factor = p->K_gradient_factor;
    f.dist_grad_factor = p->distortion_gradient_factor, f.mask_value = p->output_background_mask_value;
    f.accept_blend = p->depth_accept_blend, f.depth_accept = p->depth_accept, f.ghost = p->ghost_gradients;
    f.P  = pyramid(f.w, f.h, f.L, f.lw, f.lh, f.lbase, f.rbase, &f.Prm);
    f.PT = f.P * n_views;
    if (f.lw[f.L - 1] < 1 || f.lh[f.L - 1] < 1) return VETR_E_INVALID_ARG;  // the reference asserts w > 0 && h > 0 per level
    for (int l = 0; l < f.L; ++l) f.inv_lw[l] = 1.f / (float)f.lw[l], f.inv_band[l] = 1.f / (float)(kBand * f.lw[l]);
    if (f.PT > 0x7fffffffLL || (long long)f.lw[0] * f.lh[0] * f.C * n_views > 0x7fffffffLL) return VETR_E_TOO_LARGE;
    f.position = (const float4*)cloud->position, f.index = cloud->index;
    f.texture = tex->texture, f.confidence = tex->confidence, f.background = tex->background;
    f.poses = cams->poses_se3, f.intr = cams->intrinsics;
    f.counts = lists->counts, f.ends = lists->ends, f.recs = (uint4*)lists->frags;
    f.capacity = lists->capacity, f.status = lists->status;
    long long n_tiles = (f.PT + kScanTile - 1) / kScanTile;
    if (!lists->items || lists->items_capacity < vetr_item_table_entries(lists->capacity, f.PT)) return VETR_E_INVALID_ARG;
    VETR_CUDA(ctx, cudaSetDevice(ctx->device));
    int rc = ensure_scratch(ctx, n_tiles);
    if (rc != VETR_OK) return rc;
    f.item_start = lists->items;
    f.next_item  = lists->items + (lists->items_capacity - 1);
    f.level_mask = lists->level_mask;
    f.point_grad = (float2*)lists->point_grad;
    f.img4       = (float4*)lists->pixel_scratch;
    f.grad4      = f.img4 ? f.img4 + f.PT : nullptr;
    return VETR_OK;
}

// The two kernels of the scan.  *ticket and status[0..3] are zero on the stream before it (a ticket that is not would have the sums of
// the tiles scanned too early).
static void launch_scan(const int* counts, long long n, long long capacity, long long* tile_sums, unsigned* ticket, int n_tiles, int* ends,
                        int* status, int* items, int* next_item, cudaStream_t st, bool overlap)
{
    const bool vec = (((uintptr_t)counts | (uintptr_t)ends) & 15) == 0;
    launch(overlap, vec ? scan_tile_sums_kernel<true> : scan_tile_sums_kernel<false>, n_tiles, 256, 0, st, counts, n, tile_sums, status, capacity, items, next_item, ticket);
    launch(overlap, vec ? scan_apply_kernel<true> : scan_apply_kernel<false>, n_tiles, 256, 0, st, counts, n, tile_sums, ends, status, items);
}

// Launches zero_buffers_kernel on the context's stream; `bytes` are multiples of 4, as are the addresses.
static int zero_buffers(vetr_ctx* ctx, void* const* buffers, const int64_t* bytes, int n)
{
    ZeroArgs a;
    a.n = 0;
    long long total = 0;
    for (int i = 0; i < n; ++i)
    {
        if (bytes[i] == 0) continue;
        const long long words = bytes[i] / 4, units = (words + 3) / 4;
        total += units;
        a.ptr[a.n] = (unsigned*)buffers[i], a.end[a.n] = total, a.words[a.n] = (int)(words - 4 * (units - 1));
        ++a.n;
    }
    if (a.n == 0) return VETR_OK;
    ctx->launches += 1;
    launch(total <= kOverlapUnits, zero_buffers_kernel, (unsigned)std::min<long long>((total + 255) / 256, ctx->sm_count * 32ll), 256, 0, ctx->stream, a);
    VETR_CUDA(ctx, cudaGetLastError());
    return VETR_OK;
}

extern "C" int vetr_zero_buffers(vetr_ctx* ctx, void* const* buffers, const int64_t* bytes, int n)
{
    if (!ctx || n < 0 || n > VETR_MAX_ZERO || (n > 0 && (!buffers || !bytes))) return VETR_E_INVALID_ARG;
    for (int i = 0; i < n; ++i)
        if (bytes[i] < 0 || bytes[i] % 4 != 0 || (bytes[i] > 0 && (!buffers[i] || ((uintptr_t)buffers[i] & 3) != 0))) return VETR_E_INVALID_ARG;
    VETR_CUDA(ctx, cudaSetDevice(ctx->device));
    return zero_buffers(ctx, buffers, bytes, n);
}

// Fragments per level, at most, from which on the long lists go first, with sort_blend_kernel beside them from the start and its items handed out by a
// counter.  3 M points forward only 297 -> 292 us, 8 M points and four views 3855 -> 3806, 20 M and eight 17410 -> 17290, mode 3 with 1 M
// points 394 -> 381 and with 3 M and two views 2933 -> 2840; below it the late blocks and the counter cost more: 99 k points in mode 1 46 -> 47,
// 39 k in mode 3 58 -> 72, 114 k 122 -> 131, mode 2 with 1 M points the same.
constexpr long long kQueueFragments = 1 << 21;

// Blocks of sort_blend_kernel.  As many as are resident leave the SMs finishing at different times, however evenly the items are cut:
// neighbouring items lie on the same stretch of the image.  Four times as many are taken by the SMs as they come free, at the price of a first
// item that nothing was requested ahead for, so each block should still have one or more.  How many items there are is known only on
// the device; the pixels alone give at least `items`.  us with 1 / 2 / 4 / 8 / 16 times the resident blocks, items per resident block in front:
//   2.3 (100 k points, 512 x 512) 12.3 / 11.5 / 13.3 / 14.1 / 24.0      4.2 (mode 2, 1 M points, 801 x 603) 72.8 / 65.4 / 57.4 / 61.4 / 62.3
//   18 (3 M points, 1920 x 1080) 163 / 157 / 144 / 149 / 161            27 (8 M points x 4 views) 860 / 859 / 857 / 859 / 867
// (The backward kernel gains as well, mode 2 170 -> 125, but adds each block's share of the terms that all pixels send to one address:
// with more blocks their fp32 sum left its bound.)
static int blend_blocks(long long pixels, int resident)
{
    const long long items = pixels * kPixelWork / kQuantum;
    return items < 3ll * resident ? resident : 4 * resident;
}
extern "C" int vetr_forward(vetr_ctx* ctx, const vetr_params* params, const vetr_cloud* cloud, const vetr_texture* texture,
                            const vetr_cameras* cameras, const vetr_view* views, int n_views, const float* dropout,
                            const vetr_lists* lists, float* const* out_color, float* const* out_weight,
                            float* const* out_mask, float* const* out_depth)
{
    Frame f;
    int rc = fill_frame(ctx, f, params, cloud, texture, cameras, views, n_views, lists);
    if (rc != VETR_OK) return rc;
    if (!out_color) return VETR_E_INVALID_ARG;
    f.dropout = dropout;
    OutPtrs out;
    memset(&out, 0, sizeof(out));
    for (int l = 0; l < f.L; ++l)
    {
        if (!out_color[l]) return VETR_E_INVALID_ARG;
        out.color[l] = out_color[l];
        if ((out_weight && !out_weight[l]) || (out_mask && !out_mask[l]) || (out_depth && !out_depth[l])) return VETR_E_INVALID_ARG;
        if (out_weight) out.weight[l] = out_weight[l];
        if (out_mask) out.mask[l] = out_mask[l];
        if (out_depth) out.depth[l] = out_depth[l];
    }
    cudaStream_t st    = ctx->stream;
    const bool overlap = (long long)f.n * n_views <= kOverlapPoints;
    if (f.mode == VETR_MODE_FUZZY_DT)
    {
        if (f.capacity < f.PT) return VETR_E_INVALID_ARG;  // the fragment buffer holds one accumulator record per pixel
        const int ctas = (f.n + kProjThreads - 1) / kProjThreads;
        {
            PassScope t(ctx, VETR_T_COUNT, 1 + (ctas > 0));
            launch(overlap, fuzzy_dt_clear_kernel, (unsigned)((f.PT + 255) / 256), 256, 0, st, f);
            if (ctas > 0) launch(overlap, fuzzy_dt_point_kernel<0>, dim3(ctas, n_views), kProjThreads, 0, st, f);
        }
        if (ctas > 0)
        {
            PassScope t(ctx, VETR_T_COLLECT, 1);
            launch(overlap, fuzzy_dt_point_kernel<1>, dim3(ctas, n_views), kProjThreads, 0, st, f);
        }
        {
            PassScope t(ctx, VETR_T_SORT_BLEND, 1);
            launch(overlap, fuzzy_dt_combine_kernel, (unsigned)((f.PT + 255) / 256), 256, 0, st, f, out);
        }
        VETR_CUDA(ctx, cudaGetLastError());
        return VETR_OK;
    }
    {
        void* const buffers[3] = {f.counts, f.status, ctx->tile_sums + ctx->tile_cap};
        const int64_t bytes[3] = {(int64_t)(f.PT * sizeof(int)), 4 * sizeof(int), sizeof(long long)};
        rc = zero_buffers(ctx, buffers, bytes, 3);
        if (rc != VETR_OK) return rc;
    }
    const bool bilinear = f.mode == VETR_MODE_BILINEAR_BLEND;
    if (f.n > 0)
    {
        PassScope t(ctx, VETR_T_COUNT, 1);
        const bool one    = (long long)f.n * n_views < kCountSeveral;
        const int per     = kProjThreads * (one ? 1 : count_points(bilinear));
        const auto kernel = bilinear ? (one ? project_kernel<false, 1, true> : project_kernel<false, count_points(true), true>)
                                     : (one ? project_kernel<false, 1, false> : project_kernel<false, count_points(false), false>);
        launch(overlap, kernel, dim3((f.n + per - 1) / per, n_views), kProjThreads, 0, st, f);
    }
    const int n_tiles = (int)((f.PT + kScanTile - 1) / kScanTile);
    {
        PassScope t(ctx, VETR_T_SCAN, 2);
        launch_scan(f.counts, f.PT, f.capacity, ctx->tile_sums, reinterpret_cast<unsigned*>(ctx->tile_sums + ctx->tile_cap), n_tiles, f.ends, f.status, f.item_start, f.next_item, st, overlap);
    }
    if (f.n > 0)
    {
        PassScope t(ctx, VETR_T_COLLECT, 1);
        const bool one    = (long long)f.n * n_views < (bilinear ? kCollectPairsBilinear : kCollectPairs);
        const int per     = kCollectThreads * (one ? 1 : 2);
        const auto kernel = bilinear ? (one ? project_kernel<true, 1, true> : project_kernel<true, 2, true>)
                                     : (one ? project_kernel<true, 1, false> : project_kernel<true, 2, false>);
        launch(overlap, kernel, dim3((f.n + per - 1) / per, n_views), kCollectThreads, 0, st, f);
    }
    {
        PassScope t(ctx, VETR_T_SORT_BLEND, 2);
        const int grid = blend_blocks(f.PT, ctx->sm_count * ctx->blend_ctas_per_sm);
        const int long_grid = ctx->sm_count * ctx->blend_long_ctas_per_sm;
        if ((long long)f.n * n_views * (f.mode == VETR_MODE_BILINEAR_BLEND ? 4 : 1) >= kQueueFragments)
        {
            sort_blend_long_kernel<true><<<long_grid, kLongThreads, sizeof(LongBlendSmem), st>>>(f, out);
            launch(true, sort_blend_kernel<true>, grid, kThreads, sizeof(BlendSmem), st, f, out);
        }
        else
        {
            sort_blend_kernel<false><<<grid, kThreads, sizeof(BlendSmem), st>>>(f, out);
            launch(true, sort_blend_long_kernel<false>, long_grid, kLongThreads, sizeof(LongBlendSmem), st, f, out);
        }
    }
    VETR_CUDA(ctx, cudaGetLastError());
    return VETR_OK;
}

extern "C" int vetr_backward(vetr_ctx* ctx, const vetr_params* params, const vetr_cloud* cloud, const vetr_texture* texture,
                             const vetr_cameras* cameras, const vetr_view* views, int n_views, const float* dropout,
                             const vetr_lists* lists, const float* const* out_color, const float* const* grad_color,
                             float* g_desc, float* g_conf,
                             float* g_points, float* g_background, double* g_pose, float* g_pose_count, float* g_intr,
                             float* g_intr_count)
{
    return vetr_backward_phase(ctx, params, cloud, texture, cameras, views, n_views, dropout, lists, out_color, grad_color,
                               g_desc, g_conf, g_points, g_background, g_pose, g_pose_count, g_intr, g_intr_count,
                               VETR_BACKWARD_FRAGMENTS | VETR_BACKWARD_POINTS);
}

extern "C" int vetr_backward_phase(vetr_ctx* ctx, const vetr_params* params, const vetr_cloud* cloud,
                                   const vetr_texture* texture, const vetr_cameras* cameras, const vetr_view* views,
                                   int n_views, const float* dropout, const vetr_lists* lists,
                                   const float* const* out_color, const float* const* grad_color, float* g_desc,
                                   float* g_conf, float* g_points, float* g_background, double* g_pose,
                                   float* g_pose_count, float* g_intr, float* g_intr_count, int phases)
{
    const bool use_scratch = phases & VETR_BACKWARD_PIXEL_SCRATCH;
    if (use_scratch && !(phases & VETR_BACKWARD_FRAGMENTS)) return VETR_E_INVALID_ARG;
    phases &= ~VETR_BACKWARD_PIXEL_SCRATCH;
    if ((phases & ~(VETR_BACKWARD_FRAGMENTS | VETR_BACKWARD_POINTS)) != 0 || phases == 0) return VETR_E_INVALID_ARG;
    Frame f;
    int rc = fill_frame(ctx, f, params, cloud, texture, cameras, views, n_views, lists);
    if (rc != VETR_OK) return rc;
    if (!out_color || !grad_color || !g_desc || !g_conf || !g_background) return VETR_E_INVALID_ARG;
    if ((g_pose != nullptr) != (g_pose_count != nullptr) || (g_intr != nullptr) != (g_intr_count != nullptr))
        return VETR_E_INVALID_ARG;
    if (((uintptr_t)g_desc & 15) != 0 || ((uintptr_t)g_points & 15) != 0) return VETR_E_INVALID_ARG;
    BackPtrs bp;
    memset(&bp, 0, sizeof(bp));
    for (int l = 0; l < f.L; ++l)
    {
        if (!out_color[l] || !grad_color[l]) return VETR_E_INVALID_ARG;
        bp.out_color[l] = out_color[l], bp.grad_color[l] = grad_color[l];
    }
    bp.g_desc = (float4*)g_desc, bp.g_conf = g_conf, bp.g_points = (float4*)g_points, bp.g_background = g_background;
    bp.g_pose = g_pose, bp.g_pose_count = g_pose_count, bp.g_intr = g_intr, bp.g_intr_count = g_intr_count;
    if (!f.need_point_grad && f.mode != VETR_MODE_BILINEAR_BLEND && f.mode != VETR_MODE_FUZZY_DT) bp.g_points = nullptr;
    f.dropout          = dropout;
    const bool overlap = (long long)f.n * n_views <= kOverlapPoints;
    if (f.mode == VETR_MODE_FUZZY_DT)
    {
        if (!(phases & VETR_BACKWARD_FRAGMENTS)) return VETR_OK;  // mode 0 has one phase
        // Channel-interleaved copies: 9 gathers of 16 bytes per fragment instead of 36 of 4.  They cost 11 ps per pixel and save
        // 13 ps per point and view (2 M points, 2 views 1280x720: 234 -> 181 + 27 us), hence only where points are no fewer
        // than pixels; and only with the caller's word that the scratch is there, because mode 0 can do without.
        if (!use_scratch || ((uintptr_t)f.img4 & 15) != 0 || f.n < f.Prm) f.img4 = f.grad4 = nullptr;
        const int ctas = (f.n + kProjThreads - 1) / kProjThreads;
        PassScope t(ctx, VETR_T_BACKWARD, 1 + (ctas > 0));
        cudaStream_t st = ctx->stream;
        if (f.img4)
            launch(overlap, fuzzy_dt_pack_kernel, ctx->sm_count * 16, 256, 0, st, f, bp);
        else
            launch(overlap, fuzzy_dt_background_kernel, ctx->sm_count * 4, 256, 0, st, f, bp);
        if (ctas > 0)
        {
            const auto kernel = g_intr ? fuzzy_dt_backward_kernel<2> : g_pose ? fuzzy_dt_backward_kernel<1> : fuzzy_dt_backward_kernel<0>;
            launch(overlap, kernel, dim3(ctas, n_views), kProjThreads, 0, st, f, bp);
        }
        VETR_CUDA(ctx, cudaGetLastError());
        return VETR_OK;
    }
    const bool bilinear = f.mode == VETR_MODE_BILINEAR_BLEND;
    // position / camera gradients (and mode 3's confidence gradient) come from the per-point pass over what the
    // per-fragment kernel parks
    const bool spatial    = f.need_point_grad && (bp.g_points || g_pose || g_intr);
    const bool point_pass = bilinear || spatial;
    if (!spatial) f.need_point_grad = 0;
    if (point_pass && (!f.level_mask || !f.point_grad || ((uintptr_t)f.point_grad & 15) != 0)) return VETR_E_INVALID_ARG;
    if (bilinear && f.n_tex > kTexMask) return VETR_E_TOO_LARGE;
    if (!f.img4 || ((uintptr_t)f.img4 & 15) != 0) return VETR_E_INVALID_ARG;
    if (phases & VETR_BACKWARD_FRAGMENTS)
    {
        PassScope t(ctx, VETR_T_BACKWARD, f.mode == VETR_MODE_FUZZY_BLEND ? 4 : 3);
        cudaStream_t st = ctx->stream;
        launch(overlap, pack_images_kernel, (unsigned)((f.Prm * n_views + 255) / 256), 256, 0, st, f, bp);
        if (f.mode == VETR_MODE_FUZZY_BLEND)
        {
            const int grid = ctx->sm_count * ctx->fuzzy_ctas_per_sm;
            backward_kernel<true, false><<<grid, kThreads, sizeof(BackSmemFuzzy), st>>>(f, bp);
            launch(true, backward_fuzzy_long_kernel<kLongList, kFuzzyMidMax>, ctx->sm_count * ctx->fuzzy_mid_ctas_per_sm, kThreads, sizeof(FuzzyLongSmem<kFuzzyMidMax>), st, f, bp);
            launch(true, backward_fuzzy_long_kernel<kFuzzyMidMax, kFuzzyLongMax>, ctx->sm_count, kThreads, sizeof(FuzzyLongSmem<kFuzzyLongMax>), st, f, bp);
        }
        else if (bilinear)
        {
            const int grid = ctx->sm_count * ctx->bilinear_ctas_per_sm;
            backward_kernel<false, true><<<grid, kThreads, sizeof(BackSmemSuffix), st>>>(f, bp);
            launch(true, backward_long_kernel<true>, ctx->sm_count * ctx->bilinear_long_ctas_per_sm, kThreads, sizeof(BackSmemSuffix), st, f, bp);
        }
        else
        {
            const int grid = ctx->sm_count * ctx->back_ctas_per_sm;
            backward_kernel<false, false><<<grid, kThreads, sizeof(BackSmem), st>>>(f, bp);
            launch(true, backward_long_kernel<false>, ctx->sm_count * ctx->back_long_ctas_per_sm, kThreads, sizeof(BackSmemSuffix), st, f, bp);
        }
    }
    if ((phases & VETR_BACKWARD_POINTS) && point_pass && f.n > 0)
    {
        PassScope t(ctx, VETR_T_POINT_BACKWARD, 1);
        // several runs of 256 points per CTA share one camera reduction, as long as that leaves four CTAs per SM
        const int tiles   = std::max(1, std::min(kPointTilesMax, f.n / (kProjThreads * ctx->sm_count * 4)));
        const int ctas    = (f.n + kProjThreads * tiles - 1) / (kProjThreads * tiles);
        const size_t smem = (size_t)tiles * kProjThreads * sizeof(float4);
        const auto kernel = bilinear ? (g_intr ? point_backward_kernel<2, true> : g_pose ? point_backward_kernel<1, true> : point_backward_kernel<0, true>)
                                     : (g_intr ? point_backward_kernel<2, false> : g_pose ? point_backward_kernel<1, false> : point_backward_kernel<0, false>);
        launch(overlap, kernel, ctas, kProjThreads, smem, ctx->stream, f, bp, tiles);
    }
    VETR_CUDA(ctx, cudaGetLastError());
    return VETR_OK;
}

extern "C" int vetr_finalize_gradients(vetr_ctx* ctx, int channels, int n_tex, const float* g_desc, float* g_texture,
                                       int n, float* g_points, float* g_points_count, int n_img, double* g_pose,
                                       const float* g_pose_count, int n_cam, float* g_intr, const float* g_intr_count)
{
    if (!ctx) return VETR_E_INVALID_ARG;
    VETR_CUDA(ctx, cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    if (g_desc && g_texture && n_tex > 0 && channels != 3 && channels != 4) return VETR_E_INVALID_ARG;
    const auto blocks = [](bool wanted, int rows) { return wanted && rows > 0 ? (unsigned)((rows + 255ll) / 256) : 0u; };
    FinalizeArgs a;
    a.g_desc = (const float4*)g_desc, a.g_texture = g_texture, a.g_points = (float4*)g_points, a.g_points_count = g_points_count;
    a.g_pose = g_pose, a.g_pose_count = g_pose_count, a.g_intr = g_intr, a.g_intr_count = g_intr_count;
    a.C = channels, a.n_tex = n_tex, a.n = n, a.n_img = n_img, a.n_cam = n_cam;
    a.desc_end   = blocks(g_desc && g_texture, n_tex);
    a.points_end = a.desc_end + blocks(g_points != nullptr, n);
    a.pose_end   = a.points_end + blocks(g_pose && g_pose_count, n_img);
    const unsigned grid = a.pose_end + blocks(g_intr && g_intr_count, n_cam);
    PassScope t(ctx, VETR_T_FINALIZE, grid > 0);
    if (grid > 0) launch((long long)n + n_tex <= kOverlapPoints, finalize_kernel, grid, 256, 0, st, a);
    VETR_CUDA(ctx, cudaGetLastError());
    return VETR_OK;
}

extern "C" int64_t vetr_exchange_raw_floats(int n_tex, int n)
{
    if (n_tex < 0 || n < 0) return -1;
    return 5LL * n_tex + 4LL * n;
}

static long long exchange_out_points(int channels, int n_tex) { return ((long long)channels * n_tex + 3) / 4 * 4; }

extern "C" int64_t vetr_exchange_out_floats(int channels, int n_tex, int n)
{
    if ((channels != 3 && channels != 4) || n_tex < 0 || n < 0) return -1;
    return exchange_out_points(channels, n_tex) + 4LL * n + n_tex;
}

extern "C" int vetr_exchange_finalize(vetr_ctx* ctx, const vetr_exchange* ex, int channels, int n_tex, int n)
{
    return vetr_exchange_finalize_part(ctx, ex, channels, n_tex, n, VETR_SEG_DESC | VETR_SEG_POINTS | VETR_SEG_CONF, 4);
}

extern "C" int vetr_exchange_finalize_part(vetr_ctx* ctx, const vetr_exchange* ex, int channels, int n_tex, int n,
                                           int segments, int ctas_per_sm)
{
    if (!ctx || !ex || (channels != 3 && channels != 4) || n_tex < 1 || n < 0) return VETR_E_INVALID_ARG;
    if (segments <= 0 || (segments & ~(VETR_SEG_DESC | VETR_SEG_POINTS | VETR_SEG_CONF)) != 0) return VETR_E_INVALID_ARG;
    if (ctas_per_sm < 1 || ctas_per_sm > 8) return VETR_E_INVALID_ARG;
    if (ex->world < 1 || ex->world > VETR_MAX_RANKS || ex->rank < 0 || ex->rank >= ex->world) return VETR_E_INVALID_ARG;
    ExchangeArgs a;
    memset(&a, 0, sizeof(a));
    a.rank = ex->rank, a.world = ex->world, a.C = channels, a.n_tex = n_tex, a.n = n;
    a.out_points = exchange_out_points(channels, n_tex);
    a.out_conf   = a.out_points + 4LL * n;
    for (int k = 0; k < ex->world; ++k)
    {
        if (!ex->raw[k] || !ex->out[k] || ((uintptr_t)ex->raw[k] & 15) != 0 || ((uintptr_t)ex->out[k] & 15) != 0)
            return VETR_E_INVALID_ARG;
        a.raw[k] = ex->raw[k], a.out[k] = ex->out[k];
    }
    if ((ex->raw_multicast != nullptr) != (ex->out_multicast != nullptr)) return VETR_E_INVALID_ARG;
    if (((uintptr_t)ex->raw_multicast & 15) != 0 || ((uintptr_t)ex->out_multicast & 15) != 0) return VETR_E_INVALID_ARG;
    a.raw_mc = ex->raw_multicast, a.out_mc = ex->out_multicast;
    a.segments = segments;
    VETR_CUDA(ctx, cudaSetDevice(ctx->device));
    PassScope t(ctx, VETR_T_EXCHANGE, 1);
    if (a.raw_mc)
        exchange_finalize_kernel<true><<<ctx->sm_count * ctas_per_sm, 32 * kExchangeWarps, 0, ctx->stream>>>(a);
    else
        exchange_finalize_kernel<false><<<ctx->sm_count * ctas_per_sm, 32 * kExchangeWarps, 0, ctx->stream>>>(a);
    VETR_CUDA(ctx, cudaGetLastError());
    return VETR_OK;
}

// Room for n running sums, or nullptr where none is to be had: while the stream is being recorded, which forbids allocation,
// or when the device is full.
static double* grid_prefix(vetr_ctx* ctx, long long n)
{
    if (n > ctx->grid_prefix_cap)
    {
        cudaStreamCaptureStatus recording = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(ctx->stream, &recording) != cudaSuccess || recording != cudaStreamCaptureStatusNone)
        {
            cudaGetLastError();
            return nullptr;
        }
        const long long twice = 2 * ctx->grid_prefix_cap, cap = std::max(n, twice);
        double* p = nullptr;
        if (ctx->grid_prefix_n == 32 || cudaMalloc(&p, (size_t)cap * sizeof(double)) != cudaSuccess)
        {
            cudaGetLastError();
            return nullptr;
        }
        ctx->grid_prefix[ctx->grid_prefix_n++] = p;
        ctx->grid_prefix_cap = cap;
    }
    return ctx->grid_prefix[ctx->grid_prefix_n - 1];
}

extern "C" int vetr_grid_loss(vetr_ctx* ctx, const vetr_cameras* cams, const vetr_view* view, float dist_cutoff, int n_cells,
                              const float* cell_bb_min, const float* cell_bb_len, const float* loss_img, int channels,
                              float* cell_value, int32_t* cell_access_count)
{
    if (!ctx || !cams || !view || !cams->poses_se3 || !cams->intrinsics || n_cells < 0 || channels < 1) return VETR_E_INVALID_ARG;
    if (n_cells > 0 && (!cell_bb_min || !cell_bb_len || !loss_img || !cell_value || !cell_access_count)) return VETR_E_INVALID_ARG;
    if (view->w <= 0 || view->h <= 0) return VETR_E_INVALID_ARG;
    if (view->camera_model != 0) return VETR_E_UNSUPPORTED;
    if (view->image_index < 0 || view->image_index >= cams->n_img || view->camera_index < 0 || view->camera_index >= cams->n_cam)
        return VETR_E_INVALID_ARG;
    if ((long long)channels * view->w * view->h > 0x7fffffffLL) return VETR_E_TOO_LARGE;
    Frame f;
    memset(&f, 0, sizeof(f));
    f.n_views = 1, f.w = view->w, f.h = view->h, f.dist_cutoff = dist_cutoff;
    f.views[0].image_index = view->image_index, f.views[0].camera_index = view->camera_index;
    memcpy(f.views[0].crop, view->crop, sizeof(view->crop));
    memcpy(f.views[0].rot, view->rot, sizeof(view->rot));
    f.poses = cams->poses_se3, f.intr = cams->intrinsics;
    GridArgs a;
    a.bb_min = cell_bb_min, a.bb_len = cell_bb_len, a.loss = loss_img, a.value = cell_value, a.count = cell_access_count;
    a.n_cells = n_cells, a.channels = channels, a.h = view->h, a.w = view->w, a.view = 0;
    VETR_CUDA(ctx, cudaSetDevice(ctx->device));
    if (n_cells > 0)
    {
        if (!ctx->grid_queue)
        {
            VETR_CUDA(ctx, cudaMalloc(&ctx->grid_queue, (size_t)kGridQueueCap * sizeof(int2) + 256));
            ctx->grid_queue_count = reinterpret_cast<unsigned long long*>(ctx->grid_queue + kGridQueueCap);
        }
        a.prefix = grid_prefix(ctx, (long long)view->h * (view->w + 1)), a.no_rows = reinterpret_cast<int*>(ctx->grid_queue_count + 1);
        VETR_CUDA(ctx, cudaMemsetAsync(ctx->grid_queue_count, 0, 3 * sizeof(unsigned long long), ctx->stream));
        if (!a.prefix) VETR_CUDA(ctx, cudaMemsetAsync(a.no_rows, 1, sizeof(int), ctx->stream));
        ctx->launches += 2 + (a.prefix != nullptr);
        if (a.prefix) grid_row_sums_kernel<<<view->h, 256, 0, ctx->stream>>>(a);
        const int resident = ctx->sm_count * kGridCtas;
        const int groups = (int)((n_cells + (long long)kGridGroup - 1) / kGridGroup);
        const int each   = std::min(32 / kGridGroup, std::max(1, groups / (resident * kGridWarps)));
        const int ctas   = std::min((groups + kGridWarps - 1) / kGridWarps, resident);
        grid_loss_kernel<false><<<ctas, 32 * kGridWarps, 0, ctx->stream>>>(f, a, ctx->grid_queue, ctx->grid_queue_count, each);
        grid_loss_kernel<true><<<resident, 32 * kGridWarps, 0, ctx->stream>>>(f, a, ctx->grid_queue, ctx->grid_queue_count, 0);
    }
    VETR_CUDA(ctx, cudaGetLastError());
    return VETR_OK;
}

// Shared argument checks and parameter block of the two environment map calls, for views [v0, v0 + nv).
static int envmap_args(const vetr_cameras* cams, const vetr_view* views, int n_views, int num_layers, const vetr_envmap* env,
                       const float* const* weight, int flags, int v0, int nv, EnvArgs& a)
{
    if (!cams || !views || !env || !weight || !cams->poses_se3 || !cams->intrinsics || !env->density || !env->color)
        return VETR_E_INVALID_ARG;
    if (n_views < 1 || num_layers < 1 || num_layers > VETR_MAX_LAYERS) return VETR_E_INVALID_ARG;
    if (env->n_spheres < 1 || env->n_spheres > kEnvMaxSpheres || env->channels < 1 || env->channels > 4 || env->resolution < 1 ||
        env->up_axis < 0 || env->up_axis > 2 || (flags & ~15) != 0)
        return VETR_E_INVALID_ARG;
    if ((long long)env->n_spheres * env->resolution * env->resolution > 0x7fffffffLL) return VETR_E_TOO_LARGE;
    const int w = views[0].w, h = views[0].h;
    if (w <= 0 || h <= 0 || (w >> (num_layers - 1)) < 1 || (h >> (num_layers - 1)) < 1) return VETR_E_INVALID_ARG;
    memset(&a, 0, sizeof(a));
    a.n_views = nv, a.L = num_layers, a.S = env->n_spheres, a.R = env->resolution, a.C = env->channels;
    a.up_axis = env->up_axis, a.non_subzero = env->non_subzero_texture, a.flags = flags;
    memcpy(a.radii, env->radii, sizeof(a.radii));
    a.poses = cams->poses_se3, a.intr = cams->intrinsics, a.density = env->density, a.color = env->color;
    for (int b = 0; b < nv; ++b)
    {
        const vetr_view& v = views[v0 + b];
        if (v.w != w || v.h != h) return VETR_E_INVALID_ARG;
        if (v.camera_model != 0) return VETR_E_UNSUPPORTED;
        if (v.image_index < 0 || v.image_index >= cams->n_img || v.camera_index < 0 || v.camera_index >= cams->n_cam)
            return VETR_E_INVALID_ARG;
        a.views[b].image_index = v.image_index, a.views[b].camera_index = v.camera_index;
        memcpy(a.views[b].crop, v.crop, sizeof(v.crop));
        memcpy(a.views[b].rot, v.rot, sizeof(v.rot));
    }
    int run = 0, lw = w, lh = h;
    float scale = 1.f;
    for (int l = 0; l < num_layers; ++l, lw /= 2, lh /= 2, scale *= 0.5f)
    {
        if (!weight[l]) return VETR_E_INVALID_ARG;
        if ((long long)n_views * 4 * lw * lh > 0x7fffffffLL) return VETR_E_TOO_LARGE;
        a.lw[l] = lw, a.lh[l] = lh, a.scale[l] = scale, a.inv_lw[l] = 1.f / (float)lw;
        run += nv * lw * lh;  // a quarter of 2^31 on the largest level, a third more over all of them
        a.lend[l]   = run;
        a.weight[l] = weight[l] + (long long)v0 * lw * lh;
    }
    return VETR_OK;
}

// The cameras' distortion coefficients must all be zero: read back once per call (a few hundred bytes; synchronises).
static int envmap_check_distortion(vetr_ctx* ctx, const vetr_cameras* cams, const vetr_view* views, int n_views)
{
    std::vector<float> k((size_t)cams->n_cam * 13);
    VETR_CUDA(ctx, cudaMemcpyAsync(k.data(), cams->intrinsics, k.size() * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    VETR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (int b = 0; b < n_views; ++b)
    {
        if (views[b].camera_index < 0 || views[b].camera_index >= cams->n_cam) return VETR_E_INVALID_ARG;
        for (int i = 5; i < 13; ++i)
            if (k[(size_t)views[b].camera_index * 13 + i] != 0.f) return VETR_E_UNSUPPORTED;
    }
    return VETR_OK;
}

extern "C" int vetr_envmap_forward(vetr_ctx* ctx, const vetr_cameras* cams, const vetr_view* views, int n_views, int num_layers,
                                   const vetr_envmap* env, const float* const* weight, float* const* out, int flags)
{
    if (!ctx || !out) return VETR_E_INVALID_ARG;
    VETR_CUDA(ctx, cudaSetDevice(ctx->device));
    PassScope scope(ctx, VETR_T_ENVMAP, 0);
    for (int v0 = 0; v0 < n_views || v0 == 0; v0 += VETR_MAX_VIEWS)
    {
        const int nv = std::min(VETR_MAX_VIEWS, n_views - v0);
        EnvArgs a;
        int rc = envmap_args(cams, views, n_views, num_layers, env, weight, flags, v0, nv, a);
        if (rc != VETR_OK) return rc;
        if (v0 == 0 && !(flags & VETR_ENV_NO_DISTORTION_CHECK) && (rc = envmap_check_distortion(ctx, cams, views, n_views)) != VETR_OK) return rc;
        for (int l = 0; l < num_layers; ++l)
        {
            if (!out[l]) return VETR_E_INVALID_ARG;
            a.out[l] = out[l] + (long long)v0 * env->channels * a.lw[l] * a.lh[l];
        }
        const int grid = std::min((a.lend[num_layers - 1] + kEnvThreads - 1) / kEnvThreads, ctx->sm_count * 32);
        ctx->launches += 1;
        if (a.S <= kEnvFlatSpheres)
            envmap_forward_kernel<true><<<grid, kEnvThreads, 0, ctx->stream>>>(a);
        else
            envmap_forward_kernel<false><<<grid, kEnvThreads, 0, ctx->stream>>>(a);
    }
    VETR_CUDA(ctx, cudaGetLastError());
    return VETR_OK;
}

extern "C" int vetr_envmap_backward(vetr_ctx* ctx, const vetr_cameras* cams, const vetr_view* views, int n_views, int num_layers,
                                    const vetr_envmap* env, const float* const* weight, const float* const* grad_out, int flags,
                                    float* g_density, float* g_color)
{
    if (!ctx || !grad_out || !g_density || !g_color) return VETR_E_INVALID_ARG;
    VETR_CUDA(ctx, cudaSetDevice(ctx->device));
    PassScope scope(ctx, VETR_T_ENVMAP, 0);
    for (int v0 = 0; v0 < n_views || v0 == 0; v0 += VETR_MAX_VIEWS)
    {
        const int nv = std::min(VETR_MAX_VIEWS, n_views - v0);
        EnvArgs a;
        int rc = envmap_args(cams, views, n_views, num_layers, env, weight, flags, v0, nv, a);
        if (rc != VETR_OK) return rc;
        if (v0 == 0 && !(flags & VETR_ENV_NO_DISTORTION_CHECK) && (rc = envmap_check_distortion(ctx, cams, views, n_views)) != VETR_OK) return rc;
        for (int l = 0; l < num_layers; ++l)
        {
            if (!grad_out[l]) return VETR_E_INVALID_ARG;
            a.grad[l] = grad_out[l] + (long long)v0 * env->channels * a.lw[l] * a.lh[l];
        }
        a.g_density = g_density, a.g_color = g_color;
        ctx->launches += 1;
        const int grid = std::min((a.lend[num_layers - 1] + kEnvBackThreads - 1) / kEnvBackThreads, ctx->sm_count * 72);
        if (a.S <= kEnvFlatSpheres)
            envmap_backward_kernel<kEnvFlatSpheres><<<grid, kEnvBackThreads, 0, ctx->stream>>>(a);
        else
            envmap_backward_kernel<kEnvMaxSpheres><<<grid, kEnvBackThreads, 0, ctx->stream>>>(a);
    }
    VETR_CUDA(ctx, cudaGetLastError());
    return VETR_OK;
}

template <int KMAX>
static void knn_launch_search(vetr_ctx* ctx, const KnnSearch& a)
{
    knn_near_kernel<KMAX><<<(a.n + 127) / 128, 128, 0, ctx->stream>>>(a);
    knn_far_kernel<KMAX><<<ctx->sm_count * kKnnFarCtas, 128, 0, ctx->stream>>>(a);
}

extern "C" int vetr_knn_radius(vetr_ctx* ctx, const float* position, int position_stride, int n, int k, float* radius, int radius_stride)
{
    if (!ctx || n < 0 || k < 1 || k > kKnnMaxK || position_stride < 3 || radius_stride < 1) return VETR_E_INVALID_ARG;
    if (n == 0) return VETR_OK;
    if (!position || !radius) return VETR_E_INVALID_ARG;
    VETR_CUDA(ctx, cudaSetDevice(ctx->device));
    PassScope scope(ctx, VETR_T_KNN, 0);
    cudaStream_t st = ctx->stream;
    if (n > ctx->knn_cap_points)
    {
        cudaFree(ctx->knn_sorted), cudaFree(ctx->knn_point_cell), cudaFree(ctx->knn_queue);
        ctx->knn_sorted = nullptr, ctx->knn_point_cell = nullptr, ctx->knn_queue = nullptr, ctx->knn_cap_points = 0;
        VETR_CUDA(ctx, cudaMalloc(&ctx->knn_sorted, ((size_t)n + kKnnSortedPad) * sizeof(float4)));
        VETR_CUDA(ctx, cudaMalloc(&ctx->knn_point_cell, (size_t)n * sizeof(int)));
        VETR_CUDA(ctx, cudaMalloc(&ctx->knn_queue, (size_t)n * sizeof(int)));
        ctx->knn_cap_points = n;
    }
    if (!ctx->knn_tile_sums) VETR_CUDA(ctx, cudaMalloc(&ctx->knn_tile_sums, (16384 + 16) * sizeof(int)));
    unsigned* d_bounds          = reinterpret_cast<unsigned*>(ctx->knn_tile_sums + 16384);
    unsigned long long* d_occ   = reinterpret_cast<unsigned long long*>(ctx->knn_tile_sums + 16384 + 8);
    int* d_queue_count          = ctx->knn_tile_sums + 16384 + 10;

    // bounding box
    const unsigned init[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
    unsigned keys[6];
    VETR_CUDA(ctx, cudaMemcpyAsync(d_bounds, init, sizeof(init), cudaMemcpyHostToDevice, st));
    const int sweep = std::min((n + 255) / 256, ctx->sm_count * 8);
    knn_bounds_kernel<<<sweep, 256, 0, st>>>(position, position_stride, n, d_bounds);
    VETR_CUDA(ctx, cudaMemcpyAsync(keys, d_bounds, sizeof(keys), cudaMemcpyDeviceToHost, st));
    VETR_CUDA(ctx, cudaStreamSynchronize(st));
    float lo[3], hi[3], ext = 0.f, maxabs = 0.f;
    for (int a = 0; a < 3; ++a)
    {
        lo[a] = knn_unkey(keys[a]), hi[a] = knn_unkey(keys[3 + a]);
        if (!(lo[a] <= hi[a]) || std::isinf(lo[a]) || std::isinf(hi[a])) return VETR_E_INVALID_ARG;  // NaN or infinite coordinates
        ext    = std::max(ext, hi[a] - lo[a]);
        maxabs = std::max(maxabs, std::max(std::fabs(lo[a]), std::fabs(hi[a])));
    }

    // cell size: halve from 1/32 of the longest extent until an occupied cell holds 8 points or fewer on average
    KnnGrid g;
    g.ox = lo[0], g.oy = lo[1], g.oz = lo[2];
    auto dims_for = [&](float cell, int d[3]) -> long long
    {
        long long cells = 1;
        for (int a = 0; a < 3; ++a)
        {
            const double c = std::floor((double)(hi[a] - lo[a]) / cell) + 1.0;
            d[a] = (int)std::min(c, 1.0e9);
            cells = cells > (1ll << 40) ? cells : cells * d[a];
        }
        return cells;
    };
    float cell = ext > 0.f ? ext / 32.f : 1.f;
    int d[3];
    long long cells = dims_for(cell, d);
    bool counted = false;  // knn_cells and knn_point_cell hold the counts and cells of the current cell size
    for (int iter = 0; iter < 24 && ext > 0.f; ++iter)
    {
        int d2[3];
        const long long finer = dims_for(cell * 0.5f, d2);
        // fewer cells than n / 8: more than 8 points in an occupied cell, whatever the counts are
        if ((double)n / (double)cells > 8.0 && finer <= kKnnMaxCells)
        {
            cell *= 0.5f, cells = finer;
            d[0] = d2[0], d[1] = d2[1], d[2] = d2[2];
            continue;
        }
        if (cells > ctx->knn_cap_cells)
        {
            cudaFree(ctx->knn_cells);
            ctx->knn_cells = nullptr, ctx->knn_cap_cells = 0;
            const long long cap = std::min(kKnnMaxCells, std::max(cells * 8, 1ll << 20));
            VETR_CUDA(ctx, cudaMalloc(&ctx->knn_cells, (size_t)(cap + kKnnCellsPad) * sizeof(int)));
            ctx->knn_cap_cells = cap;
        }
        g.cell = cell, g.inv_cell = 1.f / cell, g.nx = d[0], g.ny = d[1], g.nz = d[2];
        VETR_CUDA(ctx, cudaMemsetAsync(ctx->knn_cells, 0, (size_t)(cells + kKnnCellsPad) * sizeof(int), st));
        VETR_CUDA(ctx, cudaMemsetAsync(d_occ, 0, sizeof(unsigned long long), st));
        knn_count_kernel<<<sweep, 256, 0, st>>>(position, position_stride, n, g, ctx->knn_cells + kKnnCellsPad, ctx->knn_point_cell);
        knn_occupied_kernel<<<(int)std::min<long long>((cells + 1023) / 1024, ctx->sm_count * 8), 256, 0, st>>>(ctx->knn_cells + kKnnCellsPad, cells, d_occ);
        unsigned long long occupied = 0;
        VETR_CUDA(ctx, cudaMemcpyAsync(&occupied, d_occ, sizeof(occupied), cudaMemcpyDeviceToHost, st));
        VETR_CUDA(ctx, cudaStreamSynchronize(st));
        ctx->launches += 2;
        counted = true;
        if (occupied == 0 || (double)n / (double)occupied <= 8.0) break;
        if (finer > kKnnMaxCells) break;
        counted = false;
        cell *= 0.5f, cells = finer;
        d[0] = d2[0], d[1] = d2[1], d[2] = d2[2];
    }
    if (cells > ctx->knn_cap_cells)  // all points coincide: no iteration ran
    {
        cudaFree(ctx->knn_cells);
        ctx->knn_cells = nullptr, ctx->knn_cap_cells = 0;
        const long long cap = std::max(cells, 1ll << 20);
        VETR_CUDA(ctx, cudaMalloc(&ctx->knn_cells, (size_t)(cap + kKnnCellsPad) * sizeof(int)));
        ctx->knn_cap_cells = cap;
    }
    g.cell = cell, g.inv_cell = 1.f / cell, g.nx = d[0], g.ny = d[1], g.nz = d[2];

    // counting sort into the chosen grid
    const int n_tiles = (int)((cells + kKnnScanTile - 1) / kKnnScanTile);
    // the scatter advances every cell's first slot to the next cell's: one entry further down they are first slots again
    int* const cursor = ctx->knn_cells + kKnnCellsPad;
    VETR_CUDA(ctx, cudaMemsetAsync(d_queue_count, 0, sizeof(int), st));
    if (!counted)
    {
        VETR_CUDA(ctx, cudaMemsetAsync(ctx->knn_cells, 0, (size_t)(cells + kKnnCellsPad) * sizeof(int), st));
        knn_count_kernel<<<sweep, 256, 0, st>>>(position, position_stride, n, g, ctx->knn_cells + kKnnCellsPad, ctx->knn_point_cell);
        ctx->launches += 1;
    }
    knn_tile_sums_kernel<true><<<n_tiles, 256, 0, st>>>(cursor, cells, ctx->knn_tile_sums);
    knn_spine_kernel<<<1, 1024, 0, st>>>(ctx->knn_tile_sums, n_tiles);
    knn_apply_kernel<true><<<n_tiles, 256, 0, st>>>(cursor, cells, ctx->knn_tile_sums, cursor);
    knn_scatter_kernel<<<sweep, 256, 0, st>>>(position, position_stride, n, ctx->knn_point_cell, cursor, ctx->knn_sorted);

    // search
    KnnSearch a;
    a.g = g, a.sorted = ctx->knn_sorted, a.first = cursor - 1, a.n = n;
    const int k1 = std::min(k, n - 1) + 1;  // list entries that count: the point itself and its k nearest
    a.slack = 1e-3f * cell + 4e-6f * (maxabs + ext);
    a.radius = radius, a.radius_stride = radius_stride, a.queue = ctx->knn_queue, a.queue_count = d_queue_count;
    if (k1 <= 5)
        a.dummies = 5 - k1, knn_launch_search<5>(ctx, a);
    else if (k1 <= 9)
        a.dummies = 9 - k1, knn_launch_search<9>(ctx, a);
    else
        a.dummies = 17 - k1, knn_launch_search<17>(ctx, a);
    ctx->launches += 7;
    VETR_CUDA(ctx, cudaGetLastError());
    return VETR_OK;
}

extern "C" int vetr_remove_points_plan(vetr_ctx* ctx, int n, const int64_t* remove, int m, int32_t* new_index, int* n_kept)
{
    if (!ctx || n < 0 || m < 0 || !n_kept || (n > 0 && !new_index) || (m > 0 && !remove)) return VETR_E_INVALID_ARG;
    if ((long long)n > kKnnMaxCells) return VETR_E_TOO_LARGE;  // one spine block scans 16384 tiles of 4096 flags
    *n_kept = 0;
    if (n == 0) return m == 0 ? VETR_OK : VETR_E_INVALID_ARG;
    VETR_CUDA(ctx, cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    if (n > ctx->points_cap)
    {
        cudaFree(ctx->points_flags);
        ctx->points_flags = nullptr, ctx->points_cap = 0;
        VETR_CUDA(ctx, cudaMalloc(&ctx->points_flags, (size_t)n * sizeof(int) + 16));
        ctx->points_cap = n;
    }
    if (!ctx->knn_tile_sums) VETR_CUDA(ctx, cudaMalloc(&ctx->knn_tile_sums, (16384 + 16) * sizeof(int)));
    int* d_small = ctx->knn_tile_sums + 16384 + 12;  // {bad index flag, survivors}
    VETR_CUDA(ctx, cudaMemsetAsync(d_small, 0, 2 * sizeof(int), st));
    const int sweep = std::min((n + 255) / 256, ctx->sm_count * 8);
    const int n_tiles = (n + kKnnScanTile - 1) / kKnnScanTile;
    points_fill_kernel<<<sweep, 256, 0, st>>>(ctx->points_flags, n, 1);
    if (m > 0) points_mark_removed_kernel<<<std::min((m + 255) / 256, ctx->sm_count * 8), 256, 0, st>>>((const long long*)remove, m, n, ctx->points_flags, d_small);
    knn_tile_sums_kernel<true><<<n_tiles, 256, 0, st>>>(ctx->points_flags, n, ctx->knn_tile_sums);
    knn_spine_kernel<<<1, 1024, 0, st>>>(ctx->knn_tile_sums, n_tiles);
    (((uintptr_t)new_index & 15) == 0 ? knn_apply_kernel<true> : knn_apply_kernel<false>)<<<n_tiles, 256, 0, st>>>(ctx->points_flags, n, ctx->knn_tile_sums, new_index);
    points_new_index_kernel<<<sweep, 256, 0, st>>>(ctx->points_flags, n, new_index, d_small + 1);
    ctx->launches += 6;
    int host[2] = {0, 0};
    VETR_CUDA(ctx, cudaMemcpyAsync(host, d_small, sizeof(host), cudaMemcpyDeviceToHost, st));
    VETR_CUDA(ctx, cudaStreamSynchronize(st));
    if (host[0]) return VETR_E_INVALID_ARG;
    *n_kept = host[1];
    return VETR_OK;
}

// Launches `kernel` for the arrays of which a row is units_of(width) > 0 units of work, up to kGatherArrays of them at a time.
template <typename Total, typename Kernel, typename Units>
static void gather_arrays(vetr_ctx* ctx, Kernel kernel, int n, int n_kept, const int32_t* new_index, const vetr_point_array* arrays, int n_arrays,
                          Units units_of)
{
    GatherArgs<Total> g;
    memset(&g, 0, sizeof(g));
    g.new_index = new_index, g.n = n, g.n_kept = n_kept;
    long long total   = 0;
    const auto flush = [&]()
    {
        if (g.arrays == 0) return;
        const int blocks = (int)(((long long)n + kGatherBlock - 1) / kGatherBlock);
        const int share  = std::max(1, ctx->sm_count * 16 / blocks);  // sixteen blocks per SM
        kernel<<<dim3(blocks, (unsigned)std::min<long long>(std::min(share, 65535), total)), 256, 0, ctx->stream>>>(g);
        ctx->launches += 1;
        g.arrays = 0, total = 0;
    };
    for (int k = 0; k < n_arrays; ++k)
    {
        const vetr_point_array& a = arrays[k];
        const long long units     = (long long)a.rows * units_of(a.width);
        if (units == 0) continue;
        // a launch when the table is full, and where one more array would leave the counter's range
        if (g.arrays == kGatherArrays || total + units > (long long)std::numeric_limits<Total>::max()) flush();
        total += units;
        g.src[g.arrays] = (const uint32_t*)a.src, g.dst[g.arrays] = (uint32_t*)a.dst;
        g.end[g.arrays] = (Total)total, g.width[g.arrays] = a.width;
        ++g.arrays;
    }
    flush();
}

extern "C" int vetr_gather_points(vetr_ctx* ctx, int n, int n_kept, const int32_t* new_index, const vetr_point_array* arrays, int n_arrays)
{
    if (!ctx || n < 0 || n_kept < 0 || n_kept > n || n_arrays < 0 || (n_arrays > 0 && !arrays) || (n > 0 && !new_index))
        return VETR_E_INVALID_ARG;
    for (int k = 0; k < n_arrays; ++k)
    {
        const vetr_point_array& a = arrays[k];
        if (a.rows < 1 || a.width < 1 || (n > 0 && !a.src) || (n_kept > 0 && !a.dst)) return VETR_E_INVALID_ARG;
        if (a.width == 4 && ((((uintptr_t)a.src | (uintptr_t)a.dst) & 15) != 0)) return VETR_E_INVALID_ARG;
    }
    if (n == 0 || n_kept == 0) return VETR_OK;
    VETR_CUDA(ctx, cudaSetDevice(ctx->device));
    gather_arrays<int>(ctx, points_gather_kernel, n, n_kept, new_index, arrays, n_arrays, [](int width) { return width <= kGatherNarrow ? 1 : 0; });
    gather_arrays<long long>(ctx, points_gather_pieces_kernel, n, n_kept, new_index, arrays, n_arrays,
                             [](int width) { return width <= kGatherNarrow ? 0 : gather_pieces(width); });
    VETR_CUDA(ctx, cudaGetLastError());
    return VETR_OK;
}

extern "C" int vetr_l1_loss_grad(vetr_ctx* ctx, int num_levels, const float* const* image, const float* const* target,
                                 float* const* grad, const int64_t* numel, float* loss)
{
    if (!ctx || num_levels < 1 || num_levels > VETR_MAX_LAYERS || !image || !target || !grad || !numel || !loss)
        return VETR_E_INVALID_ARG;
    L1Args a;
    memset(&a, 0, sizeof(a));
    long long run = 0;
    for (int l = 0; l < num_levels; ++l)
    {
        if (!image[l] || !target[l] || !grad[l] || numel[l] < 1) return VETR_E_INVALID_ARG;
        if ((((uintptr_t)image[l] | (uintptr_t)target[l] | (uintptr_t)grad[l]) & 15) != 0) return VETR_E_INVALID_ARG;
        a.image[l] = image[l], a.target[l] = target[l], a.grad[l] = grad[l];
        run += numel[l];
        a.end[l]       = run;
        a.inv_numel[l] = 1.f / (float)numel[l];
    }
    a.levels = num_levels, a.loss = loss;
    VETR_CUDA(ctx, cudaSetDevice(ctx->device));
    VETR_CUDA(ctx, cudaMemsetAsync(loss, 0, sizeof(float), ctx->stream));
    ctx->launches += 1;
    launch(run <= kOverlapPoints, l1_loss_grad_kernel, ctx->sm_count * 8, 256, 0, ctx->stream, a);
    VETR_CUDA(ctx, cudaGetLastError());
    return VETR_OK;
}

extern "C" int vetr_apply_tangent(vetr_ctx* ctx, double* tangent, double* poses_se3, int n)
{
    if (!ctx || !tangent || !poses_se3 || n < 0) return VETR_E_INVALID_ARG;
    VETR_CUDA(ctx, cudaSetDevice(ctx->device));
    if (n > 0)
    {
        ctx->launches += 1;
        apply_tangent_kernel<<<(n + 127) / 128, 128, 0, ctx->stream>>>(tangent, poses_se3, n);
    }
    VETR_CUDA(ctx, cudaGetLastError());
    return VETR_OK;
}

extern "C" int vetr_read_status(vetr_ctx* ctx, const vetr_lists* lists, int64_t* total_fragments, int32_t* longest_list)
{
    if (!ctx || !lists || !lists->status) return VETR_E_INVALID_ARG;
    int h[4];
    VETR_CUDA(ctx, cudaSetDevice(ctx->device));
    VETR_CUDA(ctx, cudaMemcpyAsync(h, lists->status, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
    VETR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (total_fragments) *total_fragments = h[0];
    if (longest_list) *longest_list = h[2];
    if (h[1] & 1) return VETR_E_LIST_OVERFLOW;
    return (h[1] & 2) ? VETR_E_TOO_LARGE : VETR_OK;
}

// ---------------------------------------------------------------------------------------------------------
// Scan without any allocation.
//
// Some hosts must not allocate device memory while they render: an interactive viewer whose frame loop cannot afford
// the device-wide stall of cudaMalloc / cudaFree, a process whose device memory is handed out once at start-up by an
// arena it does not own, or code running inside a region where the driver forbids allocation.  For them the scan's
// only scratch (one partial sum per tile of 4096 pixels, and the ticket) lives in a fixed array inside the library image instead of a
// buffer grown on demand.  Every GPU that loads the library carries these 128 KB until the process exits.
namespace vetr
{
constexpr int kStaticScanTiles = 16384;  // 16384 tiles x 4096 pixels = 67 108 864 pixels per call
static __device__ __align__(256) long long g_static_tile_sums[kStaticScanTiles + 1];  // and the ticket
}  // namespace vetr
static long long* g_static_tile_ptr[64] = {};  // device address of the array above, per device ordinal

extern "C" int vetr_scan_counts_static(int device, void* cuda_stream, const int32_t* counts, int64_t n_pixels,
                                       int64_t capacity, int32_t* ends, int32_t* status, int32_t* items,
                                       int64_t items_capacity)
{
    if (device < 0 || device >= 64 || !counts || !ends || !status || !items || n_pixels < 1 || capacity < 0)
        return VETR_E_INVALID_ARG;
    if (n_pixels > 0x7fffffffLL) return VETR_E_TOO_LARGE;
    const long long n_tiles = (n_pixels + kScanTile - 1) / kScanTile;
    if (n_tiles > kStaticScanTiles) return VETR_E_TOO_LARGE;  // more pixels than the fixed scratch covers
    if (items_capacity < vetr_item_table_entries(capacity, n_pixels)) return VETR_E_INVALID_ARG;
    // the launches below go to `device`; the caller's current device is put back before returning
    int caller_device = device;
    if (cudaGetDevice(&caller_device) != cudaSuccess) return VETR_E_CUDA;
    struct RestoreDevice
    {
        int to, from;
        ~RestoreDevice()
        {
            if (to != from) cudaSetDevice(to);
        }
    } restore{caller_device, device};
    if (caller_device != device && cudaSetDevice(device) != cudaSuccess) return VETR_E_CUDA;
    if (!g_static_tile_ptr[device])
    {
        // The array's name is only a handle on the host; kernels need its address on THIS device.
        long long* p = nullptr;
        if (cudaGetSymbolAddress((void**)&p, g_static_tile_sums) != cudaSuccess || !p) return VETR_E_CUDA;
        g_static_tile_ptr[device] = p;
    }
    long long* tile_sums = g_static_tile_ptr[device];
    cudaStream_t st      = (cudaStream_t)cuda_stream;
    // the status words are accumulated into (longest list is an atomic maximum): start them at zero
    if (cudaMemsetAsync(status, 0, 4 * sizeof(int), st) != cudaSuccess) return VETR_E_CUDA;
    if (cudaMemsetAsync(tile_sums + kStaticScanTiles, 0, sizeof(long long), st) != cudaSuccess) return VETR_E_CUDA;
    launch_scan(counts, n_pixels, capacity, tile_sums, reinterpret_cast<unsigned*>(tile_sums + kStaticScanTiles), (int)n_tiles, ends, status, items, items + (items_capacity - 1), st, false);
    return cudaGetLastError() == cudaSuccess ? VETR_OK : VETR_E_CUDA;
}

// Parity / debugging: the lists of one (view, level) in the reference's layout.  The reference keeps its lists in
// row-major pixel order; here they are stored in the banded order of the pixel space, so the level is brought to the
// host, reordered there and copied back (a debugging call: it synchronises and is not meant for large scenes).
extern "C" int vetr_get_lists(vetr_ctx* ctx, const vetr_lists* lists, int w, int h, int num_layers, int n_views, int view,
                              int layer, int32_t* out_collections, int32_t* out_scanned_counting, int64_t* n_fragments)
{
    if (!ctx || !lists || num_layers < 1 || num_layers > VETR_MAX_LAYERS || view < 0 || view >= n_views || layer < 0 ||
        layer >= num_layers)
        return VETR_E_INVALID_ARG;
    int lw[VETR_MAX_LAYERS], lh[VETR_MAX_LAYERS];
    long long lbase[VETR_MAX_LAYERS];
    const long long P    = pyramid(w, h, num_layers, lw, lh, lbase);
    const long long g0   = (long long)view * P + lbase[layer];
    const int W = lw[layer], H = lh[layer];
    const long long npad = (long long)W * ((H + kBand - 1) / kBand * kBand);  // pixels of the level in the pixel space
    if ((long long)W * H == 0)
    {
        if (n_fragments) *n_fragments = 0;
        return VETR_OK;
    }
    VETR_CUDA(ctx, cudaSetDevice(ctx->device));
    std::vector<int> counts((size_t)npad), ends((size_t)npad);
    VETR_CUDA(ctx, cudaMemcpyAsync(counts.data(), lists->counts + g0, npad * 4, cudaMemcpyDeviceToHost, ctx->stream));
    VETR_CUDA(ctx, cudaMemcpyAsync(ends.data(), lists->ends + g0, npad * 4, cudaMemcpyDeviceToHost, ctx->stream));
    VETR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    const long long first = (long long)ends[0] - counts[0];
    const long long n     = (long long)ends[(size_t)npad - 1] - first;
    if (n_fragments) *n_fragments = n;
    if (!out_collections && !out_scanned_counting) return VETR_OK;
    std::vector<uint4> recs;
    if (out_collections && n > 0)
    {
        recs.resize((size_t)(2 * n));
        VETR_CUDA(ctx, cudaMemcpyAsync(recs.data(), (const uint4*)lists->frags + 2 * first, (size_t)n * 32, cudaMemcpyDeviceToHost,
                                       ctx->stream));
        VETR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    }
    std::vector<int> scanned((size_t)W * H), coll(out_collections ? (size_t)(2 * n) : 0);
    long long run = 0;
    for (int y = 0; y < H; ++y)
        for (int x = 0; x < W; ++x)
        {
            const size_t k = (size_t)(y >> kBandShift) * ((size_t)W << kBandShift) + ((size_t)x << kBandShift) + (y & (kBand - 1));  // pixel_offset
            scanned[(size_t)y * W + x] = (int)run;
            if (out_collections)
                for (int j = 0; j < counts[k]; ++j)
                {
                    const uint4 r = recs[(size_t)(2 * ((long long)ends[k] - counts[k] - first + j))];
                    coll[(size_t)(run + j)]     = (int)r.y;  // row 0: depth bits
                    coll[(size_t)(n + run + j)] = (int)r.x;  // row 1: point index
                }
            run += counts[k];
        }
    if (out_collections && n > 0)
        VETR_CUDA(ctx, cudaMemcpyAsync(out_collections, coll.data(), (size_t)(2 * n) * 4, cudaMemcpyHostToDevice, ctx->stream));
    if (out_scanned_counting)
        VETR_CUDA(ctx, cudaMemcpyAsync(out_scanned_counting, scanned.data(), (size_t)W * H * 4, cudaMemcpyHostToDevice, ctx->stream));
    VETR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return VETR_OK;
}

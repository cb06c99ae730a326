// Error-grid rasterisation (FillSceneGridWithLossRasterize, rendering/RenderForward.cu:639-791): the step between a training
// epoch and the point spawning.  Every cell of the scene grid whose eight corners lie in front of the camera adds the L1
// loss of the pixels its projected box covers and their number.
//
// The reference tests every pixel of a cell's screen rectangle against the twelve triangles of the box (two per face) and
// issues two global atomics per covered pixel.  Those tests are what bounds a per-pixel form (twelve triangles of three
// edge functions in strict fp32 for each of some 600 M pixels at 128^3 cells and 1920 x 1080: 7.9 ms).  Here a lane owns one
// pixel ROW of a cell: the twelve triangles are a closed surface, so what they cover of a row is the run of pixels between its
// leftmost and rightmost crossing with the 18 segments (12 edges, 6 face diagonals), and the run's loss is a difference
// of two running sums of that image row (fp64, formed once per call).  0.63 ms at the same sizes.
//
// Why one run: a row cuts the surface in a connected set if the part of the surface above it and the part below are both
// connected (the surface is a sphere), and they are for every row if only one corner has no higher neighbour along the 18
// segments and only one has no lower neighbour.  grid_prepare counts them.  Nothing else is asked of the corners: faces may be
// bent, as they are far from the origin, where the corners are rounded to the grid of the world coordinates.
//
// The numbers stay those of the per-pixel tests, rounding included: a row in which any pixel comes so close to one of the
// 18 segments that the strict fp32 edge functions could disagree with it goes through the per-pixel test
// (grid_exact_row), and cells for which the argument does not hold - several highest or lowest corners, a face seen
// nearly edge-on, corners far outside the image, a lens distortion, rectangles whose fp32 pixel coordinates may skip a
// number, a loss image with Inf or NaN, no room for the running sums - are walked pixel by pixel as a whole.
#pragma once
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

namespace vetr
{
struct GridArgs
{
    const float* bb_min;
    const float* bb_len;
    const float* loss;
    float* value;
    int* count;
    double* prefix;   // [h][w + 1]: sum over the channels of |loss| of the pixels left of x in the row
    int* no_rows;     // not 0: no running sums, either for want of room or because a pixel's loss is Inf or NaN (they would
                      // carry it to the right)
    int n_cells, channels, h, w, view;
};

__device__ __forceinline__ float tri_sign(float2 p1, float2 p2, float2 p3)
{
    return VS(VM(VS(p1.x, p3.x), VS(p2.y, p3.y)), VM(VS(p2.x, p3.x), VS(p1.y, p3.y)));
}
__device__ __forceinline__ bool point_in_triangle(float2 pt, float2 v1, float2 v2, float2 v3)
{
    const float d1 = tri_sign(pt, v1, v2), d2 = tri_sign(pt, v2, v3), d3 = tri_sign(pt, v3, v1);
    const bool has_neg = (d1 < 0) || (d2 < 0) || (d3 < 0);
    const bool has_pos = (d1 > 0) || (d2 > 0) || (d3 > 0);
    return !(has_neg && has_pos);
}
// The reference's coverage test: faces of the box as pairs of triangles (RenderForward.cu:676-677).
__device__ __forceinline__ bool point_in_box(float2 pt, const float2 pp[8])
{
    bool in = false;
    in |= point_in_triangle(pt, pp[0], pp[1], pp[4]) || point_in_triangle(pt, pp[0], pp[4], pp[2]);
    in |= point_in_triangle(pt, pp[1], pp[5], pp[7]) || point_in_triangle(pt, pp[1], pp[7], pp[4]);
    in |= point_in_triangle(pt, pp[5], pp[3], pp[6]) || point_in_triangle(pt, pp[5], pp[6], pp[7]);
    in |= point_in_triangle(pt, pp[3], pp[0], pp[6]) || point_in_triangle(pt, pp[0], pp[6], pp[2]);
    in |= point_in_triangle(pt, pp[3], pp[0], pp[5]) || point_in_triangle(pt, pp[0], pp[5], pp[1]);
    in |= point_in_triangle(pt, pp[2], pp[4], pp[6]) || point_in_triangle(pt, pp[4], pp[6], pp[7]);
    return in;
}
__device__ __forceinline__ float grid_pixel_loss(const GridArgs& a, int x, int y)
{
    float g = 0.f;
    for (int i = 0; i < a.channels; ++i) g += fabsf(__ldg(a.loss + ((long long)i * a.h + y) * a.w + x));
    return g;
}

constexpr int kGridWarps    = 4;
constexpr int kGridGroup    = 4;                // cells a warp takes together: eight lanes each
constexpr int kGridRowBits    = 6;              // 64 rows of a queued chunk; cells of up to that many rows are not queued (32: 702 instead of 655 us,
                                                // 35^3 cells at 160x120 45 instead of 37; 128: 835 instead of 805)
constexpr int kGridRowChunk   = 1 << kGridRowBits;
constexpr int kGridChunkBits  = 6;              // 64 pixels of a rectangle, at least, that one warp walks in the per-pixel form
constexpr int kGridExactLanes = 6;              // rows of a warp with pixels to be tested from which on their own lanes test them (2: the same; never: 128^3
                                                // cells at 1920x1080 the same to 767 instead of 612 us in twelve views, 64^3 287 instead of 216)
constexpr int kGridQueueCap = 4 * 1024 * 1024;  // (cell, chunk) pairs handed to the second kernel
// Sizes of the per-pixel form's chunks, 64 << 0 to kGridCoarsest pixels: see grid_coarse.
constexpr int kGridCoarsest   = 3;
constexpr int kGridCoarseFrom = kGridQueueCap / 8;  // chunks in the queue
constexpr int kGridVast       = 1 << 16;        // pixels of a cell
constexpr int kGridMarkAt     = 28;             // bit of a chunk's number from which on the shift stands (an image has no more than 2^31 / 64 chunks)
constexpr int kGridSegments = 18;               // 12 edges, then 6 face diagonals
constexpr int kGridCtas     = 6;                // resident CTAs per SM the kernels are compiled for (5: the same, 8: 10 % slower)

// Running sums of |loss| along every image row, one CTA per row, four pixels per thread and step.  A sum is formed in fp64 from
// what lies to its left and nothing else, in at most 8 w / 1024 + 17 additions one after the other: it is off by less than
// that many times 2^-53 of itself (1920 pixels: 33, 16384 pixels: 145).
__global__ void __launch_bounds__(256) grid_row_sums_kernel(const __grid_constant__ GridArgs a)
{
    __shared__ double s_warp[8];
    const int y = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* row   = a.prefix + (long long)y * (a.w + 1);
    double before = 0.0;  // sum of the steps already done
    bool bad      = false;
    for (int base = 0; base < a.w; base += 1024)
    {
        const int x0 = base + 4 * threadIdx.x;
        double v[4], sum = 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            const float g = x0 + k < a.w ? grid_pixel_loss(a, x0 + k, y) : 0.f;
            bad |= !(g <= 3.402823466e38f);
            v[k] = sum;
            sum += (double)g;
        }
        double inc = sum;
        for (int o = 1; o < 32; o <<= 1)
        {
            const double t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) s_warp[warp] = inc;
        __syncthreads();
        double off = __shfl_up_sync(0xffffffffu, inc, 1);  // (not inc - sum: what lies to the right must leave no rounding here)
        off        = before + (lane == 0 ? 0.0 : off);
        for (int w = 0; w < 8; ++w)
        {
            if (w < warp) off += s_warp[w];
            before += s_warp[w];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (x0 + k <= a.w) row[x0 + k] = off + v[k];
        __syncthreads();
    }
    if (threadIdx.x == 0 && (a.w & 1023) == 0) row[a.w] = before;
    if (__any_sync(0xffffffffu, bad) && lane == 0) *a.no_rows = 1;
}

#define VETR_GRID_SEGMENTS                                                                                                                  \
    {{0, 1}, {2, 4}, {3, 5}, {6, 7}, {0, 2}, {1, 4}, {3, 6}, {5, 7}, {0, 3}, {1, 5}, {2, 6}, {4, 7}, {0, 4}, {1, 7}, {5, 6}, {0, 6}, {0, 5}, {4, 6}}
#define VETR_GRID_TRIANGLES                                                                                                                 \
    {{0, 1, 4}, {0, 4, 2}, {1, 5, 7}, {1, 7, 4}, {5, 3, 6}, {5, 6, 7}, {3, 0, 6}, {0, 6, 2}, {3, 0, 5}, {0, 5, 1}, {2, 4, 6}, {4, 6, 7}}
__constant__ signed char kGridSegEnds[kGridSegments][2] = VETR_GRID_SEGMENTS;
__constant__ signed char kGridTriangles[12][3]          = VETR_GRID_TRIANGLES;
// The same for loops that are unrolled.
struct GridTables
{
    int ends[kGridSegments][2] = VETR_GRID_SEGMENTS, triangles[12][3] = VETR_GRID_TRIANGLES;
    int sides[12][3] = {};  // segments between corners 0 1, 0 2 and 1 2 of a triangle
    constexpr GridTables()
    {
        for (int t = 0; t < 12; ++t)
            for (int k = 0; k < 3; ++k)
                for (int g = 0; g < kGridSegments; ++g)
                {
                    const int p = triangles[t][k == 2], q = triangles[t][k == 0 ? 1 : 2];
                    if ((ends[g][0] == p && ends[g][1] == q) || (ends[g][0] == q && ends[g][1] == p)) sides[t][k] = g;
                }
    }
};

struct GridWarpSmem
{
    float2 corner[8][33];                   // projected corners of up to 32 cells, a lane's cell per column
    float2 pp[kGridGroup][8];               // those of the group in work
    float4 seg[kGridSegments][kGridGroup];   // {x at row 0, dx/dy, middle row, half the rows (rounded up)}, relative to the rectangle's first pixel
    float2 band[kGridSegments][kGridGroup];  // {half-width of the band along the row, half the rows with what the band adds to them}
    int4 rect[kGridGroup];                   // first column, first row, columns, rows
    int2 spot[kGridGroup][8];                // {row, column} of the pixel next to a corner, row -1 if it is far enough away
    int spots[kGridGroup];                   // not 0: there are some
    int2 todo[64];                          // {cell, chunk} to be prepared
    int queued;                             // chunks in the queue when the warp looked last
};

// Corner order of the reference: (0,0,0) (1,0,0) (0,1,0) (0,0,1) (1,1,0) (1,0,1) (0,1,1) (1,1,1).
__device__ __forceinline__ float2 grid_project_corner(const Frame& f, const Camera& cam, const float (&box)[3], const float (&len)[3], int corner,
                                                       bool& behind)
{
    const float fx = 0xb2 >> corner & 1 ? 1.f : 0.f, fy = 0xd4 >> corner & 1 ? 1.f : 0.f, fz = 0xe8 >> corner & 1 ? 1.f : 0.f;
    const float4 pos   = make_float4(VA(box[0], VM(len[0], fx)), VA(box[1], VM(len[1], fy)), VA(box[2], VM(len[2], fz)), 0.f);
    const Projected pr = project_point(pos, cam, f.dist_cutoff);
    behind |= pr.z <= 0.f;
    return pr.ip;
}

// Clamped screen rectangle from the corners' bounding box (mn is clamped in place); returns the number of pixels to test.
__device__ __forceinline__ long long grid_rectangle(const GridArgs& a, float2& mn, float2 mx, int& x_size, int& y_size)
{
    const float border = 32.f, W = (float)a.w, H = (float)a.h;
    x_size = y_size = 0;
    if (mx.x < border || mn.x >= VS(W, border) || mx.y < border || mn.y >= VS(H, border)) return 0;
    mn.x = fmaxf(mn.x, border), mn.y = fmaxf(mn.y, border);
    mx.x = fminf(mx.x, VS(W, border)), mx.y = fminf(mx.y, VS(H, border));
    y_size = (int)VS(mx.y, mn.y);
    x_size = (int)VS(mx.x, mn.x);
    return (long long)y_size * x_size;
}

// Per-pixel form: pixels [first, last) of a cell's rectangle, one per lane and step; adds the warp's totals to the cell.
__device__ __noinline__ void grid_cell_pixels(const GridArgs& a, int c, int lane, const float2* s_pp, float2 mn, int x_size, long long first,
                                              long long last)
{
    float2 pp[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) pp[i] = s_pp[i];
    float sum = 0.f;
    int hits  = 0;
    // (a rectangle has no more pixels than the image, hence 32 bits; in images below 64 pixels across x_size can be negative)
    const int width = abs(x_size), turn = x_size < 0 ? -1 : 1, dx = 32 % width, dy = 32 / width * turn;
    int x = ((int)first + lane) % width, y = ((int)first + lane) / width * turn;
    for (unsigned xy = (unsigned)first + lane; xy < (unsigned)last; xy += 32, x += dx, y += dy)
    {
        if (x >= width) x -= width, y += turn;
        const int x_c = (int)VA((float)x, mn.x);
        const int y_c = (int)VA((float)y, mn.y);
        if (!point_in_box(make_float2((float)x_c, (float)y_c), pp)) continue;
        sum += grid_pixel_loss(a, x_c, y_c);
        ++hits;
    }
    for (int o = 16; o > 0; o >>= 1)
    {
        sum += __shfl_down_sync(0xffffffffu, sum, o);
        hits += __shfl_down_sync(0xffffffffu, hits, o);
    }
    if (lane == 0 && hits > 0)
    {
        atomicAdd(a.value + c, sum);
        atomicAdd(a.count + c, hits);
    }
}

// Base run of a row: the pixels between its leftmost and rightmost crossing.  Its loss is a difference of two running sums, whose
// rounding goes with the larger one.  A difference 2^20 times smaller than that - a run behind a pixel a million times
// brighter, or over pixels without loss - is formed pixel by pixel instead (grid_run_pixels; for a row with pixels in a band the
// whole cell is, see grid_rows).  Any other is off by less than 145 x 2^-52 x 2^20 = 3.4e-8 of itself up to 16384 pixels a row, half a
// unit in the last place of the fp32 result.  (Letting grid_exact_row repeat such a row by itself cost registers: 995 instead
// of 915 us at the sizes above.)
constexpr int kGridCancelBits = 20;

__device__ __forceinline__ bool grid_cancels(double sum, double scale)  // (high words: the exponent and 20 bits behind it)
{
    return __double2hiint(sum) < __double2hiint(scale) - (kGridCancelBits << 20);
}
__device__ __forceinline__ bool grid_run_ends(const int4 rect, float L, float R, int& xl, int& xr)
{
    xl = (int)fmaxf(ceilf(L), 0.f), xr = (int)fminf(floorf(R), (float)(rect.z - 1));
    return xl <= xr;
}
__device__ __forceinline__ const double* grid_prefix(const GridArgs& a, int y) { return a.prefix + (long long)y * (a.w + 1); }
__device__ __forceinline__ int grid_run(const GridArgs& a, const int4 rect, int j, float L, float R, double& sum, bool* cancels = nullptr)
{
    int xl, xr;
    if (!grid_run_ends(rect, L, R, xl, xr)) return 0;
    const double* p  = grid_prefix(a, rect.y + j) + rect.x;
    const double end = p[xr + 1], run = end - p[xl];
    if (cancels) *cancels = grid_cancels(run, end);
    sum += run;
    return xr - xl + 1;
}
__device__ __noinline__ double grid_run_pixels(const GridArgs& a, const GridWarpSmem& s, int slot, int j, float L, float R)
{
    int xl, xr;
    double sum = 0.0;
    const int4 rect = s.rect[slot];
    if (!grid_run_ends(rect, L, R, xl, xr)) return sum;
    for (int x = xl; x <= xr; ++x) sum += (double)grid_pixel_loss(a, rect.x + x, rect.y + j);
    return sum;
}

// Crossing of row y with segment k of a slot's cell, extended beyond its ends; true if it lies on the segment.
__device__ __forceinline__ bool grid_crossing(const GridWarpSmem& s, int k, int slot, float y, float& xs)
{
    const float4 g = s.seg[k][slot];
    xs             = __fmaf_rn(g.y, y, g.x);
    return fabsf(y - g.z) <= g.w;
}
// Pixels [x0, x1] of the row that lie in the segment's band.
__device__ __forceinline__ void grid_band(const GridWarpSmem& s, const int4 rect, int k, int slot, float y, float xs, int& x0, int& x1)
{
    const float2 b = s.band[k][slot];
    x0 = 1, x1 = 0;
    if (fabsf(y - s.seg[k][slot].z) <= b.y) x0 = (int)fmaxf(ceilf(xs - b.x), 0.f), x1 = (int)fminf(floorf(xs + b.x), (float)(rect.z - 1));
}

// Leftmost and rightmost crossing of row j with the segments of a cell; true if a pixel lies in the band of one.  Bound by instruction
// issue, 13 per segment.
__device__ __forceinline__ bool grid_crossings(const GridWarpSmem& s, int slot, int j, float& L, float& R)
{
    const float y = (float)j;
    bool close = false;
    L = CUDART_INF_F, R = -CUDART_INF_F;
#pragma unroll 6
    for (int q = 0; q < kGridSegments; ++q)
    {
        const float4 g = s.seg[q][slot];
        const float2 b = s.band[q][slot];
        const float t = fabsf(y - g.z), xs = __fmaf_rn(g.y, y, g.x);
        const float column = (xs + 12582912.f) - 12582912.f;  // the nearest whole number up to 2^22; beyond that the row is not near the segment
        close |= t <= b.y && fabsf(xs - column) <= b.x;
        if (t <= g.w) L = fminf(L, xs), R = fmaxf(R, xs);
    }
    if (s.spots[slot])
        for (int k = 0; k < 8; ++k) close |= s.spot[slot][k].x == j;
    return close;
}

// One row whose bands hold no more than four pixels, by the lane it belongs to, where several rows of a warp's have some: the run L to R of
// pixels, corrected where the per-pixel test disagrees.  False, and nothing done, if there are more pixels.
__device__ __noinline__ bool grid_exact_lane(const GridArgs& a, const GridWarpSmem& s, int slot, int j, float L, float R, double& sum, int& hits)
{
    const int4 rect = s.rect[slot];
    const float y   = (float)j;
    int at[4] = {-1, -1, -1, -1};
#pragma unroll 1
    for (int k = 0; k < kGridSegments + 8; ++k)
    {
        float xs;
        int x0 = 1, x1 = 0;
        if (k < kGridSegments)
        {
            grid_crossing(s, k, slot, y, xs);
            grid_band(s, rect, k, slot, y, xs, x0, x1);
        }
        else
        {
            const int2 spot = s.spot[slot][k - kGridSegments];
            if (spot.x == j && spot.y >= 0 && spot.y < rect.z) x0 = x1 = spot.y;
        }
        if (x1 - x0 > 3) return false;
        for (int x = x0; x <= x1; ++x)
        {
            if (x == at[0] || x == at[1] || x == at[2] || x == at[3]) continue;
            if (at[3] >= 0) return false;
            at[3] = at[2], at[2] = at[1], at[1] = at[0], at[0] = x;
        }
    }
    sum  = 0.0;
    hits = grid_run(a, rect, j, L, R, sum);
#pragma unroll 1
    for (int n = 0; n < 4; ++n)
    {
        const int x = at[0];
        if (x < 0) break;
        at[0] = at[1], at[1] = at[2], at[2] = at[3], at[3] = -1;
        const int change = (int)point_in_box(make_float2((float)(rect.x + x), (float)(rect.y + j)), s.pp[slot]) - (int)((float)x >= L && (float)x <= R);
        if (change != 0) sum += (double)change * (double)grid_pixel_loss(a, rect.x + x, rect.y + j), hits += change;
    }
    return true;
}

// One row of one cell in which pixels lie in the band of a segment (a whole warp): the run of pixels, corrected
// where the per-pixel test disagrees.  Lane k owns segment k.  The pixels of a short band are taken one by one, a triangle per
// lane; those of a long one (a nearly horizontal segment) 32 at a time, a pixel per lane.
__device__ __noinline__ void grid_exact_row(const GridArgs& a, const GridWarpSmem& s, int slot, int j, double& sum, int& hits)
{
    const int lane  = threadIdx.x & 31;
    const float y   = (float)j;
    const int4 rect = s.rect[slot];
    float L = CUDART_INF_F, R = -CUDART_INF_F;
    int x0 = 1, x1 = 0;  // pixels in the band of the lane's segment
    if (lane < kGridSegments)
    {
        float xs;
        const bool crossed = grid_crossing(s, lane, slot, y, xs);
        grid_band(s, rect, lane, slot, y, xs, x0, x1);
        if (crossed) L = R = xs;
    }
    else if (lane < kGridSegments + 8)
    {
        const int2 spot = s.spot[slot][lane - kGridSegments];
        if (spot.x == j && spot.y >= 0 && spot.y < rect.z) x0 = x1 = spot.y;
    }
    for (int o = 16; o > 0; o >>= 1)
    {
        L = fminf(L, __shfl_xor_sync(0xffffffffu, L, o));
        R = fmaxf(R, __shfl_xor_sync(0xffffffffu, R, o));
    }
    if (lane == 0) hits += grid_run(a, rect, j, L, R, sum);
    const unsigned all = __ballot_sync(0xffffffffu, x0 <= x1);
    const int t = min(lane, 11);
    const float2 v0 = s.pp[slot][kGridTriangles[t][0]], v1 = s.pp[slot][kGridTriangles[t][1]], v2 = s.pp[slot][kGridTriangles[t][2]];
    for (unsigned todo = all; todo; todo &= todo - 1)
    {
        const int k    = __ffs(todo) - 1;
        const int from = __shfl_sync(0xffffffffu, x0, k), last = __shfl_sync(0xffffffffu, x1, k);
        if (last - from < 6)
        {
            for (int x = from; x <= last; ++x)
            {
                const unsigned bands = __ballot_sync(0xffffffffu, x >= x0 && x <= x1);
                const bool in_one    = point_in_triangle(make_float2((float)(rect.x + x), (float)(rect.y + j)), v0, v1, v2);
                const bool in        = __any_sync(0xffffffffu, in_one);
                const bool taken     = (bands & ((1u << k) - 1u)) != 0;  // with a segment before this one
                const int change     = taken ? 0 : (int)in - (int)((float)x >= L && (float)x <= R);
                if (change != 0 && lane == 0)
                    sum += (double)change * (double)grid_pixel_loss(a, rect.x + x, rect.y + j), hits += change;
            }
            continue;
        }
        for (int base = from; base <= last; base += 32)
        {
            const int x = base + lane;
            bool taken  = x > last;
            for (unsigned before = all & ((1u << k) - 1u); before; before &= before - 1)
            {
                const int b  = __ffs(before) - 1;
                const int c0 = __shfl_sync(0xffffffffu, x0, b), c1 = __shfl_sync(0xffffffffu, x1, b);
                taken |= x >= c0 && x <= c1;
            }
            if (!taken)
            {
                const bool in    = point_in_box(make_float2((float)(rect.x + x), (float)(rect.y + j)), s.pp[slot]);
                const int change = (int)in - (int)((float)x >= L && (float)x <= R);
                if (change != 0) sum += (double)change * (double)grid_pixel_loss(a, rect.x + x, rect.y + j), hits += change;
            }
            __syncwarp();
        }
    }
}

// What is known of a cell.
struct GridCell
{
    float2 mn;            // first pixel of the rectangle (fp32, not truncated)
    int x_size, y_size;   // of the rectangle
    bool by_rows;         // row form; otherwise per-pixel form
    float rho, zone;      // reach of a segment's band and of a corner's
    __device__ __forceinline__ long long total() const { return (long long)x_size * y_size; }  // pixels; 0: nothing to do
};

// Projects the corners of the lane's cell c (-1: none) and forms its rectangle and bands.
//
// Bands.  With all differences of coordinates below E (the box's extent on the screen, plus one pixel) the strict fp32 edge
// function of an edge of length l is off by less than 8.4 E l 2^-24, i.e. its sign is certain farther than 5e-7 E pixels from
// the edge's line, and a crossing computed here is off by less than 4e-7 E (1 + |dx/dy|) along the row.  A pixel of the run
// that is farther than 5e-7 E from all segments lies inside some triangle with all three signs certain.  A pixel outside
// the run lies in no triangle.  It fails one whose side is nearest for certain if it is farther than 5e-7 E from that side,
// and one whose corner is nearest if it is farther than 5e-7 E / sin(half the smallest angle) <= 1e-6 E kappa from that
// corner, kappa = the largest (product of the two longer sides) / (2 area) of the twelve triangles, 1 / the sine of the smallest
// angle.  So the band of a segment is rho = 1e-6 E wide, which along a row of slope dx/dy = k reaches rho (1 + |k|) to either side,
// and that of a corner (kappa + 0.5) rho (the half more than covers the rounding of kappa, some 1e-6 kappa: corners' bands above
// a quarter pixel are refused) and at least 7 rho: a pixel above or below a segment of |k| <= 4 that is nearest to a point inside it is at
// most sqrt(17) rho away from its end, so that only flatter segments have to be followed beyond their ends.  (All of the edges' bands
// as wide as the corners' want 3 % of the rows tested pixel by pixel, a sixth of the whole call.)
// A row crosses a segment if it is no farther from the segment's middle row than half its rows.  Middle, half and distance are rounded, by less
// than 1.8e-7 E together, so 2.4e-7 E are added to the half: without them a corner on a whole row can lie outside every segment that meets
// there, and the run then ends at an inner one.  A row that is let in without crossing lies within 4.2e-7 E of the segment's end.  With
// |k| <= 4 its extended crossing is off the end by less than 4 of these and the crossing's own 2e-6 E, inside the corner's band (7e-6 E and
// more); with a steeper k by less than 4.2e-7 E |k| and 4e-7 E |k|, inside the 1.25e-6 E |k| by which the segment's band is longer.  So any
// pixel that such a crossing adds to the run is tested.
// All this takes the projected corners as they are, whatever rounding went into them.  Cells whose corners' bands would be wider than a
// quarter pixel, or with a triangle as thin as a few units in the last place of a pixel coordinate, take the per-pixel form.
__device__ __forceinline__ GridCell grid_prepare(const Frame& f, const GridArgs& a, const Camera& cam, GridWarpSmem& s, int c, bool no_rows)
{
    constexpr GridTables kTab;
    const int lane = threadIdx.x & 31;
    GridCell cell;
    cell.x_size = cell.y_size = 0, cell.by_rows = false, cell.mn = make_float2(0.f, 0.f), cell.rho = cell.zone = 0.f;
    if (c < 0) return cell;
    float box[3], len[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) box[k] = a.bb_min[3 * (size_t)c + k], len[k] = a.bb_len[3 * (size_t)c + k];
    bool behind = false;  // one corner behind the camera: the whole cell is ignored
    float2 lo = make_float2(10000000.f, 10000000.f), hi = make_float2(-10000000.f, -10000000.f);
#pragma unroll 1
    for (int k = 0; k < 8; ++k)
    {
        const float2 ip   = grid_project_corner(f, cam, box, len, k, behind);
        s.corner[k][lane] = ip;
        lo.x = fminf(lo.x, ip.x), lo.y = fminf(lo.y, ip.y), hi.x = fmaxf(hi.x, ip.x), hi.y = fmaxf(hi.y, ip.y);
    }
    cell.mn = lo;
    if (behind || grid_rectangle(a, cell.mn, hi, cell.x_size, cell.y_size) <= 0)
    {
        cell.x_size = cell.y_size = 0;
        return cell;
    }
    if (no_rows) return cell;
    float2 p[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) p[k] = s.corner[k][lane];
    const float E = fmaxf(hi.x - lo.x, hi.y - lo.y) + 1.f;
    // squared lengths, and which corners have a higher or a lower neighbour; equal rows are told apart by the corner's number
    float len2[kGridSegments];
    unsigned higher = 0, lower = 0;
#pragma unroll
    for (int k = 0; k < kGridSegments; ++k)
    {
        const int i = kTab.ends[k][0], j = kTab.ends[k][1];  // i < j
        const float dx = p[j].x - p[i].x, dy = p[j].y - p[i].y;
        len2[k]       = __fmaf_rn(dx, dx, dy * dy);
        const bool up = p[j].y >= p[i].y;
        higher |= up ? 1u << i : 1u << j, lower |= up ? 1u << j : 1u << i;
    }
    const bool one_run = __popc(higher) == 7 && __popc(lower) == 7;
    float sine = 1.f, thin = CUDART_INF_F;  // of the smallest angle; smallest altitude of a triangle (0: without area, or a NaN corner)
#pragma unroll
    for (int t = 0; t < 12; ++t)
    {
        const float2 p0 = p[kTab.triangles[t][0]], p1 = p[kTab.triangles[t][1]], p2 = p[kTab.triangles[t][2]];
        const float area2 = fabsf((p1.x - p0.x) * (p2.y - p0.y) - (p1.y - p0.y) * (p2.x - p0.x));
        const float a2 = len2[kTab.sides[t][0]], b2 = len2[kTab.sides[t][1]], c2 = len2[kTab.sides[t][2]];
        const float l2 = fmaxf(a2, fmaxf(b2, c2)), m2 = fmaxf(fminf(a2, b2), fminf(fmaxf(a2, b2), c2));  // longest, second longest
        const float altitude = area2 > 0.f ? area2 * rsqrtf(l2) : 0.f;
        thin = fminf(thin, altitude), sine = fminf(sine, area2 > 0.f ? altitude * rsqrtf(m2) : 0.f);
    }
    const float size = (float)max(a.w, a.h);
    cell.rho = 1e-6f * E, cell.zone = cell.rho * fmaxf(1.f / sine + 0.5f, 7.f);
    const float skip = 1.f - size * 2.4e-7f;  // fp32 column / row numbers count up without a gap below this fraction
    // (a NaN or infinite corner selects the per-pixel form through thin, or through E)
    cell.by_rows = cell.x_size > 0 && cell.y_size > 0 && one_run && E < 2e4f && cell.zone < 0.25f &&
                   thin > 4e-3f * (1.f + (size + E) * (1.f / 2048.f)) && cell.mn.x - floorf(cell.mn.x) < skip && cell.mn.y - floorf(cell.mn.y) < skip;
    return cell;
}

// What lane `from` knows of its cell.
__device__ __forceinline__ GridCell grid_cell_of(const GridCell& cell, int from)
{
    GridCell g;
    g.mn      = make_float2(__shfl_sync(0xffffffffu, cell.mn.x, from), __shfl_sync(0xffffffffu, cell.mn.y, from));
    g.x_size  = __shfl_sync(0xffffffffu, cell.x_size, from), g.y_size = __shfl_sync(0xffffffffu, cell.y_size, from);
    g.by_rows = __shfl_sync(0xffffffffu, (int)cell.by_rows, from) != 0;
    g.rho     = __shfl_sync(0xffffffffu, cell.rho, from), g.zone = __shfl_sync(0xffffffffu, cell.zone, from);
    return g;
}

// Corners, segments and rectangles of a group of four cells, eight lanes each; from: the lane that the slot's cell was prepared by.
__device__ __forceinline__ void grid_segments(GridWarpSmem& s, const GridCell& cell, int from)
{
    const int lane = threadIdx.x & 31, slot = lane >> 3, corner = lane & 7;
    __syncwarp();  // the previous group's have been read, this one's corners written
    s.pp[slot][corner] = s.corner[corner][from];
    __syncwarp();
    if (cell.by_rows)
    {
        const float bx = floorf(cell.mn.x), by = floorf(cell.mn.y);
        for (int k = corner; k < kGridSegments; k += 8)
        {
            float2 p = s.pp[slot][kGridSegEnds[k][0]], q = s.pp[slot][kGridSegEnds[k][1]];
            if (p.y > q.y)
            {
                const float2 t = p;
                p = q, q = t;
            }
            p.x -= bx, p.y -= by, q.x -= bx, q.y -= by;
            const float dx = q.x - p.x, dy = q.y - p.y, rho = cell.rho;
            const bool flat = dy < 1e-3f;  // as good as horizontal: the band covers the whole segment
            const float k_  = flat ? 0.f : dx / dy, middle = 0.5f * dy, steep = fabsf(k_);
            const float rows = middle + 0.24f * rho;  // half the rows, and what the roundings can take from them
            s.seg[k][slot]  = make_float4(flat ? p.x + 0.5f * dx : __fmaf_rn(-k_, p.y, p.x), k_, p.y + middle, rows);
            const bool beyond = flat || steep > 4.f;  // followed beyond its ends: by rho in height, the last term of its reach along the row
            // (which is also for the rounding of the crossing where the reach is cut: 1.2e-7 E |dx/dy|)
            float half = flat ? 0.5f * fabsf(dx) + 4.f * rho : fminf(rho * (1.f + steep), fabsf(dx) + 2.f * rho);
            if (beyond) half += 1.25f * rho * steep;
            s.band[k][slot] = make_float2(half, beyond ? middle + rho : rows);
        }
        const float2 c = s.pp[slot][corner];
        const float x = rintf(c.x), y = rintf(c.y);
        const bool next = fabsf(c.x - x) <= cell.zone && fabsf(c.y - y) <= cell.zone;
        s.spot[slot][corner] = next ? make_int2((int)y - (int)by, (int)x - (int)bx) : make_int2(-1, 0);
        if (corner == 0) s.spots[slot] = 0;
        __syncwarp(0xffu << (8 * slot));
        if (next) s.spots[slot] = 1;
        if (corner == 0)
            s.rect[slot] = make_int4((int)bx, (int)by, cell.x_size, cell.y_size);
    }
    __syncwarp();
}

// Rows [row0, row0 + rows) of the cell of every slot, eight at a time; adds each cell's totals.  Returns true (in all eight lanes) if
// they are not to be had like this - a row with pixels in a band comes out small against the running sums, or against pixels
// taken out of its run - and adds nothing then.
__device__ __forceinline__ bool grid_rows(const GridArgs& a, const GridWarpSmem& s, int row0, int rows, int c)
{
    const int lane = threadIdx.x & 31, slot = lane >> 3, corner = lane & 7;
    const int most = __reduce_max_sync(0xffffffffu, rows);
    double sum  = 0.0;
    int hits    = 0;
    bool refuse = false;
    for (int base = 0; base < most; base += 8)
    {
        const int i = base + corner, j = row0 + i;
        bool close  = false;
        float L = 0.f, R = 0.f;
        if (i < rows)
        {
            close = grid_crossings(s, slot, j, L, R);
            if (!close)
            {
                double run   = 0.0;
                bool cancels = false;
                hits += grid_run(a, s.rect[slot], j, L, R, run, &cancels);
                if (cancels) run = grid_run_pixels(a, s, slot, j, L, R);
                sum += run;
            }
        }
        unsigned todo = __ballot_sync(0xffffffffu, close);
        if (__popc(todo) >= kGridExactLanes)
        {
            double rs = 0.0;
            int rh    = 0;
            if (close && grid_exact_lane(a, s, slot, j, L, R, rs, rh))
            {
                close = false;
                if (rh > 0) refuse |= grid_cancels(rs, grid_prefix(a, s.rect[slot].y + j)[a.w]), sum += rs, hits += rh;
            }
            todo = __ballot_sync(0xffffffffu, close);
        }
        while (todo)
        {
            const int from = __ffs(todo) - 1;
            todo &= todo - 1;
            const int je = __shfl_sync(0xffffffffu, j, from);
            double rs = 0.0;
            int rh    = 0;
            grid_exact_row(a, s, from >> 3, je, rs, rh);
            __syncwarp();
            for (int o = 16; o > 0; o >>= 1) rs += __shfl_xor_sync(0xffffffffu, rs, o);
            rh = __reduce_add_sync(0xffffffffu, rh);
            if (lane == from && rh > 0)
            {
                refuse |= grid_cancels(rs, grid_prefix(a, s.rect[slot].y + je)[a.w]);
                sum += rs, hits += rh;
            }
        }
    }
    refuse = (__ballot_sync(0xffffffffu, refuse) >> (8 * slot) & 0xffu) != 0;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
    {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        hits += __shfl_xor_sync(0xffffffffu, hits, o);
    }
    if (corner == 0 && hits > 0 && !refuse)
    {
        atomicAdd(a.value + c, (float)sum);
        atomicAdd(a.count + c, hits);
    }
    return refuse;
}

// Per-pixel form of the cells of the slots in `which` (bits 0, 8, 16, 24).
__device__ __forceinline__ void grid_pixels(const GridArgs& a, const GridWarpSmem& s, const GridCell& cell, int c, unsigned which, long long first,
                                            long long last)
{
    const int lane = threadIdx.x & 31;
    while (which)
    {
        const int from = __ffs(which) - 1;
        which &= which - 1;
        const int ci         = __shfl_sync(0xffffffffu, c, from), xs = __shfl_sync(0xffffffffu, cell.x_size, from);
        const float mx       = __shfl_sync(0xffffffffu, cell.mn.x, from), my = __shfl_sync(0xffffffffu, cell.mn.y, from);
        const long long b    = __shfl_sync(0xffffffffu, first, from), e = __shfl_sync(0xffffffffu, last, from);
        grid_cell_pixels(a, ci, lane, s.pp[from >> 3], make_float2(mx, my), xs, b, e);
        __syncwarp();
    }
}

// Half-spaces that hold no cell to be drawn: behind the camera, and left, right, above and below what grid_rectangle keeps of the
// image.  The image position of a point with z > 0 is A (x / z, y / z) + b (no distortion), so "left of u" is n . v < 0 with
// n = (A11, A12, b1 - u) for the point v in camera space, and w . p + d < 0 for the point p in the world.  A box lies in it if
// its support w . c + d + |w| . h does (c centre, h half extents).  A cell with a corner behind the camera is not drawn, so the
// other corners' z need not be looked at.  Bounds are moved outwards by two pixels and by what fp32 may be off.
struct GridPlane
{
    float w[3], d, size;  // size: |n| . |t|, what the rounding of d is measured by
};
constexpr int kGridPlanes = 5;
__device__ __forceinline__ GridPlane grid_plane(const GridArgs& a, const Camera& cam, int k)
{
    // K, crop and rotation about the image centre, one after the other
    const float a11 = cam.crop[0] * cam.K[0], a12 = cam.crop[0] * cam.K[4] + cam.crop[4] * cam.K[1];
    const float b1  = cam.crop[0] * cam.K[2] + cam.crop[4] * cam.K[3] + cam.crop[2] - cam.cx;
    const float a22 = cam.crop[1] * cam.K[1], b2 = cam.crop[1] * cam.K[3] + cam.crop[3] - cam.cy;
    const float A[2][2] = {{cam.rot[0] * a11, cam.rot[0] * a12 + cam.rot[1] * a22}, {cam.rot[2] * a11, cam.rot[2] * a12 + cam.rot[3] * a22}};
    const float b[2]    = {cam.rot[0] * b1 + cam.rot[1] * b2 + cam.cx, cam.rot[2] * b1 + cam.rot[3] * b2 + cam.cy};
    float n[3] = {0.f, 0.f, 1.f};
    if (k > 0)
    {
        const int axis     = (k - 1) >> 1;
        const float size   = (float)(axis ? a.h : a.w), border = 32.f, out = 2.f + 1e-5f * (fabsf(b[axis]) + size);
        const bool far     = !(k & 1);
        const float sign   = far ? -1.f : 1.f;
        n[0] = sign * A[axis][0], n[1] = sign * A[axis][1];
        n[2] = far ? size - border + out - b[axis] : b[axis] - border + out;
    }
    GridPlane p;
    for (int j = 0; j < 3; ++j) p.w[j] = n[0] * cam.R[j] + n[1] * cam.R[3 + j] + n[2] * cam.R[6 + j];
    p.d    = n[0] * cam.V.tx + n[1] * cam.V.ty + n[2] * cam.V.tz;
    p.size = fabsf(n[0] * cam.V.tx) + fabsf(n[1] * cam.V.ty) + fabsf(n[2] * cam.V.tz);
    return p;
}

// True if the cell is not drawn (false for anything that is not a number).
__device__ __forceinline__ bool grid_out_of_sight(const GridArgs& a, const GridPlane* planes, int c)
{
    float centre[3], half[3];
    bool number = true;
#pragma unroll
    for (int j = 0; j < 3; ++j)
    {
        const float b = __ldg(a.bb_min + 3 * (size_t)c + j), e = b + __ldg(a.bb_len + 3 * (size_t)c + j);
        centre[j] = 0.5f * b + 0.5f * e, half[j] = fabsf(0.5f * e - 0.5f * b);
        number &= fabsf(e) < 1e30f;
    }
    bool out = false;
#pragma unroll
    for (int k = 0; k < kGridPlanes; ++k)
    {
        const GridPlane p = planes[k];
        float v = p.d, size = p.size;
#pragma unroll
        for (int j = 0; j < 3; ++j)
        {
            const float reach = fabsf(p.w[j]) * half[j], at = p.w[j] * centre[j];
            v += at + reach, size += fabsf(at) + reach;
        }
        out |= v < -1e-5f * size;
    }
    return number && out;
}

// A chunk of the per-pixel form holds 64 << grid_coarse(...) pixels.  Few cells in that form: small ones, because the warps with the last chunks of
// 512 end late (128^3 cells at 1920x1080 without distortion 706 instead of 600 us).  But a chunk costs its cell's segments and additions to the cell's
// two words anew, a third of the time with 64 pixels, and 64 of them fill the queue with 268 million pixels, after which a warp is left alone with
// its cell.  So they are larger
// - where no cell goes by rows, by the size of the image.  Eight distortion coefficients, 64 pixels / 256 / 512: 128^3 cells at 1920x1080 64 / 7.0 / 6.8 ms,
//   64^3 4.1 / 3.4 / 3.3, 16^3 1.01 / 0.88 / 0.80, 96^3 at 1237x823 3.2 / 2.6 / 2.5, 48^3 at 960x540 0.76 / 0.68 / 0.75, 32^3 at 640x480
//   0.32 / 0.30 / 0.36, 16^3 at 320x240 0.08 / 0.11 / 0.18, 128^3 at 160x120 0.38 / 0.47 / 0.45;
// - from kGridCoarseFrom chunks on.  Without distortion, 4e6 units from the origin, 64 pixels / 512 / like this: 128^3 71 / 13.9 / 14.1 ms, 64^3 2.45 /
//   2.1 / 2.43.  Views near a face of the grid, where 30 million pixels are in that form, stay below it: half of that line 1051 -> 1233 us;
// - in vast cells, by the pixels of all of them so far.  Flat boxes, always 64 / like this: four over the whole view 396 / 185 us, 300 of them
//   112 / 6.5 ms, 20 of 700x700 pixels 290 / 200 us, one 90 / 86.  Up to 512 pixels only where there are 33 million, because the few of a
//   grid among cells by rows are the last to end (200 views of 128^3 cells, against always 64: 0.996 of the time on average and 1.02 at most; with
//   512 from four million on 1.17 at most).
__device__ __forceinline__ int grid_coarse(const GridArgs& a, bool no_rows, int queued)
{
    if (queued >= kGridCoarseFrom) return kGridCoarsest;
    const int pixels = a.w * a.h;
    return !no_rows || pixels < 1 << 17 ? 0 : pixels < 1 << 20 ? 2 : kGridCoarsest;
}
__device__ __forceinline__ int grid_coarse_vast(unsigned long long pixels)
{
    return pixels >= 1ull << 25 ? kGridCoarsest : min(64 - __clzll((long long)(pixels >> 20)), 2);
}

// First kernel (kChunks = false): a warp takes `each` groups of four cells at a time, leaves out those that lie out of sight and prepares the others, a
// lane per cell, as soon as it has 32 of them; what is left of these is drawn in groups of four, eight lanes per cell.  Cells with many rows
// (next to the camera a cell covers 10^5 pixels) and large rectangles in the per-pixel form are cut into chunks that go to a queue,
// so that the second kernel (kChunks = true) can spread them over all SMs.  If the queue is full the warp does the whole cell itself.
//
// Bound by instruction issue: at 128^3 cells and 1920x1080 80 us go into looking at and preparing the cells, 160 into the groups' segments and
// what surrounds them, 270 into the rows, 50 to 100 into pixels tested one by one.  The whole call, before and after: 128^3 cells at 1920x1080 946 -> 631 us,
// 117^3 at 373x249 274 -> 222, 112^3 at 160x120 171 -> 127, 47^3 at 369x277 149 -> 87, 58^3 at 308x173 74 -> 70 (before: preparation with eight
// lanes per cell, a band kappa times as wide along all edges, chunks of 32 rows, an even stride, which gave a warp the same part of an axis of a power
// of two of cells again and again).  Handing the groups out by an atomic counter as warps come for them: 890 us without the rows alone.
template <bool kChunks>
__global__ void __launch_bounds__(32 * kGridWarps, kGridCtas) grid_loss_kernel(const __grid_constant__ Frame f, const __grid_constant__ GridArgs a,
                                                                               int2* queue, unsigned long long* queue_count, int each)
{
    __shared__ Camera s_cam;
    __shared__ GridWarpSmem s_warp[kGridWarps];
    __shared__ GridPlane s_planes[kGridPlanes];
    int n = a.n_cells;
    if (kChunks)
    {
        // reservations past the capacity were never written: those cells were done by the first kernel
        n = (int)min(*queue_count, (unsigned long long)kGridQueueCap);
        if (n == 0) return;
        each = min(32 / kGridGroup, max(1, n / ((int)gridDim.x * kGridWarps * kGridGroup)));
    }
    if (threadIdx.x == 0) s_cam = load_camera(f, a.view);
    __syncthreads();
    if (!kChunks)
    {
        if (threadIdx.x < kGridPlanes) s_planes[threadIdx.x] = grid_plane(a, s_cam, threadIdx.x);
        __syncthreads();
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    GridWarpSmem& s    = s_warp[warp];
    const bool no_rows = s_cam.has_dist || *a.no_rows != 0;
    // A warp's groups lie far apart, because cells of much work lie next to one another; the stride is odd (one warp stays idle), because
    // grids tend to have a power of two of cells along an axis, and an even one would give a warp the same part of that axis again and again.
    const long long stride = max(1, (int)gridDim.x * kGridWarps - 1);
    int waiting            = 0;  // in s.todo, whole groups
    if (lane == 0) s.queued = 0;
    for (long long first = blockIdx.x * kGridWarps + warp;; first += each * stride)
    {
        if (blockIdx.x * kGridWarps + warp < stride && first * kGridGroup < n)
        {
            const long long at = (first + lane / kGridGroup * stride) * kGridGroup + lane % kGridGroup;
            int2 q             = make_int2(-1, 0);
            if (lane < each * kGridGroup && at < n) q = kChunks ? queue[at] : make_int2((int)at, 0);
            if (!kChunks && q.x >= 0 && !s_cam.has_dist && grid_out_of_sight(a, s_planes, q.x)) q.x = -1;
            unsigned kept = __ballot_sync(0xffffffffu, q.x >= 0);
            kept |= kept >> 1 & 0x55555555u, kept |= kept >> 2 & 0x11111111u;  // bit 0 of a group: one of its four
            kept = (kept & 0x11111111u) * 15u;
            if (kept >> lane & 1) s.todo[waiting + __popc(kept & ((1u << lane) - 1u))] = q;
            waiting += __popc(kept);
            __syncwarp();
            if (waiting < 32) continue;
        }
        if (waiting == 0) break;
        int2 mine = make_int2(-1, 0);
        if (lane < waiting) mine = s.todo[lane];
        const int2 later = s.todo[lane + 32];
        __syncwarp();
        if (lane + 32 < waiting) s.todo[lane] = later;
        waiting = max(waiting - 32, 0);
        const GridCell prepared = grid_prepare(f, a, s_cam, s, mine.x, no_rows);
        unsigned todo           = __ballot_sync(0xffffffffu, prepared.total() > 0);
        while (todo)
        {
            const int group = (__ffs(todo) - 1) & -kGridGroup, from = group + (lane >> 3);  // the lane that prepared the slot's cell
            todo &= ~(15u << group);
            const GridCell cell = grid_cell_of(prepared, from);
            const int c = __shfl_sync(0xffffffffu, mine.x, from), part = __shfl_sync(0xffffffffu, mine.y, from);
            grid_segments(s, cell, from);
            if constexpr (kChunks)
            {
                const int chunk       = part & ((1 << kGridMarkAt) - 1), row0 = chunk * kGridRowChunk;
                const bool refused    = grid_rows(a, s, row0, cell.by_rows ? min(kGridRowChunk, cell.y_size - row0) : 0, c);
                const unsigned slow   = __ballot_sync(0xffffffffu, (lane & 7) == 0 && cell.total() > 0 && (!cell.by_rows || refused));
                const int size        = cell.by_rows ? kGridRowChunk * cell.x_size : 1 << (kGridChunkBits + (part >> kGridMarkAt));  // pixels of a chunk
                const long long begin = (long long)chunk * size;
                grid_pixels(a, s, cell, c, slow, begin, min(begin + size, cell.total()));
            }
            else
            {
                bool here = cell.total() > 0;  // this warp does the cell itself
                const int parts = cell.by_rows ? cell.y_size : (int)cell.total();
                int coarse      = cell.by_rows ? 0 : grid_coarse(a, no_rows, s.queued);
                const bool vast = (lane & 7) == 0 && !cell.by_rows && parts > kGridVast;
                if (__any_sync(0xffffffffu, vast))
                {
                    const int pixels = __reduce_add_sync(0xffffffffu, vast ? min(parts, 1 << 28) : 0);
                    unsigned long long all = 0;
                    if (lane == 0) all = atomicAdd(queue_count + 2, (unsigned long long)pixels);
                    all = __shfl_sync(0xffffffffu, all, 0) + pixels;
                    if (vast) coarse = max(coarse, grid_coarse_vast(all));
                }
                const int n_chunks = ((parts - 1) >> (cell.by_rows ? kGridRowBits : kGridChunkBits + coarse)) + 1;
                unsigned large     = __ballot_sync(0xffffffffu, (lane & 7) == 0 && n_chunks > 1);
                while (large)
                {
                    const int head = __ffs(large) - 1;
                    large &= large - 1;
                    const int chunks = __shfl_sync(0xffffffffu, n_chunks, head), ci = __shfl_sync(0xffffffffu, c, head);
                    const int mark   = __shfl_sync(0xffffffffu, coarse, head) << kGridMarkAt;
                    // (in 64 bits: the counter adds up what finds no room as well, and 2^31 cells of 2^31 pixels are not 2^63 chunks)
                    unsigned long long at = 0;
                    if (lane == 0) at = atomicAdd(queue_count, (unsigned long long)chunks), s.queued = (int)min(at, (unsigned long long)kGridQueueCap);
                    at = __shfl_sync(0xffffffffu, at, 0);
                    // no room for all chunks: whatever part of the reservation lies inside the queue is marked unused
                    const bool fits = at + chunks <= kGridQueueCap;
                    for (int k = lane; k < chunks && at + k < kGridQueueCap; k += 32) queue[at + k] = fits ? make_int2(ci, k | mark) : make_int2(-1, 0);
                    if (fits && (lane >> 3) == (head >> 3)) here = false;
                }
                const bool refused  = grid_rows(a, s, 0, here && cell.by_rows ? cell.y_size : 0, c);
                const unsigned slow = __ballot_sync(0xffffffffu, (lane & 7) == 0 && here && (!cell.by_rows || refused));
                grid_pixels(a, s, cell, c, slow, 0, cell.total());
            }
        }
    }
}

}  // namespace vetr

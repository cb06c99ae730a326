// Error-grid rasterisation (FillSceneGridWithLossRasterize, rendering/RenderForward.cu:639-791): the step between a training
// epoch and the point spawning.  Every cell of the scene grid whose eight corners lie in front of the camera adds the L1
// loss of the pixels its projected box covers and their number.
//
// The reference tests every pixel of a cell's screen rectangle against the twelve triangles of the box (two per face) and
// issues two global atomics per covered pixel.  Those tests are what bounds a per-pixel form (twelve triangles of three
// edge functions in strict fp32 for each of some 600 M pixels at 128^3 cells and 1920 x 1080: 7.9 ms).  Here a lane owns one
// pixel ROW of a cell: the twelve triangles are a closed surface, so what they cover of a row is the run of pixels between its
// leftmost and rightmost crossing with the 18 segments (12 edges, 6 face diagonals), and the run's loss is a difference
// of two running sums of that image row (fp64, formed once per call).  0.92 ms at the same sizes.
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
constexpr int kGridChunk    = 512;              // pixels of a rectangle one warp walks in the per-pixel form (4096: a warp with
                                                // four such chunks ends 0.3 ms after the others)
constexpr int kGridRowChunk = 32;               // rows of a queued chunk; cells of up to that many rows are not queued
constexpr int kGridQueueCap = 4 * 1024 * 1024;  // (cell, chunk) pairs handed to the second kernel
constexpr int kGridSegments = 18;               // 12 edges, then 6 face diagonals
constexpr unsigned long long kGridNeighbours = 0x72bdcbc76151b17eull;  // byte c: the corners that share a segment with corner c
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

__constant__ signed char kGridSegEnds[kGridSegments][2] = {{0, 1}, {2, 4}, {3, 5}, {6, 7}, {0, 2}, {1, 4}, {3, 6}, {5, 7}, {0, 3},
                                                           {1, 5}, {2, 6}, {4, 7}, {0, 4}, {1, 7}, {5, 6}, {0, 6}, {0, 5}, {4, 6}};
__constant__ signed char kGridTriangles[12][3] = {{0, 1, 4}, {0, 4, 2}, {1, 5, 7}, {1, 7, 4}, {5, 3, 6}, {5, 6, 7},
                                                  {3, 0, 6}, {0, 6, 2}, {3, 0, 5}, {0, 5, 1}, {2, 4, 6}, {4, 6, 7}};

struct GridWarpSmem
{
    float2 pp[kGridGroup][8];               // projected corners
    float4 seg[kGridSegments][kGridGroup];  // {x at y0, y0, y1, dx/dy}, relative to the rectangle's first pixel
    float half[kGridSegments][kGridGroup];  // half-width of the band around the segment, along the row
    int4 rect[kGridGroup];                  // first column, first row, columns, rows
    float rho[kGridGroup];                  // height of the band beyond the segment's ends
};

// Corner order of the reference: (0,0,0) (1,0,0) (0,1,0) (0,0,1) (1,1,0) (1,0,1) (0,1,1) (1,1,1).
__device__ __forceinline__ float2 grid_project_corner(const Frame& f, const GridArgs& a, const Camera& cam, int c, int corner, bool& behind)
{
    const float fx = (corner == 1 || corner == 4 || corner == 5 || corner == 7) ? 1.f : 0.f;
    const float fy = (corner == 2 || corner == 4 || corner == 6 || corner == 7) ? 1.f : 0.f;
    const float fz = (corner == 3 || corner == 5 || corner == 6 || corner == 7) ? 1.f : 0.f;
    const float4 pos = make_float4(VA(a.bb_min[3 * c], VM(a.bb_len[3 * c], fx)), VA(a.bb_min[3 * c + 1], VM(a.bb_len[3 * c + 1], fy)),
                                   VA(a.bb_min[3 * c + 2], VM(a.bb_len[3 * c + 2], fz)), 0.f);
    const Projected pr = project_point(pos, cam, f.dist_cutoff);
    behind = pr.z <= 0.f;  // one corner behind the camera: the whole cell is ignored
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
    for (long long xy = first + lane; xy < last; xy += 32)
    {
        const int x_c = (int)VA((float)(int)(xy % x_size), mn.x);
        const int y_c = (int)VA((float)(int)(xy / x_size), mn.y);
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
        const float4 q = s.seg[lane][slot];
        const float yc = fminf(fmaxf(y, q.y), q.z);
        const float xs = fmaf(yc - q.y, q.w, q.x), h = s.half[lane][slot];
        if (fabsf(y - yc) <= s.rho[slot]) x0 = (int)fmaxf(ceilf(xs - h), 0.f), x1 = (int)fminf(floorf(xs + h), (float)(rect.z - 1));
        if (y == yc) L = R = xs;
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

// What eight lanes know of their cell.
struct GridCell
{
    float2 mn;  // first pixel of the rectangle (fp32, not truncated)
    int x_size, y_size;
    long long total;  // pixels of the rectangle; 0: nothing to do
    bool by_rows;     // row form; otherwise per-pixel form
};

// Projects the corners of the cells of a warp (cell c of the lane's slot, or -1), forms rectangles and segments.
//
// Bands.  With all differences of coordinates below E (the box's extent on the screen, plus one pixel) the strict fp32 edge
// function of an edge of length l is off by less than 8.4 E l 2^-24, i.e. its sign is certain farther than 5e-7 E pixels from
// the edge's line, and a crossing computed here is off by less than 4e-7 E (1 + |dx/dy|) along the row.  A pixel of the run
// that is farther than 5e-7 E from all segments lies inside some triangle with all three signs certain.  A pixel outside
// the run lies in no triangle.  It fails one whose side is nearest for certain if it is farther than 5e-7 E from that side,
// and one whose corner is nearest if it is farther than 5e-7 E / sin(half the smallest angle) <= 1e-6 E kappa from that
// corner, kappa = the largest (product of the two longer sides) / (2 area) of the twelve triangles.  So the
// band of a diagonal is rho = 1e-6 E wide, that of an edge (kappa + 0.5) rho, which also covers all corners, and along a row
// of slope dx/dy = k a band of height rho reaches rho (1 + |k|) to either side.
// All this takes the projected corners as they are, whatever rounding went into them.  Cells whose band would be wider than a
// quarter pixel, or with a triangle as thin as a few units in the last place of a pixel coordinate, take the per-pixel form.
__device__ __forceinline__ GridCell grid_prepare(const Frame& f, const GridArgs& a, const Camera& cam, GridWarpSmem& s, int c, bool no_rows)
{
    const int lane = threadIdx.x & 31, slot = lane >> 3, corner = lane & 7;
    GridCell cell;
    cell.x_size = cell.y_size = 0, cell.total = 0, cell.by_rows = false, cell.mn = make_float2(0.f, 0.f);
    bool behind = true;
    float2 ip   = make_float2(0.f, 0.f);
    if (c >= 0) ip = grid_project_corner(f, a, cam, c, corner, behind);
    const unsigned behind_lanes = __ballot_sync(0xffffffffu, behind);
    const bool visible          = (behind_lanes >> (8 * slot) & 0xffu) == 0;
    if (!__any_sync(0xffffffffu, visible)) return cell;
    float2 lo = make_float2(fminf(ip.x, 10000000.f), fminf(ip.y, 10000000.f));
    float2 hi = make_float2(fmaxf(ip.x, -10000000.f), fmaxf(ip.y, -10000000.f));
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
    {
        lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, o)), lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, o));
        hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, o)), hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, o));
    }
    cell.mn = lo;
    if (visible) cell.total = grid_rectangle(a, cell.mn, hi, cell.x_size, cell.y_size);
    if (!__any_sync(0xffffffffu, cell.total > 0)) return cell;
    __syncwarp();  // the previous cells' segments have been read
    s.pp[slot][corner] = ip;
    __syncwarp();
    if (no_rows) return cell;
    const float2 mn = cell.mn;
    const float E   = fmaxf(hi.x - lo.x, hi.y - lo.y) + 1.f;
    float kappa = 0.f, thin = CUDART_INF_F;  // thin: smallest altitude of a triangle, 0 if one has no area or a corner is NaN
    for (int t = corner; t < 12; t += 8)
    {
        const float2 p0 = s.pp[slot][kGridTriangles[t][0]], p1 = s.pp[slot][kGridTriangles[t][1]], p2 = s.pp[slot][kGridTriangles[t][2]];
        const float ux = p1.x - p0.x, uy = p1.y - p0.y, vx = p2.x - p0.x, vy = p2.y - p0.y, wx = vx - ux, wy = vy - uy;
        const float area2 = fabsf(ux * vy - uy * vx);
        const float a2 = ux * ux + uy * uy, b2 = vx * vx + vy * vy, c2 = wx * wx + wy * wy;
        const float l2 = fmaxf(a2, fmaxf(b2, c2)), m2 = fmaxf(fminf(a2, b2), fminf(fmaxf(a2, b2), c2));  // longest, second longest
        kappa = fmaxf(kappa, sqrtf(l2 * m2) / area2), thin = fminf(thin, area2 > 0.f ? area2 * rsqrtf(l2) : 0.f);
    }
    __syncwarp();
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
    {
        kappa = fmaxf(kappa, __shfl_xor_sync(0xffffffffu, kappa, o));
        thin  = fminf(thin, __shfl_xor_sync(0xffffffffu, thin, o));
    }
    // corners without a higher (lower) neighbour; equal rows are told apart by the corner's number
    unsigned higher = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k)
    {
        const float y = s.pp[slot][k].y;
        if (y > ip.y || (y == ip.y && k > corner)) higher |= 1u << k;
    }
    const unsigned near = (unsigned)(kGridNeighbours >> (8 * corner)) & 0xffu;
    const unsigned tops = __ballot_sync(0xffffffffu, (higher & near) == 0), bottoms = __ballot_sync(0xffffffffu, (~higher & near) == 0);
    const bool one_run  = __popc(tops >> (8 * slot) & 0xffu) == 1 && __popc(bottoms >> (8 * slot) & 0xffu) == 1;
    const float size = (float)max(a.w, a.h);
    const float rho = 1e-6f * E, rho_edge = rho * (kappa + 0.5f);
    const float skip = 1.f - size * 2.4e-7f;  // fp32 column / row numbers count up without a gap below this fraction
    // (a NaN or infinite corner selects the per-pixel form through thin, or through E)
    cell.by_rows = cell.total > 0 && cell.x_size > 0 && cell.y_size > 0 && one_run && E < 2e4f && rho_edge < 0.25f &&
                   thin > 4e-3f * (1.f + (size + E) * (1.f / 2048.f)) && mn.x - floorf(mn.x) < skip && mn.y - floorf(mn.y) < skip;
    if (cell.by_rows)
    {
        const float bx = floorf(mn.x), by = floorf(mn.y);
        for (int k = corner; k < kGridSegments; k += 8)
        {
            float2 p = s.pp[slot][kGridSegEnds[k][0]], q = s.pp[slot][kGridSegEnds[k][1]];
            if (p.y > q.y)
            {
                const float2 t = p;
                p = q, q = t;
            }
            p.x -= bx, p.y -= by, q.x -= bx, q.y -= by;
            const float dx = q.x - p.x, dy = q.y - p.y, r = k < 12 ? rho_edge : rho;
            const bool flat = dy < 1e-3f;  // as good as horizontal: the band covers the whole segment
            const float k_  = flat ? 0.f : dx / dy;
            s.seg[k][slot]  = make_float4(flat ? p.x + 0.5f * dx : p.x, p.y, q.y, k_);
            s.half[k][slot] = flat ? 0.5f * fabsf(dx) + 4.f * r : fminf(r * (1.f + fabsf(k_)), fabsf(dx) + 2.f * r);
        }
    }
    if (corner == 0)
    {
        s.rect[slot] = make_int4((int)floorf(mn.x), (int)floorf(mn.y), cell.x_size, cell.y_size);
        s.rho[slot]  = rho_edge;
    }
    __syncwarp();
    return cell;
}

// Leftmost and rightmost crossing of row j with the segments of a cell; true if a pixel lies in the band of one.
__device__ __forceinline__ bool grid_crossings(const GridWarpSmem& s, int slot, int j, float& L, float& R)
{
    const float y = (float)j, rho = s.rho[slot];
    bool close = false;
    L = CUDART_INF_F, R = -CUDART_INF_F;
#pragma unroll 6
    for (int q = 0; q < kGridSegments; ++q)
    {
        const float4 g = s.seg[q][slot];
        const float yc = fminf(fmaxf(y, g.y), g.z), dy = fabsf(y - yc);
        const float xs = fmaf(yc - g.y, g.w, g.x);
        close |= dy <= rho && fabsf(xs - rintf(xs)) <= s.half[q][slot];
        if (dy == 0.f) L = fminf(L, xs), R = fmaxf(R, xs);
    }
    return close;
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
        if (i < rows)
        {
            float L, R;
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

// True if no cell of the group is drawn (false for anything that is not a number).
__device__ __forceinline__ bool grid_out_of_sight(const GridArgs& a, const GridPlane* planes, int group)
{
    float lo[3] = {CUDART_INF_F, CUDART_INF_F, CUDART_INF_F}, hi[3] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
    bool number     = true;
    const auto take = [&](int j, float b, float e)
    {
        lo[j] = fminf(lo[j], fminf(b, e)), hi[j] = fmaxf(hi[j], fmaxf(b, e));
        number &= fabsf(e) < 1e30f;
    };
    const int c0 = group * kGridGroup;
    if (c0 + kGridGroup <= a.n_cells && (((uintptr_t)a.bb_min | (uintptr_t)a.bb_len) & 15) == 0)
    {
        // the group's four boxes are three 16-byte words of either array (the lanes' groups lie far apart: a load per number would
        // be 32 accesses each)
        const float4* m = reinterpret_cast<const float4*>(a.bb_min) + 3 * (size_t)group;
        const float4* s = reinterpret_cast<const float4*>(a.bb_len) + 3 * (size_t)group;
        const float4 m0 = __ldg(m), m1 = __ldg(m + 1), m2 = __ldg(m + 2), s0 = __ldg(s), s1 = __ldg(s + 1), s2 = __ldg(s + 2);
        take(0, m0.x, m0.x + s0.x), take(1, m0.y, m0.y + s0.y), take(2, m0.z, m0.z + s0.z), take(0, m0.w, m0.w + s0.w);
        take(1, m1.x, m1.x + s1.x), take(2, m1.y, m1.y + s1.y), take(0, m1.z, m1.z + s1.z), take(1, m1.w, m1.w + s1.w);
        take(2, m2.x, m2.x + s2.x), take(0, m2.y, m2.y + s2.y), take(1, m2.z, m2.z + s2.z), take(2, m2.w, m2.w + s2.w);
    }
    else
        for (int c = c0; c < min(c0 + kGridGroup, a.n_cells); ++c)
#pragma unroll
            for (int j = 0; j < 3; ++j) take(j, a.bb_min[3 * c + j], a.bb_min[3 * c + j] + a.bb_len[3 * c + j]);
    bool out = false;
#pragma unroll
    for (int k = 0; k < kGridPlanes; ++k)
    {
        const GridPlane p = planes[k];
        float v = p.d, size = p.size;
#pragma unroll
        for (int j = 0; j < 3; ++j)
        {
            const float centre = 0.5f * lo[j] + 0.5f * hi[j], half = 0.5f * hi[j] - 0.5f * lo[j], reach = fabsf(p.w[j]) * half;
            v += p.w[j] * centre + reach, size += fabsf(p.w[j] * centre) + reach;
        }
        out |= v < -1e-5f * size;
    }
    return number && out;
}

// First kernel: one warp per group of four cells.  kCull: a warp's next 32 groups are looked at first, a lane each; groups that lie
// altogether out of sight are left out before their corners are projected, which costs about 200 instructions per group.
// Cells with many rows (next to the camera a cell covers 10^5 pixels) and large rectangles in the per-pixel form are cut into
// chunks that go to a queue, so that the second kernel can spread them over all SMs.  If the queue is full the warp does the
// whole cell itself.
//
// Looking ahead wants groups to look at: with few per warp it saves less than the half-spaces and the second reading of the boxes cost,
// unless the image is so small that there is little but the projection.  The whole call without and with it, camera on an orbit inside
// the grid: 1920x1080 64^3 cells (9 groups a warp) 406 to 535 and 397 to 544 us (three cameras), 96^3 556 to 737 and 510 to 705, 128^3 941
// to 1096 and 825 to 1006; 640x480 48^3 (4) 213 to 268 and 211 to 270, 56^3 (6) 167 to 208 and 154 to 205, 96^3 311 to 445 and 278 to
// 412; 160x120 48^3 60 to 84 and 57 to 79, 40^3 (2) no difference.  All cells in sight: 64^3 186 and 189, 128^3 903 and 901, 48^3 at
// 640x480 71 and 73.  (With a load per number instead of 16 bytes at a time all of that was 5 % slower than without looking.)
constexpr int kGridCullGroups = 6, kGridCullGroupsSmall = 3, kGridCullCells = 4;  // groups per warp; in images of no more than a
                                                                                  // pixel per kGridCullCells cells
template <bool kCull>
__global__ void __launch_bounds__(32 * kGridWarps, kGridCtas) grid_loss_kernel(const __grid_constant__ Frame f, const __grid_constant__ GridArgs a,
                                                                     int2* queue, int* queue_count)
{
    __shared__ Camera s_cam;
    __shared__ GridWarpSmem s_warp[kGridWarps];
    if (threadIdx.x == 0) s_cam = load_camera(f, a.view);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    GridWarpSmem& s    = s_warp[warp];
    const bool no_rows = s_cam.has_dist || *a.no_rows != 0;
    const int n_groups = (a.n_cells + kGridGroup - 1) / kGridGroup, stride = gridDim.x * kGridWarps;
    __shared__ GridPlane s_planes[kCull ? kGridPlanes : 1];
    if (kCull)
    {
        if (threadIdx.x < kGridPlanes) s_planes[threadIdx.x] = grid_plane(a, s_cam, threadIdx.x);
        __syncthreads();
    }
    unsigned todo = 0;  // groups first + k stride still to do (bit k)
    int first = blockIdx.x * kGridWarps + warp - 32 * stride;
    for (;;)
    {
        if (todo == 0)
        {
            first += 32 * stride;
            if (first >= n_groups) break;
            const int mine = first + lane * stride;
            todo = __ballot_sync(0xffffffffu, mine < n_groups && (!kCull || s_cam.has_dist || !grid_out_of_sight(a, s_planes, mine)));
            continue;
        }
        const int group = first + (__ffs(todo) - 1) * stride;
        todo &= todo - 1;
        const int c         = group * kGridGroup + (lane >> 3);
        const GridCell cell = grid_prepare(f, a, s_cam, s, c < a.n_cells ? c : -1, no_rows);
        if (!__any_sync(0xffffffffu, cell.total > 0)) continue;
        bool here = cell.total > 0;  // this warp does the cell itself
        const long long units = cell.by_rows ? cell.y_size : cell.total;
        const int unit        = cell.by_rows ? kGridRowChunk : kGridChunk;
        const int n_chunks    = (int)((units + unit - 1) / unit);
        unsigned large        = __ballot_sync(0xffffffffu, (lane & 7) == 0 && units > unit);
        while (large)
        {
            const int from = __ffs(large) - 1;
            large &= large - 1;
            const int chunks = __shfl_sync(0xffffffffu, n_chunks, from);
            int at = 0;
            if (lane == 0) at = atomicAdd(queue_count, chunks);
            at = __shfl_sync(0xffffffffu, at, 0);
            // no room for all chunks: whatever part of the reservation lies inside the queue is marked unused
            const bool fits = at + chunks <= kGridQueueCap;
            const int ci    = group * kGridGroup + (from >> 3);
            for (int k = lane; k < chunks && at + k < kGridQueueCap; k += 32) queue[at + k] = fits ? make_int2(ci, k) : make_int2(-1, 0);
            if (fits && (lane >> 3) == (from >> 3)) here = false;
        }
        const bool refused  = grid_rows(a, s, 0, here && cell.by_rows ? cell.y_size : 0, c);
        const unsigned slow = __ballot_sync(0xffffffffu, (lane & 7) == 0 && here && (!cell.by_rows || refused));
        grid_pixels(a, s, cell, c, slow, 0, cell.total);
    }
}

// Second kernel: one warp per four queued (cell, chunk of rows or pixels).
__global__ void __launch_bounds__(32 * kGridWarps, kGridCtas) grid_loss_chunk_kernel(const __grid_constant__ Frame f, const __grid_constant__ GridArgs a,
                                                                           const int2* queue, const int* queue_count)
{
    __shared__ Camera s_cam;
    __shared__ GridWarpSmem s_warp[kGridWarps];
    if (threadIdx.x == 0) s_cam = load_camera(f, a.view);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    GridWarpSmem& s    = s_warp[warp];
    const bool no_rows = s_cam.has_dist || *a.no_rows != 0;
    // reservations past the capacity were never written: those cells were done by the first kernel
    const int n = min(*queue_count, kGridQueueCap);
    for (int e = blockIdx.x * kGridWarps + warp; e * kGridGroup < n; e += gridDim.x * kGridWarps)
    {
        const int mine = e * kGridGroup + (lane >> 3);
        const int2 q   = mine < n ? queue[mine] : make_int2(-1, 0);
        const GridCell cell = grid_prepare(f, a, s_cam, s, q.x, no_rows);
        const int row0      = q.y * kGridRowChunk;
        const bool refused  = grid_rows(a, s, row0, cell.by_rows ? min(kGridRowChunk, cell.y_size - row0) : 0, q.x);
        const unsigned slow = __ballot_sync(0xffffffffu, (lane & 7) == 0 && cell.total > 0 && (!cell.by_rows || refused));
        const int unit      = cell.by_rows ? kGridRowChunk * cell.x_size : kGridChunk;  // pixels of a chunk
        const long long first = (long long)q.y * unit;
        grid_pixels(a, s, cell, q.x, slow, first, min(first + unit, cell.total));
    }
}

}  // namespace vetr

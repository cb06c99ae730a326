// Drop-out radius of a point cloud: SceneData::ComputeRadius (data/SceneData.cpp:554-597), the distance from every point
// to its k-th nearest other point.  The reference builds a KD-tree on the host and queries it per point; here the points
// are binned into a uniform grid by a counting sort (count per cell, exclusive scan, scatter), and every point searches
// the cells around its own in growing cubes until the k-th nearest distance found so far is smaller than the distance to
// the cube's faces, beyond which nothing has been looked at.  Most points end after the first cube of 3 x 3 x 3 cells,
// with one thread per point; the rest (isolated points, whose cubes grow to tens of cells a side) go to a queue and are
// finished by one warp per point, whose lanes split the candidates of a cube that grows from stage to stage.
//
// The result is the (k+1)-th smallest of a multiset of fp32 squared distances, each formed as (dx dx + dy dy) + dz dz
// without contraction, so it does not depend on the order in which candidates are met and is bit-equal to an all-pairs
// evaluation on the host.
#pragma once
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

namespace vetr
{
constexpr int kKnnMaxK       = 16;
constexpr int kKnnScanTile   = 4096;       // cells per thread block of the scan (256 threads x 16)
constexpr int kKnnCellsPad   = 4;          // zeros in front of the per-cell array (the first cell begins at slot 0), a whole 16 bytes
constexpr int kKnnSortedPad    = 3;        // entries behind the sorted points, read with the last of them and not used
constexpr long long kKnnMaxCells = 1ll << 26;  // 64 Mi cells: 16384 scan tiles, one spine block

struct KnnGrid
{
    float ox, oy, oz;  // origin: the cloud's minimum corner
    float cell, inv_cell;
    int nx, ny, nz;
};

// Order-preserving map between floats and unsigned integers, for atomicMin / atomicMax on coordinates.
__device__ __forceinline__ unsigned knn_key(float f)
{
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__host__ __device__ inline float knn_unkey(unsigned k)
{
    const unsigned b = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float f;
    memcpy(&f, &b, 4);
    return f;
#endif
}

// (rows of four floats on a 16-byte boundary in one load: 1 us of a call of 1500 for 4 M points)
__device__ __forceinline__ float3 knn_load(const float* __restrict__ pos, int stride, int i)
{
    const float* p = pos + (size_t)i * stride;
    return make_float3(p[0], p[1], p[2]);
}

// bounds[0..2] = min keys (initialised to 0xffffffff), bounds[3..5] = max keys (initialised to 0; all ones if a coordinate is not finite:
// the keys alone are not enough, nvcc 12.9 turns their maxima into maxima of floats, which pass over a NaN).  One atomic per
// block and value: with one per warp the six addresses took longer than the points.
__global__ void __launch_bounds__(256) knn_bounds_kernel(const float* __restrict__ pos, int stride, int n, unsigned* bounds)
{
    __shared__ unsigned s_part[8][6];
    unsigned lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[3] = {0u, 0u, 0u};
    bool finite          = true;
    const long long step = gridDim.x * 256;
    for (long long i = blockIdx.x * 256 + threadIdx.x; i < n; i += 4 * step)
    {
        float3 p[4];  // requested together; behind the last point the first of them once more
#pragma unroll
        for (int u = 0; u < 4; ++u) p[u] = knn_load(pos, stride, (int)(i + u * step < n ? i + u * step : i));
#pragma unroll
        for (int u = 0; u < 4; ++u)
        {
            const unsigned k[3] = {knn_key(p[u].x), knn_key(p[u].y), knn_key(p[u].z)};
#pragma unroll
            for (int a = 0; a < 3; ++a) lo[a] = min(lo[a], k[a]), hi[a] = max(hi[a], k[a]);
            finite &= fabsf(p[u].x) < CUDART_INF_F && fabsf(p[u].y) < CUDART_INF_F && fabsf(p[u].z) < CUDART_INF_F;
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
        if (!finite) hi[a] = 0xffffffffu;
        lo[a] = __reduce_min_sync(0xffffffffu, lo[a]), hi[a] = __reduce_max_sync(0xffffffffu, hi[a]);
        if (lane == 0) s_part[warp][a] = lo[a], s_part[warp][3 + a] = hi[a];
    }
    __syncthreads();
    if (threadIdx.x < 6)
    {
        unsigned v = s_part[0][threadIdx.x];
        for (int w = 1; w < 8; ++w) v = threadIdx.x < 3 ? min(v, s_part[w][threadIdx.x]) : max(v, s_part[w][threadIdx.x]);
        if (threadIdx.x < 3)
            atomicMin(bounds + threadIdx.x, v);
        else
            atomicMax(bounds + threadIdx.x, v);
    }
}

__device__ __forceinline__ int knn_cell_coord(float p, float origin, float inv_cell, int n)
{
    const float c = floorf((p - origin) * inv_cell);
    return (int)fminf(fmaxf(c, 0.f), (float)(n - 1));  // also sends NaN to cell 0: every access stays inside the grid
}

__device__ __forceinline__ int knn_cell_of(const KnnGrid& g, float x, float y, float z, int& cx, int& cy, int& cz)
{
    cx = knn_cell_coord(x, g.ox, g.inv_cell, g.nx);
    cy = knn_cell_coord(y, g.oy, g.inv_cell, g.ny);
    cz = knn_cell_coord(z, g.oz, g.inv_cell, g.nz);
    return (cz * g.ny + cy) * g.nx + cx;
}

// counts[cell] += 1 for every point; point_cell[i] = its cell.
__global__ void __launch_bounds__(256) knn_count_kernel(const float* __restrict__ pos, int stride, int n, const __grid_constant__ KnnGrid g,
                                                        int* counts, int* point_cell)
{
    for (long long i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256)
    {
        const float3 p = knn_load(pos, stride, (int)i);
        int cx, cy, cz;
        const int c   = knn_cell_of(g, p.x, p.y, p.z, cx, cy, cz);
        point_cell[i] = c;
        atomicAdd(counts + c, 1);
    }
}

// Number of non-empty cells (the cell size is chosen from the points per occupied cell).  counts: 16-byte aligned.
__global__ void __launch_bounds__(256) knn_occupied_kernel(const int* __restrict__ counts, long long n_cells, unsigned long long* occupied)
{
    int mine = 0;
    for (long long i = ((long long)blockIdx.x * 256 + threadIdx.x) * 4; i < n_cells; i += (long long)gridDim.x * 1024)
    {
        const int4 c = scan_load<true>(counts, i, n_cells);
        mine += (c.x > 0) + (c.y > 0) + (c.z > 0) + (c.w > 0);
    }
    mine = __reduce_add_sync(0xffffffffu, mine);
    __shared__ int s_part[8];
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = mine;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        unsigned long long sum = 0;
        for (int w = 0; w < 8; ++w) sum += s_part[w];
        if (sum) atomicAdd(occupied, sum);
    }
}

// Exclusive scan of the cell counts in three kernels: sums of tiles, scan of the tile sums by one block, scan inside the tiles.
template <bool kVec>
__global__ void __launch_bounds__(256) knn_tile_sums_kernel(const int* __restrict__ counts, long long n_cells, int* tile_sums)
{
    const long long base = (long long)blockIdx.x * kKnnScanTile;
    int s = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r)
    {
        const int4 c = scan_load<kVec>(counts, base + r * 1024 + threadIdx.x * 4, n_cells);
        s += c.x + c.y + c.z + c.w;
    }
    __shared__ int part[8];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        int t = 0;
        for (int w = 0; w < 8; ++w) t += part[w];
        tile_sums[blockIdx.x] = t;
    }
}

__global__ void __launch_bounds__(1024) knn_spine_kernel(int* tile_sums, int n_tiles)
{
    // 1024 threads x 16 consecutive tiles each = 16384 tiles at most
    __shared__ int warp_tot[32];
    const int first = threadIdx.x * 16;
    int local[16], s = 0;
#pragma unroll
    for (int k = 0; k < 16; ++k)
    {
        local[k] = first + k < n_tiles ? tile_sums[first + k] : 0;
        s += local[k];
    }
    int incl = s;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1)
    {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    if (warp == 0)
    {
        int w = warp_tot[lane], wi = w;
        for (int o = 1; o < 32; o <<= 1)
        {
            const int v = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += v;
        }
        warp_tot[lane] = wi - w;  // exclusive
    }
    __syncthreads();
    int run = warp_tot[warp] + incl - s;
#pragma unroll
    for (int k = 0; k < 16; ++k)
        if (first + k < n_tiles)
        {
            tile_sums[first + k] = run;
            run += local[k];
        }
}

// starts[cell] = exclusive scan of counts (in place is allowed: starts may alias counts).  17 M cells: 80 -> 16 us (before: 16 consecutive
// cells per thread).
template <bool kVec>
__global__ void __launch_bounds__(256) knn_apply_kernel(const int* counts, long long n_cells, const int* __restrict__ tile_sums, int* starts)
{
    __shared__ int s_warp[32];
    const long long base = (long long)blockIdx.x * kKnnScanTile;
    int4 c[4];
    int before[4];
    scan_tile<kVec>(counts, base, n_cells, s_warp, c, before);
    const int offset = tile_sums[blockIdx.x];
#pragma unroll
    for (int r = 0; r < 4; ++r)
    {
        const int s0 = offset + before[r], s1 = s0 + c[r].x, s2 = s1 + c[r].y;
        scan_store<kVec>(starts, base + r * 1024 + threadIdx.x * 4, n_cells, make_int4(s0, s1, s2, s2 + c[r].z));
    }
}

// Counting sort, last step: sorted[slot] = (x, y, z, index bits); cursor[cell] starts at the cell's first slot and ends
// at its last + 1, the first slot of the next cell.
__global__ void __launch_bounds__(256) knn_scatter_kernel(const float* __restrict__ pos, int stride, int n, const int* __restrict__ point_cell,
                                                          int* cursor, float4* sorted)
{
    for (long long i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256)
    {
        // (four points of a thread together: 60 us instead of 57 for 3.8 M points, 126 instead of 118 for 7.6 M)
        const int slot = atomicAdd(cursor + point_cell[i], 1);
        const float3 p = knn_load(pos, stride, (int)i);
        sorted[slot]   = make_float4(p.x, p.y, p.z, __int_as_float((int)i));
    }
}

struct KnnSearch
{
    KnnGrid g;
    const float4* sorted;
    const int* first;  // [cells + 1]: first slot of a cell, which ends where the cell behind it begins
    int n;
    int dummies;   // list entries pre-filled with -inf so that the (k+1)-th smallest distance sits in the last entry
    float slack;   // rounding allowance of the cube-face distances
    float* radius;
    int radius_stride;
    int* queue;        // sorted indices of the points the first pass could not finish
    int* queue_count;
};

// best[] ascending; inserts d and drops the largest.
template <int KMAX>
__device__ __forceinline__ void knn_insert(float (&best)[KMAX], float d)
{
    float v = d;
#pragma unroll
    for (int j = 0; j < KMAX; ++j)
    {
        const float lo = fminf(best[j], v);
        v              = fmaxf(best[j], v);
        best[j]        = lo;
    }
}

template <int KMAX>
__device__ __forceinline__ void knn_scan_slots(const KnnSearch& a, int b, int e, float x, float y, float z, float (&best)[KMAX])
{
    // Four candidates at a time: their loads are in flight together, and one comparison passes over most groups.  (Candidates closer than
    // the k-th put by in shared memory and inserted together, because lanes rarely meet one at the same time: 575 -> 744 us.)
    for (int j = b; j < e; j += 4)
    {
        float d[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            const float4 q = __ldg(a.sorted + j + k);  // there are kKnnSortedPad entries behind the last
            const float dx = x - q.x, dy = y - q.y, dz = z - q.z;
            d[k]           = j + k < e ? dx * dx + dy * dy + dz * dz : CUDART_INF_F;
        }
        if (fminf(fminf(d[0], d[1]), fminf(d[2], d[3])) < best[KMAX - 1])
        {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (d[k] < best[KMAX - 1]) knn_insert<KMAX>(best, d[k]);
        }
    }
}

// Distance from p to the nearest face of the cube of cells [c - r, c + r]^3 behind which unvisited cells remain
// (+inf if the cube covers the grid), minus the rounding allowance.
__device__ __forceinline__ float knn_margin(const KnnSearch& a, float x, float y, float z, int cx, int cy, int cz, int r)
{
    float m = CUDART_INF_F;
    const KnnGrid& g = a.g;
    if (cx - r > 0) m = fminf(m, x - (g.ox + (float)(cx - r) * g.cell));
    if (cx + r < g.nx - 1) m = fminf(m, (g.ox + (float)(cx + r + 1) * g.cell) - x);
    if (cy - r > 0) m = fminf(m, y - (g.oy + (float)(cy - r) * g.cell));
    if (cy + r < g.ny - 1) m = fminf(m, (g.oy + (float)(cy + r + 1) * g.cell) - y);
    if (cz - r > 0) m = fminf(m, z - (g.oz + (float)(cz - r) * g.cell));
    if (cz + r < g.nz - 1) m = fminf(m, (g.oz + (float)(cz + r + 1) * g.cell) - z);
    return m - a.slack;
}

__device__ __forceinline__ bool knn_done(float kth_d2, float margin) { return margin > 0.f && kth_d2 <= margin * margin; }

// Square of a distance to a cell's face, rounding allowance taken off.
__device__ __forceinline__ float knn_gap2(const KnnSearch& a, float d)
{
    d = fmaxf(d - a.slack, 0.f);
    return d * d;
}

// First pass: one thread per point (in cell order, so that a warp's points share their cells), the cube of 3^3 cells.  The
// point's own cell comes first: in a dense cell it holds neighbours closer than the cell's faces, and the other cells, nearest
// first, are passed over where they lie beyond the k-th distance found so far (a later candidate would have to be smaller, so
// the result is the same).  Bound by instruction issue, 82 % of the slots with ten of 32 lanes.  4 M points of a planar scene with
// 5 % outliers, k = 4: 969 us with all 27 cells, row by row from one corner, 769 with all lanes going through the rows that any of them
// needs, 575 like this.
template <int KMAX>
__global__ void __launch_bounds__(128) knn_near_kernel(const __grid_constant__ KnnSearch a)
{
    const int i = blockIdx.x * 128 + threadIdx.x;
    if (i >= a.n) return;
    const float4 p   = a.sorted[i];
    const KnnGrid& g = a.g;
    int cx, cy, cz;
    const int own = knn_cell_of(g, p.x, p.y, p.z, cx, cy, cz);
    float best[KMAX];
#pragma unroll
    for (int j = 0; j < KMAX; ++j) best[j] = j < a.dummies ? -CUDART_INF_F : CUDART_INF_F;
    const float xlo = knn_gap2(a, p.x - (g.ox + (float)cx * g.cell)), xhi = knn_gap2(a, (g.ox + (float)(cx + 1) * g.cell) - p.x);
    const float ylo = knn_gap2(a, p.y - (g.oy + (float)cy * g.cell)), yhi = knn_gap2(a, (g.oy + (float)(cy + 1) * g.cell) - p.y);
    const float zlo = knn_gap2(a, p.z - (g.oz + (float)cz * g.cell)), zhi = knn_gap2(a, (g.oz + (float)(cz + 1) * g.cell) - p.z);
    knn_scan_slots<KMAX>(a, a.first[own], a.first[own + 1], p.x, p.y, p.z, best);
    // Steps 0, 1: the neighbours along x; 2..9: the other rows of three cells, those that share a face with the own row first.  Each lane
    // goes through the steps that it needs and not through all of the warp's: with the own cell done these are two or three of ten.
    const bool y0 = cy > 0, y1 = cy < g.ny - 1, z0 = cz > 0, z1 = cz < g.nz - 1;
    const float k0 = best[KMAX - 1];
    unsigned rest  = 0;
    if (cx > 0 && xlo < k0) rest |= 1u << 0;
    if (cx < g.nx - 1 && xhi < k0) rest |= 1u << 1;
    if (y0 && ylo < k0) rest |= 1u << 2;
    if (y1 && yhi < k0) rest |= 1u << 3;
    if (z0 && zlo < k0) rest |= 1u << 4;
    if (z1 && zhi < k0) rest |= 1u << 5;
    if (y0 && z0 && ylo + zlo < k0) rest |= 1u << 6;
    if (y1 && z0 && yhi + zlo < k0) rest |= 1u << 7;
    if (y0 && z1 && ylo + zhi < k0) rest |= 1u << 8;
    if (y1 && z1 && yhi + zhi < k0) rest |= 1u << 9;
#pragma unroll 1
    while (rest)
    {
        const int t = __ffs(rest) - 1;
        rest &= rest - 1;
        const int dy = (int)(0x88585u >> (2 * t) & 3) - 1, dz = (int)(0xa0855u >> (2 * t) & 3) - 1;  // two bits a step
        const float gap = (dy < 0 ? ylo : dy > 0 ? yhi : 0.f) + (dz < 0 ? zlo : dz > 0 ? zhi : 0.f);
        const float kth = best[KMAX - 1];
        if (!(gap < kth)) continue;
        const bool left = cx > 0 && gap + xlo < kth, right = cx < g.nx - 1 && gap + xhi < kth;
        int c0 = cx - left, c1 = cx + right;  // the row's cells are consecutive slots
        if (t == 0)
        {
            if (!left) continue;
            c1 = c0;
        }
        else if (t == 1)
        {
            if (!right) continue;
            c0 = c1;
        }
        const int row = ((cz + dz) * g.ny + cy + dy) * g.nx;
        knn_scan_slots<KMAX>(a, a.first[row + c0], a.first[row + c1 + 1], p.x, p.y, p.z, best);
    }
    if (knn_done(best[KMAX - 1], knn_margin(a, p.x, p.y, p.z, cx, cy, cz, 1)))
        a.radius[(size_t)__float_as_int(p.w) * a.radius_stride] = sqrtf(best[KMAX - 1]);
    else
        a.queue[atomicAdd(a.queue_count, 1)] = i;
}

// Second pass: one warp per queued point.  The cube [c - R, c + R]^3 grows from stage to stage.  The rows (y, z) of the cube that
// lie inside the grid are dealt to the lanes; the cells of a row are consecutive in the sorted array, so a row is one range of
// slots, or two (left and right of the cube already visited), and rows or their ends that lie beyond the k-th distance known so
// far are left out.  The ranges of 32 rows are then laid end to end and every lane takes every 32nd candidate of them.
// After each stage the stopping rule is applied to the cube's faces.
//
// From stage to stage: 2, 4, 8, ... until there are k candidates, then the cube that holds the k-th of them.  4 M points of a planar
// scene with 5 % outliers, k = 4: 553 us with the stages 2, 4, 6, 9, 13, ..., row coordinates by division and a k-th distance formed by shuffles
// for every 32 rows, 470 like this; a first stage of 3 instead of 2 is 12 us faster there and slower with 30 to 200 k points (the whole call by 3 %).
//
// Where the cube of an isolated point meets a dense surface, a few rows hold hundreds of candidates: with a lane scanning
// the whole of its row the others waited for it.  4 M points of a planar scene with 5 % outliers, k = 4: 1054 -> 557 us.
//
// Points next to each other in the queue lie next to each other and cost alike, from a few rows to thousands, so the blocks are many more than
// fit at once and the SMs take them as they come free: 8 / 32 / 64 / 128 / 256 blocks per SM 474 / 442 / 425 / 426 / 433 us there (8 M points 769 /
// 727 / 687 / 668 / 681; 30 k points 16 us, 21 with 256).  Ten blocks per SM at a time (48 registers, 12 bytes spilled) instead of nine: 408 (658);
// twelve lose: 506.  For more than four neighbours the compiler's own choice is faster (200 k points, k = 8: 91 us).
constexpr int kKnnFarCtas = 64;
template <int KMAX>
__global__ void __launch_bounds__(128, KMAX <= 5 ? 10 : 0) knn_far_kernel(const __grid_constant__ KnnSearch a)
{
    constexpr unsigned kAll = 0xffffffffu;
    const int lane   = threadIdx.x & 31;
    const int n_q    = *a.queue_count;
    const KnnGrid& g = a.g;
    for (int w = blockIdx.x * 4 + (threadIdx.x >> 5); w < n_q; w += gridDim.x * 4)
    {
        const float4 p = a.sorted[a.queue[w]];
        int cx, cy, cz;
        knn_cell_of(g, p.x, p.y, p.z, cx, cy, cz);
        float best[KMAX];
#pragma unroll
        for (int j = 0; j < KMAX; ++j) best[j] = (lane == 0 && j < a.dummies) ? -CUDART_INF_F : CUDART_INF_F;
        float kth       = CUDART_INF_F;  // k-th smallest of all lanes' candidates so far
        const int r_max = max(max(max(cx, g.nx - 1 - cx), max(cy, g.ny - 1 - cy)), max(cz, g.nz - 1 - cz));
        bool closer = false;  // the lane has a new candidate since kth was formed
        int r_prev  = -1;     // half-width of the cube already visited (-1: nothing yet)
        for (int r = min(2, max(r_max, 1));;)
        {
            const int ylo = max(cy - r, 0), yhi = min(cy + r, g.ny - 1), zlo = max(cz - r, 0), zhi = min(cz + r, g.nz - 1);
            const int wz = zhi - zlo + 1, rows = (yhi - ylo + 1) * wz;  // <= ny nz <= 2^26
            const int dy = 32 / wz, dz = 32 % wz;                       // from one of the lane's rows to its next
            int y = ylo + lane / wz, z = zlo + lane % wz;
            for (int base = 0; base < rows; base += 32, y += dy, z += dz)
            {
                if (z > zhi) z -= wz, ++y;
                int b0 = 0, n0 = 0, b1 = 0, n1 = 0;  // the lane's row: its one or two ranges of slots
                if (base + lane < rows)
                {
                    float gap = 0.f;
                    if (y != cy) gap += knn_gap2(a, y < cy ? p.y - (g.oy + (float)(y + 1) * g.cell) : (g.oy + (float)y * g.cell) - p.y);
                    if (z != cz) gap += knn_gap2(a, z < cz ? p.z - (g.oz + (float)(z + 1) * g.cell) : (g.oz + (float)z * g.cell) - p.z);
                    if (gap < kth)
                    {
                        const float reach = sqrtf(kth - gap) + a.slack;  // cells follow the coordinate: none beyond it can count
                        const int x0 = max(cx - r, knn_cell_coord(p.x - reach, g.ox, g.inv_cell, g.nx));
                        const int x1 = min(cx + r, knn_cell_coord(p.x + reach, g.ox, g.inv_cell, g.nx));
                        const int* row   = a.first + (z * g.ny + y) * g.nx;
                        const bool inner = abs(y - cy) <= r_prev && abs(z - cz) <= r_prev;
                        // the cells next to the visited piece
                        const int end = inner ? min(cx - r_prev - 1, x1) : x1, begin = max(cx + r_prev + 1, x0);
                        if (x0 <= end) b0 = row[x0], n0 = row[end + 1] - b0;
                        if (inner && begin <= x1) b1 = row[begin], n1 = row[x1 + 1] - b1;
                    }
                }
                int upto = n0 + n1;  // candidates of this lane's row and the rows before it
                for (int o = 1; o < 32; o <<= 1)
                {
                    const int v = __shfl_up_sync(kAll, upto, o);
                    if (lane >= o) upto += v;
                }
                const int total = __shfl_sync(kAll, upto, 31);
                if (total == 0) continue;
                const int before = upto - n0 - n1;
                for (int first = 0; first < total; first += 32)
                {
                    const int c = first + lane;
                    int owner   = 0;  // first lane whose rows reach beyond candidate c (31 behind the last)
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1)
                        if (__shfl_sync(kAll, upto, owner + o - 1) <= c) owner += o;
                    const int at = c - __shfl_sync(kAll, before, owner), n_left = __shfl_sync(kAll, n0, owner);
                    const int left = __shfl_sync(kAll, b0, owner), right = __shfl_sync(kAll, b1, owner);
                    if (c < total)
                    {
                        const float4 q = __ldg(a.sorted + (at < n_left ? left + at : right + at - n_left));
                        const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
                        const float d  = dx * dx + dy * dy + dz * dz;
                        if (d < best[KMAX - 1] && d < kth) knn_insert<KMAX>(best, d), closer = true;
                    }
                }
                // the k-th smallest of all lanes: k times, take the smallest head off its list (of a copy).  Squares of distances order
                // like their bits, and the one -inf of a lane's head comes before them.
                if (!__any_sync(kAll, closer)) continue;
                closer = false;
                float rest[KMAX];
#pragma unroll
                for (int j = 0; j < KMAX; ++j) rest[j] = best[j];
#pragma unroll 1
                for (int j = 0; j < KMAX; ++j)
                {
                    const int head         = __reduce_min_sync(kAll, __float_as_int(rest[0]));
                    const unsigned holders = __ballot_sync(kAll, __float_as_int(rest[0]) == head);
                    kth                    = __int_as_float(head);
                    if (lane == __ffs(holders) - 1)
                    {
#pragma unroll
                        for (int q = 0; q + 1 < KMAX; ++q) rest[q] = rest[q + 1];
                        rest[KMAX - 1] = CUDART_INF_F;
                    }
                }
            }
            if (r >= r_max || knn_done(kth, knn_margin(a, p.x, p.y, p.z, cx, cy, cz, r)))
            {
                if (lane == 0) a.radius[(size_t)__float_as_int(p.w) * a.radius_stride] = sqrtf(kth);
                break;
            }
            // as far as the k-th distance reaches, or twice as far while there are not k candidates
            r_prev     = r;
            const int next = kth < CUDART_INF_F ? (int)fminf(ceilf((sqrtf(kth) + a.slack) * g.inv_cell), 1e6f) : 2 * r;
            r          = min(max(next, r + 1), max(r_max, 1));
        }
    }
}

}  // namespace vetr

// Removing points from a cloud on the device: NeuralScene::RemovePoints (data/NeuralScene.cpp:1156-1239).  The reference
// sorts the indices on the host, builds the list of indices to keep in a host loop (:1169-1181), rebuilds the cloud through
// a CPU mesh (:1191-1193) and index_selects every per-point tensor with the keep list: texture, confidence
// (NeuralTexture.cpp:160-173) and the optimizer's moments (my_adam.cpp:107-135).  Here: flag the removed points, one
// exclusive scan gives every surviving point its new index, and one gather kernel per tensor copies the survivors, in
// their old order, exactly as index_select with the sorted keep list does.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace vetr
{
// flags[i] = 0 for every listed point (duplicates allowed); an index outside [0, n) sets *bad.
__global__ void __launch_bounds__(256) points_mark_removed_kernel(const long long* __restrict__ remove, int m, int n, int* flags, int* bad)
{
    for (int j = blockIdx.x * 256 + threadIdx.x; j < m; j += gridDim.x * 256)
    {
        const long long i = remove[j];
        if (i < 0 || i >= n)
            *bad = 1;
        else
            flags[i] = 0;
    }
}

__global__ void __launch_bounds__(256) points_fill_kernel(int* a, int n, int v)
{
    for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) a[i] = v;
}

// new_index[i] (the exclusive scan of the flags on entry) becomes -1 for removed points; *n_kept = survivors.
__global__ void __launch_bounds__(256) points_new_index_kernel(const int* __restrict__ flags, int n, int* new_index, int* n_kept)
{
    for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256)
    {
        const int f = flags[i], s = new_index[i];
        if (i == n - 1) *n_kept = s + f;
        if (!f) new_index[i] = -1;
    }
}

// dst[r, new_index[i], :] = src[r, i, :] for the survivors, of up to kGatherArrays arrays [rows, points, width] of 4-byte elements
// in one launch.
//
// Bound by HBM: every element is read once and survivors are written once, both nearly coalesced (survivors keep their order).  A
// thread takes four points, looks up where they go once and then moves them in row after row; rows are dealt to gridDim.y as
// well where the points alone do not fill the GPU.  4 M points, 20 words each in eight arrays, 5 % removed: 321 -> 114 us (before: a launch
// per array, a 64-bit division and a look-up per element).  For widths of up to four words; more go to points_gather_pieces_kernel.
constexpr int kGatherArrays = 16;
constexpr int kGatherPoints = 4;                    // points per thread
constexpr int kGatherBlock  = 256 * kGatherPoints;  // points per block
template <typename Total>
struct GatherArgs
{
    const uint32_t* src[kGatherArrays];
    uint32_t* dst[kGatherArrays];
    Total end[kGatherArrays];  // running total of the rows (int), or of the pieces of rows (long long)
    int width[kGatherArrays];
    const int* new_index;
    int n, n_kept, arrays;
};

__global__ void __launch_bounds__(256) points_gather_kernel(const __grid_constant__ GatherArgs<int> a)
{
    const unsigned first = blockIdx.x * kGatherBlock + threadIdx.x;
    int to[kGatherPoints];
#pragma unroll
    for (int k = 0; k < kGatherPoints; ++k) to[k] = first + k * 256 < (unsigned)a.n ? a.new_index[first + k * 256] : -1;
    int q = 0;
    for (unsigned u = blockIdx.y; u < (unsigned)a.end[a.arrays - 1]; u += gridDim.y)
    {
        while (u >= (unsigned)a.end[q]) ++q;
        const int r = (int)u - (q ? a.end[q - 1] : 0), width = a.width[q];
        const uint32_t* src = a.src[q] + (long long)r * a.n * width;
        uint32_t* dst       = a.dst[q] + (long long)r * a.n_kept * width;
        if (width == 1)
        {
            uint32_t v[kGatherPoints];
#pragma unroll
            for (int k = 0; k < kGatherPoints; ++k)
                if (to[k] >= 0) v[k] = src[first + k * 256];
#pragma unroll
            for (int k = 0; k < kGatherPoints; ++k)
                if (to[k] >= 0) dst[to[k]] = v[k];
        }
        else if (width == 4)  // [N,4] rows are 16-byte aligned by contract
        {
            uint4 v[kGatherPoints];
#pragma unroll
            for (int k = 0; k < kGatherPoints; ++k)
                if (to[k] >= 0) v[k] = reinterpret_cast<const uint4*>(src)[first + k * 256];
#pragma unroll
            for (int k = 0; k < kGatherPoints; ++k)
                if (to[k] >= 0) reinterpret_cast<uint4*>(dst)[to[k]] = v[k];
        }
        else
        {
#pragma unroll
            for (int k = 0; k < kGatherPoints; ++k)
                for (int e = 0; to[k] >= 0 && e < width; ++e)
                    dst[(long long)to[k] * width + e] = src[(long long)(first + k * 256) * width + e];
        }
    }
}

// Wider elements: a row of a block's 1024 points is cut into pieces of 4096 words, whose consecutive words go to consecutive threads.
// The whole removal, a tenth of the points removed: 1 M points of 16 words 189 -> 92 us, 200 k of 64 words 204 -> 88, 10 k of 1024
// words 1207 -> 78 (before: by the kernel above, word after word in the element's thread); 2 M points of six words 106 -> 95, of two or
// three 72 to 83 in either.  A kernel of its own, because in one kernel the table in shared memory and its barrier cost the
// narrow elements: 4 M points, 95 % removed, 200 -> 255 us.
constexpr int kGatherNarrow = 4;                 // widest element of points_gather_kernel
constexpr int kGatherPiece  = 4 * kGatherBlock;  // words
__host__ __device__ inline int gather_pieces(int width) { return width / 4 + (width % 4 != 0); }

__global__ void __launch_bounds__(256) points_gather_pieces_kernel(const __grid_constant__ GatherArgs<long long> a)
{
    __shared__ int s_to[kGatherBlock];
    const unsigned block = blockIdx.x * kGatherBlock;
#pragma unroll
    for (int k = threadIdx.x; k < kGatherBlock; k += 256) s_to[k] = block + k < (unsigned)a.n ? a.new_index[block + k] : -1;
    __syncthreads();
    int q = 0;
    for (long long u = blockIdx.y; u < a.end[a.arrays - 1]; u += gridDim.y)
    {
        while (u >= a.end[q]) ++q;
        const int width      = a.width[q], pieces = gather_pieces(width);
        const long long unit = u - (q ? a.end[q - 1] : 0), row = unit / pieces, piece = unit - row * pieces;
        const uint32_t* src  = a.src[q] + (row * a.n + block) * width;
        uint32_t* dst        = a.dst[q] + row * a.n_kept * width;
        // the thread's words are 256 apart: word `o` of the element of point `p` of the block
        const long long word = piece * kGatherPiece + threadIdx.x;
        unsigned p = (unsigned)(word / width), o = (unsigned)(word - (long long)p * width);
        const unsigned dp = 256u / (unsigned)width, dq = 256u % (unsigned)width;
        constexpr int kTogether = 8;
#pragma unroll 1
        for (int k = 0; k < kGatherPiece / 256; k += kTogether)
        {
            uint32_t v[kTogether];
            long long at[kTogether];
#pragma unroll
            for (int j = 0; j < kTogether; ++j)
            {
                const int t = p < (unsigned)kGatherBlock ? s_to[p] : -1;
                at[j]       = t >= 0 ? (long long)t * width + o : -1;
                if (t >= 0) v[j] = src[(long long)p * width + o];
                p += dp, o += dq;
                if (o >= (unsigned)width) o -= width, ++p;
            }
#pragma unroll
            for (int j = 0; j < kTogether; ++j)
                if (at[j] >= 0) dst[at[j]] = v[j];
        }
    }
}
}  // namespace vetr

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
// per array, a 64-bit division and a look-up per element).
constexpr int kGatherArrays = 16;
constexpr int kGatherPoints = 4;  // points per thread
struct GatherArgs
{
    const uint32_t* src[kGatherArrays];
    uint32_t* dst[kGatherArrays];
    int row_end[kGatherArrays];  // running total of the rows
    int width[kGatherArrays];
    const int* new_index;
    int n, n_kept, arrays;
};

__global__ void __launch_bounds__(256) points_gather_kernel(const __grid_constant__ GatherArgs a)
{
    const unsigned first = blockIdx.x * (256 * kGatherPoints) + threadIdx.x;
    int to[kGatherPoints];
#pragma unroll
    for (int k = 0; k < kGatherPoints; ++k) to[k] = first + k * 256 < (unsigned)a.n ? a.new_index[first + k * 256] : -1;
    int q = 0;
    for (unsigned u = blockIdx.y; u < (unsigned)a.row_end[a.arrays - 1]; u += gridDim.y)
    {
        while (u >= (unsigned)a.row_end[q]) ++q;
        const int r = (int)u - (q ? a.row_end[q - 1] : 0), width = a.width[q];
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
}  // namespace vetr

// Layout helpers that let the voxel-per-lane kernels take jobs whose rows or grid they could not
// otherwise use: a copy of the channel data with padded frame rows, and the contiguous extent of
// an unannounced voxel grid, found on the device.
#include <algorithm>
#include <cstdint>

#include "das_launch.cuh"
#include "das_tiles.h"

namespace mach_b200 {
namespace {

// One 16-byte vector of the padded rows per thread.  The copy is one pass over the channel data
// (HBM-bound, 10-20 us per 40 MB); the rows it makes are read by 256-bit loads in chunks of 8 or 16
// frames, hundreds of times each.
template <typename T>
__global__ void __launch_bounds__(256) pad_frames_kernel(const T* __restrict__ src, uint4* __restrict__ dst,
                                                         int64_t n_vec, int n, int vec_per_row) {
    constexpr int kPer = 16 / sizeof(T);
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n_vec;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t row = i / vec_per_row;
        const int f0 = static_cast<int>(i - row * vec_per_row) * kPer;
        const T* s = src + row * n;
        union {
            uint4 v;
            T t[kPer];
        } u;
        u.v = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            if (f0 + k < n) u.t[k] = __ldg(s + f0 + k);
        }
        dst[i] = u.v;
    }
}

constexpr int kProbeThreads = 512;
constexpr int kProbeLimit = 1 << 16;  // longest contiguous extent looked for

// One CTA: the first point whose x or y differ from point 0's.
__global__ void __launch_bounds__(kProbeThreads) das_probe_grid_kernel(const float* __restrict__ scan, int64_t n_vox,
                                                                       int32_t* fast) {
    __shared__ int s_first;
    if (threadIdx.x == 0) s_first = 0x7fffffff;
    __syncthreads();
    const float x0 = __ldg(scan), y0 = __ldg(scan + 1);
    const int limit = static_cast<int>(n_vox < kProbeLimit ? n_vox : kProbeLimit);
    for (int base = 0; base < limit; base += kProbeThreads) {
        const int v = base + threadIdx.x;
        if (v < limit && (__ldg(scan + 3 * static_cast<int64_t>(v)) != x0 ||
                          __ldg(scan + 3 * static_cast<int64_t>(v) + 1) != y0)) {
            atomicMin(&s_first, v);
        }
        if (__syncthreads_or(s_first != 0x7fffffff)) break;  // the same for every thread
    }
    if (threadIdx.x == 0) {
        const int f = s_first;
        *fast = (f != 0x7fffffff && f >= kProbeMinFast && n_vox % f == 0 && n_vox / f >= kProbeMinOuter) ? f : 0;
    }
}

}  // namespace

cudaError_t launch_pad_frames(const void* src, void* dst, int64_t rows, int n, int p, int esz, cudaStream_t st) {
    const int vec_per_row = p * esz / 16;
    const int64_t n_vec = rows * vec_per_row;
    if (n_vec <= 0) return cudaSuccess;
    const unsigned blocks = static_cast<unsigned>(std::min<int64_t>((n_vec + 255) / 256, 148 * 64));
    uint4* d = static_cast<uint4*>(dst);
    switch (esz) {
        case 2: pad_frames_kernel<<<blocks, 256, 0, st>>>(static_cast<const unsigned short*>(src), d, n_vec, n, vec_per_row); break;
        case 4: pad_frames_kernel<<<blocks, 256, 0, st>>>(static_cast<const unsigned*>(src), d, n_vec, n, vec_per_row); break;
        default: pad_frames_kernel<<<blocks, 256, 0, st>>>(static_cast<const unsigned long long*>(src), d, n_vec, n, vec_per_row); break;
    }
    return cudaGetLastError();
}

cudaError_t launch_probe_grid(const float* scan, int64_t n_vox, int32_t* fast, cudaStream_t st) {
    das_probe_grid_kernel<<<1, kProbeThreads, 0, st>>>(scan, n_vox, fast);
    return cudaGetLastError();
}

}  // namespace mach_b200

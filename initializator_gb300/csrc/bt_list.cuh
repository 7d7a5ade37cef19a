// Pore lists: which voxels (or groups of four along x) a step has to touch.
//
// A step's work is on pore voxels only, and a rock is 20 to 70 % pore: the
// list kernels give one thread to each pore voxel (generic kernel) or to each
// group of four voxels along x that holds one (FP32 fast path), so no lane
// idles over solid and no byte of solid is streamed. The solid voxels of both
// field buffers hold zero, which the dense kernels wrote every step (the
// reference never updates them, cpp:3174, 2501-2506) and which the host
// runtime now keeps (bt_api.cu, solid_check).
//
// Order: columns of LT_X x LT_Y voxels, each marching in z, x fastest within a
// plane, so that the entries one CTA takes in a row are a compact block whose
// neighbours in y and z come from its own L1.
#pragma once
#include <algorithm>

#include "bt_internal.h"

namespace bt {

constexpr int LT_X = 64;  // voxels along x of a list column (16 groups of four)
constexpr int LT_Y = 8;   // rows of a list column
constexpr int LT_Q = LT_X / 4;
// generic list kernels: threads of a CTA, and resident CTAs a SM (a launch has
// as many chunks, one wave: every SM gets the same share of the list)
constexpr int LIST_THREADS = 128;
constexpr int list_ctas_per_sm(size_t esz) { return esz == 8 ? 4 : 5; }

// the coordinates of element `idx` of a pitched component
struct Cell {
    int x, y, z;
};
__host__ __device__ inline uint32_t fast_div(uint32_t n, const FastDiv& d) {
#ifdef __CUDA_ARCH__
    return d.mul ? __umulhi(n, d.mul) >> d.shift : n;
#else
    return d.mul ? (uint32_t)(((uint64_t)n * d.mul) >> 32) >> d.shift : n;
#endif
}
// exact for n < 2^31: mul = ceil(2^(32 + shift) / d), 2^shift < d <= 2^(shift + 1)
inline FastDiv make_fast_div(uint32_t d) {
    FastDiv f{0u, 0u};
    if (d <= 1) return f;
    uint32_t s = 0;
    while ((2u << s) < d) ++s;
    f.shift = s;
    f.mul = (uint32_t)((((uint64_t)1 << (32 + s)) + d - 1) / d);
    return f;
}
__host__ __device__ inline Cell cell_of(uint32_t idx, const FastDiv& by_pitch, const FastDiv& by_ny, int pitch, int ny) {
    Cell c;
    const uint32_t row = fast_div(idx, by_pitch);
    c.z = (int)fast_div(row, by_ny);
    c.y = (int)row - c.z * ny;
    c.x = (int)(idx - row * (uint32_t)pitch);
    return c;
}

// ---- built on the device (bt_list.cu) ----
// planes of list columns; offs of list_offsets holds one more
uint32_t list_segments(int nx, int ny, int nz);
// offs[segments + 1]: where each segment's entries begin, and how many there are
// (pore voxels, or groups of four along x that hold one)
cudaError_t list_offsets(const uint8_t* code, int nx, int ny, int nz, int cpitch, bool groups, uint32_t* offs,
                         cudaStream_t s);
cudaError_t fill_pore_list(const uint8_t* code, int nx, int ny, int nz, int pitch, int cpitch, const uint32_t* offs,
                           uint32_t* idx, uint8_t* pcode, cudaStream_t s);
// the bounding box of each chunk of a list of element indices
cudaError_t chunk_boxes(const uint32_t* idx, uint32_t n, uint32_t chunks, const FastDiv& by_pitch, const FastDiv& by_ny,
                        int pitch, int ny, int* box, cudaStream_t s);
// a field's solid voxels looked over (*flag = 1 where one is not zero), after
// dense arrays were copied in when src is given
template <typename T>
cudaError_t field_in(T* field, const T* const* src, const uint8_t* code, int nx, int ny, int nz, int pitch, int cpitch,
                     long long comp, int members, int* flag, cudaStream_t s);
template <typename T>
cudaError_t solid_clear(T* field, const uint8_t* code, int nx, int ny, int nz, int pitch, int cpitch, long long comp,
                        int members, cudaStream_t s);

}  // namespace bt

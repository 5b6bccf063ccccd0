/*
 * bp_shapes.cuh - pixel tiles of the tiled backprojectors (udev_bp_tiles.cu,
 * udev_siddon.cu): launch shapes, the rule that picks one, and the staging of
 * a chunk of angles' detector windows in shared memory.
 */
#ifndef UFOIR_BP_SHAPES_CUH
#define UFOIR_BP_SHAPES_CUH

#include <cuda_runtime.h>

#include <cstdint>

#include "udev_internal.cuh"

namespace bp {

constexpr int kTX = 32;
constexpr int kAC = 32;              /* angles per chunk: one per lane of a warp */

/* A launch shape: 32 x TY threads, each with COLS pixel columns (32 apart) of
 * PR rows (TY apart); W detectors staged per angle. */
template <int COLS_, int PR_, int TY_, int CTAS_, int UNROLL_>
struct BpShape {
    static constexpr int COLS = COLS_, PR = PR_, TY = TY_, CTAS = CTAS_, Unroll = UNROLL_;
    static constexpr int H = COLS / 2;                 /* packed pairs per row */
    static constexpr int TileX = kTX * COLS, TileY = TY * PR, Threads = kTX * TY;
    /* a tile spans at most its diagonal; 2 bins of margin and up to 3 of
     * alignment before it, 2 for the second tap after it */
    static constexpr int span(int d) { return d * d >= TileX * TileX + TileY * TileY ? d : span(d + 1); }
    static constexpr int Win = (span(TileX) + 8 + 3) / 4 * 4;
};

/* Fewer pixels per thread cost more instructions per sample but leave more,
 * smaller tiles for launches with few of them (see bp_shape). */
typedef BpShape<4, 8, 8, 2, 4> ShapeL;      /* 128 x 64 tiles */
typedef BpShape<4, 4, 8, 3, 4> ShapeM;      /* 128 x 32 */
typedef BpShape<2, 4, 4, 7, 4> ShapeS;      /* 64 x 16 */
typedef BpShape<2, 2, 4, 8, 8> ShapeT;      /* 64 x 8 */

__device__ __forceinline__ void cp_async4(float *dst, const float *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t) __cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}

__device__ __forceinline__ void cp_async16(float *dst, const float *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t) __cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}

__device__ __forceinline__ void cp_async_commit()
{
    asm volatile("cp.async.commit_group;" ::: "memory");
}

template <int N>
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

/*
 * Copies the T::Win detectors from src on (a window that starts at detector
 * w0 of a row of n, at a 16-byte aligned address) to dst with the lanes of
 * one warp: 16-byte cp.async copies, and element by element, with zeros
 * outside [0, n), where a group of 4 crosses the ends of the row.
 */
template <class T>
__device__ __forceinline__ void copy_window(float *dst, const float *src, int w0, int n)
{
#pragma unroll
    for (int g = 0; g < T::Win / 4; g += 32) {
        const int e = 4 * (g + (int) threadIdx.x), d = w0 + e;
        if (e >= T::Win)
            continue;
        if (d >= 0 && d + 4 <= n) {
            cp_async16(dst + e, src + e);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (d + q >= 0 && d + q < n)
                    cp_async4(dst + e + q, src + e + q);
                else
                    dst[e + q] = 0.0f;
            }
        }
    }
}

/* The largest detector index <= d whose address in `row` is 16-byte aligned. */
__device__ __forceinline__ int align_window(int d, const float *row)
{
    const int mis = (int) ((reinterpret_cast<uintptr_t>(row) >> 2) & 3);
    return d - ((d + mis) & 3);
}

/*
 * The launch shape by how many waves of tiles a launch has (ms, GB300, at
 * L / M / S / T):
 *   16 x 1448^2 x 1200 (14.5 waves of L)  13.69 / 14.06 / 14.74 / -
 *    2 x 2900^2 x 360  (7.0)               2.04 /  2.05 /  2.24 / -
 *    6 x 1001^2 x 451  (2.5; 3.4 of M)     1.08 /  1.03 /  1.06 / 1.26
 *    3 x 1448^2 x 1200 (2.7; 3.6 of M)     2.86 /  2.77 /  2.85 / 3.62
 *    2 x 1448^2 x 1200 (2.4 of M)          1.99 /  1.96 /  1.93 / 2.43
 *    1 x 1448^2 x 1200 (1.2 of M)          1.05 /  1.05 /  1.01 / 1.26
 *    4 x 367^2 x 180   (3.6 S tiles per SM) 0.112 / 0.067 / 0.062 / 0.067
 *    1 x 512^2 x 400   (1.7)               0.220 / 0.117 / 0.080 / 0.078
 *    1 x 367^2 x 180   (0.9)               0.112 / 0.067 / 0.037 / 0.030
 */
inline int bp_shape(udev *d, int n, int n_slices)
{
    const long long sms = udev_sm_count(d);
    const long long l = (long long) udev_div_up(n, ShapeL::TileX) * udev_div_up(n, ShapeL::TileY) * n_slices;
    const long long m = (long long) udev_div_up(n, ShapeM::TileX) * udev_div_up(n, ShapeM::TileY) * n_slices;
    const long long s = (long long) udev_div_up(n, ShapeS::TileX) * udev_div_up(n, ShapeS::TileY) * n_slices;
    return l >= 6 * ShapeL::CTAS * sms ? 0 : m >= 3 * ShapeM::CTAS * sms ? 1 : s >= 2 * sms ? 2 : 3;
}

}  // namespace bp

#endif

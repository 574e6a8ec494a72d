// Output-raster helper of the wrapped-phase workflow: grow_nodata_region
// (utils.py:613-660), which the block loop applies to the strided outputs before
// writing them (workflows/single.py:352-362).
//
// k_grow_nodata<T> -- one thread per pixel: the pixel becomes `nodata` if any pixel of
// the (2n + 1) x (2n + 1) square around it (clipped to the image: scipy's
// binary_dilation pads with False) is nodata.  A pixel is nodata where it equals the
// nodata value, or, for a NaN nodata value, where it is NaN (integer arrays then have
// none).  Out of place: `out` must not alias `in`.  HBM-bound on the output rasters,
// which are small next to the stack.
#include <algorithm>
#include <cstdio>
#include <limits>
#include <type_traits>

#include "dpl_common.cuh"

namespace dpl {

// The nodata value in the raster's own type; `mode` 0: no pixel can be nodata (a NaN on
// integers, a value that the type does not hold), 1: equal to `value`, 2: NaN.
template <class T>
struct Nodata {
    T value;
    int mode;
    __device__ __forceinline__ bool operator()(T v) const {
        if constexpr (std::is_floating_point<T>::value) {
            if (mode == 2) return isnan(v);
        }
        return mode == 1 && v == value;
    }
};

// Compared in the raster's type: in double (as the reference's promotion does, with the
// same outcome) the 25 comparisons of a 5 x 5 square run at the FP64 rate: 27 us for a
// 512 x 512 raster instead of 5.7.
template <class T>
__global__ void __launch_bounds__(256) k_grow_nodata(const T* __restrict__ in, T* __restrict__ out, int rows, int cols,
                                                      Nodata<T> nodata, int n) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (int64_t)rows * cols) return;
    const int r = (int)(p / cols), c = (int)(p - (int64_t)r * cols);
    const int r0 = max(r - n, 0), r1 = min(r + n, rows - 1), c0 = max(c - n, 0), c1 = min(c + n, cols - 1);
    bool hit = false;
    for (int rr = r0; rr <= r1 && !hit; ++rr) {
        const T* row = in + (int64_t)rr * cols;
#pragma unroll 4
        for (int cc = c0; cc <= c1; ++cc) hit |= nodata(row[cc]);
    }
    out[p] = hit ? nodata.value : in[p];
}

template <class T>
static dpl_status grow_launch(const void* in, void* out, int64_t rows, int64_t cols, double nodata, int nan_nodata,
                              int n, cudaStream_t st) {
    if (((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) % alignof(T)) != 0)
        return fail(DPL_ERR_INVALID_ARGUMENT, "dpl_grow_nodata_region: arrays must be aligned to their element size");
    Nodata<T> nd{T(0), 0};
    if (std::is_floating_point<T>::value) {
        nd.value = nan_nodata ? std::numeric_limits<T>::quiet_NaN() : (T)nodata;
        nd.mode = nan_nodata ? 2 : (double)nd.value == nodata ? 1 : 0;
    } else if (!nan_nodata && nodata >= (double)std::numeric_limits<T>::lowest() &&
               nodata <= (double)std::numeric_limits<T>::max()) {
        nd.value = (T)nodata;
        nd.mode = (double)nd.value == nodata ? 1 : 0;
    }
    const int64_t npix = rows * cols;
    n = (int)std::min<int64_t>(n, std::max(rows, cols));  // the whole raster
    k_grow_nodata<T><<<(unsigned)ceil_div(npix, 256), 256, 0, st>>>(static_cast<const T*>(in), static_cast<T*>(out),
                                                                     (int)rows, (int)cols, nd, n);
    return check_launch("k_grow_nodata");
}

}  // namespace dpl

using namespace dpl;

extern "C" dpl_status dpl_grow_nodata_region(const void* in, void* out, int dtype, int64_t rows, int64_t cols,
                                             double nodata, int nodata_is_nan, int n_pixels, dpl_stream_t stream) {
    if (rows < 0 || cols < 0 || n_pixels < 0)
        return fail(DPL_ERR_INVALID_ARGUMENT, "dpl_grow_nodata_region: bad shape or n_pixels");
    if (rows > INT32_MAX || cols > INT32_MAX) return fail(DPL_ERR_UNSUPPORTED, "dpl_grow_nodata_region: too large");
    if (rows * cols == 0) return DPL_OK;
    if (!in || !out) return fail(DPL_ERR_INVALID_ARGUMENT, "dpl_grow_nodata_region: null pointer");
    if (in == out) return fail(DPL_ERR_INVALID_ARGUMENT, "dpl_grow_nodata_region: out must not alias in");
    cudaStream_t st = (cudaStream_t)stream;
    const int nan = nodata_is_nan != 0;
    switch (dtype) {
        case DPL_DTYPE_F32: return grow_launch<float>(in, out, rows, cols, nodata, nan, n_pixels, st);
        case DPL_DTYPE_U8: return grow_launch<uint8_t>(in, out, rows, cols, nodata, nan, n_pixels, st);
        case DPL_DTYPE_I8: return grow_launch<int8_t>(in, out, rows, cols, nodata, nan, n_pixels, st);
        case DPL_DTYPE_I16: return grow_launch<int16_t>(in, out, rows, cols, nodata, nan, n_pixels, st);
        case DPL_DTYPE_U16: return grow_launch<uint16_t>(in, out, rows, cols, nodata, nan, n_pixels, st);
        case DPL_DTYPE_I32: return grow_launch<int32_t>(in, out, rows, cols, nodata, nan, n_pixels, st);
        default: return fail(DPL_ERR_INVALID_ARGUMENT, "dpl_grow_nodata_region: unknown dtype");
    }
}

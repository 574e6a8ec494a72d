// SHP kernel arguments and host launchers shared with the phase-linking pipeline.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/dpl.h"
#include "dpl_common.cuh"

namespace dpl {

struct GlrtArgs {
    int rows, cols, hy, hx, sy, sx, out_rows, out_cols, nslc;
    float thr;
    int tile_r, tile_c;  // output pixels per CTA
    int box_w, box_h;    // TMA box (floats x rows)
    uint8_t* is_shp;     // (out_rows, out_cols, wy, wx) bytes
    int ratio;           // no logarithms: the ratio test applies,
    int interval;        //   as an interval of s2
    float four_c;        // 4 exp(thr / nslc)
    float center, half;  // the interval of s2 / s1
    float ratio_max;     // largest scale^2 of either test
    int* status;         // set to DPL_ERR_TIMEOUT if a bounded wait gives up
};

struct KsArgs {
    const float* sorted;  // (n, rows, cols)
    int8_t lo[kMaxNslc + 1], hi[kMaxNslc + 1];  // admissible i2 per i1 of the merge walk
    int8_t env_lo[kMaxNslc], env_hi[kMaxNslc];  // envelope of sample t: indices into x1 (-1: none)
    int ns;               // samples with a lower bound (n minus the first index that has one)
    int pitch;            // floats per pixel's samples in shared memory
    int off_bits;         // the mask bits, in 4-byte words from the start of shared memory
    int n, rows, cols, hy, hx, sy, sx, out_rows, out_cols;
    int tile_r, tile_c;
    uint8_t* is_shp;
};

int64_t glrt_pitch(int64_t cols);
size_t glrt_workspace_size(int64_t rows, int64_t cols);
size_t ks_workspace_size(int64_t nslc, int64_t rows, int64_t cols);

// scale2: rows x glrt_pitch(cols) floats.
dpl_status launch_glrt(const float* mean, const float* var, int64_t rows, int64_t cols, int hy, int hx, int sy,
                       int sx, int nslc, float threshold, uint8_t* is_shp, int* status, float* scale2,
                       cudaStream_t s);

}  // namespace dpl

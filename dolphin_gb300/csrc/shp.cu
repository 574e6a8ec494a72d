// Statistically homogeneous pixel (SHP) selection.
//
// GLRT (shp/_glrt.py:13-130): the Rayleigh scale^2 = (var + mean^2)/2 is written to a
// pitched buffer, and each CTA stages its input region into shared memory with one
// TMA tiled copy (cp.async.bulk.tensor.2d, completion on an mbarrier with a bounded
// wait).  Window starts follow lax.dynamic_slice (clamped into the image: windows shift
// at the edges), validity follows the unclamped origin and the window centre is always
// False -- the reference's semantics.  The reference's float32 statistic
// nslc * (2*log(pooled) - log(s1) - log(s2)) < threshold is, exactly,
//     (s1 + s2)^2 < 4 c s1 s2,  c = exp(threshold / nslc),
// which needs no logarithm: s2 has to lie within 2 sqrt(c (c - 1)) s1 of (2 c - 1) s1, two
// subtractions per (pixel, offset).  They carry less than 2.7e-7 of the centre in error;
// where the distance to the interval's end is within 5e-7 of it, the decision is taken in
// double precision on nslc * log1p((s1 - s2)^2 / (4 s1 s2)) (algebraically equal, no
// cancellation), so every mask bit is the exact comparison on the float32 scale^2.  Few
// dates (c > 64) compare the two sides, within 2e-6 likewise.  Scales whose products would
// overflow float32 and thresholds outside the usual range take the statistic with its
// logarithms (glrt_test), refined in the same way where its rounding could reach the cutoff.
//
// KS (shp/_ks.py:22-239): amplitudes are sorted per pixel (NaN last, like np.sort).  The
// reference walks the two-sample merge of each (pixel, neighbour) pair and rejects it
// where the ECDFs come apart by the cutoff.  It accumulates the ECDFs by repeated
// float64 additions of 1/n, so after i steps an ECDF equals T[i] (the i-fold sum) and a
// walk position (i1, i2) is admissible where i2 lies in the interval
// {i2 : |T[i1] - T[i2]| < cutoff}, T being increasing.  Without ties the walk leaves the
// band exactly where some sample of the neighbour lies outside its envelope,
//     lo_t < x2[t] < hi_t,  lo_t = x1[m(t) - 1],  hi_t = x1[min {i : m(i) - 1 = t}],
// with m(t) the smallest i1 that admits i2 = t + 1: x2[t] is taken before x1[m(t) - 1]
// when it is smaller, and the lower bound is the same statement with the two series
// exchanged.  A violated bound rejects, all bounds strictly met accept, and only a pair
// with an equality (a tie decides by the walk's order) or with a non-finite sample is
// walked step by step.  The decision is therefore bit-identical to the float64 walk.
//
// Both kernels gather the decisions as bits, consecutive pixels on consecutive lanes
// (conflict-free reads of the staged tile): a pixel's whole window is one stream, filled
// by the pixel's thread (GLRT) or by items of 32 offsets of a window row (KS).  The mask
// bytes of each output row are written afterwards, up to 32 per store.
#include <cuda.h>

#include <algorithm>
#include <vector>

#include "dpl_common.cuh"
#include "shp.cuh"

namespace dpl {

// ---------------------------------------------------------------------------------
// TMA / mbarrier helpers (inline PTX)
// ---------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

constexpr uint32_t kWaitLimit = 1u << 24;  // bounded mbarrier wait (iterations)

__device__ __forceinline__ int clamp_start(int center, int half, int size, int dim) {
    int s = center - half;
    s = s < 0 ? 0 : s;
    return s > dim - size ? dim - size : s;
}

// ---------------------------------------------------------------------------------
// GLRT
// ---------------------------------------------------------------------------------
__global__ void k_glrt_scale(const float* __restrict__ mean, const float* __restrict__ var, int64_t rows,
                             int64_t cols, int64_t pitch, float* __restrict__ scale2) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows * cols) return;
    int64_t r = i / cols, c = i - r * cols;
    float m = mean[i];
    scale2[r * pitch + c] = fdiv(fadd(var[i], fmul(m, m)), 2.f);
}

// threshold > statistic in double precision on the float32 scales
__device__ __noinline__ bool glrt_exact(float s1, float s2, float nslc, float thr) {
    const double d = (double)s1 - (double)s2;
    const double t = (double)nslc * log1p(d * d / (4.0 * (double)s1 * (double)s2));
    return (double)thr > t;
}

// One (pixel, offset) test with the float32 statistic, refined in double precision near
// the cutoff (see above).  NaN statistics stay False.
__device__ __noinline__ bool glrt_test(float s1, float s2, float nslc, float thr) {
    // (s1 + s2) / 2 == (s1 + s2) * 0.5 exactly in IEEE arithmetic
    const float pooled = fmul(fadd(s1, s2), 0.5f);
    const float lp = fmul(2.f, logf(pooled)), l1 = logf(s1), l2 = logf(s2);
    const float stat = fmul(nslc, fsub(fsub(lp, l1), l2));
    bool shp = thr > stat;
    // the rounding of the three logarithms and of their cancelling sum
    const float err = nslc * 3e-7f * (fabsf(lp) + fabsf(l1) + fabsf(l2));
    // (a scale of 0 has an infinite logarithm and error, and no neighbour)
    if (s1 > 0.f && s2 > 0.f && fabsf(stat - thr) <= fmaf(1e-5f, thr, err)) shp = glrt_exact(s1, s2, nslc, thr);
    return shp;
}

// Bytes (0/1) of an output row's masks from their bits: run r of the tile row (a pixel's
// window row, or its whole window) has its wx bits in the nw words at bits + r * nw, zero
// beyond wx; the bytes go to dst[0 .. rows * wx).  C bytes (4 to 32, at most wx + 1, so
// that they touch two runs at most) per aligned store, by the threads t, t + nt, ...
template <int C>
__device__ __forceinline__ void write_masks(uint8_t* dst, const uint32_t* bits, int rows, int wx, int nw, int t,
                                            int nt) {
    const int len = rows * wx;
    const int head = min(len, (int)((C - (uint32_t)(reinterpret_cast<uintptr_t>(dst) & (C - 1))) & (C - 1)));
    const int chunks = (len - head) / C, tail = head + C * chunks;
    auto bit = [&](int k) -> uint32_t {
        const int r = k / wx, wb = k - r * wx;
        return (bits[r * nw + (wb >> 5)] >> (wb & 31)) & 1u;
    };
    const float inv_wx = 1.f / (float)wx;
    for (int q = t; q < chunks; q += nt) {
        const int k = head + C * q;
        int r = (int)((float)k * inv_wx);  // k / wx: the float quotient is off by one at most
        int wb = k - r * wx;
        if (wb < 0) {
            --r;
            wb += wx;
        } else if (wb >= wx) {
            ++r;
            wb -= wx;
        }
        const uint32_t* w = bits + r * nw + (wb >> 5);
        const int sh = wb & 31, left = wx - wb;
        uint32_t v = w[0] >> sh;
        if (sh > 32 - C && left > 32 - sh) v |= w[1] << (32 - sh);  // into the run's next word
        if (left < C) v |= bits[(r + 1) * nw] << left;              // into the next run
        uint32_t o[C / 4];
#pragma unroll
        for (int i = 0; i < C / 4; ++i) o[i] = (((v >> (4 * i)) & 0xfu) * 0x00204081u) & 0x01010101u;
        if constexpr (C == 32)
            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst + k), "r"(o[0]), "r"(o[1]),
                         "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7])
                         : "memory");
        else if constexpr (C == 16) *reinterpret_cast<uint4*>(dst + k) = make_uint4(o[0], o[1], o[2], o[3]);
        else if constexpr (C == 8) *reinterpret_cast<uint2*>(dst + k) = make_uint2(o[0], o[1]);
        else *reinterpret_cast<uint32_t*>(dst + k) = o[0];
    }
    if (t < head) dst[t] = (uint8_t)bit(t);  // head, len - tail < C <= nt
    if (t < len - tail) dst[tail + t] = (uint8_t)bit(tail + t);
}

__device__ __forceinline__ void write_mask_row(uint8_t* dst, const uint32_t* bits, int rows, int wx, int nw, int t,
                                               int nt) {
    if (wx >= 31) write_masks<32>(dst, bits, rows, wx, nw, t, nt);
    else if (wx >= 15) write_masks<16>(dst, bits, rows, wx, nw, t, nt);
    else if (wx >= 7) write_masks<8>(dst, bits, rows, wx, nw, t, nt);
    else if (wx >= 3) write_masks<4>(dst, bits, rows, wx, nw, t, nt);
    else
        for (int k = t; k < rows; k += nt) dst[k] = (uint8_t)(bits[k] & 1u);  // wx == 1
}

// A pixel per thread, its window's bits one stream of words; 32 mask bytes per store.
// Bound by instruction issue in the tests (~110 us) and by the mask bytes' stores (65 us),
// which overlap in part: 1024 x 2048 pixels, 11 x 23 windows: 167 us (3.2 TB/s of mask
// bytes).  The ratio test with an item per (pixel, window row) took 345 us, the interval
// with such items and 16-byte stores 253, a logarithm per test and one byte per store
// 1098.  kPlain (a window row is one word, every pixel has a thread of its own) drops the
// loop over a row's words and the shared words' atomics: 212 -> 167 us.
template <bool kPlain>
__global__ void __launch_bounds__(256, 4) k_glrt(const __grid_constant__ CUtensorMap tmap, GlrtArgs a) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar;
    // 128-byte aligned base (TMA destination), offset within the shared array so that
    // the accesses below stay shared-memory accesses
    const uint32_t mis = (uint32_t)__cvta_generic_to_shared(smem_raw) & 127u;
    float* raw = reinterpret_cast<float*>(smem_raw + ((128u - mis) & 127u));
    const int n_tile = a.box_w * a.box_h;
    uint32_t* bits = reinterpret_cast<uint32_t*>(raw + n_tile);  // [pixel][nw]: its window's bits
    const int wy = 2 * a.hy + 1, wx = 2 * a.hx + 1, W = wy * wx, nw = (W + 31) >> 5;
    const int or0 = blockIdx.y * a.tile_r, oc0 = blockIdx.x * a.tile_c;
    const int or1 = min(or0 + a.tile_r, a.out_rows), oc1 = min(oc0 + a.tile_c, a.out_cols);
    const int rr0 = clamp_start(a.sy / 2 + or0 * a.sy, a.hy, wy, a.rows);
    const int cc0 = clamp_start(a.sx / 2 + oc0 * a.sx, a.hx, wx, a.cols);
    const int x0 = cc0 & ~3;  // TMA inner coordinate: multiple of 4 floats (16 bytes)
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        mbar_expect_tx(&bar, (uint32_t)(n_tile * sizeof(float)));
        tma_load_2d(raw, &tmap, x0, rr0, &bar);
    }
    bool timed_out = false;
    for (uint32_t spins = 0; !mbar_try_wait(&bar, 0);) {
        if (++spins > kWaitLimit) {
            timed_out = true;
            break;
        }
    }
    if (__syncthreads_or(timed_out)) {
        if (threadIdx.x == 0) {
            atomicExch(a.status, (int)DPL_ERR_TIMEOUT);
            // the copy may still be in flight: give it a second bounded wait before exit
            for (uint32_t more = 0; !mbar_try_wait(&bar, 0) && more < kWaitLimit; ++more) {
            }
        }
        __syncthreads();
        return;
    }
    // a negative scale has a NaN logarithm: never an SHP.  Finite scales above the
    // bound (their products overflow) send the tile to the logarithms.
    bool large = !a.ratio;
    for (int i = threadIdx.x; i < n_tile; i += blockDim.x) {
        const float v = raw[i];
        if (v < 0.f) raw[i] = nanf("");
        large |= v > a.ratio_max && v < INFINITY;
    }
    const bool use_log = __syncthreads_or(large);

    const float nslc = (float)a.nslc;
    const int tc = oc1 - oc0, npix = (or1 - or0) * tc;
    // a pixel per thread; a small tile's pixels have their window rows spread over nsub
    // threads, which share the words where one's rows end and the next one's begin
    const int threads = blockDim.x, step = kPlain ? threads : min(npix, threads), nsub = kPlain ? 1 : threads / step;
    const int sub = kPlain ? 0 : (int)threadIdx.x / step, pix0 = (int)threadIdx.x - sub * step;
    const int wa0 = sub * wy / nsub, wa1 = sub < nsub ? (sub + 1) * wy / nsub : wa0;
    if (nsub > 1) {
        for (int i = threadIdx.x; i < npix * nw; i += threads) bits[i] = 0u;
        __syncthreads();
    }
    for (int pix = pix0; wa0 < wa1 && pix < npix; pix += step) {
        const int pr = pix / tc;
        const int in_r = a.sy / 2 + (or0 + pr) * a.sy, in_c = a.sx / 2 + (oc0 + pix - pr * tc) * a.sx;
        const int r0 = clamp_start(in_r, a.hy, wy, a.rows), c0 = clamp_start(in_c, a.hx, wx, a.cols);
        const int ur0 = in_r - a.hy, uc0 = in_c - a.hx;
        const float s1 = raw[(in_r - rr0) * a.box_w + (in_c - x0)];
        const float* row = raw + (r0 + wa0 - rr0) * a.box_w + (c0 - x0);
        // a pixel of scale 0 (no data) or NaN is nobody's neighbour: the statistic is NaN or
        // infinite.  No column of it is valid and no distance near the interval's end: each
        // of its tests would else take the double-precision route (1024 x 2048 pixels, a
        // quarter of them 0: 8.5 ms instead of 0.24).
        const bool live = s1 > 0.f || a.nslc < 0;  // (a negative count: the statistic is -inf)
        const float center = a.center * s1, half = a.half * s1;
        const float margin = live ? fmaf(5e-7f, center, 1e-40f) : -1.f;
        const float k1 = a.four_c * s1;
        // valid window columns v0 .. v1 - 1 and rows of the unclamped origin
        const int v0 = max(0, -uc0), v1 = live ? min(wx, a.cols - uc0) : 0;
        const auto columns = [&](int b0, int nb) {
            const int lo = max(v0 - b0, 0), hi = min(v1 - b0, nb);
            return hi > lo ? (0xffffffffu >> (32 - (hi - lo))) << lo : 0u;
        };
        const uint32_t first = columns(0, min(wx, 32));
        // the bits of the rows so far, from word `w` of the pixel on
        uint32_t* w = bits + pix * nw + (wa0 * wx >> 5);
        uint64_t acc = 0u;
        int fill = wa0 * wx & 31;
        const auto flush = [&](uint32_t v) {
            if (nsub > 1) atomicOr(w, v);
            else *w = v;
            ++w;
        };
        for (int wa = wa0; wa < wa1; ++wa, row += a.box_w) {
            const bool row_ok = (wa >= -ur0) && (wa < a.rows - ur0);
            const float* span = row;
            for (int b0 = 0; b0 < (kPlain ? 1 : wx); b0 += 32, span += 32) {
                const int nb = kPlain ? wx : min(wx - b0, 32);
                uint32_t valid = row_ok ? (b0 ? columns(b0, nb) : first) : 0u;
                if (wa == a.hy && a.hx >= b0 && a.hx < b0 + 32) valid &= ~(1u << (a.hx - b0));
                uint32_t shp = 0u;
                if (!use_log && a.interval) {
                    // each decision is the sign of a difference, shifted into a word (first offset
                    // highest); NaN differences are positive (canonical NaN)
                    float nearest = INFINITY;
                    auto distance = [&](int wb) { return fabsf(span[wb] - center) - half; };
                    auto test = [&](int wb) {
                        const float d = distance(wb);
                        shp = __funnelshift_l(__float_as_uint(d), shp, 1);
                        nearest = fminf(nearest, fabsf(d));
                    };
                    int wb = 0;
                    for (; wb + 8 <= nb; wb += 8) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) test(wb + i);
                    }
                    if (nb & 4) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) test(wb + i);
                        wb += 4;
                    }
                    if (nb & 2) {
                        test(wb);
                        test(wb + 1);
                        wb += 2;
                    }
                    if (nb & 1) test(wb);
                    shp = __brev(shp) >> (32 - nb);
                    if (nearest <= margin) {
#pragma unroll 1
                        for (int i = 0; i < nb; ++i)
                            if ((valid >> i & 1u) && fabsf(distance(i)) <= margin)
                                shp = (shp & ~(1u << i)) | (uint32_t)glrt_exact(s1, span[i], nslc, a.thr) << i;
                    }
                } else if (!use_log) {
                    uint32_t close = 0u;
#pragma unroll 4
                    for (int wb = 0; wb < nb; ++wb) {
                        const float s2 = span[wb];
                        const float sum = s1 + s2;
                        const float r = k1 * s2;
                        const float diff = fmaf(sum, sum, -r);
                        // 1e-40 covers products that lose bits below the normal range
                        const float gap = fabsf(diff) - fmaf(2e-6f, r, 1e-40f);
                        shp = __funnelshift_l(__float_as_uint(diff), shp, 1);
                        close = __funnelshift_l(__float_as_uint(gap), close, 1);
                    }
                    shp = __brev(shp) >> (32 - nb);
                    close = __brev(close) >> (32 - nb);
                    close &= valid;
                    while (close) {
                        const int wb2 = __ffs(close) - 1;
                        close &= close - 1u;
                        shp = (shp & ~(1u << wb2)) | (uint32_t)glrt_exact(s1, span[wb2], nslc, a.thr) << wb2;
                    }
                } else {
                    for (int wb = 0; wb < nb; ++wb)
                        if ((valid >> wb) & 1u) shp |= (uint32_t)glrt_test(s1, span[wb], nslc, a.thr) << wb;
                }
                acc |= (uint64_t)(shp & valid) << fill;
                fill += nb;
                if (fill >= 32) {
                    flush((uint32_t)acc);
                    acc >>= 32;
                    fill -= 32;
                }
            }
        }
        if (fill > 0) flush((uint32_t)acc);
    }
    __syncthreads();
    // an output row per warp, or (few rows) the CTA on one after the other
    const bool by_warp = 32 * (or1 - or0) >= threads;
    const int first_row = by_warp ? (int)threadIdx.x >> 5 : 0, row_step = by_warp ? threads >> 5 : 1;
    for (int r = first_row; r < or1 - or0; r += row_step)
        write_mask_row(a.is_shp + ((int64_t)(or0 + r) * a.out_cols + oc0) * W, bits + r * tc * nw, tc, W, nw,
                       by_warp ? threadIdx.x & 31 : threadIdx.x, by_warp ? 32 : threads);
}

// ---------------------------------------------------------------------------------
// KS
// ---------------------------------------------------------------------------------
__device__ __forceinline__ bool nan_last_greater(float a, float b) {
    // np.sort order: NaN after every number
    return (isnan(a) && !isnan(b)) || a > b;
}

template <int NMAX>
__global__ void __launch_bounds__(128) k_sort_pixels(const float* __restrict__ in, int n, int64_t npix,
                                                     float* __restrict__ out) {
    int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npix) return;
    float v[NMAX];
#pragma unroll
    for (int t = 0; t < NMAX; ++t) v[t] = t < n ? in[(int64_t)t * npix + p] : __int_as_float(0x7fc00000);
    // odd-even transposition sort (NMAX passes) on a fixed-size register array; the
    // padding NaNs sort to the end and are never stored
#pragma unroll
    for (int pass = 0; pass < NMAX; ++pass) {
#pragma unroll
        for (int i = pass & 1; i + 1 < NMAX; i += 2) {
            float x = v[i], y = v[i + 1];
            bool sw = nan_last_greater(x, y);
            v[i] = sw ? y : x;
            v[i + 1] = sw ? x : y;
        }
    }
#pragma unroll
    for (int t = 0; t < NMAX; ++t)
        if (t < n) out[(int64_t)t * npix + p] = v[t];
}

// The reference's merge walk of two sorted series.
__device__ __noinline__ bool ks_walk(const float* x1, const float* x2, int n, const KsArgs& a) {
    int i1 = 0, i2 = 0;
    for (int iout = 0; iout < 2 * n;) {
        if (i1 == n) {
            ++i2;
        } else if (i2 == n || x1[i1] < x2[i2]) {
            ++i1;
        } else if (x1[i1] > x2[i2]) {
            ++i2;
        } else {  // a tie (or a comparison with NaN): both step
            ++i1;
            ++i2;
            ++iout;
        }
        ++iout;
        if (i2 < a.lo[i1] || i2 > a.hi[i1]) return false;
    }
    return true;
}

// A thread keeps the envelope of its pixel in registers and takes up to 32 neighbours
// through it.  With d the smallest t that has a lower bound, sample t has an upper bound
// only for t < n - d, so the bounds pair up: x2[s + d] > low[s], x2[s] < high[s] for
// s < ns = n - d, NS being ns rounded up to a multiple of 4.  The samples of a pixel are
// contiguous in shared memory (immediate offsets), at an odd pitch (consecutive pixels
// fall into different banks).  Bound by issue (71 % of the slots, 61 % of them for loads
// from shared memory) at 15 warps per SM: 512 x 512 pixels, 20 dates, 11 x 23 windows, 313
// us (a merge walk per thread, divergent and with bank conflicts: 3949 us).
template <int NS>
__global__ void __launch_bounds__(256) k_ks(const __grid_constant__ KsArgs a) {
    extern __shared__ float samp[];  // sorted samples [pixel][np], then the mask bits
    const int n = a.n, np = a.pitch, d = a.n - a.ns;
    const int wy = 2 * a.hy + 1, wx = 2 * a.hx + 1, W = wy * wx, nw = (wx + 31) >> 5, pw = (W + 31) >> 5;
    const int or0 = blockIdx.y * a.tile_r, oc0 = blockIdx.x * a.tile_c;
    const int or1 = min(or0 + a.tile_r, a.out_rows), oc1 = min(oc0 + a.tile_c, a.out_cols);
    // input region of the (unclamped) windows, intersected with the image
    const int rr0 = max(0, a.sy / 2 + or0 * a.sy - a.hy), cc0 = max(0, a.sx / 2 + oc0 * a.sx - a.hx);
    const int rr1 = min(a.rows, a.sy / 2 + (or1 - 1) * a.sy + a.hy + 1);
    const int cc1 = min(a.cols, a.sx / 2 + (oc1 - 1) * a.sx + a.hx + 1);
    const int rw = cc1 - cc0, rh = rr1 - rr0;
    uint32_t* bits = reinterpret_cast<uint32_t*>(samp + a.off_bits);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int tr = warp; tr < n * rh; tr += 8) {  // one warp per (date, row)
        const int t = tr / rh, r = tr - t * rh;
        const float* src = a.sorted + ((int64_t)t * a.rows + rr0 + r) * a.cols + cc0;
        float* dst = samp + r * rw * np + t;
        for (int c = lane; c < rw; c += 32)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst + c * np)), "l"(src + c)
                         : "memory");
    }
    const int tc = oc1 - oc0, npix = (or1 - or0) * tc;
    for (int i = threadIdx.x; i < npix * pw; i += blockDim.x) bits[i] = 0u;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const int items = npix * wy * nw;
    for (int it = threadIdx.x; it < items; it += blockDim.x) {
        const int rest = it / npix, pix = it - rest * npix;
        const int word = rest / wy, wa = rest - word * wy;
        const int pr = pix / tc;
        const int in_r = a.sy / 2 + (or0 + pr) * a.sy, in_c = a.sx / 2 + (oc0 + pix - pr * tc) * a.sx;
        uint32_t shp = 0u;
        if (in_r - a.hy >= 0 && in_r + a.hy + 1 <= a.rows && in_c - a.hx >= 0 && in_c + a.hx + 1 <= a.cols) {
            const float* x1 = samp + ((in_r - rr0) * rw + (in_c - cc0)) * np;
            float low[NS], high[NS];
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                const int il = s < a.ns ? a.env_lo[s + d] : -1, ih = s < a.ns ? a.env_hi[s] : -1;
                low[s] = il >= 0 ? x1[il] : -INFINITY;
                high[s] = ih >= 0 ? x1[ih] : INFINITY;
            }
            const bool special = !(fabsf(x1[n - 1] - x1[0]) < INFINITY);
            const int b0 = 32 * word, nb = min(wx - b0, 32);
            const float* q = samp + ((in_r - a.hy + wa - rr0) * rw + (in_c - a.hx - cc0) + b0) * np;
#pragma unroll 1
            for (int wb = 0; wb < nb; ++wb, q += np) {
                const float* qd = q + d;
                float f4[4] = {INFINITY, INFINITY, INFINITY, INFINITY};  // four short chains of minima
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    if (s < NS - 3 || s < a.ns) {
                        f4[2 * (s & 1)] = fminf(f4[2 * (s & 1)], qd[s] - low[s]);
                        f4[2 * (s & 1) + 1] = fminf(f4[2 * (s & 1) + 1], high[s] - q[s]);
                    }
                }
                const float f = fminf(fminf(f4[0], f4[1]), fminf(f4[2], f4[3]));
                bool ok = f > 0.f;
                // an equality, or a sample that is not finite
                if (f == 0.f || special || !(fabsf(q[n - 1] - q[0]) < INFINITY)) ok = ks_walk(x1, q, n, a);
                if (ok) shp |= 1u << wb;
            }
            if (wa == a.hy && a.hx >= b0 && a.hx < b0 + 32) shp &= ~(1u << (a.hx - b0));
        }
        if (shp) {  // into the pixel's stream, whose words the rows share
            const int at = wa * wx + 32 * word, sh = at & 31;
            uint32_t* w = bits + pix * pw + (at >> 5);
            atomicOr(w, shp << sh);
            if (sh && shp >> (32 - sh)) atomicOr(w + 1, shp >> (32 - sh));
        }
    }
    __syncthreads();
    for (int orow = or0; orow < or1; ++orow)
        write_mask_row(a.is_shp + ((int64_t)orow * a.out_cols + oc0) * W, bits + (orow - or0) * tc * pw, tc, W, pw,
                       threadIdx.x, blockDim.x);
}

template <int NS>
static dpl_status launch_ks(const KsArgs& a, dim3 grid, size_t smem, cudaStream_t s) {
    if constexpr (NS <= kMaxNslc) {
        if (a.ns > NS) return launch_ks<NS + 4>(a, grid, smem, s);
        DPL_CUDA_TRY(cudaFuncSetAttribute(k_ks<NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_ks<NS><<<grid, 256, smem, s>>>(a);
        return check_launch("k_ks");
    }
    return fail(DPL_ERR_UNSUPPORTED, "dpl_shp_ks: nslc > 64");
}

// ---------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

int64_t glrt_pitch(int64_t cols) { return (cols + 3) / 4 * 4; }

size_t glrt_workspace_size(int64_t rows, int64_t cols) {
    return align_up(256, 256) + align_up((size_t)rows * glrt_pitch(cols) * sizeof(float), 256);
}

dpl_status launch_glrt(const float* mean, const float* var, int64_t rows, int64_t cols, int hy, int hx, int sy,
                       int sx, int nslc, float threshold, uint8_t* is_shp, int* status, float* scale2,
                       cudaStream_t s) {
    const int wy = 2 * hy + 1, wx = 2 * hx + 1;
    if (wy > rows || wx > cols) return fail(DPL_ERR_INVALID_ARGUMENT, "GLRT window larger than the image");
    const int64_t pitch = glrt_pitch(cols);
    const int64_t npix = rows * cols;
    k_glrt_scale<<<ceil_div(npix, 256), 256, 0, s>>>(mean, var, rows, cols, pitch, scale2);
    DPL_CUDA_TRY(cudaGetLastError());

    GlrtArgs a{};
    a.rows = (int)rows;
    a.cols = (int)cols;
    a.hy = hy;
    a.hx = hx;
    a.sy = sy;
    a.sx = sx;
    a.out_rows = (int)(rows / sy);
    a.out_cols = (int)(cols / sx);
    a.nslc = nslc;
    a.thr = threshold;
    a.is_shp = is_shp;
    a.status = status;
    // the ratio test: 4 exp(threshold / nslc) in float32, and the largest scale whose
    // product with it stays finite.  A threshold of 0 (alpha 1) or a ratio beyond 1e12
    // leaves the float32 range in which the test's error bound holds: logarithms there.
    const double c = nslc > 0 ? std::exp((double)threshold / nslc) : 0.0;
    a.ratio = threshold > 0.f && c > 1.0 && c < 1e12;
    a.four_c = a.ratio ? (float)(4.0 * c) : 0.f;
    // the interval of s2 / s1: 2 c - 1 -+ 2 sqrt(c (c - 1)).  Its lower end is 1 / (4 c), and
    // the error bound of its test a part of the centre: up to c = 64 the two stay two orders
    // of magnitude apart (beyond, as with one or two dates, the ratio test)
    const double cm1 = nslc > 0 ? std::expm1((double)threshold / nslc) : 0.0;
    a.interval = a.ratio && c <= 64.0;
    a.center = a.interval ? (float)(2.0 * c - 1.0) : 0.f;
    a.half = a.interval ? (float)(2.0 * std::sqrt(c * cm1)) : 0.f;
    a.ratio_max = a.ratio ? (float)std::sqrt(1e37 / (4.0 * c)) : 0.f;
    if (a.out_rows == 0 || a.out_cols == 0) return DPL_OK;
    // pick the largest tile whose TMA box fits the 256-element box limit and ~96 KB smem
    int tr = 16, tc = 32;
    auto box_w = [&](int t) { return (int)((((int64_t)(t - 1) * sx + wx + 3) + 3) / 4 * 4); };
    auto box_h = [&](int t) { return (t - 1) * sy + wy; };
    while (tc > 1 && box_w(tc) > 256) tc /= 2;
    while (tr > 1 && box_h(tr) > 256) tr /= 2;
    // staged scale^2, then the tile's mask bits
    auto smem_for = [&](int r, int c) {
        return (size_t)box_w(c) * box_h(r) * sizeof(float) + 128 +
               (size_t)r * c * ((wy * wx + 31) / 32) * sizeof(uint32_t);
    };
    while (smem_for(tr, tc) > 96 * 1024 && (tr > 1 || tc > 1)) {
        if (tr >= tc && tr > 1) tr /= 2;
        else tc /= 2;
    }
    if (box_w(tc) > 256 || box_h(tr) > 256) return fail(DPL_ERR_UNSUPPORTED, "GLRT window too large for a TMA box");
    // the interface's limit, well above one pixel's needs here
    if ((size_t)2 * box_w(1) * box_h(1) * sizeof(float) + 128 + (size_t)wy * wx > 227 * 1024)
        return fail(DPL_ERR_UNSUPPORTED, "GLRT window too large for shared memory");
    a.tile_r = tr;
    a.tile_c = tc;
    a.box_w = box_w(tc);
    a.box_h = box_h(tr);

    EncodeTiledFn enc = get_encode_fn();
    if (!enc) return fail(DPL_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
    CUtensorMap map;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)(pitch * sizeof(float))};
    cuuint32_t box[2] = {(cuuint32_t)a.box_w, (cuuint32_t)a.box_h};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, scale2, dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(DPL_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
    const size_t smem = smem_for(tr, tc);
    dim3 grid(ceil_div(a.out_cols, tc), ceil_div(a.out_rows, tr));
    // one word per window row and a pixel per thread
    const bool plain = wx <= 32 && std::min(tr, a.out_rows) * std::min(tc, a.out_cols) >= 256;
    const auto kernel = plain ? k_glrt<true> : k_glrt<false>;
    DPL_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kernel<<<grid, 256, smem, s>>>(map, a);
    return check_launch("k_glrt");
}

}  // namespace dpl

using namespace dpl;

extern "C" size_t dpl_shp_glrt_workspace_size(int64_t rows, int64_t cols) { return glrt_workspace_size(rows, cols); }

extern "C" dpl_status dpl_shp_glrt(const float* mean, const float* var, int64_t rows, int64_t cols, int hy, int hx,
                                   int sy, int sx, int nslc, float threshold, uint8_t* is_shp, void* workspace,
                                   size_t workspace_bytes, dpl_stream_t stream) {
    if (rows <= 0 || cols <= 0 || hy < 0 || hx < 0 || sy <= 0 || sx <= 0)
        return fail(DPL_ERR_INVALID_ARGUMENT, "dpl_shp_glrt: bad shape");
    if (rows > INT32_MAX || cols > INT32_MAX) return fail(DPL_ERR_UNSUPPORTED, "dpl_shp_glrt: image too large");
    if (!mean || !var || !is_shp || !workspace) return fail(DPL_ERR_INVALID_ARGUMENT, "dpl_shp_glrt: null pointer");
    if (workspace_bytes < glrt_workspace_size(rows, cols))
        return fail(DPL_ERR_WORKSPACE, "dpl_shp_glrt: workspace too small");
    cudaStream_t s = (cudaStream_t)stream;
    Workspace ws{(char*)workspace, workspace_bytes};
    int* status = ws.take<int>(64);
    float* scale2 = ws.take<float>((size_t)rows * glrt_pitch(cols));
    DPL_CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(int), s));
    return launch_glrt(mean, var, rows, cols, hy, hx, sy, sx, nslc, threshold, is_shp, status, scale2, s);
}

size_t dpl::ks_workspace_size(int64_t nslc, int64_t rows, int64_t cols) {
    return align_up((size_t)nslc * rows * cols * sizeof(float), 256);
}

// shp/_ks.py:221-239: distances from 0.01 in steps of 0.001, the first whose Kolmogorov
// series (100 terms, n / 2 effective samples) is <= alpha.  The reference's operations in
// its order, so the distance is the same double: the power of two of `value` through pow()
// and the terms through exp(), as its interpreter evaluates them.  Host code: as a Python
// loop the scan took 4-7 ms a call, longer than the kernels.
extern "C" double dpl_ks_critical_distance(double nslc, double alpha) {
    const double n_eff = nslc / 2.0, sq = std::sqrt(n_eff);
    double cur = 0.01;
    while (cur <= 1.0) {
        const double value = cur * (sq + 0.12 + 0.11 / sq);
        const double scale = -2 * std::pow(value, 2.0);
        double pvalue = 0.0;
        for (int t = 1; t <= 100; ++t) {
            const double term = std::exp(scale * (double)(t * t));
            // the terms fall: below a quarter of the last place none changes the sum
            if (term <= pvalue * 0x1p-55) break;
            pvalue = t & 1 ? pvalue + term : pvalue - term;
        }
        pvalue = std::max(0.0, std::min(1.0, 2 * pvalue));
        if (pvalue <= alpha) return cur;
        cur += 0.001;
    }
    return 0.1;
}

extern "C" size_t dpl_shp_ks_workspace_size(int64_t nslc, int64_t rows, int64_t cols) {
    return ks_workspace_size(nslc, rows, cols);
}

extern "C" dpl_status dpl_shp_ks(const float* amp_stack, int64_t nslc, int64_t rows, int64_t cols, int hy, int hx,
                                 int sy, int sx, double cutoff, int is_sorted, uint8_t* is_shp, void* workspace,
                                 size_t workspace_bytes, dpl_stream_t stream) {
    if (nslc <= 0 || rows <= 0 || cols <= 0 || hy < 0 || hx < 0 || sy <= 0 || sx <= 0)
        return fail(DPL_ERR_INVALID_ARGUMENT, "dpl_shp_ks: bad shape");
    if (nslc > kMaxNslc) return fail(DPL_ERR_UNSUPPORTED, "dpl_shp_ks: nslc > 64");
    if (rows > INT32_MAX || cols > INT32_MAX) return fail(DPL_ERR_UNSUPPORTED, "dpl_shp_ks: image too large");
    if (!amp_stack || !is_shp || !workspace) return fail(DPL_ERR_INVALID_ARGUMENT, "dpl_shp_ks: null pointer");
    if (workspace_bytes < ks_workspace_size(nslc, rows, cols))
        return fail(DPL_ERR_WORKSPACE, "dpl_shp_ks: workspace too small");
    cudaStream_t s = (cudaStream_t)stream;
    const int n = (int)nslc;
    const int wy = 2 * hy + 1, wx = 2 * hx + 1;
    const int out_rows = (int)(rows / sy), out_cols = (int)(cols / sx);
    if (out_rows == 0 || out_cols == 0) return DPL_OK;
    if (2 * (n + 1) * sizeof(int) + (size_t)wy * wx * n * sizeof(float) > 200 * 1024)
        return fail(DPL_ERR_UNSUPPORTED, "dpl_shp_ks: window too large");
    // ECDF tables: T[k] = k-fold float64 sum of 1/n; admissible partner interval per i1
    std::vector<double> T(n + 1, 0.0);
    const double step = 1.0 / n;
    for (int k = 1; k <= n; ++k) T[k] = T[k - 1] + step;
    std::vector<int> lo(n + 1), hi(n + 1);
    for (int i1 = 0; i1 <= n; ++i1) {
        int l = n + 1, h = -1;
        for (int i2 = 0; i2 <= n; ++i2) {
            if (std::fabs(T[i1] - T[i2]) < cutoff) {
                l = std::min(l, i2);
                h = std::max(h, i2);
            }
        }
        lo[i1] = l;
        hi[i1] = h;
    }
    KsArgs a{};
    for (int i = 0; i <= n; ++i) {
        a.lo[i] = (int8_t)std::min(lo[i], 127);
        a.hi[i] = (int8_t)hi[i];
    }
    // m(t): the smallest i1 that admits t + 1 neighbour samples; n + 1 if none does (a
    // cutoff <= 0, which admits nothing: the walk's first step already leaves the band)
    for (int t = 0; t < n; ++t) a.env_hi[t] = -1;
    for (int t = n - 1; t >= 0; --t) {
        int m = 0;
        while (m <= n && hi[m] < t + 1) ++m;
        a.env_lo[t] = (int8_t)(m - 1);
        if (m >= 1 && m <= n) a.env_hi[m - 1] = (int8_t)t;  // the smallest such t is written last
    }
    int d = 0;  // the first sample with a lower bound
    while (d < n && a.env_lo[d] < 0) ++d;
    a.ns = n - d;
    Workspace ws{(char*)workspace, workspace_bytes};
    float* sorted = ws.take<float>((size_t)n * rows * cols);
    if (hi[0] < 0) {
        DPL_CUDA_TRY(cudaMemsetAsync(is_shp, 0, (size_t)out_rows * out_cols * wy * wx, s));
        return DPL_OK;
    }
    const int64_t npix = rows * cols;
    const float* src = amp_stack;
    if (!is_sorted) {
        dim3 g(ceil_div(npix, 128));
        if (n <= 16) k_sort_pixels<16><<<g, 128, 0, s>>>(amp_stack, n, npix, sorted);
        else if (n <= 32) k_sort_pixels<32><<<g, 128, 0, s>>>(amp_stack, n, npix, sorted);
        else k_sort_pixels<64><<<g, 128, 0, s>>>(amp_stack, n, npix, sorted);
        DPL_CUDA_TRY(cudaGetLastError());
        src = sorted;
    }
    a.sorted = src;
    a.n = n;
    a.rows = (int)rows;
    a.cols = (int)cols;
    a.hy = hy;
    a.hx = hx;
    a.sy = sy;
    a.sx = sx;
    a.out_rows = out_rows;
    a.out_cols = out_cols;
    a.is_shp = is_shp;
    // the largest tile of up to 8 x 32 pixels whose samples and mask bits leave room for
    // two CTAs per SM; windows too large for that get what one CTA can hold
    int tr = 8, tc = 32;
    auto region = [&](int r, int c) { return ((size_t)(r - 1) * sy + wy) * ((size_t)(c - 1) * sx + wx); };
    const auto bytes_for = [&](int r, int c, int pitch) {
        return region(r, c) * pitch * sizeof(float) + (size_t)r * c * ((wy * wx + 31) / 32) * sizeof(uint32_t);
    };
    // an odd pitch (no bank conflicts) wherever one pixel's window has room for it
    a.pitch = bytes_for(1, 1, n | 1) <= 227 * 1024 ? n | 1 : n;
    const auto smem_for = [&](int r, int c) { return bytes_for(r, c, a.pitch); };
    while (smem_for(tr, tc) > 110 * 1024 && (tr > 1 || tc > 1)) {
        if (tr * sy >= tc * sx && tr > 1) tr /= 2;
        else if (tc > 1) tc /= 2;
        else tr /= 2;
    }
    a.tile_r = tr;
    a.tile_c = tc;
    a.off_bits = (int)region(tr, tc) * a.pitch;
    return launch_ks<4>(a, dim3(ceil_div(out_cols, tc), ceil_div(out_rows, tr)), smem_for(tr, tc), s);
}

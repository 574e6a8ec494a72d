// Amplitude dispersion and PS selection: calc_ps_block (ps.py:169-244).
//
// One thread per pixel streams the N magnitudes once (coalesced across the warp,
// date-major input) and keeps them in registers for the second (variance) pass.
// The arithmetic reproduces numpy's float32 nanmean / nanstd exactly: sequential
// sums along axis 0, NaN entries replaced by 0, divisions by the count rounded
// once, no FMA contraction.  4N bytes in, 9 bytes out.
//
// Bound by HBM with the loads in flight: 2048 x 4096 pixels at N = 30 take 155 us (7.0
// TB/s, part of it from L2).  A pixel whose plain sum is a number has no NaN, so the
// replacement, its bookkeeping and the count run only where that sum is NaN (on every
// sample, issue-bound, 386 us); all loads are issued before the first sum.  A pixel with
// a NaN reads its samples again, eight loads in flight: with 1 % of the samples NaN, so
// that every warp takes both routes, the call takes 347 us where it takes 219 without
// NaNs (487 one load after the other).  Keeping that route's samples in registers as
// well took 280, but 2 to 20 % longer without NaNs.  Two or four pixels per thread, for
// wider loads, were slower at every size.
#include "dpl_common.cuh"

namespace dpl {

// the reference's last steps (ps.py:221-244) and the outputs of one pixel
struct PsOut {
    float thr;
    int thr_is_f64;
    double thr64;
    int64_t min_count;
    float* mean;
    float* disp;
    uint8_t* ps;

    __device__ __forceinline__ void write(int64_t p, float m, float ss, int cnt) const {
        const float sd = fsqrt(fdiv(ss, (float)cnt));
        float d = fdiv(sd, m);
        if (cnt < min_count) d = nanf("");
        if (!isfinite(m)) m = 0.f;
        if (!isfinite(d)) d = 0.f;
        bool is_ps = thr_is_f64 ? ((double)d < thr64) : (d < thr);
        if (d == 0.f) is_ps = false;
        mean[p] = m;
        disp[p] = d;
        ps[p] = is_ps ? 1 : 0;
    }
};

// any n: NaN samples replaced by 0 and left out of the count; x(t) loads sample t
template <class Sample>
__device__ __forceinline__ void ps_pixel(Sample&& x, int n, int64_t p, const PsOut& out) {
    float sum = 0.f;
    int cnt = 0;
#pragma unroll 8
    for (int t = 0; t < n; ++t) {
        const float v = x(t);
        const bool nan = isnan(v);
        const float xv = nan ? 0.f : v;
        cnt += nan ? 0 : 1;
        sum = t == 0 ? xv : fadd(sum, xv);
    }
    const float mean = fdiv(sum, (float)cnt);
    float ss = 0.f;
#pragma unroll 8
    for (int t = 0; t < n; ++t) {
        const float v = x(t);
        const float d = isnan(v) ? 0.f : fsub(v, mean);
        const float sq = fmul(d, d);
        ss = t == 0 ? sq : fadd(ss, sq);
    }
    out.write(p, mean, ss, cnt);
}

// NMAX - 8 < n <= NMAX; NMAX = 0: any n, the samples read twice
template <int NMAX>
__global__ void __launch_bounds__(256) k_ps_block(const float* __restrict__ mag, int n, int64_t npix, const PsOut out) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npix) return;
    auto sample = [&](int t) { return __ldg(mag + (int64_t)t * npix + p); };
    if constexpr (NMAX > 0) {
        float x[NMAX];
        const float* src = mag + p;
#pragma unroll
        for (int t = 0; t < NMAX; ++t) {
            x[t] = t < NMAX - 7 || t < n ? __ldg(src) : 0.f;
            src += npix;
        }
        float sum = x[0];
#pragma unroll
        for (int t = 1; t < NMAX; ++t)
            if (t < NMAX - 7 || t < n) sum = fadd(sum, x[t]);
        if (!isnan(sum)) {
            const float mean = fdiv(sum, (float)n);
            float ss = 0.f;
#pragma unroll
            for (int t = 0; t < NMAX; ++t) {
                if (t < NMAX - 7 || t < n) {
                    const float d = fsub(x[t], mean);
                    const float sq = fmul(d, d);
                    ss = t == 0 ? sq : fadd(ss, sq);
                }
            }
            out.write(p, mean, ss, n);
            return;
        }
    }
    ps_pixel(sample, n, p, out);
}

template <int NMAX>
static void launch_ps(int nmax, const float* mag, int n, int64_t npix, const PsOut& out, cudaStream_t s) {
    if constexpr (NMAX < 64) {
        if (nmax > NMAX) return launch_ps<NMAX + 8>(nmax, mag, n, npix, out, s);
    }
    k_ps_block<NMAX><<<ceil_div(npix, 256), 256, 0, s>>>(mag, n, npix, out);
}

}  // namespace dpl

using namespace dpl;

extern "C" dpl_status dpl_ps_block(const float* stack_mag, int64_t nslc, int64_t npix, float threshold,
                                   int threshold_is_f64, double threshold64, int64_t min_count, float* mean,
                                   float* amp_disp, uint8_t* ps, dpl_stream_t stream) {
    if (nslc <= 0 || npix < 0) return fail(DPL_ERR_INVALID_ARGUMENT, "dpl_ps_block: bad shape");
    if (npix == 0) return DPL_OK;
    if (!stack_mag || !mean || !amp_disp || !ps) return fail(DPL_ERR_INVALID_ARGUMENT, "dpl_ps_block: null pointer");
    cudaStream_t s = (cudaStream_t)stream;
    const int n = (int)nslc;
    const PsOut out{threshold, threshold_is_f64, threshold64, min_count, mean, amp_disp, ps};
    if (n <= 64) launch_ps<8>(n, stack_mag, n, npix, out, s);
    else k_ps_block<0><<<ceil_div(npix, 256), 256, 0, s>>>(stack_mag, n, npix, out);
    return check_launch("k_ps_block");
}

// Register-resident per-pixel solver for N <= K: a group of G warps solves one pixel
// (K = 16 or 32 with one warp, K = 64 with two warps); thread i of the group owns row i
// of each matrix in registers.
//
// Same algorithms, iteration rules and outputs as solve_pixel (solver.cuh), laid out
// for the register file instead of shared memory:
//   |Gamma| + 1e-6 I  -> symmetric sweep (Gauss-Jordan in the "sweep" form: after
//        sweeping every index the matrix holds -A^{-1}).  A non-positive pivot is
//        the reference's Cholesky failure (_core.py:466-472, 496-515): EVD fallback.
//   CRLB: the Fisher matrix (crlb.py:132-189) is swept the same way.
//   EMI: A - 0.99 I (A = |Gamma|^{-1} o C) is inverted by the Hermitian sweep, and
//        inverse iteration (_eigenvalues.py:139-205) is a matrix-vector product per
//        step.  The sweep's pivots are those of the Cholesky/LDL^H factorisation, so
//        a non-positive pivot is exactly "not positive definite": such a pixel is
//        listed for the LU pass (the reference's LU algorithm), as in solve_pixel.
//   EVD: power iteration on C o |C| with the rows in registers (_eigenvalues.py:93-136).
//
// What bounds it: no single pipe, but issue slots, the shared-memory reads of the
// broadcast columns (a 16-byte broadcast costs the SM about two cycles) and instruction
// fetch: code that a pixel runs once, unrolled, costs several times more cycles per
// instruction than the sweep loops, so options that few runs use (baseline lag, beta,
// zero-correlation threshold, zero entries in the temporal coherence) sit in rolled loops
// apart, and divergent stores are selects.
//
// Packed arithmetic: a row's K values are held as K / 2 pairs of neighbouring columns
// (complex rows as a real and an imaginary plane), and the sweeps, the matrix-vector
// product and the element-wise builds use two-wide multiply-adds (one issue slot for two
// IEEE operations).  Every element sees the operations of the scalar form in the same
// order: phases, CRLB and estimator are the same bit for bit.  One pixel-warp at K = 30,
// alone on the SM: a real sweep 2594 -> 2041 cycles, the Hermitian one 6982 -> 5268.
//
// 1034 x 1046 pixels at N = 30: 17.3 -> 13.9 ms.
//
// Register rotation keeps the sweeps in compact loops: before the steps k, k + 1 (k
// even), slot s of a row holds column (k + s) mod K, so the pivot columns are slots 0 and
// 1.  Step k updates in place; step k + 1 writes pair q - 1 from pair q (the shift by one
// pair costs nothing).  Both columns are broadcast through shared memory at position
// (row - k) mod K, so slot s reads position s.  Rows and columns N .. K - 1 are padded
// with the identity, whose steps change nothing.
#pragma once

namespace dpl {

// two floats in one 64-bit register pair, with two IEEE operations per instruction
typedef float2 f2;
__device__ __forceinline__ f2 f2_pack(float x, float y) { return make_float2(x, y); }
__device__ __forceinline__ float f2_lo(f2 v) { return v.x; }
__device__ __forceinline__ float f2_hi(f2 v) { return v.y; }
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ f2 f2_neg(f2 v) { return make_float2(-v.x, -v.y); }  // an operand modifier
__device__ __forceinline__ f2 f2_ld(const float* p, int q) { return reinterpret_cast<const float2*>(p)[q]; }
__device__ __forceinline__ void f2_ld2(const float* p, int q, f2& a, f2& b) {  // pairs 2q, 2q + 1
    const float4 t = reinterpret_cast<const float4*>(p)[q];
    a = f2_pack(t.x, t.y);
    b = f2_pack(t.z, t.w);
}
__device__ __forceinline__ void f2_st(float* p, int q, f2 v) { reinterpret_cast<float2*>(p)[q] = v; }

// Shared memory of a pixel group: three K x LD planes (Re and Im of the full Hermitian C,
// and |Gamma| or its inverse), a buffer for the broadcast columns (two halves of two
// planes) and vectors, and (two-warp groups) reduction slots.  LD is even with LD / 2
// odd: a thread per row reading pairs is conflict-free.
template <int K, int G>
struct RegShape {
    static constexpr int LD = (K / 2) % 2 ? K : K + 2;
    static constexpr int KB = (K + 3) & ~3;  // a plane of a broadcast column or vector
    static constexpr int NP = (K * (K - 1) / 2 + G - 1) / G;  // lower pairs per thread
    static constexpr int PLANE = K * LD;
    static constexpr int OFF_U = 3 * PLANE, OFF_X = OFF_U + 4 * KB;
    static constexpr int FLOATS = (OFF_X + (G == 64 ? 16 : 0) + 31) & ~31;
};

// A pixel group of G threads: G = 8, 16 or 32 lanes of one warp (a warp holds 32 / G
// pixels) or G = 64, two whole warps: row index, synchronisation, reductions.
template <int G>
struct Grp {
    int gl;         // thread (= row) index within the group, 0 .. G - 1
    int lane;       // lane within its warp
    int wig;        // warp within the group (G == 64)
    int bar;        // named barrier of the group (G == 64)
    int base;       // first lane of the group in its warp (G <= 32)
    unsigned mask;  // the group's lanes (G <= 32)
    float* x;       // reduction slots (shared memory, 16 floats)

    __device__ __forceinline__ void sync() const {
        if (G <= 32) {
            __syncwarp(mask);
        } else {
            __syncwarp();  // bar.sync counts a warp as arrived when any of its lanes arrives
            asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(64) : "memory");
        }
    }
    // sum over the group, the same value in every thread
    __device__ __forceinline__ float sum(float v) const {
        if (G <= 32) {
#pragma unroll
            for (int o = (G >> 1); o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
            return v;
        }
        v = warp_sum(v);
        if (lane == 0) x[wig] = v;
        sync();
        const float r = x[0] + x[1];
        sync();
        return r;
    }
    __device__ __forceinline__ float max(float v) const {
#pragma unroll
        for (int o = (G <= 32 ? G >> 1 : 16); o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(mask, v, o));
        if (G <= 32) return v;
        if (lane == 0) x[wig] = v;
        sync();
        const float r = fmaxf(x[0], x[1]);
        sync();
        return r;
    }
    __device__ __forceinline__ bool any(bool v) const {
        if (G <= 32) return __any_sync(mask, v);
        v = warp_any(v);
        if (lane == 0) x[2 + wig] = v ? 1.f : 0.f;
        sync();
        const bool r = x[2] + x[3] > 0.f;
        sync();
        return r;
    }
    // value of thread k (uniform k)
    __device__ __forceinline__ cfloat bcast(cfloat v, int k) const {
        if (G <= 32) return {__shfl_sync(mask, v.re, base + k), __shfl_sync(mask, v.im, base + k)};
        if (gl == k) {
            x[4] = v.re;
            x[5] = v.im;
        }
        sync();
        const cfloat r = cmake(x[4], x[5]);
        sync();
        return r;
    }
};

// 1/p to about an ulp: the approximate reciprocal refined by one Newton step.
__device__ __forceinline__ float frcp_nr(float p) {
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(p));
    return fmaf(r, fmaf(-p, r, 1.f), r);
}

// A power of two that takes the largest diagonal entry `top` of a positive definite matrix,
// and so every pivot of its sweep, to 1 or below (1 where it is there already).
__device__ __forceinline__ float r_scale(float top) {
    return top > 1.f && top < 1e30f ? __uint_as_float((253u - (__float_as_uint(top) >> 23)) << 23) : 1.f;
}

// The sweeps broadcast the pivot column through `buf`, two halves used alternately so
// that one barrier per step suffices: step k writes half k & 1, whose readers (step
// k - 2) all passed step k - 1's barrier before this thread did.

// Real symmetric sweep of the matrix whose row `gl` is g; on success g holds row `gl` of
// -A^{-1}.  Row k's 1 - 1/p loses p units of the last place where p > 1 (the CRLB's Fisher
// matrix, the shifted EMI matrix of a coherent pixel): the strided route, which stands in
// for a solver without that loss, scales them to pivots of 1 or below.  Returns false
// (uniformly) if any pivot was <= 0 (the remaining steps then run on meaningless values,
// without branching).  buf: 2 * KB floats.
template <int K, int G>
__device__ __forceinline__ bool r_sweep(f2 (&g)[K / 2], float* buf, const Grp<G>& gr) {
    constexpr int KB = RegShape<K, G>::KB;
    bool bad = false;  // uniform: every thread reads the same pivot
    int pos = gr.gl;
    gr.sync();  // earlier users of buf are done with it
#pragma unroll 1
    for (int k = 0; k < K; k += 2) {
        {
            const float g0 = f2_lo(g[0]);
            if (gr.gl < K) buf[pos] = g0;  // A[row][k] (= A[k][row])
            gr.sync();
            const float p = buf[0];
            bad |= !(p > 0.f);
            const float ip = frcp_nr(p);
            const bool me = gr.gl == k;
            // rows i != k: a_ij - (a_ik / p) a_kj; row k: a_kj / p, written as
            // a_kj - (1 - 1/p) a_kj so that every thread runs the same FMA
            const float t = me ? 1.f - ip : g0 * ip;
            const float last = me ? -ip : g0 * ip;
            const f2 nt = f2_neg(f2_pack(t, t));
#pragma unroll
            for (int q = 0; q < K / 4; ++q) {
                f2 x, y;
                f2_ld2(buf, q, x, y);
                g[2 * q] = f2_fma(nt, x, g[2 * q]);
                g[2 * q + 1] = f2_fma(nt, y, g[2 * q + 1]);
            }
            if (K % 4) g[K / 2 - 1] = f2_fma(nt, f2_ld(buf, K / 2 - 1), g[K / 2 - 1]);
            g[0] = f2_pack(last, f2_hi(g[0]));
        }
        {
            const float g1 = f2_hi(g[0]);
            float* b1 = buf + KB;
            if (gr.gl < K) b1[pos] = g1;
            gr.sync();
            const float p = b1[1];
            bad |= !(p > 0.f);
            const float ip = frcp_nr(p);
            const bool me = gr.gl == k + 1;
            const float t = me ? 1.f - ip : g1 * ip;
            const float last = me ? -ip : g1 * ip;
            const f2 nt = f2_neg(f2_pack(t, t));
            f2 first = f2_pack(0.f, 0.f);
#pragma unroll
            for (int q = 0; q < K / 4; ++q) {
                f2 x, y;
                f2_ld2(b1, q, x, y);
                if (q == 0) first = f2_fma(nt, x, g[0]);
                else g[2 * q - 1] = f2_fma(nt, x, g[2 * q]);
                g[2 * q] = f2_fma(nt, y, g[2 * q + 1]);
            }
            if (K % 4) g[K / 2 - 2] = f2_fma(nt, f2_ld(b1, K / 2 - 1), g[K / 2 - 1]);
            g[K / 2 - 1] = f2_pack(f2_lo(first), last);
        }
        pos -= 2;
        pos = pos < 0 ? pos + K : pos;
    }
    gr.sync();
    return !bad;
}

// Hermitian sweep: on success (re, im) hold row `gl` of -A^{-1}.  False if a pivot was
// <= 0.  buf: 4 * KB floats.
template <int K, int G>
__device__ __forceinline__ bool r_sweep_c(f2 (&re)[K / 2], f2 (&im)[K / 2], float* buf, const Grp<G>& gr) {
    constexpr int KB = RegShape<K, G>::KB;
    bool bad = false;  // uniform: every thread reads the same pivot
    int pos = gr.gl;
    gr.sync();
#pragma unroll 1
    for (int k = 0; k < K; k += 2) {
        {
            const float a0 = f2_lo(re[0]), c0 = f2_lo(im[0]);
            if (gr.gl < K) {  // A[row][k] = conj(A[k][row])
                buf[pos] = a0;
                buf[KB + pos] = c0;
            }
            gr.sync();
            const float p = buf[0];
            bad |= !(p > 0.f);
            const float ip = frcp_nr(p);
            const bool me = gr.gl == k;
            const float sr = a0 * ip, si = c0 * ip;
            const float tr = me ? 1.f - ip : sr, ti = me ? 0.f : si;
            const f2 ptr = f2_pack(tr, tr), pti = f2_pack(ti, ti);
            // slot s: a_ij - t a_kj, a_kj = conj(buffer entry s)
            auto update = [&](int q, f2 br, f2 bi) {
                re[q] = f2_fma(f2_neg(ptr), br, f2_fma(f2_neg(pti), bi, re[q]));
                im[q] = f2_fma(f2_neg(pti), br, f2_fma(ptr, bi, im[q]));
            };
#pragma unroll
            for (int q = 0; q < K / 4; ++q) {
                f2 r0, r1, i0, i1;
                f2_ld2(buf, q, r0, r1);
                f2_ld2(buf + KB, q, i0, i1);
                update(2 * q, r0, i0);
                update(2 * q + 1, r1, i1);
            }
            if (K % 4) update(K / 2 - 1, f2_ld(buf, K / 2 - 1), f2_ld(buf + KB, K / 2 - 1));
            re[0] = f2_pack(me ? -ip : sr, f2_hi(re[0]));
            im[0] = f2_pack(me ? 0.f : si, f2_hi(im[0]));
        }
        {
            float* b1 = buf + 2 * KB;
            const float a1 = f2_hi(re[0]), c1 = f2_hi(im[0]);
            if (gr.gl < K) {
                b1[pos] = a1;
                b1[KB + pos] = c1;
            }
            gr.sync();
            const float p = b1[1];
            bad |= !(p > 0.f);
            const float ip = frcp_nr(p);
            const bool me = gr.gl == k + 1;
            const float sr = a1 * ip, si = c1 * ip;
            const float tr = me ? 1.f - ip : sr, ti = me ? 0.f : si;
            const f2 ptr = f2_pack(tr, tr), pti = f2_pack(ti, ti);
            f2 fr = f2_pack(0.f, 0.f), fi = f2_pack(0.f, 0.f);
            auto update = [&](int q, f2 br, f2 bi) {  // pair q into pair q - 1
                const f2 x = f2_fma(f2_neg(ptr), br, f2_fma(f2_neg(pti), bi, re[q]));
                const f2 y = f2_fma(f2_neg(pti), br, f2_fma(ptr, bi, im[q]));
                if (q == 0) {
                    fr = x;
                    fi = y;
                } else {
                    re[q - 1] = x;
                    im[q - 1] = y;
                }
            };
#pragma unroll
            for (int q = 0; q < K / 4; ++q) {
                f2 r0, r1, i0, i1;
                f2_ld2(b1, q, r0, r1);
                f2_ld2(b1 + KB, q, i0, i1);
                update(2 * q, r0, i0);
                update(2 * q + 1, r1, i1);
            }
            if (K % 4) update(K / 2 - 1, f2_ld(b1, K / 2 - 1), f2_ld(b1 + KB, K / 2 - 1));
            re[K / 2 - 1] = f2_pack(f2_lo(fr), me ? -ip : sr);
            im[K / 2 - 1] = f2_pack(f2_lo(fi), me ? 0.f : si);
        }
        pos -= 2;
        pos = pos < 0 ? pos + K : pos;
    }
    gr.sync();
    return !bad;
}

// Publishes a vector as two planes (Re, Im) of KB floats.
template <int K, int G>
__device__ __forceinline__ void r_publish(float* vb, cfloat x, const Grp<G>& gr) {
    constexpr int KB = RegShape<K, G>::KB;
    gr.sync();
    if (gr.gl < K) {
        vb[gr.gl] = x.re;
        vb[KB + gr.gl] = x.im;
    }
    gr.sync();
}

// y_row = sum_j h_j x_j (row `gl` of a matrix in registers), even and odd columns summed
// apart; x published in vb
template <int K, int G>
__device__ __forceinline__ cfloat r_matvec(const f2 (&hr)[K / 2], const f2 (&hi)[K / 2], cfloat x, float* vb,
                                           const Grp<G>& gr) {
    constexpr int KB = RegShape<K, G>::KB;
    r_publish<K, G>(vb, x, gr);
    f2 ar = f2_pack(0.f, 0.f), ai = f2_pack(0.f, 0.f);
    auto step = [&](int q, f2 r, f2 i) {
        ar = f2_fma(hr[q], r, f2_fma(hi[q], f2_neg(i), ar));
        ai = f2_fma(hr[q], i, f2_fma(hi[q], r, ai));
    };
#pragma unroll
    for (int q = 0; q < K / 4; ++q) {
        f2 r0, r1, i0, i1;
        f2_ld2(vb, q, r0, r1);
        f2_ld2(vb + KB, q, i0, i1);
        step(2 * q, r0, i0);
        step(2 * q + 1, r1, i1);
    }
    if (K % 4) step(K / 2 - 1, f2_ld(vb, K / 2 - 1), f2_ld(vb + KB, K / 2 - 1));
    if (gr.gl >= K) return cmake(0.f, 0.f);  // lanes beyond the matrix
    return cmake(f2_lo(ar) + f2_hi(ar), f2_lo(ai) + f2_hi(ai));
}

// One pixel's input in registers: the diagonal entry of row `gl` and the lower pairs
// e = gl, gl + G, ... (planar sums, or entries of a full matrix).  Fetched for the next
// pixel while the current one's temporal coherence runs, when the matrix rows are dead.
template <int K, int G>
struct RegFetch {
    float2 v[RegShape<K, G>::NP];
    float2 d;
    __device__ __forceinline__ void load(const PixArgs& a, int64_t p, const uint16_t* ptab, int gl) {
        const int n = a.n, npairs = n * (n - 1) / 2;
        d = make_float2(0.f, 0.f);
        if (a.Cplanar) {
            const float* src = a.Cplanar + p * n * n;
            if (gl < n) d.x = src[gl];
            src += n;
            if (n & 1) {  // the pairs lie on 4-byte boundaries in every other pixel
#pragma unroll
                for (int i = 0; i < RegShape<K, G>::NP; ++i) {
                    const int e = gl + i * G;
                    v[i] = e < npairs ? make_float2(src[2 * e], src[2 * e + 1]) : make_float2(0.f, 0.f);
                }
            } else {
#pragma unroll
                for (int i = 0; i < RegShape<K, G>::NP; ++i) {
                    const int e = gl + i * G;
                    v[i] = e < npairs ? reinterpret_cast<const float2*>(src)[e] : make_float2(0.f, 0.f);
                }
            }
        } else {
            const float2* src = reinterpret_cast<const float2*>(a.Cin) + p * n * n;
            if (gl < n) d = src[gl * n + gl];
#pragma unroll
            for (int i = 0; i < RegShape<K, G>::NP; ++i) {
                const int e = gl + i * G;
                const uint32_t rc = e < npairs ? ptab[e] : 0u;
                v[i] = src[(rc & 0xff) * n + (rc >> 8)];
            }
        }
    }
};

// Normalising iteration x <- op(v) / |op(v)| until |x - v| <= 1e-5 or 49 steps
// (the reference's while-loop: iteration count starts at 1, stops below 50).  Adds the
// steps taken to `steps`; returns the last step's difference (NaN also ends the loop).
template <int G, class Op>
__device__ __forceinline__ float r_iterate(cfloat& v, const Grp<G>& gr, int& steps, Op&& op) {
    float diff = 1.f;
    for (int it = 1; diff > 1e-5f && it < 50; ++it) {
        cfloat x = op(v);
        const float inv = rsqrtf(gr.sum(cabs2(x)));
        x = cscale(x, inv);
        diff = sqrtf(gr.sum(cabs2(csub(x, v))));
        v = x;
        ++steps;
    }
    return diff;
}

// Full solve for one pixel whose Hermitian coherence matrix is in the planes Cr, Ci (both
// triangles) and whose |Gamma| is in Gs off the diagonal.  A pixel whose shifted EMI
// matrix is not positive definite is listed and left for the LU pass (or the plain form).
// `fetch` loads the group's next pixel.  kScale: the matrices are scaled (r_sweep), as every
// launch with an ill_list is; that list is looked up at run time in all instances, because
// the others compile to slower code without it (N = 30 by 1 %, N = 44 by 5 %).
template <int K, int G, bool kScale, class Fetch>
__device__ __forceinline__ void solve_pixel_reg(const PixArgs& a, int64_t p, float* Cr, float* Ci, float* Gs, float* U,
                                                const uint16_t* ptab, const Grp<G>& gr, Fetch&& fetch) {
    using S = RegShape<K, G>;
    constexpr int LD = S::LD, KB = S::KB;
    const int n = a.n, me = gr.gl;
    const bool row = me < n, act = me < K;  // a row of the matrix; a row of the padded one
    const int mrow = act ? me : 0;
    float* cr = Cr + mrow * LD;
    float* ci = Ci + mrow * LD;
    float* Gi = Gs + mrow * LD;
    if (a.closure && me < n - 2) {
        const cfloat c01 = cmake(Cr[me * LD + me + 1], Ci[me * LD + me + 1]);
        const cfloat c12 = cmake(Cr[(me + 1) * LD + me + 2], Ci[(me + 1) * LD + me + 2]);
        const cfloat c02 = cmake(Cr[me * LD + me + 2], Ci[me * LD + me + 2]);
        const cfloat c = cmulc(cmul(c01, c12), c02);
        a.closure[p * (n - 2) + me] = atan2f(c.im, c.re);
    }
    const int ref = a.crlb_ref;
    bool inv_nan = true;
    bool crlb_ok = false;
    float dg = 0.f, unscale = 1.f;
    if (!(a.use_evd && !a.compute_crlb)) {
        // |Gamma| + 1e-6 I -> -|Gamma|^{-1} (round 0), then the CRLB's Fisher matrix
        // FIM = 2L (Gamma o Gamma^{-1} - I), row/col `ref` -> identity, + 1e-6 I (round 1).
        // Gs holds |Gamma| during round 0 and |Gamma|^{-1} afterwards.
        float gdiag = 0.f;
        if (row) {
            gdiag = s_gamma(a, cmake(cr[me], ci[me]), true);
            Gi[me] = fadd(gdiag, 1e-6f);
        } else if (act) {
            Gi[me] = 1.f;
        }
        f2 g[K / 2];
#pragma unroll
        for (int q = 0; q < K / 2; ++q) g[q] = f2_ld(Gi, q);
#pragma unroll 1
        for (int round = 0; round < 2; ++round) {
            const bool ok = r_sweep<K, G>(g, U, gr);
            if (round == 1) {
                crlb_ok = ok;
#pragma unroll
                for (int q = 0; q < K / 2; ++q) {
                    if (me == 2 * q) dg = f2_lo(g[q]);
                    if (me == 2 * q + 1) dg = f2_hi(g[q]);
                }
                break;
            }
            inv_nan = !ok;
            if (ok) {
                f2 z = f2_pack(0.f, 0.f);  // NaN if any entry is NaN or infinite
#pragma unroll
                for (int q = 0; q < K / 2; ++q) z = f2_fma(g[q], f2_pack(0.f, 0.f), z);
                const float zs = f2_lo(z) + f2_hi(z);
                if (gr.any(row && isnan(zs))) {
                    bool nan = false;
#pragma unroll
                    for (int q = 0; q < K / 2; ++q) nan |= isnan(f2_lo(g[q])) || isnan(f2_hi(g[q]));
                    inv_nan = gr.any(row && nan);
                }
            }
            if (inv_nan) break;  // Gs keeps its finite padding
            // keep |Gamma|^{-1} and build the FIM in place of it; the identity rows (the
            // reference's, the padding) are 0 with 1 on the diagonal
            const bool unit = me == ref || !row;
            const float f = unit ? 0.f : a.crlb_factor;
            const float dsub = unit ? 0.f : 1.f, dadd = unit ? 1.f : 1e-6f;
            if (row) {
                Gi[me] = gdiag;
                if (a.compute_crlb) Gi[ref] = 0.f;
            }
            const f2 ff = f2_pack(f, f), minus = f2_pack(-1.f, -1.f);
            float fd = 0.f;  // the diagonal entry
#pragma unroll
            for (int q = 0; q < K / 2; ++q) {
                const f2 ginv = f2_mul(g[q], minus);
                const f2 gm = f2_ld(Gi, q);
                if (act) f2_st(Gi, q, ginv);
                const f2 y = f2_mul(gm, ginv);
                float y0 = f2_lo(y), y1 = f2_hi(y);
                if (me == 2 * q) y0 = fsub(y0, dsub);
                if (me == 2 * q + 1) y1 = fsub(y1, dsub);
                const f2 x = f2_mul(ff, f2_pack(y0, y1));
                float x0 = f2_lo(x), x1 = f2_hi(x);
                if (me == 2 * q) x0 = fadd(x0, dadd);
                if (me == 2 * q + 1) x1 = fadd(x1, dadd);
                g[q] = f2_pack(x0, x1);
                if (me == 2 * q) fd = x0;
                if (me == 2 * q + 1) fd = x1;
            }
            if (!a.compute_crlb) break;
            if constexpr (kScale) {  // see r_sweep: pivots of 1 or below
                unscale = r_scale(gr.max(fd));
                const f2 c = f2_pack(unscale, unscale);
#pragma unroll
                for (int q = 0; q < K / 2; ++q) g[q] = f2_mul(g[q], c);
            }
        }
    }
    const bool evd = a.use_evd || inv_nan;
    const float var = kScale ? -dg * unscale : -dg;
    if (row) a.crlb[p * n + me] = !a.compute_crlb || me == ref ? 0.f : (crlb_ok ? sqrtf(var) : nanf(""));

    // One matrix (re, im) and one iteration for both estimators, the matrix formed as
    // C o Gs: EMI iterates with -(A - 0.99 I)^{-1} (the negated sweep result), its
    // shifted diagonal put into Gs against a diagonal of 1 in C for the time of the
    // build; EVD iterates with C o |C|, |C| put into Gs.
    const int npairs = n * (n - 1) / 2;
    const float cd = cr[mrow], gd = Gi[mrow];
    if (!evd) {
        if (act) {
            Gi[me] = row ? fsub(cd * gd, 0.99f) : 1.f;
            cr[me] = 1.f;
        }
    } else {
        gr.sync();
        for (int e = me; e < npairs; e += G) {
            const uint32_t rc = ptab[e];
            const int r = rc & 0xff, c = rc >> 8;
            const float x = Cr[r * LD + c], y = Ci[r * LD + c];
            const float m = sqrtf(fmaf(x, x, y * y));
            Gs[r * LD + c] = m;
            Gs[c * LD + r] = m;
        }
        if (row) Gi[me] = sqrtf(fmaf(cd, cd, ci[me] * ci[me]));
        gr.sync();
    }
    f2 re[K / 2], im[K / 2];
#pragma unroll
    for (int q = 0; q < K / 2; ++q) {
        const f2 gq = f2_ld(Gi, q);
        re[q] = f2_mul(f2_ld(cr, q), gq);
        im[q] = f2_mul(f2_ld(ci, q), gq);
    }
    if (!evd) {
        if constexpr (kScale) {  // see r_sweep: pivots of 1 or below (the iterates are normalised)
            const float top = gr.max(act ? Gi[me] : 0.f), scale = r_scale(top);
            const f2 c = f2_pack(scale, scale);
#pragma unroll
            for (int q = 0; q < K / 2; ++q) {
                re[q] = f2_mul(re[q], c);
                im[q] = f2_mul(im[q], c);
            }
        }
        if (act) {
            Gi[me] = gd;
            cr[me] = cd;
        }
        if (!r_sweep_c<K, G>(re, im, U, gr)) {
            // not positive definite: the LU pass, or the plain form's own decision
            if (me == 0) {
                if (a.ill_list) a.ill_list[atomicAdd(a.ill_count, 1)] = (int)p;
                else a.fb_list[atomicAdd(a.fb_count, 1)] = (int)p;
            }
            fetch();
            return;
        }
    }
    cfloat v = row ? cmake(1.f / sqrtf((float)n), 0.f) : cmake(0.f, 0.f);
    float lambda;
    int steps = 0;
    const float sgn = evd ? 1.f : -1.f;
    auto op = [&](cfloat x) { return cscale(r_matvec<K, G>(re, im, x, U, gr), sgn); };
    bool warm = false;
    if (a.vstart && !evd) {
        // learned starting vector; plain EMI (constant start) if it is unusable or the
        // iteration from it does not meet the stopping rule
        const cfloat w0 = row ? a.vstart[p * n + me] : cmake(0.f, 0.f);
        const float w2 = gr.sum(cabs2(w0));
        if (w2 > 0.f && w2 <= 3.4e38f) {
            v = cscale(w0, 1.f / sqrtf(w2));
            warm = true;
        }
    }
    float diff = r_iterate<G>(v, gr, steps, op);
    if (!(diff <= 1e-5f) && warm) {  // a warm start that misses the rule (or goes NaN): plain EMI
        v = row ? cmake(1.f / sqrtf((float)n), 0.f) : cmake(0.f, 0.f);
        diff = r_iterate<G>(v, gr, steps, op);
    }
    // ill-conditioned for the explicit inverses, or not decided by them: listed for the
    // plain form's solver.  The others' errors against FP64 are the plain form's: over N = 5 to
    // 64, windows of 63 to 253 samples, decaying, coherent (0.8 to 0.99) and EVD scenes the
    // root mean squares of the CRLB agree to 4 % and those of the phases to 5 % or, near the
    // last place (2e-7 rad), 11 %; no phase comes out more than 1e-4 rad worse.
    if (a.ill_list && (!a.use_evd || a.compute_crlb)) {
        const bool ill = gr.any(row && gd > 32.f);
        if ((inv_nan || ill || (!evd && steps > 24)) && me == 0) a.ill_list[atomicAdd(a.ill_count, 1)] = (int)p;
    }
    // 49 steps without meeting the stopping rule (a NaN difference stops the loop, as in
    // the reference): listed for the dense eigensolver
    if (diff > 1e-5f && a.nc_list && me == 0) a.nc_list[atomicAdd(a.nc_count, 1)] = (int)p;
    if (!evd) {
        // lambda = Re v^H A v, A_ij = |Gamma|^{-1}_ij C_ij
        r_publish<K, G>(U, v, gr);
        f2 ar = f2_pack(0.f, 0.f), ai = f2_pack(0.f, 0.f);
#pragma unroll
        for (int q = 0; q < K / 2; ++q) {
            const f2 gq = f2_ld(Gi, q);
            const f2 hr = f2_mul(f2_ld(cr, q), gq), hi = f2_mul(f2_ld(ci, q), gq);
            const f2 xr = f2_ld(U, q), xi = f2_ld(U + KB, q);
            ar = f2_fma(hr, xr, f2_fma(hi, f2_neg(xi), ar));
            ai = f2_fma(hr, xi, f2_fma(hi, xr, ai));
        }
        const cfloat acc = row ? cmake(f2_lo(ar) + f2_hi(ar), f2_lo(ai) + f2_hi(ai)) : cmake(0.f, 0.f);
        const float n2 = gr.sum(cabs2(v));
        lambda = gr.sum(v.re * acc.re + v.im * acc.im);
        v = cscale(v, sqrtf((float)n) / sqrtf(n2));
    } else {
        const cfloat y = op(v);
        lambda = gr.sum(v.re * y.re + v.im * y.im);
    }
    fetch();  // the matrix rows are dead: the next pixel's values travel during what follows
    // reference to reference_idx
    const cfloat rot = cconj(fphasor(gr.bcast(v, a.ref_idx)));
    v = cmul(v, rot);
    if (row) a.vout[p * n + me] = v;
    if (me == 0) {
        a.eig[p] = lambda;
        a.est[p] = evd ? 0 : 1;
        if (a.iters) a.iters[p] = (int16_t)steps;
    }
    // temporal coherence |mean over pairs c < r of conj(phasor(C_rc) w_c conj(w_r))|.
    // Thread i takes the pairs (i, j), j = i + d mod n, d = 1 .. n / 2: each pair once and
    // every thread as many.  With x = phasor(C_ij) w_j the pair adds x conj(w_i) where
    // i < j and its conjugate where i > j: the real part needs the sum of the x, the
    // imaginary part their sum with the sign of j - i.  A zero or NaN entry makes the sums
    // NaN: those pixels (and all with a baseline lag, which zeroes entries) take the
    // pairs one by one and leave NaN pairs out.
    const cfloat w = fphasor(v);
    r_publish<K, G>(U, w, gr);
    float sre = 0.f, sim = 0.f, cnt = (float)npairs;
    if (row) {
        float pr = 0.f, pi = 0.f, qr = 0.f, qi = 0.f;
        const int half = (n - 1) / 2 + ((n & 1) == 0 && me < n / 2 ? 1 : 0);
#pragma unroll 2
        for (int d = 1; d <= half; ++d) {
            int j = me + d;
            const bool wrap = j >= n;
            j = wrap ? j - n : j;
            const float xr = cr[j], xi = ci[j], wr = U[j], wi = U[KB + j];
            const float s = rsqrtf(xr * xr + xi * xi);
            const float ur = xr * wr - xi * wi, ui = xr * wi + xi * wr;
            const float t = wrap ? -s : s;
            pr = fmaf(s, ur, pr);
            pi = fmaf(s, ui, pi);
            qr = fmaf(t, ur, qr);
            qi = fmaf(t, ui, qi);
        }
        sre = w.re * pr + w.im * pi;
        sim = w.re * qi - w.im * qr;
    }
    sre = gr.sum(sre);
    sim = gr.sum(sim);
    if (a.baseline_lag > 0 || isnan(sre + sim)) {
        sre = sim = cnt = 0.f;
#pragma unroll 1
        for (int e = me; e < npairs; e += G) {
            const uint32_t rc = ptab[e];
            const int r = rc & 0xff, c = rc >> 8;
            const cfloat u = fphasor(cmake(Cr[r * LD + c], Ci[r * LD + c]));
            const cfloat t = cconj(cmulc(cmul(u, cmake(U[c], U[KB + c])), cmake(U[r], U[KB + r])));
            if (!cisnan(t)) {
                sre += t.re;
                sim += t.im;
                cnt += 1.f;
            }
        }
        sre = gr.sum(sre);
        sim = gr.sum(sim);
        cnt = gr.sum(cnt);  // exact: at most 2016 pairs
    }
    if (me == 0) {
        const float tc = hypotf(sre / cnt, sim / cnt);
        a.tcoh[p] = isfinite(tc) ? tc : 0.f;
    }
}

// Solve-only pass over all pixels with the register solver (n <= K), one pixel per
// group of G threads.  The coherence comes planar (diagonal, then (Re, Im) of the
// lower pair (i, j), i > j, at o = i(i-1)/2 + j) or as full (npix, n, n) matrices
// of which the lower triangle is read.
// Two CTAs per SM (128 registers) wherever two CTAs' shared memory fits, K <= 46: the
// two-warp instances would take more registers and one CTA.
template <int K, int G, bool kScale>
__global__ void __launch_bounds__(256, (G == 64 && K > 46) ? 1 : 2) k_solve_reg(PixArgs a) {
    using S = RegShape<K, G>;
    constexpr int LD = S::LD;
    extern __shared__ __align__(16) float reg_smem[];
    const int warp = threadIdx.x >> 5;
    Grp<G> gr;
    gr.lane = threadIdx.x & 31;
    int group, ngroups;
    if (G <= 32) {
        constexpr int per_warp = 32 / (G <= 32 ? G : 32);
        ngroups = (blockDim.x >> 5) * per_warp;
        group = warp * per_warp + gr.lane / G;
        gr.base = gr.lane & ~(G - 1);
        gr.mask = G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << gr.base;
        gr.wig = 0;
        gr.gl = gr.lane - gr.base;
        gr.bar = 0;
    } else {
        ngroups = (blockDim.x >> 5) / 2;
        group = warp / 2;
        gr.base = 0;
        gr.mask = 0xffffffffu;
        gr.wig = warp - group * 2;
        gr.gl = gr.wig * 32 + gr.lane;
        gr.bar = 1 + group;
    }
    float* Cr = reg_smem + group * S::FLOATS;
    float* Ci = Cr + S::PLANE;
    float* Gs = Ci + S::PLANE;
    float* U = Cr + S::OFF_U;
    gr.x = Cr + S::OFF_X;
    uint16_t* ptab = reinterpret_cast<uint16_t*>(reg_smem + ngroups * S::FLOATS);  // shared by the CTA: r | c << 8
    const int n = a.n, lag = a.baseline_lag, me = gr.gl;
    const int npairs = n * (n - 1) / 2;
    for (int i = threadIdx.x; i < ngroups * S::FLOATS; i += blockDim.x) reg_smem[i] = 0.f;  // the padding stays 0
    for (int o = threadIdx.x; o < npairs; o += blockDim.x) {
        int r = (int)((sqrtf(8.f * o + 1.f) + 1.f) * 0.5f);  // o = r(r-1)/2 + c, 0 <= c < r
        while (r * (r - 1) / 2 > o) --r;
        while ((r + 1) * r / 2 <= o) ++r;
        ptab[o] = (uint16_t)(r | (o - r * (r - 1) / 2) << 8);
    }
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * ngroups;
    RegFetch<K, G> in;
    int64_t p = (int64_t)blockIdx.x * ngroups + group;
    if (p < a.npix) in.load(a, p, ptab, me);
    for (; p < a.npix; p += stride) {
        gr.sync();
        // the planar sums are unnormalised: C_ij = numer_ij r_i r_j with r = 1 / sqrt(amp)
        // (amp = the diagonal sum), 0 where r_i r_j >= 1e6 (covariance.py:131-142)
        const bool raw = a.Cplanar && !a.planar_norm;
        if (raw) {
            const float rme = me < n ? __frsqrt_rn(in.d.x) : 0.f;
            if (me < n) U[me] = rme;
            gr.sync();
            const float f = rme * rme;
            in.d.x = f < 1e6f ? in.d.x * f : 0.f;
        }
        if (me < n) {
            Cr[me * LD + me] = in.d.x;
            Ci[me * LD + me] = in.d.y;
        }
#pragma unroll
        for (int i = 0; i < S::NP; ++i) {
            const int e = me + i * G;
            if (e < npairs) {
                const uint32_t rc = ptab[e];
                const int r = rc & 0xff, c = rc >> 8;
                cfloat v = cmake(in.v[i].x, in.v[i].y);
                if (raw) {
                    const float f = U[r] * U[c];
                    v = f < 1e6f ? cscale(v, f) : cmake(0.f, 0.f);
                }
                Cr[r * LD + c] = v.re;
                Ci[r * LD + c] = v.im;
                Cr[c * LD + r] = v.re;
                Ci[c * LD + r] = -v.im;
                const float gm = s_abs_approx(v);
                Gs[r * LD + c] = gm;
                Gs[c * LD + r] = gm;
            }
        }
        // options that few runs use, apart from the unrolled code: the baseline lag, and
        // |Gamma| with a beta or a zero-correlation threshold
        if (lag > 0 || a.beta_on || a.zct > 0.f) {
#pragma unroll 1
            for (int e = me; e < npairs; e += G) {
                const uint32_t rc = ptab[e];
                const int r = rc & 0xff, c = rc >> 8;
                if (lag > 0 && r - c >= lag) Cr[r * LD + c] = Ci[r * LD + c] = Cr[c * LD + r] = Ci[c * LD + r] = 0.f;
                const float gm = s_gamma(a, cmake(Cr[r * LD + c], Ci[r * LD + c]), false);
                Gs[r * LD + c] = gm;
                Gs[c * LD + r] = gm;
            }
        }
        gr.sync();
        const int64_t next = p + stride;
        solve_pixel_reg<K, G, kScale>(a, p, Cr, Ci, Gs, U, ptab, gr, [&]() {
            in.load(a, next < a.npix ? next : p, ptab, me);  // unconditional: the old values die here
        });
    }
}

// Host launch of the instance with K slots and G threads per pixel: 8 warps per CTA,
// 256 / G pixel groups; a persistent grid of at most 8 waves.
template <int K, int G, bool kScale>
dpl_status launch_solve_reg_kl(const PixArgs& a, cudaStream_t s) {
    const int warps = 8;
    const int groups = warps * 32 / G;
    const size_t smem = (size_t)groups * RegShape<K, G>::FLOATS * sizeof(float) + (size_t)a.n * (a.n - 1) / 2 * sizeof(uint16_t);
    if (smem > 227 * 1024) return fail(DPL_ERR_UNSUPPORTED, "register solver: shared memory exceeds the SM limit");
    int dev = 0, sms = 0;
    DPL_CUDA_TRY(cudaGetDevice(&dev));
    DPL_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const auto kernel = k_solve_reg<K, G, kScale>;
    DPL_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    DPL_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, warps * 32, smem));
    const int64_t resident = (int64_t)std::max(1, per_sm) * std::max(1, sms);
    const int64_t grid = std::min<int64_t>((a.npix + groups - 1) / groups, resident * 8);
    kernel<<<(unsigned)std::max<int64_t>(grid, 1), warps * 32, smem, s>>>(a);
    return check_launch("k_solve_reg");
}

template <int K, int G>
dpl_status launch_solve_reg_k(const PixArgs& a, cudaStream_t s) {
    return a.ill_list ? launch_solve_reg_kl<K, G, true>(a, s) : launch_solve_reg_kl<K, G, false>(a, s);
}

}  // namespace dpl

// Non-convergence fallback: a dense Hermitian eigensolver for the pixels whose eigen-
// iteration missed its stopping rule.
//
// The reference iterates at most 49 times and returns the last iterate, with no flag
// (phase_link/_eigenvalues.py:194-202).  Where the two eigenvalues nearest the target
// are close, that iterate is still a mix of their eigenvectors.  Here such pixels are
// listed by the solvers and solved again, by one, two or four warps per pixel:
//   EMI: |Gamma| (+ beta I, zero threshold) + 1e-6 I is inverted in double precision
//        (the symmetric sweep operator on its lower triangle), A = |Gamma|^{-1} o C,
//        and the eigenvector is the one whose eigenvalue is nearest the inverse
//        iteration's shift 0.99 (the vector that iteration converges to), scaled to
//        norm sqrt(N) (_core.py:486-490).
//   EVD: A = C o |C|; the eigenvector of the eigenvalue of largest magnitude (the one
//        power iteration converges to), unit norm.
// Only one eigenpair is wanted, so the solver is the one LAPACK's subset drivers use
// (Golub & Van Loan, Matrix Computations, sections 8.3-8.4): Householder reduction of A
// to a real symmetric tridiagonal T = Q^H A Q, the wanted eigenvalue of T by Sturm-
// sequence multisection (32 shifts per round, one per lane), its eigenvector by inverse
// iteration on T - lambda I (Gaussian elimination with partial pivoting), and Q applied
// to it.  It runs in float32 on the float32 A.  The pixel is then referenced and its
// temporal coherence recomputed as in the solvers, and flagged.
#pragma once

namespace dpl {

constexpr int kEighMaxN = 64;
constexpr int kEighSmallN = 16;  // up to here one or two warps per pixel, above it four

// Warps of one pixel's CTA.  A pixel is a chain of ~3 n dependent phases and the list is
// mostly short, so the kernel's time is a pixel's latency, not its arithmetic: the phases
// that have n^2 / 2 independent elements are spread over the CTA's threads, and the FP64
// pipe, which takes 64 cycles for any warp instruction and has one unit per quarter of the
// SM, is used in all four quarters.  244 pixels at N = 45 and 1882 at N = 30 take 181 and
// 250 us with four warps and a table of the triangle (two warps: 222 and 239; one warp that
// walks the triangles by division-free row steps: 483 and 389).  At N <= 16 a second warp
// brings 3 pixels of N = 10 from 37 to 30 us, but 14839 pixels of N = 15, where the SM's
// issue slots are the limit, from 279 to 490 us: k_eigh_small takes one warp per pixel
// (274 us) once the list is longer than the grid.  Between N = 17 and 28 the two kernels
// lie close: the small one takes 2 to 8 % off a whole call with long lists (400 x 400
// pixels, EVD) and adds up to 3 % to one with short lists (64 x 64).
template <int W>
struct EighCta {
    static constexpr int T = 32 * W;
    int tid, lane, warp;
    __device__ __forceinline__ void sync() const {
        if (W == 1) __syncwarp();
        else __syncthreads();
    }
};

// Shared-memory layout of one pixel: C and A (n x ld complex, ld odd; the double |Gamma|
// work matrix shares A's storage, element for element, until A is formed), the per-pixel
// vectors, and the (row, column) of each element of a lower triangle walked row by row.
struct EighLayout {
    int ld;
    size_t off_C, off_A, off_vec, off_tri, bytes;
};

// the vectors of one pixel, each n long (padded to a multiple of two)
struct EighVec {
    cfloat* pw0;    // p = A v of the current Householder step, even and odd columns' sums;
    cfloat* pw1;    //   before that the inverse's column k and its multiple (doubles)
    cfloat* tau;    // Householder scalars
    cfloat* u;      // the current Householder vector; phasors of the result
    cfloat* w;      // each warp's copy of the current step's w
    float* d;       // diagonal of T
    float* e;       // off-diagonal of T
    float* e2;      // its squares
    float* r;       // right-hand side, then the eigenvector of T
    float* u0;      // elimination rows of T - lambda I (in pw0 and pw1, which are free then)
    float* u1;
    float* u2;
    float* m;       // elimination multipliers
    float* pair;    // the eigenvalues on both sides of the shift
    unsigned short* tri;  // row << 8 | column of the triangle's elements
};

inline int eigh_pad(int n) { return (n + 1) & ~1; }

inline EighLayout make_eigh_layout(int n, int warps) {
    EighLayout L{};
    L.ld = n | 1;
    const size_t np = (size_t)eigh_pad(n);
    size_t o = 0;
    auto take = [&](size_t bytes) {
        size_t at = o;
        o = align_up(o + bytes, 16);
        return at;
    };
    L.off_C = take((size_t)n * L.ld * sizeof(cfloat));
    L.off_A = take((size_t)n * L.ld * sizeof(cfloat));
    L.off_vec = take(np * ((4 + warps) * sizeof(cfloat) + 4 * sizeof(float)) + 4 * sizeof(float));
    L.off_tri = take((size_t)n * (n + 1) / 2 * sizeof(unsigned short));
    L.bytes = align_up(o, 128);
    return L;
}

template <int W>
__device__ inline EighVec eigh_vectors(unsigned char* smem, const EighLayout& L, int n) {
    const int np = (n + 1) & ~1;
    EighVec v;
    v.pw0 = reinterpret_cast<cfloat*>(smem + L.off_vec);
    v.pw1 = v.pw0 + np;
    v.tau = v.pw1 + np;
    v.u = v.tau + np;
    v.w = v.u + np;
    v.d = reinterpret_cast<float*>(v.w + W * np);
    v.e = v.d + np;
    v.e2 = v.e + np;
    v.r = v.e2 + np;
    v.pair = v.r + np;
    v.u0 = reinterpret_cast<float*>(v.pw0);
    v.u1 = v.u0 + np;
    v.u2 = reinterpret_cast<float*>(v.pw1);
    v.m = v.u2 + np;
    v.tri = reinterpret_cast<unsigned short*>(smem + L.off_tri);
    return v;
}

// In-place inverse of the symmetric positive definite n x n double matrix G (row stride
// ld; lower triangle read and written) by the sweep operator: sweeping pivot k maps
// g_kk -> -1/g_kk, g_ik -> g_ik/g_kk, g_ij -> g_ij - g_ik g_kj / g_kk; after all n pivots
// G holds -G^{-1}.  col and cinv are n-long double work vectors (column k, and column
// k / g_kk, so that each update is one fused multiply-add on the narrow FP64 pipe).  False
// on a non-positive pivot (not positive definite).
template <int W>
__device__ inline bool e_inverse_spd(double* G, int ld, double* col, double* cinv, const unsigned short* tri, int n,
                                     const EighCta<W>& t) {
    const int ne = n * (n + 1) / 2;
    for (int k = 0; k < n; ++k) {
        t.sync();
        const double piv = G[k * ld + k];
        // piv > 0 by its bits: a comparison would take its turn in the FP64 pipe
        const long long pb = __double_as_longlong(piv);
        if (pb <= 0 || pb > 0x7ff0000000000000ll) return false;
        const double inv = 1.0 / piv;
        for (int i = t.tid; i < n; i += t.T) {
            const double c = i >= k ? G[i * ld + k] : G[k * ld + i];
            col[i] = c;
            cinv[i] = c * inv;
        }
        t.sync();
#pragma unroll 2
        for (int e = t.tid; e < ne; e += t.T) {
            const int i = tri[e] >> 8, j = tri[e] & 255;
            double* g = G + i * ld + j;
            double v;
            if (i == k) v = j == k ? -inv : cinv[j];
            else if (j == k) v = cinv[i];
            else v = fma(-col[i], cinv[j], *g);
            *g = v;
        }
    }
    t.sync();
    return true;
}

// Householder reduction of the Hermitian A (n x ld; the lower triangle is read and
// updated) to the real symmetric tridiagonal T (V.d, V.e), A = Q T Q^H with
// Q = H_0 ... H_{n-2}, H_k = I - tau_k u_k u_k^H acting on rows k+1..n-1, u_k = (1, v)
// with v kept in column k below the subdiagonal.  Each H_k^H maps column k's part below
// the diagonal, x, to (beta, 0, ...): beta = -sign(Re x_0) ||x||, tau = (beta - x_0) /
// beta, v = x_{1:} / (x_0 - beta), and with p = A22 u, s = u^H p, w = tau p -
// |tau|^2 s u / 2 the trailing block becomes A22 - w u^H - u w^H.  What a step needs of
// all rows (the norm, s, w) every warp computes for itself, in the same order.
template <int W>
__device__ inline void e_tridiag(cfloat* A, int n, int ld, const EighVec& V, const EighCta<W>& t) {
    const int lane = t.lane;
    cfloat* wv = V.w + t.warp * ((n + 1) & ~1);
    for (int k = 0; k + 1 < n; ++k) {
        t.sync();
        const cfloat alpha = A[(k + 1) * ld + k];
        float xn2 = 0.f;
        for (int i = k + 2 + lane; i < n; i += 32) xn2 += cabs2(A[i * ld + k]);
        xn2 = warp_sum(xn2);  // butterfly: the same value on every lane
        if (xn2 == 0.f && alpha.im == 0.f) {
            if (t.tid == 0) {
                V.tau[k] = cmake(0.f, 0.f);
                V.e[k] = alpha.re;
            }
            continue;
        }
        const float beta = -copysignf(sqrtf(alpha.re * alpha.re + alpha.im * alpha.im + xn2), alpha.re);
        const cfloat tau = cmake((beta - alpha.re) / beta, -alpha.im / beta);
        const cfloat den = cmake(alpha.re - beta, alpha.im);
        const float dd = 1.f / cabs2(den);
        const cfloat scal = cmake(den.re * dd, -den.im * dd);  // 1 / (x_0 - beta)
        if (t.warp == 0) {
            for (int i = k + 2 + lane; i < n; i += 32) V.u[i] = cmul(A[i * ld + k], scal);
            if (lane == 0) {
                V.u[k + 1] = cmake(1.f, 0.f);
                V.tau[k] = tau;
                V.e[k] = beta;
            }
        }
        t.sync();
        // p = A22 u from the lower triangle, in two chains (columns k+2, k+4, ... after
        // column k+1, and k+3, k+5, ...); from two warps on each takes one of them
        auto a22 = [&](int i, int j) {
            cfloat x = j <= i ? A[i * ld + j] : A[j * ld + i];
            if (j > i) x.im = -x.im;
            return x;
        };
        constexpr int kChains = W == 1 ? 1 : 2;
        const int chain = W == 1 ? 0 : t.warp & 1;
        for (int i = k + 1 + lane + 32 * (t.warp / kChains); i < n; i += 32 * (W / kChains)) {
            if (chain == 0) {
                cfloat acc = A[i * ld + k + 1];  // u_{k+1} = 1
                if (i == k + 1) acc.im = 0.f;
#pragma unroll 4
                for (int j = k + 2; j < n; j += 2) acc = cfma(acc, a22(i, j), V.u[j]);
                V.pw0[i] = acc;
            }
            if (W == 1 || chain == 1) {
                cfloat acc = cmake(0.f, 0.f);
#pragma unroll 4
                for (int j = k + 3; j < n; j += 2) acc = cfma(acc, a22(i, j), V.u[j]);
                V.pw1[i] = acc;
            }
        }
        if (t.warp == W - 1)
            for (int i = k + 2 + lane; i < n; i += 32) A[i * ld + k] = V.u[i];
        t.sync();
        // s = u^H p
        float s = 0.f;
        for (int i = k + 1 + lane; i < n; i += 32) {
            const cfloat vi = V.u[i], p = cadd(V.pw0[i], V.pw1[i]);
            s += vi.re * p.re + vi.im * p.im;
        }
        s = warp_sum(s);
        const float h = 0.5f * cabs2(tau) * s;
        for (int i = k + 1 + lane; i < n; i += 32) {
            const cfloat vi = V.u[i], pi = cadd(V.pw0[i], V.pw1[i]);
            wv[i] = cmake(tau.re * pi.re - tau.im * pi.im - h * vi.re, tau.re * pi.im + tau.im * pi.re - h * vi.im);
        }
        __syncwarp();
        // A22 -= w u^H + u w^H on the lower triangle (i, j relative to k + 1)
        const int m = n - k - 1, o = k + 1;
        const int ne = m * (m + 1) / 2;
#pragma unroll 2
        for (int e = t.tid; e < ne; e += t.T) {
            const int i = o + (V.tri[e] >> 8), j = o + (V.tri[e] & 255);
            const cfloat wi = wv[i], wj = wv[j], vi = V.u[i], vj = V.u[j];
            cfloat& x = A[i * ld + j];
            x = csub(x, cadd(cmulc(wi, vj), cmulc(vi, wj)));  // w_i conj(v_j) + v_i conj(w_j)
        }
    }
    t.sync();
    for (int i = t.tid; i < n; i += t.T) {
        V.d[i] = A[i * ld + i].re;
        if (i + 1 < n) V.e2[i] = V.e[i] * V.e[i];
    }
    t.sync();
}

// Number of eigenvalues of T below x (Sturm sequence of the LDL^T pivots).
__device__ __forceinline__ int e_sturm(const float* d, const float* e2, int n, float x, float pivmin) {
    float q = d[0] - x;
    if (fabsf(q) < pivmin) q = -pivmin;
    int c = q < 0.f;
#pragma unroll 4
    for (int i = 1; i < n; ++i) {
        q = (d[i] - x) - __fdividef(e2[i - 1], q);
        if (fabsf(q) < pivmin) q = -pivmin;
        c += q < 0.f;
    }
    return c;
}

// The k-th smallest eigenvalue of T (k from 0): each round splits [lo, hi) into 33
// parts at the lanes' shifts and keeps the part that holds it.
__device__ inline float e_kth(const float* d, const float* e2, int n, int k, float lo, float hi, float pivmin,
                              int lane) {
    for (int it = 0; it < 12; ++it) {
        if (!(hi - lo > 2.4e-7f * fmaxf(fabsf(lo), fabsf(hi)) + pivmin)) break;
        const float x = lo + (hi - lo) * ((float)(lane + 1) * (1.f / 33.f));
        const unsigned above = __ballot_sync(0xffffffffu, e_sturm(d, e2, n, x, pivmin) > k);
        const int jx = above ? __ffs(above) - 1 : 32;
        const float xl = __shfl_sync(0xffffffffu, x, jx > 0 ? jx - 1 : 0);
        const float xh = __shfl_sync(0xffffffffu, x, jx < 32 ? jx : 31);
        if (jx > 0) lo = xl;
        if (jx < 32) hi = xh;
    }
    return 0.5f * (lo + hi);
}

// Eigenvector of T for the eigenvalue lam by three steps of inverse iteration (one lane):
// (T - lam I) y = b by Gaussian elimination with partial pivoting, pivots below tiny
// replaced by tiny.  The elimination does not depend on b: it runs once, and the later
// steps apply its multipliers and row exchanges to their right-hand side.  The result is
// left in V.r; the factor that scales it to a largest entry of 1 is returned.
__device__ inline float e_inverse_iteration(const EighVec& V, int n, float lam, float tiny) {
    const float* __restrict__ d = V.d;
    const float* __restrict__ e = V.e;
    float* __restrict__ r = V.r;
    float* __restrict__ u0 = V.u0;
    float* __restrict__ u1 = V.u1;
    float* __restrict__ u2 = V.u2;
    float* __restrict__ mul = V.m;
    unsigned long long swapped = 0;
    {
        float p0 = d[0] - lam, p1 = n > 1 ? e[0] : 0.f;
        for (int i = 0; i + 1 < n; ++i) {
            const float q0 = e[i], q1 = d[i + 1] - lam, q2 = i + 2 < n ? e[i + 1] : 0.f;
            if (fabsf(p0) >= fabsf(q0)) {
                if (fabsf(p0) < tiny) p0 = p0 < 0.f ? -tiny : tiny;
                const float m = q0 / p0;
                u0[i] = p0, u1[i] = p1, u2[i] = 0.f, mul[i] = m;
                p0 = q1 - m * p1, p1 = q2;
            } else {
                const float m = p0 / q0;
                u0[i] = q0, u1[i] = q1, u2[i] = q2, mul[i] = m;
                swapped |= 1ull << i;
                p0 = p1 - m * q1, p1 = -(m * q2);
            }
        }
        if (fabsf(p0) < tiny) p0 = p0 < 0.f ? -tiny : tiny;
        u0[n - 1] = p0;
    }
    float sc = 1.f;
    for (int step = 0; step < 3; ++step) {
        auto rhs = [&](int i) { return step == 0 ? 1.f + 0.1f * (float)((7 * i) % 5) : __fmul_rn(r[i], sc); };
        float rr = rhs(0);
        for (int i = 0; i + 1 < n; ++i) {
            const float rq = rhs(i + 1), m = mul[i];
            const bool sw = swapped >> i & 1;
            const float top = sw ? rq : rr, bottom = sw ? rr : rq;
            r[i] = top;
            rr = bottom - m * top;
        }
        float big = 0.f, r1 = 0.f, r2 = 0.f;
        float uu0 = u0[n - 1], uu1 = 0.f, uu2 = 0.f, t = rr;
        for (int i = n - 1; i >= 0; --i) {
            // the next row's entries, before the division that this row waits for
            float nu0 = 1.f, nu1 = 0.f, nu2 = 0.f, nt = 0.f;
            if (i > 0) {
                nu0 = u0[i - 1], nu1 = u1[i - 1], nt = r[i - 1];
                if (i + 1 < n) nu2 = u2[i - 1];
            }
            if (i + 1 < n) t -= uu1 * r1;
            if (i + 2 < n) t -= uu2 * r2;
            r2 = r1;
            r1 = t / uu0;
            r[i] = r1;
            big = fmaxf(big, fabsf(r1));
            uu0 = nu0, uu1 = nu1, uu2 = nu2, t = nt;
        }
        sc = big > 0.f && isfinite(big) ? 1.f / big : 1.f;
    }
    return sc;
}

// The wanted eigenpair of the Hermitian A (n x ld, lower triangle; destroyed): EMI
// (evd false) the eigenvalue nearest 0.99, ties to the smaller; EVD the largest in
// magnitude, ties to the smaller.  Returns lambda; the eigenvector (unnormalised)
// is left in xv by the first warp, which alone goes on from there.
template <int W>
__device__ inline float e_eigpair(cfloat* A, int n, int ld, bool evd, const EighVec& V, cfloat* xv,
                                  const EighCta<W>& t) {
    const int lane = t.lane;
    e_tridiag<W>(A, n, ld, V, t);
    // Gershgorin bounds of T
    float lo = INFINITY, hi = -INFINITY, tn = 0.f, e2max = 0.f;
    for (int i = lane; i < n; i += 32) {
        const float rad = (i > 0 ? fabsf(V.e[i - 1]) : 0.f) + (i + 1 < n ? fabsf(V.e[i]) : 0.f);
        lo = fminf(lo, V.d[i] - rad);
        hi = fmaxf(hi, V.d[i] + rad);
        tn = fmaxf(tn, fabsf(V.d[i]) + rad);
        if (i + 1 < n) e2max = fmaxf(e2max, V.e2[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        tn = fmaxf(tn, __shfl_xor_sync(0xffffffffu, tn, o));
        e2max = fmaxf(e2max, __shfl_xor_sync(0xffffffffu, e2max, o));
    }
    const float pivmin = 1.18e-38f * fmaxf(1.f, e2max);
    const float pad = 2.4e-7f * (float)n * fmaxf(fabsf(lo), fabsf(hi)) + 2.f * pivmin;
    lo -= pad;
    hi += pad;
    // the two candidates, one per warp where there are two
    const int m = evd ? 0 : e_sturm(V.d, V.e2, n, 0.99f, pivmin);
    const bool both = evd || (m > 0 && m < n);
    const int ka = evd ? 0 : max(m - 1, 0), kb = evd ? n - 1 : m;
    float la = 0.f, lb = 0.f;
    if (W == 1 || t.warp == 0) la = e_kth(V.d, V.e2, n, ka, lo, hi, pivmin, lane);
    if (both && (W == 1 || t.warp == 1)) lb = e_kth(V.d, V.e2, n, kb, lo, hi, pivmin, lane);
    if (W > 1) {
        if (t.warp == 1 && lane == 0) V.pair[0] = lb;
        t.sync();
        if (t.warp != 0) return 0.f;
        lb = V.pair[0];
    }
    float lam = la;
    if (evd) lam = fabsf(lb) > fabsf(la) ? lb : la;
    else if (both) lam = fabsf(lb - 0.99f) < fabsf(la - 0.99f) ? lb : la;
    float sc = 1.f;
    if (lane == 0) sc = e_inverse_iteration(V, n, lam, 1.2e-7f * fmaxf(tn, 1.18e-38f));
    __syncwarp();
    sc = __shfl_sync(0xffffffffu, sc, 0);
    // x = Q y = H_0 (H_1 (... H_{n-2} y)), two rows per lane in registers
    cfloat x[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int i = lane + 32 * h;
        x[h] = cmake(i < n ? __fmul_rn(V.r[i], sc) : 0.f, 0.f);
    }
    cfloat un[2], tn1;  // the next step's column and scalar, loaded one step ahead
    auto fetch = [&](int k) {
        tn1 = V.tau[k];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = lane + 32 * h;
            un[h] = i == k + 1 ? cmake(1.f, 0.f) : i > k && i < n ? A[i * ld + k] : cmake(0.f, 0.f);
        }
    };
    if (n > 1) fetch(n - 2);
    for (int k = n - 2; k >= 0; --k) {
        const cfloat tk = tn1, u0 = un[0], u1 = un[1];
        if (k > 0) fetch(k - 1);
        if (tk.re == 0.f && tk.im == 0.f) continue;
        float dre = 0.f, dim = 0.f;  // u^H x
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = lane + 32 * h;
            if (i > k && i < n) {
                const cfloat u = h ? u1 : u0;
                dre += u.re * x[h].re + u.im * x[h].im;
                dim += u.re * x[h].im - u.im * x[h].re;
            }
        }
        const cfloat dot = cmake(warp_sum(dre), warp_sum(dim));
        const cfloat td = cmul(tk, dot);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = lane + 32 * h;
            if (i > k && i < n) x[h] = csub(x[h], cmul(h ? u1 : u0, td));
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int i = lane + 32 * h;
        if (i < n) xv[i] = x[h];
    }
    __syncwarp();
    return lam;
}

}  // namespace dpl

// SHP-masked coherence matrices on the CUDA cores, float32 throughout, for the shapes
// whose tiles do not fit the tensor-core kernel's shared memory (strided outputs with a
// large input region per tile: the mask bits of 256 pixels over it).
//
// One warp per output pixel.  The lower triangle of the N x N matrix is cut into B x B
// blocks, one per lane (B = ceil(N / 7): 28 blocks; above N = 49, B = ceil(N / 10) and two
// passes over 55 blocks), whose sums stay in registers; a sample costs a lane 2 B loads
// from shared memory for B^2 complex products.  The window's rows, contiguous in the
// pixel-major stack, are staged with cp.async one row ahead.
//
// Bound by issue (87 % of the slots, the FP32 pipe 64 %): six operations per complex
// product, a product, a fused multiply-add and an addition per component, rounded and
// ordered as in warp_covariance.  Both give the same sums bit for bit, but for the imaginary
// residues of the diagonal, which are left out here, and, above N = 32, the imaginary parts
// of rows 32 .. by columns 0 .. 31, which warp_covariance sums as the conjugate pair
// (warp_residues restores both where the plain form's solver reads the matrices).  A thread
// per matrix row over all 32 columns, as in warp_covariance, computes 1024 products per
// sample where N = 21 needs 231; the blocks compute 252.  512 x 384 outputs, 11 x 23
// windows, N = 21: 3.55 ms, 21 T operations/s (a fully set window row skips the search for
// set bits and takes two samples per turn: 4.0 ms without).  The whole call against the
// fused plain form, 200 x 150 outputs: N = 21 0.36 of its time, N = 45 0.26, and with the
// two passes above N = 49, N = 50 0.27 and N = 64 0.23.
//
// Output: planar per pixel and normalised, Cg[p][0 .. N^2): diagonal, then (Re, Im) per
// lower pair, C_ij = numer_ij / sqrt(amp_i amp_j) where that root is > 1e-6, else 0
// (covariance.py:131-142).
#pragma once

namespace dpl {

constexpr int kCovSimtPad = 16;  // elements behind a staged row that a last block may read

inline int cov_simt_block(int n) { return n <= 49 ? (n + 6) / 7 : (n + 9) / 10; }

template <int B>
__global__ void __launch_bounds__(256, B <= 3 ? 3 : B <= 5 ? 2 : 1) k_cov_simt(const PixArgs a, float* __restrict__ Cg, int row_elems) {
    extern __shared__ __align__(16) unsigned char cov_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    cfloat* buf = reinterpret_cast<cfloat*>(cov_smem) + (size_t)warp * 2 * row_elems;
    const int n = a.n, wy = 2 * a.hy + 1, wx = 2 * a.hx + 1;
    const int T = (n + B - 1) / B, nblocks = T * (T + 1) / 2;
    const int row_len = wx * n;
    const uint64_t full_row = wx >= 64 ? ~0ull : (1ull << wx) - 1ull;
    for (int64_t p = (int64_t)blockIdx.x * nwarps + warp; p < a.npix; p += (int64_t)gridDim.x * nwarps) {
        const int out_r = (int)(p / a.out_cols), out_c = (int)(p - (int64_t)out_r * a.out_cols);
        const int r0 = clamp_start_i(a.sy / 2 + out_r * a.sy, a.hy, wy, a.rows);
        const int c0 = clamp_start_i(a.sx / 2 + out_c * a.sx, a.hx, wx, a.cols);
        const cfloat* win = a.zt + ((int64_t)r0 * a.cols + c0) * n;
        auto stage = [&](int wa) {
            const cfloat* src = win + (int64_t)wa * a.cols * n;
            cfloat* dst = buf + (wa & 1) * row_elems;
            for (int i = lane; i < row_len; i += 32)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + i)),
                             "l"(src + i)
                             : "memory");
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        float* out = Cg + p * n * n;
        for (int first = 0; first < nblocks; first += 32) {
            // this lane's block (bi, bj), bj <= bi
            const int blk = first + lane;
            int bi = 0;
            while ((bi + 1) * (bi + 2) / 2 <= blk) ++bi;
            const bool active = blk < nblocks;
            const int bj = active ? blk - bi * (bi + 1) / 2 : 0;
            if (!active) bi = 0;
            float are[B][B], aim[B][B];
#pragma unroll
            for (int x = 0; x < B; ++x)
#pragma unroll
                for (int y = 0; y < B; ++y) are[x][y] = aim[x][y] = 0.f;
            int count = 0;
            __syncwarp();
            stage(0);
            for (int wa = 0; wa < wy; ++wa) {
                if (wa + 1 < wy) {
                    stage(wa + 1);
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                } else {
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                }
                __syncwarp();
                const uint64_t rm = row_mask(a, p, wa, wx, lane);
                count += __popcll(rm);
                const cfloat* row = buf + (wa & 1) * row_elems;
                auto add = [&](const cfloat* si, const cfloat* sj) {
                    cfloat zi[B], zj[B];
#pragma unroll
                    for (int x = 0; x < B; ++x) {
                        zi[x] = si[x];
                        zj[x] = sj[x];
                    }
#pragma unroll
                    for (int x = 0; x < B; ++x)
#pragma unroll
                        for (int y = 0; y < B; ++y) {
                            are[x][y] = fadd(are[x][y], fmaf(zi[x].re, zj[y].re, fmul(zi[x].im, zj[y].im)));
                            aim[x][y] = fadd(aim[x][y], fmaf(zi[x].im, zj[y].re, -fmul(zi[x].re, zj[y].im)));
                        }
                };
                const cfloat *si = row + bi * B, *sj = row + bj * B;
                if (rm == full_row) {
#pragma unroll(B <= 3 ? 2 : 1)
                    for (int b = 0; b < wx; ++b, si += n, sj += n) add(si, sj);
                } else {
#pragma unroll 1
                    for (int half = 0; half < 2; ++half) {
#pragma unroll 1
                        for (uint32_t m = (uint32_t)(rm >> (32 * half)); m; m &= m - 1u) {
                            const int b = (__ffs(m) - 1 + 32 * half) * n;
                            add(si + b, sj + b);
                        }
                    }
                }
                __syncwarp();  // the row's buffer is refilled by the next stage
            }
            // the diagonal sums first: published (with two passes, those of the other pass are
            // summed again from global memory), then every entry normalised
            float* amp = reinterpret_cast<float*>(buf);
            if (first == 0 && a.counts && lane == 0) a.counts[p] = count;
            if (active && bi == bj) {
#pragma unroll
                for (int x = 0; x < B; ++x)
                    if (bi * B + x < n) amp[bi * B + x] = are[x][x];
            }
            __syncwarp();
            if (nblocks > 32) {
                // two passes: sums of all rows' squares that this pass's blocks do not hold
                for (int i = lane; i < n; i += 32) {
                    const int d = i / B, db = d * (d + 1) / 2 + d;
                    if (db >= first && db < first + 32) continue;
                    float s = 0.f;
                    for (int wa = 0; wa < wy; ++wa) {
                        const cfloat* src = win + (int64_t)wa * a.cols * n + i;
                        for (int b = 0; b < wx; ++b) {
                            if (a.nb_u8 && !a.nb_u8[(p * wy + wa) * wx + b]) continue;
                            const cfloat z = src[(int64_t)b * n];
                            s = fadd(s, fmaf(z.re, z.re, fmul(z.im, z.im)));
                        }
                    }
                    amp[i] = s;
                }
                __syncwarp();
            }
            if (active) {
#pragma unroll
                for (int x = 0; x < B; ++x) {
                    const int i = bi * B + x;
#pragma unroll
                    for (int y = 0; y < B; ++y) {
                        const int j = bj * B + y;
                        if (i < n && j <= i) {
                            const float s = fsqrt(fmul(amp[i], amp[j]));
                            const bool ok = s > 1e-6f;
                            const float re = ok ? fdiv(are[x][y], s) : 0.f, im = ok ? fdiv(aim[x][y], s) : 0.f;
                            if (i == j) {
                                out[i] = re;
                            } else {
                                float* o = out + n + i * (i - 1) + 2 * j;
                                o[0] = re;
                                o[1] = im;
                            }
                        }
                    }
                }
            }
            __syncwarp();
        }
    }
}

template <int B>
static dpl_status launch_cov_simt(int block, const PixArgs& a, float* Cg, cudaStream_t s) {
    if constexpr (B <= 7) {
        if (block != B) return launch_cov_simt<B + 1>(block, a, Cg, s);
        const int row_elems = (int)align_up((size_t)(2 * a.hx + 1) * a.n + kCovSimtPad, 2);
        const size_t per_warp = 2 * (size_t)row_elems * sizeof(cfloat);
        const int warps = (int)std::max<size_t>(1, std::min<size_t>(8, (size_t)(100 * 1024) / per_warp));
        const size_t smem = (size_t)warps * per_warp;
        int dev = 0, sms = 0, per_sm = 0;
        DPL_CUDA_TRY(cudaGetDevice(&dev));
        DPL_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        DPL_CUDA_TRY(cudaFuncSetAttribute(k_cov_simt<B>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        DPL_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cov_simt<B>, warps * 32, smem));
        const int64_t want = (a.npix + warps - 1) / warps;
        const int64_t grid = std::min<int64_t>(want, (int64_t)std::max(1, per_sm) * sms * 8);
        k_cov_simt<B><<<(unsigned)std::max<int64_t>(grid, 1), warps * 32, smem, s>>>(a, Cg, row_elems);
        return check_launch("k_cov_simt");
    }
    return fail(DPL_ERR_UNSUPPORTED, "covariance: no block size for this depth");
}

}  // namespace dpl

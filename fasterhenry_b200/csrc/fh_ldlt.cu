// Batched FP64 factorization of the mesh system without interchanges,
// A = L D L^T with a unit lower triangular L (no conjugation), for the FP64
// sweep and the gradient.
//
// Z_ee = R_ee + j w L_ee is complex symmetric, and with both parts positive
// definite elimination without pivoting is stable (N. J. Higham, Math. Comp.
// 67, 1998).  Against the pivoted LU this leaves out half of the arithmetic
// (only the lower triangle is updated) and the pivot search, whose exchange
// among a matrix's CTAs in every column was most of the time of small orders
// and a quarter of large ones.
//
// The matrix is the whole mesh system, the port rows last (order M = m + p);
// the first m columns are eliminated.  The rows of L below them then hold
// (D^-1 L^-1 Z_ep)^T, and the trailing p x p block is the Schur complement
// Z_pp - Z_ep^T Z_ee^-1 Z_ep = Z(w) itself, so a sweep needs no triangular
// solve; X = Z_ee^-1 Z_ep, where it is wanted, is one backward substitution.
//
// Nothing is assumed of the matrix: the factors' backward error is bounded by
// u |L| |D| |L|^T, whose diagonal sum_k |l_ik|^2 |d_k| is accumulated row by
// row as the panels go.  A matrix with a row above kGrowthLimit |a_ii| (it is
// about |a_ii| for the class above), or with a zero or non-finite pivot, is
// reported as failed, and the caller factors it with partial pivoting.
//
// Per panel of 64 columns, launches over all matrices:
//   ldlt_diag_kernel    the 64 x 64 diagonal block's L and D, and L^-1;
//   ldlt_panel_kernel   B = A21 L11^-T, L21 = B D^-1 for the rows below;
// and A22 -= L21 B^T by ldlt_update_kernel on the tiles on and below the
// diagonal: of the next panel's columns alone within a group of up to four
// panels (ldlt_depth), of the rest of the matrix once per group.
// The products run on the FP64 tensor cores (mma.sync f64: tcgen05 has no FP64
// kind), as four real products of split real and imaginary parts.
#include <cuda_runtime.h>

#include <algorithm>

#include "fh_device.cuh"
#include "fh_ldlt.cuh"
#include "fh_lu.cuh"

namespace fhb {
namespace {

constexpr int kLd = kLdltPanel;       // panel width and tile edge
constexpr int kLdPad = kLd + 2;       // row of a staged chunk: four k and two rows of a fragment load hit all banks once
constexpr int kLdK = 16;              // k per stage of the update
constexpr int kLdThreads = 256;
constexpr int kDiagThreads64 = 512;
// From this order on the next group's panels run beside the update of the rest
// of the matrix, on a stream of the highest priority, whose blocks take the
// slots that the update's leave: their chain of small launches is a fifth of
// the time at order 2,321.  Without and with, in ms: order 6,787, 1 matrix 20.3
// and 17.4, 4 matrices 56.5 and 52.5; order 2,321, 2 matrices 3.98 and 3.50,
// 32 matrices 22.4 and 21.2; order 464, 32 matrices 0.89 and 0.82; 232, 1
// matrix 0.37 and 0.37.
constexpr int64_t kAheadOrder = 256;

// A = R + j w L on the tiles on and below the diagonal, order M, and the
// diagonal's 1-norms.
__global__ void __launch_bounds__(256) ldlt_form_kernel(const double *__restrict__ R, const double *__restrict__ L,
                                                        int64_t M, const double *__restrict__ omega, int count,
                                                        double2 *__restrict__ a, double *__restrict__ diag) {
    const int64_t col = blockIdx.x, first = col / kLd * kLd;
    for (int64_t row = first + (int64_t)blockIdx.y * blockDim.x + threadIdx.x; row < M;
         row += (int64_t)gridDim.y * blockDim.x) {
        const double r = R[row + col * M], l = L[row + col * M];
        for (int f = 0; f < count; ++f) {
            const double x = omega[f] * l;
            a[(int64_t)f * M * M + row + col * M] = make_double2(r, x);
            if (row == col) diag[(int64_t)f * M + row] = fabs(r) + fabs(x);
        }
    }
}

// The diagonal block [k0, k0 + nb)^2 of every matrix, one CTA each (DiagBlock).
__global__ void __launch_bounds__(kDiagThreads64) ldlt_diag_kernel(double2 *__restrict__ a, int64_t M, int64_t k0,
                                                                   int nb, double2 *__restrict__ xinv,
                                                                   int64_t xinv_stride, double2 *__restrict__ dinv,
                                                                   double *__restrict__ growth,
                                                                   int *__restrict__ failed) {
    __shared__ double2 v[2 * kLd];
    DiagBlock<kLd, kDiagThreads64 / 32, true> block;
    block.factor(v, a + (int64_t)blockIdx.x * M * M + k0 + k0 * M, M, nb, nb,
                 xinv + (int64_t)blockIdx.x * xinv_stride, kLd, dinv + (int64_t)blockIdx.x * kLd,
                 growth + (int64_t)blockIdx.x * M + k0, failed + blockIdx.x);
}

// Rows [c0, M) of the panel [k0, k0 + nb): B = A21 L11^-T into `panel`
// (column-major, ld M, by absolute row), L21 = B D^-1 in place, and the rows'
// growth.  A CTA takes 64 rows; it has read them all before it writes.
__global__ void __launch_bounds__(kLdThreads, 2)
    ldlt_panel_kernel(double2 *__restrict__ a, int64_t M, int64_t k0, int nb, const double2 *__restrict__ xinv,
                      int64_t xinv_stride, const double2 *__restrict__ dinv, double2 *__restrict__ panel,
                      int64_t panel_stride, double *__restrict__ growth) {
    extern __shared__ __align__(16) unsigned char ld_smem[];
    double2 *Ls = reinterpret_cast<double2 *>(ld_smem), *Us = Ls + 32 * kLdPad;
    __shared__ double rowsum[kLd];
    double2 *A = a + (int64_t)blockIdx.y * M * M;
    const double2 *X = xinv + (int64_t)blockIdx.y * xinv_stride, *D = dinv + (int64_t)blockIdx.y * kLd;
    double2 *P = panel + (int64_t)blockIdx.y * panel_stride;
    const int64_t r0 = k0 + nb + (int64_t)blockIdx.x * kLd;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3, wr = warp >> 2, wc = warp & 3;
    double re[4][2][2] = {}, im[4][2][2] = {};
    if (tid < kLd) rowsum[tid] = 0.0;
    for (int kc = 0; kc < kLd; kc += 32) {
        __syncthreads();
        for (int idx = tid; idx < 32 * kLd; idx += kLdThreads) {
            const int r = idx & (kLd - 1), k = idx / kLd;
            copy16(&Ls[k * kLdPad + r], A, r0 + r + (k0 + kc + k) * M, r0 + r < M && kc + k < nb);
            Us[k * kLdPad + r] = X[r + (kc + k) * kLd];  // L^-1 at (column r of B, k)
        }
        copy_commit();
        copy_wait<0>();
        __syncthreads();
        // L^-1 is lower triangular: its columns k >= 32 reach only B's columns >= 32
        if (kc == 0 || wc >= 2) {
#pragma unroll 2
            for (int k4 = 0; k4 < 32; k4 += 4)
                tile_step<1>(Ls + k4 * kLdPad, kLdPad, Us + k4 * kLdPad, kLdPad, 32 * wr, 16 * wc, g, t, re, im);
        }
    }
#pragma unroll
    for (int fm = 0; fm < 4; ++fm) {
        const int r = 32 * wr + 8 * fm + g;
        double sum = 0.0;
#pragma unroll
        for (int fn = 0; fn < 2; ++fn)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int c = 16 * wc + 8 * fn + 2 * t + e;
                if (r0 + r >= M || c >= nb) continue;
                const double2 b = make_double2(re[fm][fn][e], im[fm][fn][e]), d = D[c];
                const double2 l = make_double2(b.x * d.x - b.y * d.y, b.x * d.y + b.y * d.x);
                P[r0 + r + (int64_t)c * M] = b;
                A[r0 + r + (k0 + c) * M] = l;
                sum += (fabs(b.x) + fabs(b.y)) * (fabs(l.x) + fabs(l.y));  // |l|^2 |d|
            }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        if (t == 0) atomicAdd(&rowsum[r], sum);
    }
    __syncthreads();
    if (tid < kLd && r0 + tid < M) growth[(int64_t)blockIdx.y * M + r0 + tid] += rowsum[tid];
}

// A -= L B^T over the columns [k0, k0 + nb) of L on rows and columns from base:
// the whole lower triangle (end = M) or its columns [base, end); one 64 x 64
// tile on or below the diagonal per CTA, k in stages of 16 through two buffers
// of asynchronous copies, both operands [k][row] with re and im side by side
// (one 16-byte load per fragment).
//
// Bound by the FP64 tensor pipe: 8 nb operations per complex entry against 32
// bytes of C.  Order 2,321 x 32 matrices with nb = 64: 19.0 ms in all, 29
// TFLOP/s of the 37 that the instruction reaches alone (33.5 with the kernel's
// memory traffic taken out; a third buffer, a fixed or random start delay per
// CTA against lockstep, and m8n8k4 fragments measured the same or slower; the
// full update of the pivoted form takes 38.4 ms); with nb = 256 (ldlt_depth)
// 17.5, 31.5 TFLOP/s.
__global__ void __launch_bounds__(kLdThreads, 2)
    ldlt_update_kernel(double2 *__restrict__ a, int64_t M, int64_t k0, int nb, int64_t base, int64_t end,
                       const double2 *__restrict__ panel, int64_t panel_stride) {
    extern __shared__ __align__(16) unsigned char ld_smem[];
    double2 *smem = reinterpret_cast<double2 *>(ld_smem);  // stage s: L at 2 s kLdK kLdPad, B after it
    double2 *A = a + (int64_t)blockIdx.y * M * M;
    const double2 *P = panel + (int64_t)blockIdx.y * panel_stride;
    // tile index to (ti >= tj)
    const int tile = blockIdx.x;
    int ti, tj;
    if (end < M) {
        const int rows = (int)((M - base + kLd - 1) / kLd);
        tj = tile / rows;
        ti = tile - tj * rows;
        if (ti < tj) return;
    } else {
        ti = (int)((sqrt(8.0 * (double)tile + 1.0) - 1.0) * 0.5);
        while ((int64_t)ti * (ti + 1) / 2 > tile) --ti;
        while ((int64_t)(ti + 1) * (ti + 2) / 2 <= tile) ++ti;
        tj = tile - (int)((int64_t)ti * (ti + 1) / 2);
    }
    const int64_t i0 = base + (int64_t)ti * kLd, j0 = base + (int64_t)tj * kLd;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3, wr = warp >> 2, wc = warp & 3;
    const int stages = (nb + kLdK - 1) / kLdK;
    auto load = [&](int st) {
        double2 *L = smem + (st & 1) * 2 * kLdK * kLdPad, *U = L + kLdK * kLdPad;
#pragma unroll
        for (int idx = tid; idx < kLdK * kLd; idx += kLdThreads) {
            const int r = idx & (kLd - 1), k = idx / kLd, kk = st * kLdK + k;
            const bool live = kk < nb;
            copy16(&L[k * kLdPad + r], A, i0 + r + (k0 + kk) * M, live && i0 + r < M);
            copy16(&U[k * kLdPad + r], P, j0 + r + (int64_t)kk * M, live && j0 + r < M);
        }
        copy_commit();
    };
    load(0);
    double re[4][2][2], im[4][2][2];
#pragma unroll
    for (int fm = 0; fm < 4; ++fm)
#pragma unroll
        for (int fn = 0; fn < 2; ++fn)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int64_t row = i0 + 32 * wr + 8 * fm + g, col = j0 + 16 * wc + 8 * fn + 2 * t + e;
                double2 c = make_double2(0.0, 0.0);
                if (row < M && col < M) c = A[row + col * M];
                re[fm][fn][e] = c.x;
                im[fm][fn][e] = c.y;
            }
    for (int st = 0; st < stages; ++st) {
        if (st + 1 < stages) {
            load(st + 1);
            copy_wait<1>();
        } else {
            copy_wait<0>();
        }
        __syncthreads();
        const double2 *L = smem + (st & 1) * 2 * kLdK * kLdPad, *U = L + kLdK * kLdPad;
#pragma unroll
        for (int k4 = 0; k4 < kLdK; k4 += 4)
            tile_step<-1>(L + k4 * kLdPad, kLdPad, U + k4 * kLdPad, kLdPad, 32 * wr, 16 * wc, g, t, re, im);
        __syncthreads();  // before the stage after next overwrites this buffer
    }
#pragma unroll
    for (int fm = 0; fm < 4; ++fm)
#pragma unroll
        for (int fn = 0; fn < 2; ++fn)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int64_t row = i0 + 32 * wr + 8 * fm + g, col = j0 + 16 * wc + 8 * fn + 2 * t + e;
                if (row < M && col < end) A[row + col * M] = make_double2(re[fm][fn][e], im[fm][fn][e]);
            }
}

// failed[f] = 1 for a row whose growth is above the limit (or not a number).
__global__ void __launch_bounds__(256) ldlt_growth_kernel(const double *__restrict__ growth,
                                                          const double *__restrict__ diag, int64_t M, int64_t m,
                                                          int *__restrict__ failed) {
    bool bad = false;
    for (int64_t i = threadIdx.x; i < m; i += blockDim.x)
        bad = bad || !(growth[blockIdx.x * M + i] <= kGrowthLimit * diag[blockIdx.x * M + i]);
    if (__syncthreads_or(bad) && threadIdx.x == 0) failed[blockIdx.x] = 1;
}

// Z from the trailing block: [f][i][j], symmetric; real at zero frequency
// (solve.rs:811-815).
__global__ void ldlt_z_kernel(const double2 *__restrict__ a, int64_t M, int64_t m, int p,
                              const double *__restrict__ omega, int count, double2 *__restrict__ z) {
    const int64_t total = (int64_t)count * p * p;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t f = idx / (p * p), ij = idx % (p * p);
        const int64_t i = max(ij / p, ij % p), j = min(ij / p, ij % p);
        double2 v = a[f * M * M + (m + i) + (m + j) * M];
        if (omega[f] == 0.0) v.y = 0.0;
        z[idx] = v;
    }
}

// x (f, q) <- row m + q of L: the right-hand side of L^T x = .
__global__ void ldlt_rows_kernel(const double2 *__restrict__ a, int64_t M, int64_t m, int p, int count,
                                 double2 *__restrict__ x) {
    const int64_t total = (int64_t)count * p * m;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t fq = idx / m, k = idx % m, f = fq / p, q = fq % p;
        x[idx] = a[f * M * M + (m + q) + k * M];
    }
}

__device__ __forceinline__ double2 warp_sum(double2 v) {
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    return v;
}

// x[k0 .. k0 + nb) <- (L11^-1)^T x, a warp per entry.
__global__ void __launch_bounds__(256) ldlt_back_block_kernel(const double2 *__restrict__ xinv, int64_t xinv_stride,
                                                              int64_t m, int p, int64_t k0, int nb,
                                                              double2 *__restrict__ x) {
    __shared__ double2 s[kLd];
    const int64_t f = blockIdx.x / p;
    const double2 *X = xinv + f * xinv_stride;
    double2 *xs = x + (int64_t)blockIdx.x * m + k0;
    const int lane = threadIdx.x & 31;
    for (int r = threadIdx.x; r < kLd; r += blockDim.x) s[r] = r < nb ? xs[r] : make_double2(0.0, 0.0);
    __syncthreads();
    for (int c = threadIdx.x >> 5; c < nb; c += blockDim.x >> 5) {
        double2 acc = make_double2(0.0, 0.0);
        for (int r = lane; r < kLd; r += 32) {
            const double2 l = X[r + c * kLd], v = s[r];
            acc.x += l.x * v.x - l.y * v.y;
            acc.y += l.x * v.y + l.y * v.x;
        }
        acc = warp_sum(acc);
        if (lane == 0) xs[c] = acc;
    }
}

// x_j -= sum_r L[k0 + r][j] x[k0 + r] for the columns j < k0, a warp per
// column (its nb rows are one run of memory), all right-hand sides of a
// matrix from one read.
__global__ void __launch_bounds__(256) ldlt_back_update_kernel(const double2 *__restrict__ a, int64_t M, int64_t m,
                                                               int p, int64_t k0, int nb, double2 *__restrict__ x) {
    const int64_t f = blockIdx.y, j = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (j >= k0) return;
    const int lane = threadIdx.x & 31;
    const double2 *L = a + f * M * M + k0 + j * M;
    double2 l[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) l[h] = lane + 32 * h < nb ? L[lane + 32 * h] : make_double2(0.0, 0.0);
    for (int q = 0; q < p; ++q) {
        double2 *xq = x + (f * p + q) * m;
        double2 acc = make_double2(0.0, 0.0);
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (lane + 32 * h < nb) {
                const double2 v = xq[k0 + lane + 32 * h];
                acc.x += l[h].x * v.x - l[h].y * v.y;
                acc.y += l[h].x * v.y + l[h].y * v.x;
            }
        acc = warp_sum(acc);
        if (lane == 0) {
            xq[j].x -= acc.x;
            xq[j].y -= acc.y;
        }
    }
}

// The stream of the panels and the events between it and the updates'.
struct Ahead {
    cudaStream_t s = nullptr;
    cudaEvent_t e[2] = {};
    bool joined = false;  // the caller's stream waits for all of it
    ~Ahead() {
        if (s && !joined) cudaStreamSynchronize(s);  // an error return: the buffers are the caller's
        for (cudaEvent_t x : e)
            if (x) cudaEventDestroy(x);
        if (s) stream_release(s);
    }
};

// Panels per group: the trailing matrix is updated once per group, by all its
// columns, and a panel within a group just before its turn, so the traffic of
// C falls with the depth; but a panel's own update has only the panel's tiles,
// and the first panels of a matrix wait for nothing else.  Where these fill the
// chip's two CTAs per SM by a margin four panels are best, below a third of it
// one (ms for depths 1, 2, 4: order 6,787, 4 matrices 57.9, 53.9, 52.5; 1
// matrix 18.2, 17.4, 17.8; order 2,321, 32 matrices 23.1, 21.7, 21.2; 8
// matrices 6.98, 6.74, 7.04; 2 matrices 3.50, 3.69, 4.15).
int ldlt_depth(int64_t m, int64_t p, int count) {
    const int64_t tiles = (m + p + kLd - 1) / kLd * count;
    return tiles >= 384 ? 4 : tiles >= 96 ? 2 : 1;
}

}  // namespace

size_t ldlt_bytes(int64_t m, int64_t p, int count) {
    const int64_t M = m + p, blocks = (m + kLd - 1) / kLd;
    // two groups of panels, the diagonal blocks' inverses, D^-1, the rows' growth and diagonal
    return (size_t)count * (32 * (size_t)M * kLd * ldlt_depth(m, p, count) + 16 * (size_t)blocks * kLd * kLd +
                            16 * (size_t)blocks * kLd + 16 * (size_t)M + 16);
}

fh_status ldlt_factor(const double *Rm, const double *Lm, int64_t m, int64_t p, const double *d_omega, int count,
                      double *a, void *work, double *z, double *x, int *d_failed, cudaStream_t s,
                      fh_error_info *err) {
    const int64_t M = m + p, blocks = (m + kLd - 1) / kLd;
    double2 *A = reinterpret_cast<double2 *>(a);
    double2 *panel = static_cast<double2 *>(work);
    double2 *xinv = panel + (int64_t)count * M * kLd * ldlt_depth(m, p, count) * 2;
    double2 *dinv = xinv + (int64_t)count * blocks * kLd * kLd;
    double *diag = reinterpret_cast<double *>(dinv + (int64_t)count * blocks * kLd);
    double *growth = diag + (int64_t)count * M;
    FHB_CUDA(cudaMemsetAsync(d_failed, 0, sizeof(int) * (size_t)count, s));
    FHB_CUDA(cudaMemsetAsync(growth, 0, sizeof(double) * (size_t)count * M, s));
    prof_begin(s, FH_PROF_FORM);
    ldlt_form_kernel<<<dim3((unsigned)M, (unsigned)std::min<int64_t>((M + 255) / 256, 8)), 256, 0, s>>>(
        Rm, Lm, M, d_omega, count, A, diag);
    prof_end(s, FH_PROF_FORM, 16.0 * (double)M * (double)M * count / 2.0);
    constexpr int panel_smem = 2 * 32 * kLdPad * (int)sizeof(double2);
    constexpr int update_smem = 4 * kLdK * kLdPad * (int)sizeof(double2);
    FHB_CUDA(cudaFuncSetAttribute(ldlt_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, panel_smem));
    FHB_CUDA(cudaFuncSetAttribute(ldlt_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, update_smem));
    const int64_t xs = blocks * kLd * kLd;
    const int depth = ldlt_depth(m, p, count);
    const int64_t ps = M * kLd * depth;
    // columns [base, end) of the trailing matrix, from the group's panels k0 ..
    auto update = [&](int64_t k0, int64_t base, int64_t end, const double2 *P, cudaStream_t q) -> fh_status {
        const int64_t rows = (M - base + kLd - 1) / kLd, cols = (end - base + kLd - 1) / kLd;
        if (rows <= 0 || cols <= 0) return FH_OK;
        const int64_t tiles = end < M ? rows * cols : rows * (rows + 1) / 2;
        const int64_t kk = std::min({base - k0, depth * (int64_t)kLd, m - k0});
        prof_begin(q, FH_PROF_GEMM_FP64);
        ldlt_update_kernel<<<dim3((unsigned)tiles, (unsigned)count), kLdThreads, update_smem, q>>>(A, M, k0, (int)kk,
                                                                                                 base, end, P, ps);
        const double width = (double)(end - base), height = (double)(M - base);
        prof_end(q, FH_PROF_GEMM_FP64, 8.0 * (width * height - 0.5 * width * width) * (double)kk * count);
        FHB_CUDA(cudaGetLastError());
        return FH_OK;
    };
    // the panels of the group from column g0 on
    auto panels = [&](int64_t g0, double2 *P, cudaStream_t q) -> fh_status {
        for (int64_t k0 = g0; k0 < std::min(m, g0 + depth * kLd); k0 += kLd) {
            const int64_t b = k0 / kLd, nb = std::min<int64_t>(kLd, m - k0), rest = M - k0 - nb;
            double2 *xb = xinv + b * kLd * kLd, *db = dinv + b * count * kLd;
            if (k0 > g0) {
                const fh_status e = update(g0, k0, k0 + nb, P, q);
                if (e) return e;
            }
            prof_begin(q, FH_PROF_PANEL);
            ldlt_diag_kernel<<<(unsigned)count, kDiagThreads64, 0, q>>>(A, M, k0, (int)nb, xb, xs, db, growth,
                                                                       d_failed);
            prof_end(q, FH_PROF_PANEL, 0.0);
            if (rest > 0) {
                prof_begin(q, FH_PROF_TRSM);
                ldlt_panel_kernel<<<dim3((unsigned)((rest + kLd - 1) / kLd), (unsigned)count), kLdThreads, panel_smem,
                                    q>>>(A, M, k0, (int)nb, xb, xs, db, P + (k0 - g0) * M, ps, growth);
                prof_end(q, FH_PROF_TRSM, 4.0 * kLd * kLd * (double)rest * count);
            }
            FHB_CUDA(cudaGetLastError());
        }
        return FH_OK;
    };
    Ahead ahead;
    if (m >= kAheadOrder) {
        FHB_CUDA(stream_acquire(&ahead.s, true));
        for (cudaEvent_t &e : ahead.e) FHB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    const cudaStream_t q = ahead.s ? ahead.s : s;
    auto hand_over = [&](cudaStream_t from, cudaStream_t to, cudaEvent_t e) -> fh_status {
        if (from == to) return FH_OK;
        FHB_CUDA(cudaEventRecord(e, from));
        FHB_CUDA(cudaStreamWaitEvent(to, e, 0));
        return FH_OK;
    };
    fh_status st = hand_over(s, q, ahead.e[0]);
    if (!st && m > 0) st = panels(0, panel, q);
    for (int64_t k0 = 0, group = 0; !st && k0 < m; k0 += depth * kLd, ++group) {
        double2 *P = panel + (group & 1) * count * ps, *next = panel + ((group + 1) & 1) * count * ps;
        const int64_t base = std::min(m, k0 + depth * kLd), end = std::min(m, base + depth * kLd);
        if (!ahead.s) {
            st = update(k0, base, M, P, s);
            if (!st && base < m) st = panels(base, next, s);
            continue;
        }
        st = hand_over(q, s, ahead.e[1]);
        if (!st && base < m) {
            st = update(k0, base, end, P, s);
            if (!st) st = hand_over(s, q, ahead.e[0]);
            if (!st) st = panels(base, next, q);
        }
        if (!st && end < M) st = update(k0, end, M, P, s);
    }
    if (st) return st;
    ahead.joined = true;
    if (m > 0) ldlt_growth_kernel<<<(unsigned)count, 256, 0, s>>>(growth, diag, M, m, d_failed);
    if (p > 0)
        ldlt_z_kernel<<<(unsigned)std::min<int64_t>(((int64_t)count * p * p + 255) / 256, 1024), 256, 0, s>>>(
            A, M, m, (int)p, d_omega, count, reinterpret_cast<double2 *>(z));
    FHB_CUDA(cudaGetLastError());
    if (!x || m == 0 || p == 0) return FH_OK;
    prof_begin(s, FH_PROF_SOLVE);
    double2 *X = reinterpret_cast<double2 *>(x);
    ldlt_rows_kernel<<<(unsigned)std::min<int64_t>(((int64_t)count * p * m + 255) / 256, 148 * 8), 256, 0, s>>>(
        A, M, m, (int)p, count, X);
    for (int64_t b = blocks - 1; b >= 0; --b) {
        const int64_t k0 = b * kLd;
        const int nb = (int)std::min<int64_t>(kLd, m - k0);
        ldlt_back_block_kernel<<<(unsigned)(count * p), 256, 0, s>>>(xinv + b * kLd * kLd, xs, m, (int)p, k0, nb, X);
        if (k0 > 0)
            ldlt_back_update_kernel<<<dim3((unsigned)((k0 + 7) / 8), (unsigned)count), 256, 0, s>>>(A, M, m, (int)p,
                                                                                                    k0, nb, X);
    }
    prof_end(s, FH_PROF_SOLVE, 4.0 * (double)m * (double)m * (double)p * count);
    FHB_CUDA(cudaGetLastError());
    return FH_OK;
}

}  // namespace fhb

using namespace fhb;

extern "C" fh_status fh_test_mesh_solve(const double *r, const double *l, int64_t m, int64_t p, const double *omega,
                                        int32_t count, double *z, double *x, int32_t *failed, fh_error_info *err) {
    clear_error(err);
    if (!r || !l || !omega || !z || !x || !failed || m < 1 || p < 1 || count < 1)
        return fail(err, FH_ERR_INVALID_ARGUMENT, "null argument or empty system");
    fh_status st = ensure_device(err);
    if (st) return st;
    const size_t M = (size_t)(m + p), sym = 8 * M * M, zs = 16 * (size_t)(count * p * p),
                 xs = 16 * (size_t)(count * p * m);
    void *d[8] = {};
    struct Release {
        void **d;
        ~Release() {
            for (int k = 0; k < 8; ++k) cudaFree(d[k]);
        }
    } release{d};
    const size_t bytes[8] = {sym, sym, 8 * (size_t)count, 2 * sym * (size_t)count, ldlt_bytes(m, p, count), zs, xs,
                             4 * (size_t)count};
    for (int k = 0; k < 8; ++k) FHB_CUDA(cudaMalloc(&d[k], bytes[k]));
    FHB_CUDA(cudaMemcpy(d[0], r, sym, cudaMemcpyHostToDevice));
    FHB_CUDA(cudaMemcpy(d[1], l, sym, cudaMemcpyHostToDevice));
    FHB_CUDA(cudaMemcpy(d[2], omega, bytes[2], cudaMemcpyHostToDevice));
    st = ldlt_factor((double *)d[0], (double *)d[1], m, p, (double *)d[2], count, (double *)d[3], d[4], (double *)d[5],
                     (double *)d[6], (int *)d[7], nullptr, err);
    if (st) return st;
    FHB_CUDA(cudaMemcpy(z, d[5], zs, cudaMemcpyDeviceToHost));
    FHB_CUDA(cudaMemcpy(x, d[6], xs, cudaMemcpyDeviceToHost));
    FHB_CUDA(cudaMemcpy(failed, d[7], bytes[7], cudaMemcpyDeviceToHost));
    return FH_OK;
}

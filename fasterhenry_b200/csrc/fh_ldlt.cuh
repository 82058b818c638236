// Device pieces of the FP64 factorization A = L D L^T without interchanges,
// shared by the sweeps of one system (fh_ldlt.cu, a launch per step over all
// its matrices) and of many small ones (fh_batchsolve.cu, a CTA per matrix).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace fhb {

// A row's growth sum_k |l_ik|^2 |d_k| (1-norms of complex numbers, at most twice
// the moduli's product) above this times |a_ii| rejects the elimination.
constexpr double kGrowthLimit = 128.0;

// m16n8k4: two stacked m8n8k4 fragments of A and C.
__device__ __forceinline__ void dmma(double (&lo)[2], double (&hi)[2], double a0, double a1, double b) {
    asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
                 : "+d"(lo[0]), "+d"(lo[1]), "+d"(hi[0]), "+d"(hi[1])
                 : "d"(a0), "d"(a1), "d"(b));
}
// base[at] to shared memory, or zeros when !live (the address is then base's).
__device__ __forceinline__ void copy16(double2 *dst, const double2 *base, int64_t at, bool live) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(live ? base + at : base),
                 "r"(live ? 16 : 0));
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N));
}

// y -= l t
__device__ __forceinline__ void sub_mul(double2 &y, double2 l, double2 t) {
    y.x -= l.x * t.x - l.y * t.y;
    y.y -= l.x * t.y + l.y * t.x;
}

// The first nb steps on a diagonal block of `rows` rows (nb <= rows <= NB) by one
// CTA of WARPS warps: L below its diagonal and D on it, in place in A (leading
// dimension M) where KEEP asks for them; L^-1 (unit lower, zeros above) in X's
// first nb rows and the Schur complement of the other rows in its trailing
// corner (leading dimension ldx; without KEEP X may be A, whose places take no
// other store); D^-1; the rows' growth added to G.  v: 2 NB entries of shared
// memory.  Gauss-Jordan in one array: until step k place (i, k) holds the Schur complement's entry,
// after it the entry of L^-1, which starts as -l_ik; step j takes l_ij times v
// from row i, where v is row j of L^-1 left of the pivot and column j of the
// complement beyond it.
//
// A warp owns the columns w + WARPS c and its lanes the rows lane and lane + 32,
// in registers (columns from 32 on only the lower rows); v goes through a
// double buffer with one barrier per step, and rows at or above the pivot take
// part with l = 0.  The steps run in segments of WARPS, so that which of a
// warp's columns lie left or right of the pivot is known at compile time.
//
// Bound by its chain of NB steps of one barrier, one division and some forty
// dependent instructions: 38 us for 64 with 16 warps (88 us with a row per
// thread, whose columns' cases diverge in every step).
template <int NB, int WARPS, bool KEEP>
struct DiagBlock {
    static_assert((NB == 32 || NB == 64) && (WARPS == 8 || WARPS == 16), "rows lane and lane + 32");
    static constexpr int kLo = 32 / WARPS, kCols = NB / WARPS, kHi = NB == 64 ? kCols : 0;
    double2 lo[kLo], hi[kHi > 0 ? kHi : 1];  // rows lane and lane + 32 of column w + WARPS c
    double sum0 = 0.0, sum1 = 0.0;           // the rows' |l|^2 |d| over the block (warp 0)

    template <int JC>
    __device__ __forceinline__ void segment(double2 *v, double2 *A, int64_t M, int rows, int nb, int w, int lane,
                                            double2 *dinv, int *failed) {
        if constexpr (JC < kCols) {
            constexpr bool upper = JC < kLo;  // pivots among the rows `lane`
            constexpr int jl = upper ? JC : 0, jh = kHi > 0 ? JC : 0;
            const int r0 = lane, r1 = lane + 32;
            for (int jw = 0; jw < WARPS; ++jw) {
                const int j = WARPS * JC + jw;
                if (j >= nb) return;
                double2 *vj = v + (jw & 1) * NB;
                // row j of L^-1 and column j of the complement
                if (lane == (j & 31)) {
#pragma unroll
                    for (int c = 0; c < JC; ++c) vj[w + WARPS * c] = upper ? lo[c < kLo ? c : 0] : hi[kHi > 0 ? c : 0];
                    if (w < jw) vj[w + WARPS * JC] = upper ? lo[jl] : hi[jh];
                }
                if (w == jw) {
                    if (upper && r0 >= j) vj[r0] = lo[jl];
                    if (NB == 64 && r1 >= j) vj[r1] = hi[jh];
                }
                __syncthreads();
                const double2 d = vj[j];
                double2 q0 = make_double2(0.0, 0.0), q1 = make_double2(0.0, 0.0);
                if (upper) q0 = vj[r0];
                if (NB == 64) q1 = vj[r1];
                const double n = 1.0 / (d.x * d.x + d.y * d.y);
                const double2 inv = make_double2(d.x * n, -d.y * n);
                double2 l0 = make_double2(q0.x * inv.x - q0.y * inv.y, q0.x * inv.y + q0.y * inv.x);
                double2 l1 = make_double2(q1.x * inv.x - q1.y * inv.y, q1.x * inv.y + q1.y * inv.x);
                if (!upper || r0 <= j) l0 = make_double2(0.0, 0.0);
                if (NB != 64 || r1 <= j) l1 = make_double2(0.0, 0.0);
#pragma unroll
                for (int c = 0; c < kCols; ++c) {
                    if (c == JC && w == jw) {  // L's column, and the start of L^-1's
                        if (upper && r0 > j) {
                            if (KEEP && r0 < rows) A[r0 + (int64_t)j * M] = l0;
                            lo[jl] = make_double2(-l0.x, -l0.y);
                        }
                        if (NB == 64 && r1 > j) {
                            if (KEEP && r1 < rows) A[r1 + (int64_t)j * M] = l1;
                            hi[jh] = make_double2(-l1.x, -l1.y);
                        }
                    } else {
                        const double2 t = vj[w + WARPS * c];
                        if (c < kLo && upper) sub_mul(lo[c < kLo ? c : 0], l0, t);
                        if (NB == 64) sub_mul(hi[kHi > 0 ? c : 0], l1, t);
                    }
                }
                if (w == 0) {
                    if (upper) sum0 += (fabs(q0.x) + fabs(q0.y)) * (fabs(l0.x) + fabs(l0.y));
                    sum1 += (fabs(q1.x) + fabs(q1.y)) * (fabs(l1.x) + fabs(l1.y));
                    if (r0 == j) sum0 += fabs(d.x) + fabs(d.y);
                    if (r1 == j) sum1 += fabs(d.x) + fabs(d.y);
                }
                if (w == WARPS - 1 && lane == 0) {
                    if (KEEP) A[j + (int64_t)j * M] = d;
                    dinv[j] = inv;
                    if (!isfinite(inv.x) || !isfinite(inv.y) || !isfinite(d.x) || !isfinite(d.y)) *failed = 1;
                }
            }
        }
    }

    __device__ static __forceinline__ double2 place(int r, int k, int nb, double2 value) {
        if (r < nb) return k < r ? value : make_double2(r == k ? 1.0 : 0.0, 0.0);
        return k >= nb && k <= r ? value : make_double2(0.0, 0.0);
    }

    __device__ __forceinline__ void factor(double2 *v, double2 *A, int64_t M, int rows, int nb, double2 *X,
                                           int ldx, double2 *dinv, double *G, int *failed) {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, r0 = lane, r1 = lane + 32;
        const double2 zero = make_double2(0.0, 0.0);
        if (threadIdx.x < 2 * NB) v[threadIdx.x] = zero;  // rows that no step publishes
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
            const int k = w + WARPS * c;
            if (c < kLo) lo[c < kLo ? c : 0] = r0 >= k && r0 < rows ? A[r0 + k * M] : zero;
            if (NB == 64) hi[kHi > 0 ? c : 0] = r1 >= k && r1 < rows ? A[r1 + k * M] : zero;
        }
        __syncthreads();
        segment<0>(v, A, M, rows, nb, w, lane, dinv, failed);
        segment<1>(v, A, M, rows, nb, w, lane, dinv, failed);
        segment<2>(v, A, M, rows, nb, w, lane, dinv, failed);
        segment<3>(v, A, M, rows, nb, w, lane, dinv, failed);
        segment<4>(v, A, M, rows, nb, w, lane, dinv, failed);
        segment<5>(v, A, M, rows, nb, w, lane, dinv, failed);
        segment<6>(v, A, M, rows, nb, w, lane, dinv, failed);
        segment<7>(v, A, M, rows, nb, w, lane, dinv, failed);
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
            const int k = w + WARPS * c;
            X[r0 + k * ldx] = place(r0, k, nb, c < kLo ? lo[c < kLo ? c : 0] : zero);
            if (NB == 64) X[r1 + k * ldx] = place(r1, k, nb, hi[kHi > 0 ? c : 0]);
        }
        if (w == 0) {
            if (r0 < rows) G[r0] += sum0;
            if (NB == 64 && r1 < rows) G[r1] += sum1;
        }
    }
};

// One k4 step of a warp's part of a tile: C rows row0 .. + 8 FM, columns col0 ..
// + 8 FN.  l and u point at the step's first k of the staged operands ([k][row],
// ldl and ldu apart).  Fragment layout of m16n8k4 f64: A at (rows g and g + 8, k
// t), B at (k t, column g), C at (rows g and g + 8, columns 2 t, 2 t + 1), with
// g = lane / 4, t = lane % 4.  SIGN: +1 adds, -1 subtracts.
template <int SIGN, int FM, int FN>
__device__ __forceinline__ void tile_step(const double2 *l, int ldl, const double2 *u, int ldu, int row0, int col0,
                                          int g, int t, double (&re)[FM][FN][2], double (&im)[FM][FN][2]) {
    double2 lf[FM], uf[FN];
#pragma unroll
    for (int fm = 0; fm < FM; ++fm) {
        lf[fm] = l[t * ldl + row0 + 8 * fm + g];
        if (SIGN < 0) lf[fm].x = -lf[fm].x;
        else lf[fm].y = -lf[fm].y;
    }
#pragma unroll
    for (int fn = 0; fn < FN; ++fn) uf[fn] = u[t * ldu + col0 + 8 * fn + g];
    // SIGN < 0: lf = (-l_re, l_im); SIGN > 0: lf = (l_re, -l_im); FM FN
    // independent products between two on the same accumulator
#pragma unroll
    for (int fm = 0; fm < FM; fm += 2)
#pragma unroll
        for (int fn = 0; fn < FN; ++fn) {
            dmma(re[fm][fn], re[fm + 1][fn], lf[fm].x, lf[fm + 1].x, uf[fn].x);
            dmma(im[fm][fn], im[fm + 1][fn], lf[fm].x, lf[fm + 1].x, uf[fn].y);
        }
#pragma unroll
    for (int fm = 0; fm < FM; fm += 2)
#pragma unroll
        for (int fn = 0; fn < FN; ++fn) {
            dmma(re[fm][fn], re[fm + 1][fn], lf[fm].y, lf[fm + 1].y, uf[fn].y);
            dmma(im[fm][fn], im[fm + 1][fn], -lf[fm].y, -lf[fm + 1].y, uf[fn].x);
        }
}

}  // namespace fhb

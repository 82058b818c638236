// The precorrected-FFT operator on the device: y = L x without forming L
// (pfft/mod.rs:482-560 of the reference).
//
//   y = C x + mu0/4pi sum_c d_c . W^T (K (*) (W (d_c . x)))
//
// per product, for `count` vectors at once, taken in pairs:
//   1. sources_kernel     pairs x_v, x_v+1 side by side, and the sources
//                         d_ic x_vi of every filament likewise, so that the
//                         gathers below take one 16-byte load per pair;
//   2. near_kernel        y = C x (CSR rows of precorrected near pairs; warp
//                         per filament, up to two pairs of vectors from one
//                         pass over the row);
//   3. spread_kernel      the grid sources q_{v,c}(g) = sum_i W_ig d_ic x_vi,
//                         one thread per grid point over the transposed
//                         projection (no atomics), written to compact complex
//                         grids (two real sources per grid: real and imaginary
//                         part) in the convolution's precision;
//   4. fftconv_run        the aperiodic convolution K (*) q by pruned
//                         mixed-radix transforms on the 2N-1 padded torus
//                         (fh_fftconv.cu; FP64 or FP32);
//   5. interp_kernel      y_vi += mu0/4pi sum_c d_ic sum_g W_ig phi_{v,c}(g),
//                         warp per filament, from the compact grids.
// Real source r = v ncomp + c is part r % 2 of complex grid r / 2, so a pair
// of vectors fills ncomp whole grids.
//
// The near-field corrections C_ij = L_ij(exact) - mu0/4pi cos_ij G_ij are
// built at set-up from the device's grid approximations G_ij and the exact
// partial inductances of the same pairs, evaluated by the device fill in
// pair-list mode; the upper triangle is mirrored into full rows (near.rs:
// 263-298).  The kernel spectrum is the forward transform of the wrapped
// kernel 1/|r_g - r_h| on the padded grid, real for an even kernel.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <string>
#include <type_traits>

#include "fh_device.cuh"
#include "fh_pfft.h"

namespace fhb {

namespace {

constexpr double kMu0Over4PiP = 1e-7;

double now_s() {
    return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

template <class T>
cudaError_t upload(T **d, const std::vector<T> &h, cudaStream_t s) {
    cudaError_t e = cache_alloc((void **)d, std::max<size_t>(1, h.size()) * sizeof(T), s);
    if (e != cudaSuccess) return e;
    if (h.empty()) return cudaSuccess;
    return cudaMemcpyAsync(*d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, s);
}

// ---------------------------------------------------------------------------
// Products.
// ---------------------------------------------------------------------------
struct ApplyArgs {
    int64_t n, G;
    int comp[3];
    int count;   // vectors
    int pairs;   // (count + 1) / 2
    int grids;   // (count ncomp + 1) / 2
};

// Pair p of the vectors: xp[p n + i] = (x_2p,i, x_2p+1,i) (a missing second
// vector is zero), and its NC complex sources sp[(p n + i) NC + g].
template <int NC>
__global__ void __launch_bounds__(256) sources_kernel(const double *__restrict__ x, const double *__restrict__ dir,
                                                      double2 *__restrict__ xp, double2 *__restrict__ sp,
                                                      ApplyArgs a) {
    const int p = blockIdx.y;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.n; i += (int64_t)gridDim.x * blockDim.x) {
        const double2 v = make_double2(x[2 * (int64_t)p * a.n + i],
                                       2 * p + 1 < a.count ? x[(2 * (int64_t)p + 1) * a.n + i] : 0.0);
        xp[(int64_t)p * a.n + i] = v;
        double r[2 * (NC > 0 ? NC : 1)];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const double d = dir[3 * i + a.comp[c]];
            r[c] = v.x * d;
            r[NC + c] = v.y * d;
        }
#pragma unroll
        for (int g = 0; g < NC; ++g) sp[((int64_t)p * a.n + i) * NC + g] = make_double2(r[2 * g], r[2 * g + 1]);
    }
}

// y_v = C x_v, warp per row; the row is read once for NP pairs of vectors.
// Bound by the row stream (12 bytes an entry) and the gathers of x: at 15.1 M
// entries and two vectors 80 us with two separate 8-byte gathers, 52 us with
// one of 16 bytes.
template <int NP>
__global__ void __launch_bounds__(256) near_kernel(const int64_t *__restrict__ off, const uint32_t *__restrict__ col,
                                                   const double *__restrict__ val, const double2 *__restrict__ xp,
                                                   double *__restrict__ y, int64_t n, int p0, int count) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); row < n; row += warps) {
        const int64_t b = off[row], e = off[row + 1];
        double2 acc[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q) acc[q] = make_double2(0.0, 0.0);
#pragma unroll 4
        for (int64_t k = b + lane; k < e; k += 32) {
            const double a = val[k];
            const int64_t c = col[k];
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                const double2 v = xp[(int64_t)(p0 + q) * n + c];
                acc[q].x += a * v.x;
                acc[q].y += a * v.y;
            }
        }
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            for (int o = 16; o > 0; o >>= 1) {
                acc[q].x += __shfl_xor_sync(0xffffffffu, acc[q].x, o);
                acc[q].y += __shfl_xor_sync(0xffffffffu, acc[q].y, o);
            }
            const int v = 2 * (p0 + q) + lane;
            if (lane < 2 && v < count) y[(int64_t)v * n + row] = lane ? acc[q].y : acc[q].x;
        }
    }
}

// Grid sources into compact complex grids at the grid index g.  T: the
// convolution's precision.  Bound by latency (a few entries per point, each a
// gather): at 2.8 M points, 7.1 M entries and two grids 182 us with the
// entries read once per vector and x and the direction gathered apart, 55 us
// with one pass and one 16-byte gather per grid.
template <int NC, class T2>
__global__ void __launch_bounds__(256) spread_kernel(const int64_t *__restrict__ off,
                                                     const uint32_t *__restrict__ fil,
                                                     const double *__restrict__ w, const double2 *__restrict__ sp,
                                                     T2 *__restrict__ work, ApplyArgs a) {
    const int p = blockIdx.y;
    const double2 *__restrict__ s = sp + (int64_t)p * a.n * NC;
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < a.G; g += (int64_t)gridDim.x * blockDim.x) {
        const int64_t b = off[g], e = off[g + 1];
        double2 q[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) q[c] = make_double2(0.0, 0.0);
#pragma unroll 4
        for (int64_t t = b; t < e; ++t) {
            const int64_t f = fil[t];
            const double wt = w[t];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const double2 v = s[f * NC + c];
                q[c].x += wt * v.x;
                q[c].y += wt * v.y;
            }
        }
#pragma unroll
        for (int c = 0; c < NC; ++c)
            if (p * NC + c < a.grids) {
                T2 o;
                o.x = q[c].x;
                o.y = q[c].y;
                work[(int64_t)(p * NC + c) * a.G + g] = o;
            }
    }
}

// y_vi += mu0/4pi sum_c d_ic sum_g W_ig phi_{v,c}(g), warp per filament, from
// the compact potential grids: the two vectors' sums are formed per lane and
// reduced together.  At 7.1 M entries and two grids 112 us with a pass and a
// reduction for each vector and component, 58 us now.
template <int NC, class T2>
__global__ void __launch_bounds__(256) interp_kernel(const int64_t *__restrict__ off, const uint32_t *__restrict__ idx,
                                                     const double *__restrict__ w, const double *__restrict__ dir,
                                                     const T2 *__restrict__ work, double *__restrict__ y,
                                                     ApplyArgs a) {
    const int lane = threadIdx.x & 31, p = blockIdx.y;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < a.n; i += warps) {
        const int64_t b = off[i], e = off[i + 1];
        double acc[2 * NC] = {};
#pragma unroll 2
        for (int64_t t = b + lane; t < e; t += 32) {
            const int64_t g = idx[t];
            const double wt = w[t];
#pragma unroll
            for (int c = 0; c < NC; ++c)
                if (p * NC + c < a.grids) {
                    const T2 v = work[(int64_t)(p * NC + c) * a.G + g];
                    acc[2 * c] += wt * (double)v.x;
                    acc[2 * c + 1] += wt * (double)v.y;
                }
        }
        double f0 = 0.0, f1 = 0.0;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const double d = dir[3 * i + a.comp[c]];
            f0 += d * acc[c];
            f1 += d * acc[NC + c];
        }
        for (int o = 16; o > 0; o >>= 1) {
            f0 += __shfl_xor_sync(0xffffffffu, f0, o);
            f1 += __shfl_xor_sync(0xffffffffu, f1, o);
        }
        const int v = 2 * p + lane;
        if (lane < 2 && v < a.count) y[(int64_t)v * a.n + i] += kMu0Over4PiP * (lane ? f1 : f0);
    }
}

// The convolution's work buffer of `bytes`, from the device cache (grown on
// demand; the old buffer goes back to the cache, stream-ordered).
fh_status ensure_work(PfftDevice &op, size_t bytes, fh_error_info *err) {
    if (op.work_bytes >= bytes) return FH_OK;
    cudaStream_t s = (cudaStream_t)op.stream;
    if (op.d_work) cache_free(op.d_work, s);
    op.d_work = nullptr;
    op.work_bytes = 0;
    if (cache_alloc(&op.d_work, bytes, s) != cudaSuccess) {
        cudaGetLastError();
        return fail(err, FH_ERR_OUT_OF_MEMORY, "device allocation of " + std::to_string(bytes) + " bytes failed");
    }
    op.work_bytes = bytes;
    return FH_OK;
}

inline unsigned blocks_for(int64_t work, int threads, int64_t cap = 148 * 16) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((work + threads - 1) / threads, cap));
}

}  // namespace

fh_status pfft_apply_impl(PfftDevice &op, const double *d_x, double *d_y, int count, fh_error_info *err,
                          PfftProduct kind);

PfftDevice::~PfftDevice() {
    cudaStream_t s = (cudaStream_t)stream;
    fftconv_free(conv, s);
    fftconv_free(conv64, s);
    if (d_work) cache_free(d_work, s);
    void *ptrs[] = {d_dir, d_proj_off, d_proj_idx, d_proj_w, d_spread_off, d_spread_fil,
                    d_spread_w, d_near_off, d_near_col, d_near_val};
    for (void *p : ptrs) cache_free(p, s);
    if (own_stream) stream_release(s);
}

size_t PfftDevice::memory_bytes() const {
    return (size_t)projection_entries * 2 * (4 + 8) + (size_t)(n + 1 + G + 1) * 8 + (size_t)near_entries * (4 + 8) +
           (size_t)(n + 1) * 8 + (size_t)n * 3 * 8 + (size_t)P * 8 + work_bytes;
}

fh_status pfft_build(const fh_filament *fil, int64_t n, const PfftConfig &cfg, void *stream, PfftDevice &op,
                     fh_error_info *err) {
    const double t0 = now_s();
    PfftSetup st;
    fh_status e = pfft_setup(fil, n, cfg, st, err);
    if (e) return e;
    const double t1 = now_s();
    op.setup_host_s = t1 - t0;
    if (stream) {
        op.stream = stream;
    } else {
        cudaStream_t s;
        FHB_CUDA(stream_acquire(&s));
        op.stream = s;
        op.own_stream = true;
    }
    cudaStream_t s = (cudaStream_t)op.stream;
    op.n = n;
    if (n == 0) return FH_OK;
    op.grid = st.grid;
    for (int a = 0; a < 3; ++a) op.padded[a] = st.padded[a];
    op.G = st.grid.len();
    op.P = op.padded[0] * op.padded[1] * op.padded[2];
    op.components = st.components;

    // Near pairs (device search), projections, their transpose and the grid
    // approximations of the near pairs on the device; then the exact near
    // pairs (device fill, pair list) and the near-field matrix.
    std::vector<DevFil> hf((size_t)n);
    for (int64_t i = 0; i < n; ++i) hf[i] = make_devfil(fil[i]);
    DevFil *d_fil = nullptr;
    double *d_exact = nullptr;
    NearPairs near;
    struct Release {
        cudaStream_t s;
        DevFil **fil;
        double **exact;
        NearPairs *near;
        ~Release() {
            cache_free(*fil, s);
            cache_free(*exact, s);
            near_pairs_free(*near, s);
        }
    } release{s, &d_fil, &d_exact, &near};
    FHB_CUDA(upload(&d_fil, hf, s));
    const double tn = now_s();
    e = near_pairs_device(d_fil, n, st.radius, s, near, err);
    if (e) return e;
    op.setup_near_s = now_s() - tn;
    PfftDeviceSetup ds;
    e = pfft_device_setup(st, fil, near, s, ds, err);
    op.d_proj_off = ds.proj_off;
    op.d_proj_idx = ds.proj_idx;
    op.d_proj_w = ds.proj_w;
    op.d_spread_off = ds.spread_off;
    op.d_spread_fil = ds.spread_fil;
    op.d_spread_w = ds.spread_w;
    CacheBuf free_grid(s);
    free_grid.p = ds.pair_grid;
    if (e) return e;
    op.projection_entries = ds.entries;
    const int64_t np = near.count;
    FHB_CUDA(cache_alloc((void **)&d_exact, sizeof(double) * std::max<int64_t>(np, 1), s));
    if (np) {
        e = device_fill_pairs(d_fil, n, near.pairs, np, d_exact, s, nullptr, err);
        if (e) return e;
    }
    e = pfft_near_csr(n, np, near.pairs, d_exact, ds.pair_grid, near.cos, s, &op.d_near_off, &op.d_near_col,
                      &op.d_near_val, &op.near_entries, err);
    if (e) return e;
    FHB_CUDA(upload(&op.d_dir, st.directions, s));

    // The convolution's twiddles and the kernel's spectrum.
    FftConvShape shape;
    for (int a = 0; a < 3; ++a) {
        shape.n[a] = op.grid.dims[a];
        shape.m[a] = op.padded[a];
    }
    op.fft_fp32 = cfg.fft_fp32;
    e = op.fft_fp32 ? fftconv_setup<float>(shape, op.grid.spacing, op.conv, s, err)
                    : fftconv_setup<double>(shape, op.grid.spacing, op.conv, s, err);
    if (e) return e;
    if (op.fft_fp32) {
        e = fftconv_setup<double>(shape, op.grid.spacing, op.conv64, s, err);
        if (e) return e;
    }
    FHB_CUDA(cudaStreamSynchronize(s));
    op.setup_device_s = now_s() - t1;
    return FH_OK;
}

// Algorithmic bytes of one product of `count` vectors: the near-field CSR
// read once (12 B per entry), both passes over the projection (12 B per entry
// each), the vectors, and per complex grid (element size E: 8 B in FP32, 16 B
// in FP64) the pruned transform chain of fh_fftconv.cu: the sources A written
// and read, B = n0 n1 m2 and C = n0 m1 m2 written and read twice each, the
// spectrum (P reals), and the potentials A written and read.  The thin form
// has no B, C = n0 m1 n2 and m0 m1 n2 reals of spectrum.
double pfft_apply_bytes(const PfftDevice &op, int count, PfftProduct kind) {
    const int ncomp = (int)op.components.size();
    const double grids = (double)((count * ncomp + 1) / 2);
    const double E = op.fft_fp32 && kind != PfftProduct::Full ? 8.0 : 16.0;
    const FftConvShape &sh = op.conv.shape;
    const double A = (double)sh.n[0] * sh.n[1] * sh.n[2], B = (double)sh.n[0] * sh.n[1] * sh.m[2],
                 C = (double)sh.n[0] * sh.m[1] * sh.m[2], P = (double)op.P;
    const bool full = op.fft_fp32 && kind == PfftProduct::Full;
    const bool thin = kind != PfftProduct::Ports && (full ? op.conv64 : op.conv).thin;
    const double thinner = (double)sh.n[2] / sh.m[2];
    const double conv = thin ? E * (4.0 * A + 4.0 * C * thinner) + (E / 2.0) * P * thinner
                             : E * (4.0 * A + 4.0 * B + 4.0 * C) + (E / 2.0) * P;
    return 12.0 * (double)op.near_entries + 24.0 * (double)op.projection_entries + 32.0 * (double)op.n * count +
           grids * conv;
}

fh_status pfft_apply(PfftDevice &op, const double *d_x, double *d_y, int count, fh_error_info *err,
                     PfftProduct kind) {
    if (op.n == 0 || count <= 0) return FH_OK;
    prof_begin((cudaStream_t)op.stream, FH_PROF_PFFT_APPLY);
    fh_status st = pfft_apply_impl(op, d_x, d_y, count, err, kind);
    prof_end((cudaStream_t)op.stream, FH_PROF_PFFT_APPLY, pfft_apply_bytes(op, count, kind));
    return st;
}

namespace {
ApplyArgs apply_args(const PfftDevice &op, int count) {
    const int ncomp = (int)op.components.size();
    ApplyArgs a;
    a.n = op.n;
    a.G = op.G;
    for (int c = 0; c < 3; ++c) a.comp[c] = c < ncomp ? op.components[c] : 0;
    a.count = count;
    a.pairs = (count + 1) / 2;
    a.grids = (count * ncomp + 1) / 2;
    return a;
}

template <int NC, class T>
fh_status apply_far(PfftDevice &op, const FftConvTables &conv, const double2 *sp, T *work, double *d_y,
                    const ApplyArgs &a, PfftProduct kind, fh_error_info *err) {
    using T2 = typename std::conditional<sizeof(T) == 4, float2, double2>::type;
    cudaStream_t s = (cudaStream_t)op.stream;
    T2 *grids = reinterpret_cast<T2 *>(work);
    spread_kernel<NC, T2><<<dim3(blocks_for(op.G, 256), a.pairs), 256, 0, s>>>(op.d_spread_off, op.d_spread_fil,
                                                                              op.d_spread_w, sp, grids, a);
    FHB_CUDA(cudaGetLastError());
    const fh_status e = sizeof(T) == 4 && kind == PfftProduct::Ports ? fftconv_run_ports(conv, work, a.grids, s, err)
                                                                     : fftconv_run<T>(conv, work, a.grids, s, err);
    if (e) return e;
    interp_kernel<NC, T2><<<dim3(blocks_for(op.n * 32, 256), a.pairs), 256, 0, s>>>(
        op.d_proj_off, op.d_proj_idx, op.d_proj_w, op.d_dir, grids, d_y, a);
    FHB_CUDA(cudaGetLastError());
    return FH_OK;
}

template <int NC>
fh_status apply_components(PfftDevice &op, const double *d_x, double *d_y, int count, PfftProduct kind,
                           fh_error_info *err) {
    cudaStream_t s = (cudaStream_t)op.stream;
    const ApplyArgs a = apply_args(op, count);
    const bool fp32 = op.fft_fp32 && kind != PfftProduct::Full;
    const FftConvTables &conv = op.fft_fp32 && !fp32 ? op.conv64 : op.conv;
    // workspace: the vectors' pairs, their sources, the convolution's grids
    const size_t vectors = sizeof(double2) * (size_t)op.n * a.pairs * (1 + NC);
    const size_t grids = NC ? (fp32 ? 8 : 16) * fftconv_work_elems(conv.shape) * (size_t)a.grids : 0;
    fh_status e = ensure_work(op, vectors + grids, err);
    if (e) return e;
    double2 *xp = static_cast<double2 *>(op.d_work);
    double2 *sp = xp + op.n * a.pairs;
    void *work = sp + op.n * a.pairs * NC;
    sources_kernel<NC><<<dim3(blocks_for(op.n, 256), a.pairs), 256, 0, s>>>(d_x, op.d_dir, xp, sp, a);
    for (int p = 0; p < a.pairs; p += 2) {
        const unsigned blocks = blocks_for(op.n * 32, 256);
        if (p + 1 < a.pairs)
            near_kernel<2><<<blocks, 256, 0, s>>>(op.d_near_off, op.d_near_col, op.d_near_val, xp, d_y, op.n, p, count);
        else
            near_kernel<1><<<blocks, 256, 0, s>>>(op.d_near_off, op.d_near_col, op.d_near_val, xp, d_y, op.n, p, count);
    }
    FHB_CUDA(cudaGetLastError());
    if constexpr (NC > 0) {
        if (fp32) return apply_far<NC, float>(op, conv, sp, static_cast<float *>(work), d_y, a, kind, err);
        return apply_far<NC, double>(op, conv, sp, static_cast<double *>(work), d_y, a, kind, err);
    }
    return FH_OK;
}
}  // namespace

fh_status pfft_apply_impl(PfftDevice &op, const double *d_x, double *d_y, int count, fh_error_info *err,
                          PfftProduct kind) {
    switch (op.components.size()) {
        case 0: return apply_components<0>(op, d_x, d_y, count, kind, err);
        case 1: return apply_components<1>(op, d_x, d_y, count, kind, err);
        case 2: return apply_components<2>(op, d_x, d_y, count, kind, err);
        default: return apply_components<3>(op, d_x, d_y, count, kind, err);
    }
}

}  // namespace fhb

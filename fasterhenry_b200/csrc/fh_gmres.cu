// Device GMRES (see fh_gmres.cuh).  The Arnoldi loop, the rotations and the
// stopping rule follow gmres.rs:91-215; every vector operation is a kernel
// on the solver's stream, and the host reads back one Hessenberg column and
// one norm per Arnoldi step, on a second stream: the solver's own has the next
// step's product queued by then, so the device does not wait for the host's
// part of a step (70 us of 740 at 107,144 filaments; 15 are left).
#include <cmath>
#include <complex>
#include <string>
#include <vector>

#include "fh_device.cuh"
#include "fh_gmres.cuh"

namespace fhb {

namespace {

constexpr int kRB = 256;  // reduction blocks (fixed: the combination order never depends on n's scheduling)
constexpr int kRT = 256;  // threads per block

// Layout of GmresWork::red (doubles).
constexpr int kMaxPartial = 2 * kRB;            // kRB
constexpr int kSumPartial = 3 * kRB;            // kRB
constexpr int kScale = 4 * kRB;                 // 1
constexpr int kSum = 4 * kRB + 1;               // 1
constexpr int kRedLen = 4 * kRB + 8;

using cplx = std::complex<double>;

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }

__global__ void __launch_bounds__(kRT) maxabs_partial_kernel(const double2 *__restrict__ v, int64_t n,
                                                             double *__restrict__ partial) {
    __shared__ double sh[kRT];
    double m = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * kRT + threadIdx.x; i < n; i += (int64_t)kRB * kRT) {
        const double a = hypot(v[i].x, v[i].y);
        m = fmax(m, a);
        if (a != a) m = a;  // NaN propagates
    }
    sh[threadIdx.x] = m;
    __syncthreads();
    for (int s = kRT / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            const double o = sh[threadIdx.x + s];
            sh[threadIdx.x] = (o != o) ? o : fmax(sh[threadIdx.x], o);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

// sum |v_i / scale|^2 (gmres.rs:234-241: the scaled norm); scale is the
// largest of the kRB maxima, which every block finds for itself.
__global__ void __launch_bounds__(kRT) sumsq_partial_kernel(const double2 *__restrict__ v, int64_t n,
                                                            const double *__restrict__ maxima,
                                                            double *__restrict__ scale,
                                                            double *__restrict__ partial) {
    __shared__ double sh[kRT];
    static_assert(kRB == kRT, "one maximum per thread");
    sh[threadIdx.x] = maxima[threadIdx.x];
    __syncthreads();
    for (int s = kRT / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            const double o = sh[threadIdx.x + s];
            sh[threadIdx.x] = (o != o) ? o : fmax(sh[threadIdx.x], o);
        }
        __syncthreads();
    }
    const double sc = sh[0];
    if (blockIdx.x == 0 && threadIdx.x == 0) *scale = sc;
    double acc = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * kRT + threadIdx.x; i < n; i += (int64_t)kRB * kRT) {
        const double a = v[i].x / sc, b = v[i].y / sc;
        acc += a * a + b * b;
    }
    __syncthreads();  // sh[0] has been read
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int s = kRT / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

__global__ void __launch_bounds__(kRT) sum_final_kernel(const double *__restrict__ partial, double *__restrict__ out) {
    __shared__ double sh[kRT];
    sh[threadIdx.x] = partial[threadIdx.x];
    __syncthreads();
    for (int s = kRT / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = sh[0];
}

// The projections of w on the cnt basis vectors V_0 .. V_cnt-1 at once
// (classical Gram-Schmidt): conj(V_k) . w over one of kDotChunks chunks of
// the rows for kDotVecs vectors per block, into partial[2 (k kDotChunks +
// chunk)].
//
// Bound by reading the basis once: 1.25 MB per vector at 78,307 loops.  A
// block takes several vectors so that w is read once for them and each
// thread has kDotVecs loads in flight, and its 2 kDotVecs sums cross the warp
// in 16 exchanges (each step halves the values a lane keeps).  Over a cycle
// of 400 vectors of 78,307: 163 us on average with one vector at a time per
// block and a block-wide reduction for each, 36 us now.  The chunks depend on
// n alone, so a result does not depend on the device's scheduling.
constexpr int kDotVecs = 8;
constexpr int kDotChunks = 64;
constexpr int kDotThreads = 128;
__global__ void __launch_bounds__(kDotThreads) multidot_partial_kernel(const double2 *__restrict__ V,
                                                                       const double2 *__restrict__ w, int64_t n,
                                                                       int cnt, double *__restrict__ partial) {
    __shared__ double sh[kDotThreads / 32][2 * kDotVecs];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k0 = blockIdx.y * kDotVecs;
    const int64_t rows = (n + kDotChunks - 1) / kDotChunks;
    const int64_t begin = blockIdx.x * rows, end = begin + rows < n ? begin + rows : n;
    const double2 *vk[kDotVecs];
#pragma unroll
    for (int q = 0; q < kDotVecs; ++q) vk[q] = V + (size_t)(k0 + q < cnt ? k0 + q : cnt - 1) * n;
    double acc[2 * kDotVecs] = {};
    for (int64_t i = begin + threadIdx.x; i < end; i += kDotThreads) {
        const double2 b = w[i];
#pragma unroll
        for (int q = 0; q < kDotVecs; ++q) {
            const double2 a = vk[q][i];
            acc[2 * q] += a.x * b.x + a.y * b.y;
            acc[2 * q + 1] += a.x * b.y - a.y * b.x;
        }
    }
    // After the step of distance o a lane holds the sums over its pair of the
    // half of the values that its bit o selects; value `lane >> 1` at last.
#pragma unroll
    for (int o = 16, have = 2 * kDotVecs; o > 1; o >>= 1, have >>= 1) {
#pragma unroll
        for (int q = 0; q < kDotVecs; ++q)
            if (q < have / 2) {
                const double keep = lane & o ? acc[q + have / 2] : acc[q];
                const double give = lane & o ? acc[q] : acc[q + have / 2];
                acc[q] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
    }
    acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
    if (!(lane & 1)) sh[warp][lane >> 1] = acc[0];
    __syncthreads();
    if (threadIdx.x < 2 * kDotVecs) {
        double t = sh[0][threadIdx.x];
        for (int q = 1; q < kDotThreads / 32; ++q) t += sh[q][threadIdx.x];
        const int k = k0 + threadIdx.x / 2;
        if (k < cnt) partial[2 * ((size_t)k * kDotChunks + blockIdx.x) + (threadIdx.x & 1)] = t;
    }
}

// h[k] = the sum of vector k's kDotChunks partials (a warp each, fixed tree).
__global__ void __launch_bounds__(kRT) multidot_final_kernel(const double *__restrict__ partial, int cnt,
                                                             double2 *__restrict__ h) {
    const int lane = threadIdx.x & 31, k = blockIdx.x * (kRT / 32) + (threadIdx.x >> 5);
    if (k >= cnt) return;
    const double2 *p = reinterpret_cast<const double2 *>(partial) + (size_t)k * kDotChunks;
    double2 t = make_double2(0.0, 0.0);
    for (int c = lane; c < kDotChunks; c += 32) t = cadd(t, p[c]);
    for (int o = 16; o > 0; o >>= 1) {
        t.x += __shfl_xor_sync(0xffffffffu, t.x, o);
        t.y += __shfl_xor_sync(0xffffffffu, t.y, o);
    }
    if (lane == 0) h[k] = t;
}

// w -= sum_k h[k] V_k, the terms taken in increasing k.  Bound by reading the
// basis: over a cycle of 400 vectors of 78,307, 43 us on average with the
// compiler's four loads in flight per thread, 32 us with eight.
__global__ void multi_axpy_kernel(double2 *__restrict__ w, const double2 *__restrict__ V,
                                  const double2 *__restrict__ h, int cnt, int64_t n) {
    extern __shared__ double2 hs[];
    for (int k = threadIdx.x; k < cnt; k += blockDim.x) hs[k] = h[k];
    __syncthreads();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double2 y = w[i];
        int k = 0;
        for (; k + 8 <= cnt; k += 8) {
            double2 b[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) b[q] = V[(size_t)(k + q) * n + i];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const double2 a = hs[k + q];
                y.x += -a.x * b[q].x + a.y * b[q].y;
                y.y += -a.x * b[q].y - a.y * b[q].x;
            }
        }
        for (; k < cnt; ++k) {
            const double2 a = hs[k], b = V[(size_t)k * n + i];
            y.x += -a.x * b.x + a.y * b.y;
            y.y += -a.x * b.y - a.y * b.x;
        }
        w[i] = y;
    }
}

__global__ void div_real_kernel(double2 *__restrict__ out, const double2 *__restrict__ in, double s, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = make_double2(in[i].x / s, in[i].y / s);
}

// out = in / |in|, the norm from its scale norm[0] and the kRB partial sums;
// their total goes to norm[1] for the host.
__global__ void __launch_bounds__(kRT) normalize_kernel(double2 *__restrict__ out, const double2 *__restrict__ in,
                                                        const double *__restrict__ partial,
                                                        double *__restrict__ norm, int64_t n) {
    __shared__ double sh[kRT];
    sh[threadIdx.x] = partial[threadIdx.x];
    __syncthreads();
    for (int s = kRT / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    const double scale = norm[0], sum = sh[0];
    const double s = scale == 0.0 || !isfinite(scale) ? scale : scale * sqrt(sum);
    if (blockIdx.x == 0 && threadIdx.x == 0) norm[1] = sum;
    for (int64_t i = blockIdx.x * (int64_t)kRT + threadIdx.x; i < n; i += (int64_t)gridDim.x * kRT)
        out[i] = make_double2(in[i].x / s, in[i].y / s);
}

__global__ void sub_kernel(double2 *__restrict__ r, const double2 *__restrict__ b, const double2 *__restrict__ ax,
                           int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        r[i] = make_double2(b[i].x - ax[i].x, b[i].y - ax[i].y);
}

__global__ void add_kernel(double2 *__restrict__ x, const double2 *__restrict__ c, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        x[i] = make_double2(x[i].x + c[i].x, x[i].y + c[i].y);
}

inline unsigned grid_of(int64_t n) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 148 * 8)); }

// The reference's complex division (num-complex): (a conj(b)) / |b|^2.
cplx cdiv_ref(cplx a, cplx b) {
    const double ns = b.real() * b.real() + b.imag() * b.imag();
    return cplx((a.real() * b.real() + a.imag() * b.imag()) / ns, (a.imag() * b.real() - a.real() * b.imag()) / ns);
}
cplx cmul_ref(cplx a, cplx b) {
    return cplx(a.real() * b.real() - a.imag() * b.imag(), a.real() * b.imag() + a.imag() * b.real());
}

// The rotation G = [c s; -conj(s) c] with G [a; b] = [r; 0] (gmres.rs:244-257).
void givens(cplx a, cplx b, double &c, cplx &s, cplx &r) {
    const double abs_a = std::hypot(a.real(), a.imag()), abs_b = std::hypot(b.real(), b.imag());
    if (abs_b == 0.0) {
        c = 1.0;
        s = 0.0;
        r = a;
        return;
    }
    if (abs_a == 0.0) {
        c = 0.0;
        s = 1.0;
        r = b;
        return;
    }
    const double length = std::hypot(abs_a, abs_b);
    const cplx phase(a.real() / abs_a, a.imag() / abs_a);
    c = abs_a / length;
    s = cmul_ref(phase, cplx(b.real() / length, -b.imag() / length));
    r = cplx(phase.real() * length, phase.imag() * length);
}

struct Norm {
    double scale = 0, sum = 0;
    double value() const { return (scale == 0.0 || !std::isfinite(scale)) ? scale : scale * std::sqrt(sum); }
};

}  // namespace

GmresWork::~GmresWork() { release(); }

void GmresWork::release() {
    void *p[] = {V, w, r, t, u, h, red, part};
    for (void *q : p) cache_free(q, stream);
    V = w = r = t = u = h = nullptr;
    red = part = nullptr;
}

fh_status GmresWork::ensure(int64_t n_, int restart_, cudaStream_t s, fh_error_info *err) {
    if (n_ <= n && restart_ <= restart && V) return FH_OK;
    release();
    stream = s;
    n = n_;
    restart = restart_;
    auto alloc = [&](void **q, size_t bytes) { return cache_alloc(q, std::max<size_t>(bytes, 16), s); };
    if (alloc((void **)&V, sizeof(double2) * (size_t)(restart + 1) * n) != cudaSuccess ||
        alloc((void **)&w, sizeof(double2) * n) != cudaSuccess || alloc((void **)&r, sizeof(double2) * n) != cudaSuccess ||
        alloc((void **)&t, sizeof(double2) * n) != cudaSuccess || alloc((void **)&u, sizeof(double2) * n) != cudaSuccess ||
        alloc((void **)&h, sizeof(double2) * (2 * (restart + 1) + 1)) != cudaSuccess ||
        alloc((void **)&red, sizeof(double) * kRedLen) != cudaSuccess ||
        alloc((void **)&part, sizeof(double) * 2 * kDotChunks * (size_t)(restart + 1)) != cudaSuccess) {
        cudaGetLastError();
        return fail(err, FH_ERR_OUT_OF_MEMORY, "device allocation of the GMRES workspace failed");
    }
    return FH_OK;
}

fh_status gmres_solve(int64_t n, const DeviceOp &apply, const DeviceOp &precondition, const double2 *d_b, double2 *d_x,
                      const GmresParams &params, cudaStream_t s, GmresWork &work, GmresOutcome *out,
                      fh_error_info *err) {
    GmresOutcome oc;
    const int restart = (int)std::max<int64_t>(1, std::min<int64_t>(params.restart, n));
    fh_status st = work.ensure(n, restart, s, err);
    if (st) return st;
    auto norm_of = [&](const double2 *v, Norm &nm) -> fh_status {
        maxabs_partial_kernel<<<kRB, kRT, 0, s>>>(v, n, work.red + kMaxPartial);
        sumsq_partial_kernel<<<kRB, kRT, 0, s>>>(v, n, work.red + kMaxPartial, work.red + kScale,
                                                 work.red + kSumPartial);
        sum_final_kernel<<<1, kRT, 0, s>>>(work.red + kSumPartial, work.red + kSum);
        FHB_CUDA(cudaGetLastError());
        double hv[2];
        FHB_CUDA(cudaMemcpyAsync(hv, work.red + kScale, sizeof hv, cudaMemcpyDeviceToHost, s));
        FHB_CUDA(cudaStreamSynchronize(s));
        nm.scale = hv[0];
        nm.sum = hv[1];
        return FH_OK;
    };
    auto residual = [&](double &rn) -> fh_status {
        fh_status e = apply(d_x, work.t, err);
        if (e) return e;
        sub_kernel<<<grid_of(n), 256, 0, s>>>(work.r, d_b, work.t, n);
        FHB_CUDA(cudaGetLastError());
        Norm nm;
        e = norm_of(work.r, nm);
        rn = nm.value();
        return e;
    };
    Norm bn;
    st = norm_of(d_b, bn);
    if (st) return st;
    const double b_norm = bn.value();
    if (b_norm == 0.0) {
        FHB_CUDA(cudaMemsetAsync(d_x, 0, sizeof(double2) * n, s));
        FHB_CUDA(cudaStreamSynchronize(s));
        oc.converged = true;
        if (out) *out = oc;
        return FH_OK;
    }
    const double target = params.tolerance * b_norm;
    int64_t iterations = 0;
    double r_norm = 0.0;
    st = residual(r_norm);
    if (st) return st;
    std::vector<cplx> hcol_dev(2 * (size_t)(restart + 1) + 1);
    struct Side {  // the stream of the readbacks, and where it may start
        cudaStream_t s = nullptr;
        cudaEvent_t ready = nullptr;
        ~Side() {
            if (ready) cudaEventDestroy(ready);
            if (s) stream_release(s);
        }
    } side;
    FHB_CUDA(stream_acquire(&side.s));
    FHB_CUDA(cudaEventCreateWithFlags(&side.ready, cudaEventDisableTiming));
    for (;;) {
        oc.iterations = iterations;
        oc.relative_residual = r_norm / b_norm;
        if (r_norm <= target) {
            oc.converged = true;
            break;
        }
        if (iterations >= params.max_iterations || !std::isfinite(r_norm)) {
            oc.converged = false;
            break;
        }
        // One Arnoldi cycle from the current residual.
        div_real_kernel<<<grid_of(n), 256, 0, s>>>(work.V, work.r, r_norm, n);
        FHB_CUDA(cudaGetLastError());
        std::vector<std::vector<cplx>> hess;
        std::vector<std::pair<double, cplx>> rot;
        std::vector<cplx> g((size_t)restart + 1, cplx(0.0, 0.0));
        g[0] = cplx(r_norm, 0.0);
        auto product = [&](int j) -> fh_status {  // w = A M V_j
            fh_status e = precondition(work.V + (size_t)j * n, work.u, err);
            return e ? e : apply(work.u, work.w, err);
        };
        bool queued = false;
        while ((int)hess.size() < restart && iterations < params.max_iterations) {
            const int j = (int)hess.size();
            if (!queued && (st = product(j))) return st;
            iterations += 1;
            // Classical Gram-Schmidt twice: each pass projects w on all of
            // V_0 .. V_j in one product and removes them in one update (the
            // reference's modified Gram-Schmidt applied twice reaches the same
            // orthogonality; three launches per pass instead of three per
            // basis vector).
            for (int pass = 0; pass < 2; ++pass) {
                double2 *hp = work.h + pass * (j + 1);
                multidot_partial_kernel<<<dim3(kDotChunks, (unsigned)(j / kDotVecs + 1)), kDotThreads, 0, s>>>(
                    work.V, work.w, n, j + 1, work.part);
                multidot_final_kernel<<<j / (kRT / 32) + 1, kRT, 0, s>>>(work.part, j + 1, hp);
                multi_axpy_kernel<<<grid_of(n), 256, sizeof(double2) * (j + 1), s>>>(work.w, work.V, hp, j + 1, n);
            }
            // the norm (after the columns in h), and V_j+1 from it
            double *norm = reinterpret_cast<double *>(work.h + 2 * (j + 1));
            maxabs_partial_kernel<<<kRB, kRT, 0, s>>>(work.w, n, work.red + kMaxPartial);
            sumsq_partial_kernel<<<kRB, kRT, 0, s>>>(work.w, n, work.red + kMaxPartial, norm, work.red + kSumPartial);
            normalize_kernel<<<grid_of(n), kRT, 0, s>>>(work.V + (size_t)(j + 1) * n, work.w, work.red + kSumPartial,
                                                        norm, n);
            FHB_CUDA(cudaGetLastError());
            FHB_CUDA(cudaEventRecord(side.ready, s));
            // The next step's product, unless this step should be the last: the
            // residual falls as in the step before, with a factor 2 in hand.
            const double now = std::abs(g[(size_t)j]), rate = j > 0 ? now / std::abs(g[(size_t)j - 1]) : 1.0;
            queued = j + 1 < restart && iterations < params.max_iterations && now * rate > 2.0 * target;
            if (queued && (st = product(j + 1))) return st;
            FHB_CUDA(cudaStreamWaitEvent(side.s, side.ready, 0));
            FHB_CUDA(cudaMemcpyAsync(hcol_dev.data(), work.h, sizeof(double2) * (2 * (size_t)(j + 1) + 1),
                                     cudaMemcpyDeviceToHost, side.s));
            FHB_CUDA(cudaStreamSynchronize(side.s));
            Norm wn;
            wn.scale = hcol_dev[2 * (size_t)(j + 1)].real();
            wn.sum = hcol_dev[2 * (size_t)(j + 1)].imag();
            const double next_norm = wn.value();
            std::vector<cplx> column((size_t)j + 2, cplx(0.0, 0.0));
            for (int pass = 0; pass < 2; ++pass)
                for (int k = 0; k <= j; ++k) column[k] += hcol_dev[pass * (j + 1) + k];
            column[j + 1] = cplx(next_norm, 0.0);
            for (size_t i = 0; i < rot.size(); ++i) {
                const double c = rot[i].first;
                const cplx sr = rot[i].second;
                const cplx a = column[i], b = column[i + 1];
                column[i] = cplx(a.real() * c, a.imag() * c) + cmul_ref(sr, b);
                column[i + 1] = cplx(b.real() * c, b.imag() * c) - cmul_ref(std::conj(sr), a);
            }
            double c;
            cplx sr, rr;
            givens(column[j], column[j + 1], c, sr, rr);
            column[j] = rr;
            column[j + 1] = cplx(0.0, 0.0);
            rot.push_back({c, sr});
            const cplx gj = g[j];
            g[j] = cplx(gj.real() * c, gj.imag() * c);
            g[j + 1] = -cmul_ref(std::conj(sr), gj);
            hess.push_back(column);
            if (next_norm == 0.0 || std::abs(g[j + 1]) <= target) break;
        }
        // Back substitution, then x += M (V y).
        const int steps = (int)hess.size();
        std::vector<cplx> y((size_t)steps);
        for (int i = steps - 1; i >= 0; --i) {
            cplx sum = g[i];
            for (int k = i + 1; k < steps; ++k) sum -= cmul_ref(hess[k][i], y[k]);
            y[i] = cdiv_ref(sum, hess[i][i]);
        }
        for (cplx &v : y) v = -v;
        FHB_CUDA(cudaMemcpyAsync(work.h, y.data(), sizeof(double2) * (size_t)steps, cudaMemcpyHostToDevice, s));
        FHB_CUDA(cudaMemsetAsync(work.u, 0, sizeof(double2) * n, s));
        multi_axpy_kernel<<<grid_of(n), 256, sizeof(double2) * steps, s>>>(work.u, work.V, work.h, steps, n);
        FHB_CUDA(cudaGetLastError());
        st = precondition(work.u, work.t, err);
        if (st) return st;
        add_kernel<<<grid_of(n), 256, 0, s>>>(d_x, work.t, n);
        FHB_CUDA(cudaGetLastError());
        st = residual(r_norm);
        if (st) return st;
    }
    if (out) *out = oc;
    return FH_OK;
}

}  // namespace fhb

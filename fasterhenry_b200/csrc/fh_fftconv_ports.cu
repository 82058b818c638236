// The FP32 convolution of the port columns: L times each port's current, once
// per system, which becomes the right-hand side and Z_pp.  GMRES's FP32
// products are refined against the FP64 operator, so their rounding leaves no
// trace in Z; the port columns' rounding goes into Z as it is (3e-9 to 3e-8
// of Z at 10,000 to 107,000 filaments).  They therefore stay on the
// transform that every earlier Z was computed with -- a Stockham chain of
// radix 4, 2, 3 and 5 passes between two shared buffers -- and are not moved
// to the faster one of fh_fftconv.cu, whose rounding is as large but another
// one: Z of the same deck then agrees to 1e-12 with earlier runs instead of
// 1e-8.  Its steps are those of fh_fftconv.cu; at 1200 x 1200 x 15 torus
// points one product takes 0.9 ms against 0.3 ms, once per port.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "fh_device.cuh"
#include "fh_fftconv.h"

namespace fhb {
namespace {

using V = float2;
using T = float;
constexpr int kThreads = 512;
constexpr size_t kSmemBudget = 100 * 1024;  // two CTAs per SM
constexpr int kMaxPasses = 24;

// Radices 4, then 2, 3, 5.
struct Passes {
    int m = 1;
    int nfac = 0;
    int fac[kMaxPasses] = {};
};
Passes passes_of(int m) {
    Passes ax;
    ax.m = m;
    for (int p : {4, 2, 3, 5})
        for (; m % p == 0; m /= p) ax.fac[ax.nfac++] = p;
    return ax;
}

__device__ __forceinline__ V cmul(V a, V b) {
    V r;
    r.x = a.x * b.x - a.y * b.y;
    r.y = a.x * b.y + a.y * b.x;
    return r;
}

// R-point DFT of v in place, W = exp(sign 2 pi i / R).
template <int R>
__device__ __forceinline__ void small_dft(V (&v)[R], int sign) {
    if constexpr (R == 2) {
        V a = v[0], b = v[1];
        v[0].x = a.x + b.x;
        v[0].y = a.y + b.y;
        v[1].x = a.x - b.x;
        v[1].y = a.y - b.y;
    } else if constexpr (R == 4) {
        const V a = v[0], b = v[1], c = v[2], d = v[3];
        V s0, s1, d0, d1;
        s0.x = a.x + c.x, s0.y = a.y + c.y;
        d0.x = a.x - c.x, d0.y = a.y - c.y;
        s1.x = b.x + d.x, s1.y = b.y + d.y;
        d1.x = b.x - d.x, d1.y = b.y - d.y;
        // (b - d) times sign * i
        V jd;
        jd.x = -(T)sign * d1.y;
        jd.y = (T)sign * d1.x;
        v[0].x = s0.x + s1.x, v[0].y = s0.y + s1.y;
        v[2].x = s0.x - s1.x, v[2].y = s0.y - s1.y;
        v[1].x = d0.x + jd.x, v[1].y = d0.y + jd.y;
        v[3].x = d0.x - jd.x, v[3].y = d0.y - jd.y;
    } else {
        // cos and sin of 2 pi k / R, k = 0 .. R-1
        constexpr double c3[3] = {1.0, -0.5, -0.5};
        constexpr double s3[3] = {0.0, 0.86602540378443864676, -0.86602540378443864676};
        constexpr double c5[5] = {1.0, 0.30901699437494742410, -0.80901699437494742410, -0.80901699437494742410,
                                  0.30901699437494742410};
        constexpr double s5[5] = {0.0, 0.95105651629515357212, 0.58778525229247312917, -0.58778525229247312917,
                                  -0.95105651629515357212};
        V out[R];
#pragma unroll
        for (int b = 0; b < R; ++b) {
            V acc = v[0];
#pragma unroll
            for (int a = 1; a < R; ++a) {
                const int e = (a * b) % R;
                const T c = (T)(R == 3 ? c3[e] : c5[e]);
                const T s = (T)sign * (T)(R == 3 ? s3[e] : s5[e]);
                acc.x += v[a].x * c - v[a].y * s;
                acc.y += v[a].x * s + v[a].y * c;
            }
            out[b] = acc;
        }
#pragma unroll
        for (int b = 0; b < R; ++b) v[b] = out[b];
    }
}

// One Stockham pass of radix R over `lines` interleaved lines of length m
// (element t of line l at t * lines + l), src -> dst; tw holds
// exp(-2 pi i t / m) in shared memory.
template <int R>
__device__ void stockham_pass(const V *__restrict__ src, V *__restrict__ dst, int m, int lines, int Ns,
                              const V *__restrict__ tw, int sign) {
    const int nb = m / R;
    const int tw_step = m / (Ns * R);
    for (int idx = threadIdx.x; idx < nb * lines; idx += blockDim.x) {
        const int line = idx % lines, j = idx / lines;
        V v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = src[(j + r * nb) * lines + line];
        const int k = j % Ns;
#pragma unroll
        for (int r = 1; r < R; ++r) {
            V w = tw[k * r * tw_step];
            if (sign > 0) w.y = -w.y;
            v[r] = cmul(v[r], w);
        }
        small_dft<R>(v, sign);
        const int base = (j / Ns) * Ns * R + k;
#pragma unroll
        for (int r = 0; r < R; ++r) dst[(base + r * Ns) * lines + line] = v[r];
    }
}

// The transform of `lines` lines of length m held in a (interleaved), with b
// as the second buffer; returns the buffer holding the result.
__device__ V *stockham(V *a, V *b, int m, int lines, const Passes &ax, const V *__restrict__ tw, int sign) {
    int Ns = 1;
    for (int f = 0; f < ax.nfac; ++f) {
        const int R = ax.fac[f];
        __syncthreads();
        if (R == 4)
            stockham_pass<4>(a, b, m, lines, Ns, tw, sign);
        else if (R == 2)
            stockham_pass<2>(a, b, m, lines, Ns, tw, sign);
        else if (R == 3)
            stockham_pass<3>(a, b, m, lines, Ns, tw, sign);
        else
            stockham_pass<5>(a, b, m, lines, Ns, tw, sign);
        Ns *= R;
        V *t = a;
        a = b;
        b = t;
    }
    __syncthreads();
    return a;
}

// One pruned axis transform over a batch of arrays.  An array holds
// `outer` x len x `inner` complex elements (len = n_in for the input, keep
// for the output); line (o, c) is elements (o len + t) inner + c.  Lines are
// tiled `tile` at a time: consecutive o when inner == 1 (each line
// contiguous), else consecutive c.  With `spectrum`, the forward transform is
// multiplied by spectrum[t inner + c] (real) and transformed back (sign
// flipped) before the write.  in and out may be the same array (the fused
// axis-0 step): a CTA reads its whole tile before it writes, and tiles are
// disjoint.
__global__ void __launch_bounds__(kThreads)
    fft_lines_kernel(const V *in, V *out,
                     int64_t in_stride, int64_t out_stride, int64_t outer, int64_t inner, int n_in, int keep,
                     Passes ax, const V *__restrict__ tw_global, int sign, int tile,
                     const T *__restrict__ spectrum) {
    extern __shared__ __align__(16) unsigned char fft_smem[];
    V *bufa = reinterpret_cast<V *>(fft_smem);
    V *bufb = bufa + (size_t)tile * ax.m;
    V *tw = bufb + (size_t)tile * ax.m;  // the twiddles, read by every pass
    const int m = ax.m;
    for (int t = threadIdx.x; t < m; t += blockDim.x) tw[t] = tw_global[t];
    const V *src = in + (int64_t)blockIdx.y * in_stride;
    V *dst = out + (int64_t)blockIdx.y * out_stride;
    const bool contiguous = inner == 1;
    const int64_t tiles = contiguous ? (outer + tile - 1) / tile : outer * ((inner + tile - 1) / tile);
    for (int64_t tt = blockIdx.x; tt < tiles; tt += gridDim.x) {
        int64_t o0, c0;
        int lines;
        if (contiguous) {
            o0 = tt * tile;
            c0 = 0;
            lines = (int)(outer - o0 < tile ? outer - o0 : (int64_t)tile);
        } else {
            const int64_t per = (inner + tile - 1) / tile;
            o0 = tt / per;
            c0 = (tt % per) * tile;
            lines = (int)(inner - c0 < tile ? inner - c0 : (int64_t)tile);
        }
        __syncthreads();  // the previous tile's reads of the buffers are done
        // load (zero-padded to m)
        for (int idx = threadIdx.x; idx < lines * m; idx += blockDim.x) {
            int l, t;
            if (contiguous) {
                l = idx / m;
                t = idx % m;
            } else {
                t = idx / lines;
                l = idx % lines;
            }
            V v;
            v.x = v.y = (T)0;
            if (t < n_in)
                v = contiguous ? src[(o0 + l) * (int64_t)n_in + t] : src[(o0 * n_in + t) * inner + c0 + l];
            bufa[t * lines + l] = v;
        }
        V *res = stockham(bufa, bufb, m, lines, ax, tw, sign);
        if (spectrum) {
            for (int idx = threadIdx.x; idx < lines * m; idx += blockDim.x) {
                const int t = idx / lines, l = idx % lines;
                const T s = spectrum[(int64_t)t * inner + c0 + l];
                V v = res[idx];
                v.x *= s;
                v.y *= s;
                res[idx] = v;
            }
            V *other = res == bufa ? bufb : bufa;
            res = stockham(res, other, m, lines, ax, tw, -sign);
        }
        for (int idx = threadIdx.x; idx < lines * keep; idx += blockDim.x) {
            int l, t;
            if (contiguous) {
                l = idx / keep;
                t = idx % keep;
            } else {
                t = idx / lines;
                l = idx % lines;
            }
            const V v = res[t * lines + l];
            if (contiguous)
                dst[(o0 + l) * (int64_t)keep + t] = v;
            else
                dst[(o0 * keep + t) * inner + c0 + l] = v;
        }
    }
}

// The spectrum in natural order from the order of fh_fftconv.cu.
__global__ void spectrum_natural_kernel(const T *__restrict__ in, T *__restrict__ out, int64_t m0, int64_t m1,
                                        int64_t m2, const int *__restrict__ place) {
    const int64_t total = m0 * m1 * m2;
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < total; p += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = p % m2, rest = p / m2, j = rest % m1, i = rest / m1;
        out[p] = in[((int64_t)place[i] * m1 + place[m0 + j]) * m2 + place[m0 + m1 + k]];
    }
}

// One axis step: outer x n_in x inner -> outer x keep x inner, `batch` arrays.
fh_status axis_step(const V *in, V *out, int64_t in_stride, int64_t out_stride, int64_t outer, int64_t inner, int n_in,
                    int keep, const Passes &ax, const V *tw, int sign, const T *spectrum, int batch, cudaStream_t s,
                    fh_error_info *err) {
    // Lines per CTA: as many as two buffers of them and the twiddles fit the
    // budget, up to about 8,192 points per tile.
    const size_t line = sizeof(V) * (size_t)ax.m;
    const size_t want = std::max<size_t>(16, 8192 / (size_t)ax.m);
    const size_t room = kSmemBudget > line ? kSmemBudget - line : 0;
    const int tile = (int)std::max<size_t>(1, std::min<size_t>(want, room / (2 * line)));
    const size_t smem = line * (2 * (size_t)tile + 1);
    if (smem > 227 * 1024)
        return fail(err, FH_ERR_PFFT, "pFFT convolution: axis length " + std::to_string(ax.m) +
                                          " does not fit the transform kernel's shared memory");
    const int64_t tiles = inner == 1 ? (outer + tile - 1) / tile : outer * ((inner + tile - 1) / tile);
    FHB_CUDA(cudaFuncSetAttribute(fft_lines_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const unsigned gx = (unsigned)std::max<int64_t>(1, std::min<int64_t>(tiles, 148 * 8));
    fft_lines_kernel<<<dim3(gx, (unsigned)batch), kThreads, smem, s>>>(in, out, in_stride, out_stride, outer, inner,
                                                                       n_in, keep, ax, tw, sign, tile, spectrum);
    FHB_CUDA(cudaGetLastError());
    return FH_OK;
}

}  // namespace

fh_status fftconv_run_ports(const FftConvTables &tab, void *work, int grids, cudaStream_t s, fh_error_info *err) {
    const FftConvShape &sh = tab.shape;
    const int64_t n0 = sh.n[0], n1 = sh.n[1], n2 = sh.n[2], m0 = sh.m[0], m1 = sh.m[1], m2 = sh.m[2];
    const int64_t sa = n0 * n1 * n2, sb = n0 * n1 * m2, sc = n0 * m1 * m2;
    // twiddles exp(-2 pi i t / m) of the three axes, computed in FP64
    std::vector<V> h;
    std::vector<int> place;
    Passes ax[3];
    for (int a = 0; a < 3; ++a) {
        const int64_t m = sh.m[a];
        ax[a] = passes_of((int)m);
        for (int64_t t = 0; t < m; ++t) {
            const double ang = -2.0 * 3.14159265358979323846 * (double)t / (double)m;
            h.push_back(make_float2((float)std::cos(ang), (float)std::sin(ang)));
        }
        const std::vector<int> p = fft_places(tab.axis[a]);
        place.insert(place.end(), p.begin(), p.end());
    }
    V *tw = nullptr;
    T *spec = nullptr;
    int *d_place = nullptr;
    struct Release {
        V **tw;
        T **spec;
        int **place;
        cudaStream_t s;
        ~Release() {
            cache_free(*tw, s);
            cache_free(*spec, s);
            cache_free(*place, s);
            cudaStreamSynchronize(s);  // the host tables' copies have run
        }
    } release{&tw, &spec, &d_place, s};
    FHB_CUDA(cache_alloc(reinterpret_cast<void **>(&tw), sizeof(V) * h.size(), s));
    FHB_CUDA(cache_alloc(reinterpret_cast<void **>(&d_place), sizeof(int) * place.size(), s));
    FHB_CUDA(cache_alloc(reinterpret_cast<void **>(&spec), sizeof(T) * (size_t)(m0 * m1 * m2), s));
    FHB_CUDA(cudaMemcpyAsync(tw, h.data(), sizeof(V) * h.size(), cudaMemcpyHostToDevice, s));
    FHB_CUDA(cudaMemcpyAsync(d_place, place.data(), sizeof(int) * place.size(), cudaMemcpyHostToDevice, s));
    const int64_t P = m0 * m1 * m2;
    spectrum_natural_kernel<<<(unsigned)std::min<int64_t>((P + 255) / 256, 148 * 16), 256, 0, s>>>(
        static_cast<const T *>(tab.spectrum), spec, m0, m1, m2, d_place);
    FHB_CUDA(cudaGetLastError());
    const V *tw0 = tw, *tw1 = tw + m0, *tw2 = tw + m0 + m1;
    V *A = static_cast<V *>(work);
    V *B = A + sa * grids;
    V *C = B + sb * grids;
    fh_status e = axis_step(A, B, sa, sb, n0 * n1, 1, (int)n2, (int)m2, ax[2], tw2, -1, nullptr, grids, s, err);
    if (!e) e = axis_step(B, C, sb, sc, n0, m2, (int)n1, (int)m1, ax[1], tw1, -1, nullptr, grids, s, err);
    if (!e) e = axis_step(C, C, sc, sc, 1, m1 * m2, (int)n0, (int)n0, ax[0], tw0, -1, spec, grids, s, err);
    if (!e) e = axis_step(C, B, sc, sb, n0, m2, (int)m1, (int)n1, ax[1], tw1, +1, nullptr, grids, s, err);
    if (!e) e = axis_step(B, A, sb, sa, n0 * n1, 1, (int)m2, (int)n2, ax[2], tw2, +1, nullptr, grids, s, err);
    return e;
}

}  // namespace fhb

// The pFFT convolution K (*) q on the device, without a library FFT: pruned
// mixed-radix transforms, in FP32 or FP64 (pfft/fft.rs:155-320 of the
// reference, re-designed for the GPU).
//
// The sources q live on the n0 x n1 x n2 grid; the aperiodic convolution
// needs transforms of length m_a >= 2 n_a - 1 per axis (a torus of 2^a 3^b
// 5^c points).  Only n0 n1 lines carry data along axis 2, only n0 planes
// along axis 1, and only n0 planes of the result are read back, so the
// transform is pruned axis by axis (the reference prunes the same way):
//
//   1. axis 2 forward  A[n0][n1][n2]  -> B[n0][n1][m2]   (n0 n1 lines)
//   2. axis 1 forward  B[n0][n1][m2]  -> C[n0][m1][m2]   (n0 m2 lines)
//   3. axis 0 forward, times the kernel's real spectrum, axis 0 inverse, in
//      place in C (m1 m2 lines of n0 points in, n0 points out)
//   4. axis 1 inverse  C[n0][m1][m2]  -> B[n0][n1][m2]
//   5. axis 2 inverse  B[n0][n1][m2]  -> A[n0][n1][n2]   (the potentials)
//
// A thin grid (4 to 16 points along axis 2: a planar layout's thickness) is
// not transformed along axis 2 at all.  With d the distance along it, the
// kernel's two-axis spectrum K_d is real and the rest is y_i = sum_j K_|i-j|
// x_j over n2 points, n2 products per point against two transforms of twice
// the length:
//
//   1. axis 1 forward  A[n0][n1][n2]  -> C[n0][m1][n2]   (n0 n2 lines)
//   2. axis 0 forward, the product along axis 2, axis 0 inverse, in place in C
//      (m1 n2 lines): a tile is the n2 lines of one k1
//   3. axis 1 inverse  C[n0][m1][n2]  -> A[n0][n1][n2]
//
// which transforms n2 lines where the five steps transform m2 >= 2 n2 - 1.
// Above 16 points the tile outgrows a shared buffer of two CTAs per SM; up to
// 3 the lines of a tile are shorter than a 32-byte sector.
//
// Each step is one launch.  What bounds a step is the shared-memory traffic
// and the latency of its butterflies, not the device memory, so:
//   * a length is cut into as few stages as possible (radices up to 16 in
//     FP32, 12 in FP64, held in registers: 1200 = 8 x 10 x 15 instead of the
//     five passes of a radix-4/2/3/5 chain);
//   * the forward transform is decimated in frequency and the inverse in
//     time, so every stage reads and writes the same places: one buffer of
//     `lines` lines (a second one would halve the lines in flight), one
//     barrier per stage, and the transformed axes stay in the stages' own
//     order, which nothing but the spectrum's layout has to know;
//   * strided steps take their first stage from device memory into registers
//     and their last one back, so a line of k stages crosses shared memory
//     k - 1 times, and zero padding is never loaded or stored;
//   * in step 3 the last forward stage, the spectrum and the first inverse
//     stage stay in registers.
// Measured on 1200 x 1200 x 15 torus points (590 x 589 x 8 sources, two
// grids), in us for the steps 1 to 5, against the radix-2/3/4/5 Stockham chain
// with two buffers that came before:
//   FP32   45 + 115 + 309 + 104 + 58 =  631   (104 + 284 + 1008 + 290 + 101)
//   FP64  110 + 182 + 511 + 178 + 129 = 1110
// and the thin form's three steps on the same grid:
//   FP32   47 + 185 + 54 = 287      FP64   89 + 356 + 97 = 542
// (300 x 300 x 16 sources, 600 x 600 x 32: 163 and 321).
// FP32 issues instructions in 0.6 of the cycles (packed FP32 arithmetic, see
// cadd; twiddles in rows of 16-byte loads) at 32 warps per SM; 256 and 384
// threads per CTA measured within 5 %.
//
// The inverse runs on swapped real and imaginary parts: with s(z) the swap,
// IDFT(z) = s(DFT(s(z))) and s(conj(w) z) = w s(z), so both directions share
// one set of butterflies and twiddles.  Two real source fields travel in one
// complex grid (real and imaginary parts), as in the reference's convolver.
// The kernel's spectrum is computed at set-up by the same kernels (unpruned,
// FP64) from the wrapped kernel grid; it is real because the wrapped kernel
// is even.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <type_traits>
#include <vector>

#include "fh_device.cuh"
#include "fh_fftconv.h"

namespace fhb {
namespace {

// Threads per CTA, two CTAs per SM.
template <class T>
constexpr int fft_threads() {
    return sizeof(T) == 4 ? 512 : 256;
}
constexpr size_t kFftSmemBudget = 110 * 1024;  // two CTAs per SM
constexpr size_t kFftSmemMost = 227 * 1024;
constexpr int kFftTilePoints = 8192;
constexpr double kPi = 3.14159265358979323846;

template <class T>
struct Cplx;
template <>
struct Cplx<float> {
    using type = float2;
    using real = float;
};
template <>
struct Cplx<double> {
    using type = double2;
    using real = double;
};
__device__ __forceinline__ float2 cmake(float x, float y) { return make_float2(x, y); }
__device__ __forceinline__ double2 cmake(double x, double y) { return make_double2(x, y); }

// a + b, a - b and a + s t of complex numbers.  FP32: the packed two-element
// instructions, one issue slot instead of two (these kernels are bound by
// issue: 0.63 instructions per scheduler and cycle without them).
__device__ __forceinline__ unsigned long long pack2(float2 a) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(a)), "l"(pack2(b)));
    return unpack2(r);
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(a)), "l"(pack2(b)));
    return unpack2(r);
}
__device__ __forceinline__ float2 caxpy(float s, float2 t, float2 a) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pack2(make_float2(s, s))), "l"(pack2(t)), "l"(pack2(a)));
    return unpack2(r);
}
__device__ __forceinline__ float2 cscale(float s, float2 t) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(make_float2(s, s))), "l"(pack2(t)));
    return unpack2(r);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 caxpy(double s, double2 t, double2 a) {
    return make_double2(a.x + s * t.x, a.y + s * t.y);
}
__device__ __forceinline__ double2 cscale(double s, double2 t) { return make_double2(s * t.x, s * t.y); }
template <class V>
__device__ __forceinline__ V cmul(V a, V b) {
    return cmake(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <class V>
__device__ __forceinline__ V cswap(V a) {
    return cmake(a.y, a.x);
}

// ---------------------------------------------------------------------------
// Register transforms: v <- DFT_R v, W = exp(-2 pi i / R), natural order in
// and out.  2, 3, 4 and 5 directly; a product of coprime factors by the prime
// factor map (no twiddles), 8, 9 and 16 by their two equal-base factors.
// ---------------------------------------------------------------------------
template <class V>
__device__ __forceinline__ void dft2(V &a, V &b) {
    const V t = csub(a, b);
    a = cadd(a, b);
    b = t;
}
template <class V>
__device__ __forceinline__ void dft3(V &a, V &b, V &c) {
    using T = decltype(a.x);
    const V t = cadd(b, c), d = csub(b, c);
    const T s = (T)0.86602540378443864676;
    const V m = caxpy((T)-0.5, t, a);
    a = cadd(a, t);
    b = cmake(m.x + s * d.y, m.y - s * d.x);
    c = cmake(m.x - s * d.y, m.y + s * d.x);
}
template <class V>
__device__ __forceinline__ void dft4(V &a, V &b, V &c, V &d) {
    const V s0 = cadd(a, c), d0 = csub(a, c), s1 = cadd(b, d), d1 = csub(b, d);
    a = cadd(s0, s1);
    c = csub(s0, s1);
    b = cmake(d0.x + d1.y, d0.y - d1.x);
    d = cmake(d0.x - d1.y, d0.y + d1.x);
}
template <class V>
__device__ __forceinline__ void dft5(V &a, V &b, V &c, V &d, V &e) {
    using T = decltype(a.x);
    const T c1 = (T)0.30901699437494742410, c2 = (T)-0.80901699437494742410;
    const T s1 = (T)0.95105651629515357212, s2 = (T)0.58778525229247312917;
    const V t1 = cadd(b, e), t2 = cadd(c, d), t3 = csub(b, e), t4 = csub(c, d);
    const V m1 = caxpy(c2, t2, caxpy(c1, t1, a)), m2 = caxpy(c1, t2, caxpy(c2, t1, a));
    const V n1 = caxpy(s2, t4, cscale(s1, t3)), n2 = caxpy(-s1, t4, cscale(s2, t3));
    a = cadd(a, cadd(t1, t2));
    b = cmake(m1.x + n1.y, m1.y - n1.x);
    e = cmake(m1.x - n1.y, m1.y + n1.x);
    c = cmake(m2.x + n2.y, m2.y - n2.x);
    d = cmake(m2.x - n2.y, m2.y + n2.x);
}

template <int R, class V>
__device__ __forceinline__ void dft(V (&v)[R]);

// N = A B coprime: input (B i + A j) mod N, output (B B' k + A A' l) mod N
// with B B' = 1 mod A and A A' = 1 mod B.
constexpr int inverse_mod(int a, int n) {
    for (int k = 1; k < n; ++k)
        if (a * k % n == 1) return k;
    return 1;
}
template <int A, int B, class V>
__device__ __forceinline__ void dft_coprime(V (&v)[A * B]) {
    constexpr int N = A * B, bi = B * inverse_mod(B % A, A), ai = A * inverse_mod(A % B, B);
    V t[B][A];
#pragma unroll
    for (int j = 0; j < B; ++j) {
#pragma unroll
        for (int i = 0; i < A; ++i) t[j][i] = v[(B * i + A * j) % N];
        dft<A>(t[j]);
    }
#pragma unroll
    for (int k = 0; k < A; ++k) {
        V u[B];
#pragma unroll
        for (int j = 0; j < B; ++j) u[j] = t[j][k];
        dft<B>(u);
#pragma unroll
        for (int l = 0; l < B; ++l) v[(bi * k + ai * l) % N] = u[l];
    }
}

// cos and sin of 2 pi k / N for the equal-base products (N = 8, 9, 16).
template <int N>
__device__ constexpr double root_cos(int k) {
    constexpr double c8[4] = {1.0, 0.70710678118654752440, 0.0, -0.70710678118654752440};
    constexpr double c9[5] = {1.0, 0.76604444311897803520, 0.17364817766693034885, -0.5, -0.93969262078590838405};
    constexpr double c16[10] = {1.0, 0.92387953251128675613, 0.70710678118654752440, 0.38268343236508977173, 0.0,
                                -0.38268343236508977173, -0.70710678118654752440, -0.92387953251128675613, -1.0,
                                -0.92387953251128675613};
    return N == 8 ? c8[k & 3] : N == 9 ? c9[k % 5] : c16[k % 10];
}
template <int N>
__device__ constexpr double root_sin(int k) {
    constexpr double s8[4] = {0.0, 0.70710678118654752440, 1.0, 0.70710678118654752440};
    constexpr double s9[5] = {0.0, 0.64278760968653932632, 0.98480775301220805937, 0.86602540378443864676,
                              0.34202014332566873304};
    constexpr double s16[10] = {0.0, 0.38268343236508977173, 0.70710678118654752440, 0.92387953251128675613, 1.0,
                                0.92387953251128675613, 0.70710678118654752440, 0.38268343236508977173, 0.0,
                                -0.38268343236508977173};
    return N == 8 ? s8[k & 3] : N == 9 ? s9[k % 5] : s16[k % 10];
}
// N = A B: input i B + j, output k + A l.
template <int A, int B, class V>
__device__ __forceinline__ void dft_product(V (&v)[A * B]) {
    using T = decltype(v[0].x);
    V t[B][A];
#pragma unroll
    for (int j = 0; j < B; ++j) {
#pragma unroll
        for (int i = 0; i < A; ++i) t[j][i] = v[i * B + j];
        dft<A>(t[j]);
    }
#pragma unroll
    for (int k = 0; k < A; ++k) {
        V u[B];
#pragma unroll
        for (int j = 0; j < B; ++j) {
            if (j * k == 0)
                u[j] = t[j][k];
            else if (4 * j * k == A * B)  // -i
                u[j] = cmake(t[j][k].y, -t[j][k].x);
            else
                u[j] = cmul(t[j][k], cmake((T)root_cos<A * B>(j * k), (T)-root_sin<A * B>(j * k)));
        }
        dft<B>(u);
#pragma unroll
        for (int l = 0; l < B; ++l) v[k + A * l] = u[l];
    }
}
template <int R, class V>
__device__ __forceinline__ void dft(V (&v)[R]) {
    if constexpr (R == 2) dft2(v[0], v[1]);
    else if constexpr (R == 3) dft3(v[0], v[1], v[2]);
    else if constexpr (R == 4) dft4(v[0], v[1], v[2], v[3]);
    else if constexpr (R == 5) dft5(v[0], v[1], v[2], v[3], v[4]);
    else if constexpr (R == 6) dft_coprime<2, 3>(v);
    else if constexpr (R == 8) dft_product<4, 2>(v);
    else if constexpr (R == 9) dft_product<3, 3>(v);
    else if constexpr (R == 10) dft_coprime<2, 5>(v);
    else if constexpr (R == 12) dft_coprime<4, 3>(v);
    else if constexpr (R == 15) dft_coprime<3, 5>(v);
    else if constexpr (R == 16) dft_product<4, 4>(v);
}

// ---------------------------------------------------------------------------
// Stages.
// ---------------------------------------------------------------------------
// x / d for x < 2^16, d < 2^16, magic = ceil(2^32 / d) (d > 1): the error
// x (magic d - 2^32) / d stays below 2^32 / d.
__device__ __forceinline__ int fast_div(int x, unsigned magic) {
    return magic ? (int)__umulhi((unsigned)x, magic) : x;
}

// v_r <- v_r w^r from a row of the stage's table (r = 0 included, padded to an
// even length: 16-byte loads at constant offsets).
__host__ __device__ constexpr int twiddle_row(int R) { return (R + 1) & ~1; }
template <int R>
__device__ __forceinline__ void twiddle(float2 (&v)[R], const float2 *__restrict__ row) {
    const float4 *__restrict__ q = reinterpret_cast<const float4 *>(row);
#pragma unroll
    for (int h = 0; h < twiddle_row(R) / 2; ++h) {
        const float4 w = __ldg(q + h);
        if (h > 0) v[2 * h] = cmul(v[2 * h], make_float2(w.x, w.y));
        if (2 * h + 1 < R) v[2 * h + 1] = cmul(v[2 * h + 1], make_float2(w.z, w.w));
    }
}
template <int R>
__device__ __forceinline__ void twiddle(double2 (&v)[R], const double2 *__restrict__ row) {
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = cmul(v[r], __ldg(row + r));
}

// Where a tile's element (point t, line l) lies in the shared buffer, and which
// runs fastest over the threads.
enum Layout {
    kStrided,  // t 2^lg + l, lines first
    kWide,     // the same; places in device memory beyond 32-bit indices
    kContig,   // l pitch + t, points first
    kThin      // l pitch + t, lines first (any number of lines)
};

// Where a tile's lines lie in device memory.
template <class V>
struct Lines {
    const V *src;   // point 0 of line 0 (input), `inner` between points, 1 between lines
    V *dst;
    int inner;
    int count;      // lines of this tile
    int n_in, keep; // points read, points written; the rest is zero
    unsigned magic; // of count (kThin)
};

// One stage of radix R = ax.R[st] over the tile's lines: point b R S + k + r S
// of every block b, offset k, by one thread.
//   DIT = false: DFT then twiddle (forward); true: twiddle then DFT (inverse).
//   GIN / GOUT: from / to device memory instead of the buffer.
//   MID: the forward's last stage, the spectrum and the inverse's first.
template <int R, class T, int LAYOUT, bool DIT, bool GIN, bool GOUT, bool MID>
__device__ __forceinline__ void fft_stage(typename Cplx<T>::type *buf, const FftAxis &ax, int st, int lg, int pitch,
                                          const typename Cplx<T>::type *__restrict__ tw_all,
                                          const Lines<typename Cplx<T>::type> &g, const T *__restrict__ spectrum) {
    using V = typename Cplx<T>::type;
    const int S = ax.S[st], nb = ax.m / R;
    const V *__restrict__ tw = tw_all + ax.tw[st];
    const int total = LAYOUT == kThin ? nb * g.count : nb << lg;
    constexpr bool kLines = LAYOUT == kStrided || LAYOUT == kWide;
    auto at = [&](int t, int l) { return kLines ? (t << lg) + l : l * pitch + t; };
    auto place = [&](int t, int l) -> std::conditional_t<LAYOUT == kWide, int64_t, int> {
        if constexpr (LAYOUT == kWide) return (int64_t)t * g.inner + l;
        else return t * g.inner + l;
    };
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        int l, j;
        if (LAYOUT == kContig) {
            l = fast_div(idx, ax.magic_nb[st]);
            j = idx - l * nb;
        } else if (LAYOUT == kThin) {
            j = fast_div(idx, g.magic);
            l = idx - j * g.count;
        } else {
            l = idx & ((1 << lg) - 1);
            j = idx >> lg;
        }
        const int b = fast_div(j, ax.magic_S[st]);
        const int k = j - b * S;
        const int t0 = b * R * S + k;
        V v[R];
        const bool live = !kLines || l < g.count;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int t = t0 + r * S;
            if (GIN) {
                v[r] = cmake((T)0, (T)0);
                if (live && t < g.n_in) v[r] = g.src[place(t, l)];
                if (DIT) v[r] = cswap(v[r]);
            } else {
                v[r] = buf[at(t, l)];
            }
        }
        if (DIT && S > 1) twiddle<R>(v, tw + k * twiddle_row(R));
        dft<R>(v);
        if (MID) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const T s = live ? spectrum[place(t0 + r * S, l)] : (T)0;
                v[r] = cmake(s * v[r].y, s * v[r].x);  // swapped: the inverse begins
            }
            dft<R>(v);
        }
        if (!DIT && !MID && S > 1) twiddle<R>(v, tw + k * twiddle_row(R));
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int t = t0 + r * S;
            if (GOUT) {
                if (live && t < g.keep) g.dst[place(t, l)] = DIT || MID ? cswap(v[r]) : v[r];
            } else {
                buf[at(t, l)] = v[r];
            }
        }
    }
}

template <class T, int LAYOUT, bool DIT, bool GIN, bool GOUT, bool MID>
__device__ __forceinline__ void fft_stage_any(typename Cplx<T>::type *buf, const FftAxis &ax, int st, int lg,
                                              int pitch, const typename Cplx<T>::type *__restrict__ tw,
                                              const Lines<typename Cplx<T>::type> &g,
                                              const T *__restrict__ spectrum) {
    switch (ax.R[st]) {
#define FHB_FFT_RADIX(r)                                                                             \
    case r:                                                                                          \
        fft_stage<r, T, LAYOUT, DIT, GIN, GOUT, MID>(buf, ax, st, lg, pitch, tw, g, spectrum);       \
        break;
        FHB_FFT_RADIX(1)
        FHB_FFT_RADIX(2)
        FHB_FFT_RADIX(3)
        FHB_FFT_RADIX(4)
        FHB_FFT_RADIX(5)
        FHB_FFT_RADIX(6)
        FHB_FFT_RADIX(8)
        FHB_FFT_RADIX(9)
        FHB_FFT_RADIX(10)
        FHB_FFT_RADIX(12)
        default:
            if constexpr (sizeof(T) == 4) {
                if (ax.R[st] == 15)
                    fft_stage<15, T, LAYOUT, DIT, GIN, GOUT, MID>(buf, ax, st, lg, pitch, tw, g, spectrum);
                else
                    fft_stage<16, T, LAYOUT, DIT, GIN, GOUT, MID>(buf, ax, st, lg, pitch, tw, g, spectrum);
            }
#undef FHB_FFT_RADIX
    }
}

enum FftKind { kForward, kInverse, kFused };

// Axis 2 of at least kThinLeast and at most kThinMost points: the thin form.
constexpr int kThinLeast = 4, kThinMost = 16;

// One pruned axis transform over a batch of arrays.  An array holds
// `outer` x len x `inner` complex elements (len = n_in for the input, keep
// for the output); line (o, c) is elements (o len + t) inner + c.  A tile is
// 2^lg lines of consecutive c (tail tiles: fewer).  kFused: forward, times
// spectrum[t inner + c] (real), and back; in and out may be the same array,
// since a CTA reads its whole tile before it writes and tiles are disjoint.
// LAYOUT kWide: len x inner may pass 2^31 (axis 0 of the largest tori), for a
// sixth more time on the fused step.
template <class T, int KIND, int LAYOUT>
__global__ void __launch_bounds__(fft_threads<T>(), 2)
    fft_strided_kernel(const typename Cplx<T>::type *in, typename Cplx<T>::type *out, int64_t in_stride,
                       int64_t out_stride, int64_t outer, int inner, int n_in, int keep, FftAxis ax, int lg,
                       const typename Cplx<T>::type *__restrict__ tw, const T *__restrict__ spectrum) {
    using V = typename Cplx<T>::type;
    extern __shared__ __align__(16) unsigned char fft_smem[];
    V *buf = reinterpret_cast<V *>(fft_smem);
    const int per = (inner + (1 << lg) - 1) >> lg;
    const int64_t tiles = outer * per;
    const int last = ax.nst - 1;
    for (int64_t tt = blockIdx.x; tt < tiles; tt += gridDim.x) {
        const int64_t o = tt / per;
        const int c0 = (int)(tt - o * per) << lg;
        Lines<V> g;
        g.inner = inner;
        g.count = min(1 << lg, inner - c0);
        g.n_in = n_in;
        g.keep = keep;
        g.src = in + (int64_t)blockIdx.y * in_stride + o * n_in * inner + c0;
        g.dst = out + (int64_t)blockIdx.y * out_stride + o * keep * inner + c0;
        const T *spec = KIND == kFused ? spectrum + c0 : nullptr;
        if (last == 0) {
            fft_stage_any<T, LAYOUT, KIND == kInverse, true, true, KIND == kFused>(buf, ax, 0, lg, 0, tw, g, spec);
            continue;
        }
        if (KIND != kInverse) {
            fft_stage_any<T, LAYOUT, false, true, false, false>(buf, ax, 0, lg, 0, tw, g, spec);
            for (int st = 1; st < last; ++st) {
                __syncthreads();
                fft_stage_any<T, LAYOUT, false, false, false, false>(buf, ax, st, lg, 0, tw, g, spec);
            }
            __syncthreads();
            fft_stage_any<T, LAYOUT, false, false, KIND == kForward, KIND == kFused>(buf, ax, last, lg, 0, tw, g, spec);
        }
        if (KIND != kForward) {
            if (KIND == kInverse) fft_stage_any<T, LAYOUT, true, true, false, false>(buf, ax, last, lg, 0, tw, g, spec);
            for (int st = last - 1; st > 0; --st) {
                __syncthreads();
                fft_stage_any<T, LAYOUT, true, false, false, false>(buf, ax, st, lg, 0, tw, g, spec);
            }
            __syncthreads();
            fft_stage_any<T, LAYOUT, true, false, true, false>(buf, ax, 0, lg, 0, tw, g, spec);
        }
        __syncthreads();  // the next tile's first stage writes the buffer
    }
}

// The same for contiguous lines (inner = 1, axis 2): a tile of `lines` whole
// lines is one run of device memory, copied in and out of the buffer in order
// and transformed there.
template <class T, int KIND>
__global__ void __launch_bounds__(fft_threads<T>(), 2)
    fft_contiguous_kernel(const typename Cplx<T>::type *in, typename Cplx<T>::type *out, int64_t in_stride,
                          int64_t out_stride, int64_t outer, int n_in, int keep, FftAxis ax, int lg,
                          unsigned magic_in, unsigned magic_keep, const typename Cplx<T>::type *__restrict__ tw) {
    using V = typename Cplx<T>::type;
    extern __shared__ __align__(16) unsigned char fft_smem[];
    V *buf = reinterpret_cast<V *>(fft_smem);
    const int lines = 1 << lg, pitch = ax.m | 1;
    const int64_t tiles = (outer + lines - 1) >> lg;
    const Lines<V> none = {};
    for (int64_t tt = blockIdx.x; tt < tiles; tt += gridDim.x) {
        const int64_t o0 = tt << lg;
        const int count = (int)min((int64_t)lines, outer - o0);
        const V *src = in + (int64_t)blockIdx.y * in_stride + o0 * n_in;
        V *dst = out + (int64_t)blockIdx.y * out_stride + o0 * keep;
        const int pad = ax.m - n_in;
        for (int idx = threadIdx.x; idx < count * n_in; idx += blockDim.x) {
            const int l = fast_div(idx, magic_in);
            const V v = src[idx];
            buf[l * pitch + idx - l * n_in] = KIND == kInverse ? cswap(v) : v;
        }
        for (int idx = threadIdx.x; idx < (pad << lg); idx += blockDim.x)
            buf[(idx & (lines - 1)) * pitch + n_in + (idx >> lg)] = cmake((T)0, (T)0);
        if (count < lines)  // a tail tile: the missing lines are transformed too
            for (int idx = threadIdx.x; idx < (lines - count) * pitch; idx += blockDim.x)
                buf[count * pitch + idx] = cmake((T)0, (T)0);
        for (int k = 0; k < ax.nst; ++k) {
            __syncthreads();
            fft_stage_any<T, kContig, KIND == kInverse, false, false, false>(
                buf, ax, KIND == kInverse ? ax.nst - 1 - k : k, lg, pitch, tw, none, nullptr);
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < count * keep; idx += blockDim.x) {
            const int l = fast_div(idx, magic_keep);
            const V v = buf[l * pitch + idx - l * keep];
            dst[idx] = KIND == kInverse ? cswap(v) : v;
        }
        __syncthreads();  // the next tile's loads write the buffer
    }
}

// y_i = sum_j K_|i-j| x_j along axis 2 at every point of a tile of n2 <= N
// lines, in place, swapped (the inverse begins).  K: [d][m].
template <int N, class T>
__device__ __forceinline__ void thin_product(typename Cplx<T>::type *buf, int pitch, int n2, int m,
                                             const T *__restrict__ K) {
    using V = typename Cplx<T>::type;
    for (int t = threadIdx.x; t < m; t += blockDim.x) {
        V x[N];
        T k[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            x[i] = i < n2 ? buf[i * pitch + t] : cmake((T)0, (T)0);
            k[i] = i < n2 ? __ldg(K + i * m + t) : (T)0;
        }
#pragma unroll
        for (int i = 0; i < N; ++i) {
            V y = cscale(k[i], x[0]);
#pragma unroll
            for (int j = 1; j < N; ++j) y = caxpy(k[i > j ? i - j : j - i], x[j], y);
            if (i < n2) buf[i * pitch + t] = cswap(y);
        }
    }
}

// The strided steps of a thin grid: a tile is the n2 lines of one (i, j), whole
// in the buffer.  kFused: forward along axis 0, the product along axis 2 with
// K[k1][d][k0], and back.
template <class T, int KIND>
__global__ void __launch_bounds__(2 * fft_threads<T>(), 1)
    fft_thin_kernel(const typename Cplx<T>::type *in, typename Cplx<T>::type *out, int64_t in_stride,
                    int64_t out_stride, int64_t tiles, int64_t in_tile, int64_t out_tile, int inner, int n2,
                    unsigned magic_n2, int n_in, int keep, FftAxis ax, int pitch,
                    const typename Cplx<T>::type *__restrict__ tw, const T *__restrict__ K) {
    using V = typename Cplx<T>::type;
    extern __shared__ __align__(16) unsigned char fft_smem[];
    V *buf = reinterpret_cast<V *>(fft_smem);
    const int last = ax.nst - 1;
    for (int64_t tt = blockIdx.x; tt < tiles; tt += gridDim.x) {
        Lines<V> g;
        g.inner = inner;
        g.count = n2;
        g.magic = magic_n2;
        g.n_in = n_in;
        g.keep = keep;
        g.src = in + (int64_t)blockIdx.y * in_stride + tt * in_tile;
        g.dst = out + (int64_t)blockIdx.y * out_stride + tt * out_tile;
        if (KIND != kFused && last == 0) {
            fft_stage_any<T, kThin, KIND == kInverse, true, true, false>(buf, ax, 0, 0, pitch, tw, g, nullptr);
            continue;
        }
        if (KIND != kInverse) {
            fft_stage_any<T, kThin, false, true, false, false>(buf, ax, 0, 0, pitch, tw, g, nullptr);
            for (int st = 1; st < (KIND == kFused ? last + 1 : last); ++st) {
                __syncthreads();
                fft_stage_any<T, kThin, false, false, false, false>(buf, ax, st, 0, pitch, tw, g, nullptr);
            }
            __syncthreads();
            if (KIND == kForward)
                fft_stage_any<T, kThin, false, false, true, false>(buf, ax, last, 0, pitch, tw, g, nullptr);
        }
        if (KIND == kFused) {
            const T *k = K + tt * n2 * ax.m;
            if (n2 <= 8) thin_product<8>(buf, pitch, n2, ax.m, k);
            else thin_product<kThinMost>(buf, pitch, n2, ax.m, k);
            __syncthreads();
        }
        if (KIND != kForward) {
            if (KIND == kInverse)
                fft_stage_any<T, kThin, true, true, false, false>(buf, ax, last, 0, pitch, tw, g, nullptr);
            for (int st = KIND == kFused ? last : last - 1; st > 0; --st) {
                if (KIND == kInverse || st < last) __syncthreads();
                fft_stage_any<T, kThin, true, false, false, false>(buf, ax, st, 0, pitch, tw, g, nullptr);
            }
            if (last > 0) __syncthreads();
            fft_stage_any<T, kThin, true, false, true, false>(buf, ax, 0, 0, pitch, tw, g, nullptr);
        }
        __syncthreads();  // the next tile's first stage writes the buffer
    }
}

// The wrapped kernel 1 / (h |d|) on the padded grid (zero at the origin and
// beyond the unpadded extent), FP64 complex.
__global__ void wrapped_kernel_kernel(double2 *__restrict__ out, int64_t n0, int64_t n1, int64_t n2, int64_t m0,
                                      int64_t m1, int64_t m2, double spacing) {
    const int64_t total = m0 * m1 * m2;
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < total; p += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = p % m2, rest = p / m2, j = rest % m1, i = rest / m1;
        auto wrap = [](int64_t t, int64_t n, int64_t m, int64_t &d) {
            if (t < n) {
                d = t;
                return true;
            }
            if (t + n > m) {
                d = t - m;
                return true;
            }
            return false;
        };
        int64_t di, dj, dk;
        double v = 0.0;
        if (wrap(i, n0, m0, di) && wrap(j, n1, m1, dj) && wrap(k, n2, m2, dk)) {
            const double r2 = (double)(di * di + dj * dj + dk * dk);
            v = r2 == 0.0 ? 0.0 : 1.0 / (spacing * sqrt(r2));
        }
        out[p] = make_double2(v, 0.0);
    }
}

// The spectrum, scaled by 1 / P, from the FP64 transform's order to the
// convolution's: map[a] gives for each place of axis a the place of the same
// frequency in the FP64 transform.
template <class T>
__global__ void spectrum_store_kernel(const double2 *__restrict__ in, T *__restrict__ out, int64_t m0, int64_t m1,
                                      int64_t m2, const int *__restrict__ map) {
    const int64_t total = m0 * m1 * m2;
    const double scale = 1.0 / (double)total;
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < total; p += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = p % m2, rest = p / m2, j = rest % m1, i = rest / m1;
        out[p] = (T)(in[((int64_t)map[i] * m1 + map[m0 + j]) * m2 + map[m0 + m1 + k]].x * scale);
    }
}

// The spectrum of a thin grid, [k1][d][k0]: the kernel's distances d along
// axis 2 as they are, in the convolution's order along axes 0 and 1.
template <class T>
__global__ void thin_store_kernel(const double2 *__restrict__ in, T *__restrict__ out, int64_t m0, int64_t m1,
                                  int64_t n2, const int *__restrict__ map) {
    const int64_t total = m0 * m1 * n2;
    const double scale = 1.0 / (double)(m0 * m1);
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < total; p += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = p % m0, rest = p / m0, d = rest % n2, j = rest / n2;
        out[p] = (T)(in[((int64_t)map[i] * m1 + map[m0 + j]) * n2 + d].x * scale);
    }
}

unsigned blocks_of(int64_t work, int threads, int64_t cap = 148 * 16) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((work + threads - 1) / threads, cap));
}

unsigned magic_of(int d) { return d > 1 ? (unsigned)(((uint64_t(1) << 32) + (uint64_t)d - 1) / (uint64_t)d) : 0u; }

// log2 of the lines per tile: lines of 64 bytes or more per point (8 FP32, 4
// FP64) where two CTAs of them fit an SM, else fewer; short lines come up to
// kFftTilePoints points to a tile.
template <class T>
int tile_lg(int m, int64_t inner) {
    const size_t elem = sizeof(typename Cplx<T>::type);
    int lg = 0;
    while (lg < 9) {
        const size_t next = (size_t)2 << lg;
        if (next * (size_t)(m | 1) * elem > kFftSmemBudget) break;
        if (next * elem > 64 && next * (size_t)m > (size_t)kFftTilePoints) break;
        if (inner > 1 && (int64_t)1 << lg >= inner) break;
        ++lg;
    }
    return lg;
}

// One axis step: outer x n_in x inner -> outer x keep x inner, `batch` arrays.
template <class T, int KIND>
fh_status axis_step(const void *in, void *out, int64_t in_stride, int64_t out_stride, int64_t outer, int64_t inner,
                    int n_in, int keep, const FftAxis &ax, const void *tw, const T *spectrum, int batch,
                    cudaStream_t s, fh_error_info *err) {
    using V = typename Cplx<T>::type;
    const int lg = tile_lg<T>(ax.m, inner);
    const size_t smem = sizeof(V) * ((size_t)(ax.m | 1) << lg);
    if (smem > kFftSmemMost)
        return fail(err, FH_ERR_PFFT, "pFFT convolution: axis length " + std::to_string(ax.m) +
                                          " does not fit the transform kernel's shared memory");
    const int64_t tiles = inner == 1 && KIND != kFused ? (outer + (1 << lg) - 1) >> lg
                                                       : outer * ((inner + (1 << lg) - 1) >> lg);
    const unsigned gx = (unsigned)std::max<int64_t>(1, std::min<int64_t>(tiles, 148 * 8));
    const dim3 grid(gx, (unsigned)batch);
    // the contiguous form exists for plain transforms; a fused step of a
    // single line (m1 = m2 = 1) is a strided one with one line per tile
    if (inner == 1 && KIND != kFused) {
        constexpr int K = KIND == kFused ? kForward : KIND;
        FHB_CUDA(cudaFuncSetAttribute(fft_contiguous_kernel<T, K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
        fft_contiguous_kernel<T, K><<<grid, fft_threads<T>(), smem, s>>>(
            static_cast<const V *>(in), static_cast<V *>(out), in_stride, out_stride, outer, n_in, keep, ax, lg,
            magic_of(n_in), magic_of(keep), static_cast<const V *>(tw));
    } else {
        auto kernel = fft_strided_kernel<T, KIND, kStrided>;
        // axis 0 of more than 2^31 points; along axis 1 (inner = m2) there are
        // never as many
        if constexpr (KIND == kFused || (KIND == kForward && sizeof(T) == 8))
            if ((int64_t)ax.m * inner > INT32_MAX) kernel = fft_strided_kernel<T, KIND, kWide>;
        FHB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kernel<<<grid, fft_threads<T>(), smem, s>>>(static_cast<const V *>(in), static_cast<V *>(out), in_stride,
                                                    out_stride, outer, (int)inner, n_in, keep, ax, lg,
                                                    static_cast<const V *>(tw), spectrum);
    }
    FHB_CUDA(cudaGetLastError());
    return FH_OK;
}

// Points between two lines of a thin tile: 16 lanes (8 in FP64) of a
// shared-memory access are n2 lines times a few consecutive points, which this
// spreads over all banks.
template <class T>
int thin_pitch(int m, int64_t n2) {
    const int lanes = sizeof(T) == 4 ? 16 : 8;
    const int step = (int)std::max<int64_t>(1, (lanes + n2 - 1) / n2);
    return (m + lanes - 1) / lanes * lanes + step;
}
template <class T>
size_t thin_smem(int m, int64_t n2) {
    return sizeof(typename Cplx<T>::type) * (size_t)thin_pitch<T>(m, n2) * (size_t)n2;
}
template <class T>
bool thin_grid(const FftConvShape &sh) {
    return sh.n[2] >= kThinLeast && sh.n[2] <= kThinMost &&
           thin_smem<T>((int)std::max(sh.m[0], sh.m[1]), sh.n[2]) <= kFftSmemMost;
}

template <class T, int KIND>
fh_status thin_step(const void *in, void *out, int64_t in_stride, int64_t out_stride, int64_t tiles, int64_t in_tile,
                    int64_t out_tile, int64_t inner, int64_t n2, int n_in, int keep, const FftAxis &ax,
                    const void *tw, const T *K, int batch, cudaStream_t s, fh_error_info *err) {
    using V = typename Cplx<T>::type;
    const size_t smem = thin_smem<T>(ax.m, n2);
    // two CTAs per SM, or one of twice the threads
    const int threads = fft_threads<T>() * (smem > kFftSmemBudget ? 2 : 1);
    FHB_CUDA(cudaFuncSetAttribute(fft_thin_kernel<T, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    fft_thin_kernel<T, KIND><<<dim3((unsigned)std::min<int64_t>(tiles, 148 * 8), (unsigned)batch), threads, smem, s>>>(
        static_cast<const V *>(in), static_cast<V *>(out), in_stride, out_stride, tiles, in_tile, out_tile, (int)inner,
        (int)n2, magic_of((int)n2), n_in, keep, ax, thin_pitch<T>(ax.m, n2), static_cast<const V *>(tw), K);
    FHB_CUDA(cudaGetLastError());
    return FH_OK;
}

}  // namespace

// The place of every frequency of an axis after the forward stages: stage s
// writes residue r of the frequencies of its block to offset r S.
std::vector<int> fft_places(const FftAxis &ax) {
    std::vector<int> place((size_t)ax.m);
    for (int f = 0; f < ax.m; ++f) {
        int rest = f, at = 0;
        for (int s = 0; s < ax.nst; ++s) {
            at += rest % ax.R[s] * ax.S[s];
            rest /= ax.R[s];
        }
        place[(size_t)f] = at;
    }
    return place;
}

// Radices of a length: the fewest stages, then an odd last one (stage S = 1
// strides the shared buffer by R: an odd R keeps a half-warp's lines off each
// other's banks), then the smallest largest radix (registers).
bool fft_axis_plan(int64_t m, bool fp32, FftAxis &ax) {
    ax = FftAxis();
    if (m < 1 || m > kFftMaxLength) return false;
    static const int all[] = {2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16};
    const int count = fp32 ? 11 : 9;
    int best[kFftMaxStages], trial[kFftMaxStages], best_n = 0, best_cost = 1 << 30;
    struct Search {
        const int *radix;
        int count;
        int *trial, *best, *best_n, *best_cost;
        void go(int64_t rest, int depth, int largest) const {
            if (rest == 1) {
                const int cost = 100 * depth + (depth > 1 && trial[depth - 1] % 2 == 0 ? 20 : 0) + largest;
                if (cost < *best_cost) {
                    *best_cost = cost;
                    *best_n = depth;
                    std::copy(trial, trial + depth, best);
                }
                return;
            }
            if (depth == kFftMaxStages || 100 * (depth + 1) > *best_cost) return;
            for (int i = count - 1; i >= 0; --i)
                if (rest % radix[i] == 0) {
                    trial[depth] = radix[i];
                    go(rest / radix[i], depth + 1, std::max(largest, radix[i]));
                }
        }
    };
    if (m == 1)
        best[best_n++] = 1;  // one stage that changes nothing
    else
        Search{all, count, trial, best, &best_n, &best_cost}.go(m, 0, 0);
    if (best_n == 0) return false;
    ax.m = (int)m;
    ax.nst = best_n;
    int len = ax.m, tw = 0;
    for (int s = 0; s < best_n; ++s) {
        ax.R[s] = best[s];
        len /= best[s];
        ax.S[s] = len;
        ax.magic_S[s] = magic_of(len);
        ax.magic_nb[s] = magic_of(ax.m / best[s]);
        ax.tw[s] = tw;
        tw += twiddle_row(best[s]) * len;
    }
    ax.tw_count = tw;
    return true;
}

size_t fftconv_work_elems(const FftConvShape &sh) {
    const int64_t a = sh.n[0] * sh.n[1] * sh.n[2];
    const int64_t b = sh.n[0] * sh.n[1] * sh.m[2];
    const int64_t c = sh.n[0] * sh.m[1] * sh.m[2];
    return (size_t)(a + b + c);
}

template <class T>
fh_status fftconv_setup(const FftConvShape &sh, double spacing, FftConvTables &tab, cudaStream_t s,
                        fh_error_info *err) {
    using V = typename Cplx<T>::type;
    constexpr bool fp32 = sizeof(T) == 4;
    FftAxis ax64[3];
    for (int a = 0; a < 3; ++a)
        if (!fft_axis_plan(sh.m[a], fp32, tab.axis[a]) || !fft_axis_plan(sh.m[a], false, ax64[a]))
            return fail(err, FH_ERR_PFFT,
                        "pFFT convolution: padded axis length " + std::to_string((long long)sh.m[a]) +
                            " is not a 2^a 3^b 5^c length up to " + std::to_string(kFftMaxLength));
    // Twiddles of every stage, [k][r] = exp(-2 pi i r k / (R S)), computed in
    // FP64 on the host.
    for (int a = 0; a < 3; ++a) {
        auto stage_twiddles = [](const FftAxis &ax) {
            std::vector<double2> h((size_t)std::max(1, ax.tw_count));
            for (int st = 0; st < ax.nst; ++st)
                for (int k = 0; k < ax.S[st]; ++k)
                    for (int r = 0; r < ax.R[st]; ++r) {
                        const double ang = -2.0 * kPi * (double)r * (double)k / ((double)ax.R[st] * ax.S[st]);
                        h[(size_t)(ax.tw[st] + k * twiddle_row(ax.R[st]) + r)] =
                            make_double2(std::cos(ang), std::sin(ang));
                    }
            return h;
        };
        const std::vector<double2> h64 = stage_twiddles(ax64[a]);
        const std::vector<double2> hd = stage_twiddles(tab.axis[a]);
        std::vector<V> h(hd.size());
        for (size_t t = 0; t < hd.size(); ++t) {
            h[t].x = (T)hd[t].x;
            h[t].y = (T)hd[t].y;
        }
        FHB_CUDA(cache_alloc(&tab.tw[a], sizeof(V) * h.size(), s));
        FHB_CUDA(cudaMemcpyAsync(tab.tw[a], h.data(), sizeof(V) * h.size(), cudaMemcpyHostToDevice, s));
        if (fp32) {
            FHB_CUDA(cache_alloc(&tab.tw64[a], sizeof(double2) * h64.size(), s));
            FHB_CUDA(cudaMemcpyAsync(tab.tw64[a], h64.data(), sizeof(double2) * h64.size(), cudaMemcpyHostToDevice,
                                     s));
        } else {
            tab.tw64[a] = tab.tw[a];
        }
        FHB_CUDA(cudaStreamSynchronize(s));
    }
    // places of the FP64 transform's frequencies in the convolution's order
    std::vector<int> map;
    for (int a = 0; a < 3; ++a) {
        const std::vector<int> here = fft_places(tab.axis[a]), wide = fft_places(ax64[a]);
        std::vector<int> part((size_t)sh.m[a], 0);
        for (size_t f = 0; f < here.size(); ++f) part[(size_t)here[f]] = wide[f];
        map.insert(map.end(), part.begin(), part.end());
    }
    // Spectrum: unpruned FP64 forward transform of the wrapped kernel.
    const int64_t P = sh.m[0] * sh.m[1] * sh.m[2];
    double2 *grid = nullptr, *tmp = nullptr;
    FHB_CUDA(cache_alloc(reinterpret_cast<void **>(&grid), sizeof(double2) * (size_t)P, s));
    FHB_CUDA(cache_alloc(reinterpret_cast<void **>(&tmp), sizeof(double2) * (size_t)P, s));
    int *d_map = nullptr;
    FHB_CUDA(cache_alloc(reinterpret_cast<void **>(&d_map), sizeof(int) * map.size(), s));
    struct Release {
        void *a, *b, *c;
        cudaStream_t s;
        ~Release() {
            cache_free(a, s);
            cache_free(b, s);
            cache_free(c, s);
        }
    } release{grid, tmp, d_map, s};
    FHB_CUDA(cudaMemcpyAsync(d_map, map.data(), sizeof(int) * map.size(), cudaMemcpyHostToDevice, s));
    const int64_t m0 = sh.m[0], m1 = sh.m[1], m2 = sh.m[2], n2 = sh.n[2];
    tab.shape = sh;
    tab.fp32 = fp32;
    if (thin_grid<T>(sh)) {
        wrapped_kernel_kernel<<<blocks_of(m0 * m1 * n2, 256), 256, 0, s>>>(grid, sh.n[0], sh.n[1], n2, m0, m1, n2,
                                                                          spacing);
        FHB_CUDA(cudaGetLastError());
        fh_status e = axis_step<double, kForward>(grid, tmp, 0, 0, m0, n2, (int)m1, (int)m1, ax64[1], tab.tw64[1],
                                                  nullptr, 1, s, err);
        if (!e)
            e = axis_step<double, kForward>(tmp, grid, 0, 0, 1, m1 * n2, (int)m0, (int)m0, ax64[0], tab.tw64[0],
                                            nullptr, 1, s, err);
        if (e) return e;
        FHB_CUDA(cache_alloc(&tab.thin, sizeof(T) * (size_t)(m0 * m1 * n2), s));
        thin_store_kernel<T><<<blocks_of(m0 * m1 * n2, 256), 256, 0, s>>>(grid, static_cast<T *>(tab.thin), m0, m1, n2,
                                                                          d_map);
        FHB_CUDA(cudaGetLastError());
        if (!fp32) {
            FHB_CUDA(cudaStreamSynchronize(s));
            return FH_OK;
        }
        // the port columns of an FP32 operator take the whole spectrum
    }
    wrapped_kernel_kernel<<<blocks_of(P, 256), 256, 0, s>>>(grid, sh.n[0], sh.n[1], sh.n[2], sh.m[0], sh.m[1],
                                                           sh.m[2], spacing);
    FHB_CUDA(cudaGetLastError());
    fh_status e = axis_step<double, kForward>(grid, tmp, 0, 0, m0 * m1, 1, (int)m2, (int)m2, ax64[2], tab.tw64[2],
                                              nullptr, 1, s, err);
    if (!e)
        e = axis_step<double, kForward>(tmp, grid, 0, 0, m0, m2, (int)m1, (int)m1, ax64[1], tab.tw64[1], nullptr, 1, s,
                                        err);
    if (!e)
        e = axis_step<double, kForward>(grid, tmp, 0, 0, 1, m1 * m2, (int)m0, (int)m0, ax64[0], tab.tw64[0], nullptr,
                                        1, s, err);
    if (e) return e;
    FHB_CUDA(cache_alloc(&tab.spectrum, sizeof(T) * (size_t)P, s));
    spectrum_store_kernel<T><<<blocks_of(P, 256), 256, 0, s>>>(tmp, static_cast<T *>(tab.spectrum), m0, m1, m2,
                                                               d_map);
    FHB_CUDA(cudaGetLastError());
    FHB_CUDA(cudaStreamSynchronize(s));
    return FH_OK;
}

template <class T>
fh_status fftconv_run(const FftConvTables &tab, void *work, int grids, cudaStream_t s, fh_error_info *err) {
    using V = typename Cplx<T>::type;
    const FftConvShape &sh = tab.shape;
    const int64_t n0 = sh.n[0], n1 = sh.n[1], n2 = sh.n[2], m1 = sh.m[1], m2 = sh.m[2];
    const int64_t sa = n0 * n1 * n2, sb = n0 * n1 * m2, sc = n0 * m1 * m2;
    V *A = static_cast<V *>(work);
    V *B = A + sa * grids;
    V *C = B + sb * grids;
    if (tab.thin) {
        const T *K = static_cast<const T *>(tab.thin);
        C = A + sa * grids;
        const int64_t st = n0 * m1 * n2;
        fh_status e = thin_step<T, kForward>(A, C, sa, st, n0, n1 * n2, m1 * n2, n2, n2, (int)n1, (int)m1, tab.axis[1],
                                             tab.tw[1], nullptr, grids, s, err);
        if (!e)
            e = thin_step<T, kFused>(C, C, st, st, m1, n2, n2, m1 * n2, n2, (int)n0, (int)n0, tab.axis[0], tab.tw[0],
                                     K, grids, s, err);
        if (!e)
            e = thin_step<T, kInverse>(C, A, st, sa, n0, m1 * n2, n1 * n2, n2, n2, (int)m1, (int)n1, tab.axis[1],
                                       tab.tw[1], nullptr, grids, s, err);
        return e;
    }
    const T *spec = static_cast<const T *>(tab.spectrum);
    fh_status e = axis_step<T, kForward>(A, B, sa, sb, n0 * n1, 1, (int)n2, (int)m2, tab.axis[2], tab.tw[2], nullptr,
                                         grids, s, err);
    if (!e)
        e = axis_step<T, kForward>(B, C, sb, sc, n0, m2, (int)n1, (int)m1, tab.axis[1], tab.tw[1], nullptr, grids, s,
                                   err);
    if (!e)
        e = axis_step<T, kFused>(C, C, sc, sc, 1, m1 * m2, (int)n0, (int)n0, tab.axis[0], tab.tw[0], spec, grids, s,
                                 err);
    if (!e)
        e = axis_step<T, kInverse>(C, B, sc, sb, n0, m2, (int)m1, (int)n1, tab.axis[1], tab.tw[1], nullptr, grids, s,
                                   err);
    if (!e)
        e = axis_step<T, kInverse>(B, A, sb, sa, n0 * n1, 1, (int)m2, (int)n2, tab.axis[2], tab.tw[2], nullptr, grids,
                                   s, err);
    return e;
}

void fftconv_free(FftConvTables &tab, cudaStream_t s) {
    for (int a = 0; a < 3; ++a) {
        if (tab.tw64[a] && tab.tw64[a] != tab.tw[a]) cache_free(tab.tw64[a], s);
        if (tab.tw[a]) cache_free(tab.tw[a], s);
        tab.tw[a] = tab.tw64[a] = nullptr;
    }
    if (tab.spectrum) cache_free(tab.spectrum, s);
    if (tab.thin) cache_free(tab.thin, s);
    tab.spectrum = tab.thin = nullptr;
}

template fh_status fftconv_setup<float>(const FftConvShape &, double, FftConvTables &, cudaStream_t, fh_error_info *);
template fh_status fftconv_setup<double>(const FftConvShape &, double, FftConvTables &, cudaStream_t,
                                         fh_error_info *);
template fh_status fftconv_run<float>(const FftConvTables &, void *, int, cudaStream_t, fh_error_info *);
template fh_status fftconv_run<double>(const FftConvTables &, void *, int, cudaStream_t, fh_error_info *);

}  // namespace fhb

using namespace fhb;

extern "C" fh_status fh_test_grid_convolution(const int64_t *n, const int64_t *m, double spacing, int32_t fp32,
                                              const double *sources, int32_t fields, double *potentials,
                                              fh_error_info *err) {
    clear_error(err);
    if (!n || !m || !sources || !potentials || fields < 1)
        return fail(err, FH_ERR_INVALID_ARGUMENT, "null argument or no fields");
    FftConvShape sh;
    for (int a = 0; a < 3; ++a) {
        if (n[a] < 1 || m[a] < 2 * n[a] - 1)
            return fail(err, FH_ERR_INVALID_ARGUMENT, "padded axis shorter than 2 n - 1");
        sh.n[a] = n[a];
        sh.m[a] = m[a];
    }
    fh_status st = ensure_device(err);
    if (st) return st;
    cudaStream_t s = nullptr;
    FHB_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    struct Guard {
        cudaStream_t s;
        FftConvTables tab;
        void *work = nullptr;
        ~Guard() {
            cudaStreamSynchronize(s);
            if (work) cache_free(work, s);
            fftconv_free(tab, s);
            cudaStreamSynchronize(s);
            cudaStreamDestroy(s);
        }
    } g{s};
    st = fp32 ? fftconv_setup<float>(sh, spacing, g.tab, s, err) : fftconv_setup<double>(sh, spacing, g.tab, s, err);
    if (st) return st;
    const int grids = (fields + 1) / 2;
    const int64_t G = sh.n[0] * sh.n[1] * sh.n[2];
    const size_t elem = fp32 ? 4 : 8;
    FHB_CUDA(cache_alloc(&g.work, 2 * elem * fftconv_work_elems(sh) * (size_t)grids, s));
    // fields as real / imaginary parts of the complex source grids
    std::vector<double> h((size_t)(2 * G * grids), 0.0);
    for (int f = 0; f < fields; ++f)
        for (int64_t p = 0; p < G; ++p) h[(size_t)(2 * ((f / 2) * G + p) + (f & 1))] = sources[(size_t)(f * G + p)];
    if (fp32) {
        std::vector<float> hf(h.begin(), h.end());
        FHB_CUDA(cudaMemcpyAsync(g.work, hf.data(), 4 * hf.size(), cudaMemcpyHostToDevice, s));
        st = fftconv_run<float>(g.tab, g.work, grids, s, err);
        if (st) return st;
        FHB_CUDA(cudaMemcpyAsync(hf.data(), g.work, 4 * hf.size(), cudaMemcpyDeviceToHost, s));
        FHB_CUDA(cudaStreamSynchronize(s));
        std::copy(hf.begin(), hf.end(), h.begin());
    } else {
        FHB_CUDA(cudaMemcpyAsync(g.work, h.data(), 8 * h.size(), cudaMemcpyHostToDevice, s));
        st = fftconv_run<double>(g.tab, g.work, grids, s, err);
        if (st) return st;
        FHB_CUDA(cudaMemcpyAsync(h.data(), g.work, 8 * h.size(), cudaMemcpyDeviceToHost, s));
        FHB_CUDA(cudaStreamSynchronize(s));
    }
    for (int f = 0; f < fields; ++f)
        for (int64_t p = 0; p < G; ++p) potentials[(size_t)(f * G + p)] = h[(size_t)(2 * ((f / 2) * G + p) + (f & 1))];
    return FH_OK;
}

// The pFFT convolution without a library FFT (fh_fftconv.cu): pruned
// mixed-radix transforms, FP32 or FP64.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "fh_internal.h"

namespace fhb {

constexpr int kFftMaxStages = 8;
constexpr int64_t kFftMaxLength = 4800;  // longest padded axis

// One axis: its length and its stages (radix R over blocks of R S points),
// with the constants of the stages' index divisions and the places of their
// twiddles in the axis' table, passed by value to the kernels. 
struct FftAxis {
    int m = 1;
    int nst = 0;
    int R[kFftMaxStages] = {};
    int S[kFftMaxStages] = {};
    unsigned magic_S[kFftMaxStages] = {};
    unsigned magic_nb[kFftMaxStages] = {};  // of m / R
    int tw[kFftMaxStages] = {};
    int tw_count = 0;
};
bool fft_axis_plan(int64_t m, bool fp32, FftAxis &ax);
// The place of every frequency of an axis after its forward stages.
std::vector<int> fft_places(const FftAxis &ax);

// Unpadded grid n (axis 2 fastest) and the padded torus m (m_a >= 2 n_a - 1).
struct FftConvShape {
    int64_t n[3] = {1, 1, 1};
    int64_t m[3] = {1, 1, 1};
};

// Per-operator tables: the stages' twiddles per axis (in the convolution's
// precision, and FP64 for the set-up) and the kernel's real spectrum on the
// padded grid (times 1 / P), laid out [i][j][k], each axis in the order that
// its forward stages leave the frequencies in.
struct FftConvTables {
    FftConvShape shape;
    FftAxis axis[3];
    void *tw[3] = {nullptr, nullptr, nullptr};
    void *tw64[3] = {nullptr, nullptr, nullptr};
    void *spectrum = nullptr;
    // A thin grid's spectrum over axes 0 and 1 only (times 1 / (m0 m1)), laid
    // out [k1][distance along axis 2][k0]; FP64 tables then have no `spectrum`.
    void *thin = nullptr;
    bool fp32 = false;
};

// Complex elements of the work buffer per complex grid: the sources /
// potentials A (n0 n1 n2), then B (n0 n1 m2), then C (n0 m1 m2); a batch of
// grids keeps each part contiguous per grid (A of every grid first).  (The thin
// form has no B and n0 m1 n2 for C.)
size_t fftconv_work_elems(const FftConvShape &sh);

// T = float or double: the precision of the convolution.
template <class T>
fh_status fftconv_setup(const FftConvShape &sh, double spacing, FftConvTables &tab, cudaStream_t s,
                        fh_error_info *err);
// The convolution of `grids` complex grids in place: on entry A[g] holds the
// sources of grid g (two real fields as real and imaginary parts, [i][j][k]),
// on return the potentials.
template <class T>
fh_status fftconv_run(const FftConvTables &tab, void *work, int grids, cudaStream_t s, fh_error_info *err);
// The same with the FP32 tables for the port columns (fh_fftconv_ports.cu).
fh_status fftconv_run_ports(const FftConvTables &tab, void *work, int grids, cudaStream_t s, fh_error_info *err);
void fftconv_free(FftConvTables &tab, cudaStream_t s);

}  // namespace fhb

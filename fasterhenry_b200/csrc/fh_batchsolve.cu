// Batched sweeps of many small, unevenly sized systems in ONE
// persistent launch (the batched form of MeshSystem::sweep over many
// geometries, solve.rs:881-893 / 1039-1079; the reference sweeps them one
// after another).
//
// A work item is one (system, frequency).  Items are sorted by cost (m^3,
// largest first) on the host and handed out through an atomic counter to
// persistent CTAs, two per SM.  A CTA solves its item alone, in its own
// workspace slot, by the FP64 factorization A = L D L^T without interchanges
// of the matrix bordered with its ports (fh_ldlt.cuh), whose trailing p x p
// block is Z: the products run on the FP64 tensor instruction, which beats
// FP32 factors from the scalar pipes and their refinement.
//
// The order M = m + p is cut into tiles of E x E; tile (i, j) below the
// diagonal holds L_ij, tile (j, i) above it B_ij = L_ij D_j, both [k][row], so
// every operand is one run of memory.  Padding rows (a unit diagonal) stand
// at the front, so that the ports end the last tile, where the diagonal
// block's elimination leaves Z; E or more ports take tiles of their own.
// Block columns are taken left to right, each tile once:
//
//   C_ij = A_ij - sum_k<j L_ik B_jk^T   straight from R and L, in registers;
//   j = i: L_jj^-1 and D_j (DiagBlock), L_jj^-1 kept in tile (j, j);
//   i > j: B_ij = C_ij L_jj^-T, L_ij = B_ij D_j^-1, and the rows' growth.
//
// Taking the sum over k in one go reads each operand tile once per product
// and writes a tile once; a trailing update per panel would also read and
// write every C per panel, and the slots of all CTAs together exceed L2.
//
// Items larger than a CTA's even share of the launch would set its time on
// their own, so the leading ones are taken by clusters of CTAs: in block
// column j the tiles go round, the first CTA starting with the diagonal block
// while the others take the sums of theirs; one cluster barrier hands them
// L_jj^-1, a second ends the column.
//
// 64 spirals of orders 56-736 x 16 frequencies on one B200: 3.6 ms, 15 of
// the 37 TFLOP/s of the instruction, bound by the diagonal blocks' chains and
// by few tiles per column (7.5 ms with a CTA for every item, 36 ms with FP32
// factors from the scalar pipes and FP64 refinement).
//
// An item with a vanishing pivot or too much growth is marked; the host
// redoes it with the FP64 sweep.  E and the depth of the operand pipeline come
// per item from the autotuner's table (fh_batchtune.cpp), by order bucket.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <vector>

#include "fh_batchsolve.h"
#include "fh_device.cuh"
#include "fh_ldlt.cuh"

namespace fhb {
namespace {

constexpr int kBT = 256;  // threads per CTA: 2 x 4 warps over a tile

struct Shared {
    double2 v[2 * 64];   // the diagonal block's published rows
    double2 dinv[64];
    double rowsum[64];
    BatchSys sys;
    BatchItem item;
    int next, bad;
    int group, rank;  // CTAs on this item, and this one's place among them
};

__device__ __forceinline__ void group_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void group_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// The tiling of a bordered matrix of m internal rows and p ports.
struct Tiling {
    int tiles;     // tiles per side
    int inner;     // block columns that are eliminated
    int64_t off;   // padding rows at the front
    __host__ __device__ Tiling(int64_t m, int64_t p, int edge) {
        if (p < edge) {
            tiles = inner = (int)((m + p + edge - 1) / edge);
            off = (int64_t)tiles * edge - (m + p);
        } else {
            inner = (int)((m + edge - 1) / edge);
            tiles = inner + (int)((p + edge - 1) / edge);
            off = (int64_t)inner * edge - m;
        }
    }
};

template <int E, int KS, int BUFS>
__device__ __forceinline__ void solve_item(double2 *tiles, double *growth, double2 *dinv, double2 *smem, Shared &sh,
                                           double2 *z_all, int32_t *status) {
    constexpr int kPad = E + 2;  // row of a staged chunk (bank offsets as in fh_ldlt.cu)
    constexpr int FM = E / 16, FN = E / 32;
    static_assert(BUFS * 2 * KS >= E, "the buffers also hold a whole tile");
    const int m = (int)sh.sys.m, p = (int)sh.sys.p;
    const int64_t ld = sh.sys.ld;
    const Tiling tl(m, p, E);
    const int T = tl.tiles, off = (int)tl.off, mi = off + m;  // mi: the first port
    const double w = sh.item.omega;
    const double *R = sh.sys.R, *L = sh.sys.L;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int row0 = 8 * FM * (warp >> 2), col0 = 8 * FN * (warp & 3);
    auto tile = [&](int i, int j) { return tiles + ((int64_t)i * T + j) * (E * E); };
    auto put_z = [&](int a, int c, double2 v) {  // Z is symmetric, and real at zero frequency (solve.rs:811-815)
        if (w == 0.0) v.y = 0.0;
        double2 *z = z_all + sh.item.z_offset;
        z[(int64_t)a * p + c] = v;
        z[(int64_t)c * p + a] = v;
    };
    if (sh.rank == 0)
        for (int i = tid; i < T * E; i += kBT) growth[i] = 0.0;
    if (tid == 0) sh.bad = 0;
    __syncthreads();
    for (int j = 0; j < T; ++j) {
        const int nb = min(E, max(0, mi - j * E));
        const int stages = min(j, tl.inner) * (E / KS);
        bool joined = sh.group == 1 || nb == 0;  // past the wait for the diagonal block
        if (!joined && sh.rank != 0) group_arrive();
        for (int ti = j + sh.rank; ti < T; ti += sh.group) {
            auto load = [&](int st) {
                if (st < stages) {
                    double2 *l = smem + (st % BUFS) * 2 * KS * kPad, *u = l + KS * kPad;
                    const int kt = st / (E / KS), k0 = st % (E / KS) * KS * E;
                    const double2 *lt = tile(ti, kt) + k0, *ut = tile(kt, j) + k0;
#pragma unroll
                    for (int idx = tid; idx < KS * E; idx += kBT) {
                        const int r = idx % E, k = idx / E;
                        copy16(&l[k * kPad + r], lt, idx, true);
                        copy16(&u[k * kPad + r], ut, idx, true);
                    }
                }
                copy_commit();  // an empty group keeps the count
            };
#pragma unroll
            for (int st = 0; st < BUFS - 1; ++st) load(st);
            double re[FM][FN][2], im[FM][FN][2];
#pragma unroll
            for (int fm = 0; fm < FM; ++fm)
#pragma unroll
                for (int fn = 0; fn < FN; ++fn)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int i = ti * E + row0 + 8 * fm + g - off;
                        const int c = j * E + col0 + 8 * fn + 2 * t + e - off;
                        double2 a = make_double2(i == c ? 1.0 : 0.0, 0.0);
                        if (i >= 0 && c >= 0)
                            a = i < m + p && c < m + p ? make_double2(R[i + c * ld], w * L[i + c * ld])
                                                       : make_double2(0.0, 0.0);
                        re[fm][fn][e] = a.x;
                        im[fm][fn][e] = a.y;
                    }
            // a diagonal tile's part above the diagonal is not needed
            const bool live = ti > j || row0 + 8 * FM > col0;
            for (int st = 0; st < stages; ++st) {
                copy_wait<BUFS - 2>();
                __syncthreads();  // stage st has arrived; stage st - 1 has been read
                load(st + BUFS - 1);
                const double2 *l = smem + (st % BUFS) * 2 * KS * kPad, *u = l + KS * kPad;
                if (live) {
#pragma unroll
                    for (int k4 = 0; k4 < KS; k4 += 4)
                        tile_step<-1>(l + k4 * kPad, kPad, u + k4 * kPad, kPad, row0, col0, g, t, re, im);
                }
            }
            if (nb == 0) {  // among the ports: a block of Z
#pragma unroll
                for (int fm = 0; fm < FM; ++fm)
#pragma unroll
                    for (int fn = 0; fn < FN; ++fn)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int a = ti * E + row0 + 8 * fm + g - mi;
                            const int c = j * E + col0 + 8 * fn + 2 * t + e - mi;
                            if (a < p && c <= a) put_z(a, c, make_double2(re[fm][fn][e], im[fm][fn][e]));
                        }
                __syncthreads();  // before the next tile's copies
                continue;
            }
            __syncthreads();  // the last stage has been read
#pragma unroll
            for (int fm = 0; fm < FM; ++fm)
#pragma unroll
                for (int fn = 0; fn < FN; ++fn)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        smem[(col0 + 8 * fn + 2 * t + e) * kPad + row0 + 8 * fm + g] =
                            make_double2(re[fm][fn][e], im[fm][fn][e]);
            if (tid < E) sh.rowsum[tid] = 0.0;
            __syncthreads();
            if (ti == j) {
                DiagBlock<E, kBT / 32, false> block;
                block.factor(sh.v, smem, kPad, E, nb, smem, kPad, sh.dinv, sh.rowsum, &sh.bad);
                __syncthreads();
                if (nb < E) {  // the last tile ends with the ports
                    for (int idx = tid; idx < p * p; idx += kBT) {
                        const int a = idx / p, c = idx % p;
                        if (c <= a) put_z(a, c, smem[(nb + c) * kPad + nb + a]);
                    }
                } else {
                    double2 *x = tile(j, j);
                    for (int idx = tid; idx < E * E; idx += kBT) x[idx] = smem[idx / E * kPad + idx % E];
                    if (tid < E) dinv[tid] = sh.dinv[tid];
                }
                if (!joined) group_arrive();
            } else {
                if (!joined) {
                    group_wait();
                    joined = true;
                    if (tid < E) sh.dinv[tid] = dinv[tid];
                    __syncthreads();
                }
                // B = C X^T; X = L_jj^-1 is lower triangular: column c of B needs k <= c
                const double2 *x = tile(j, j);
                double bre[FM][FN][2] = {}, bim[FM][FN][2] = {};
#pragma unroll 1
                for (int k4 = 0; k4 < col0 + 8 * FN; k4 += 4)
                    tile_step<1>(smem + k4 * kPad, kPad, x + k4 * E, E, row0, col0, g, t, bre, bim);
                double2 *bt = tile(j, ti), *lt = tile(ti, j);
#pragma unroll
                for (int fm = 0; fm < FM; ++fm) {
                    const int r = row0 + 8 * fm + g;
                    double sum = 0.0;
#pragma unroll
                    for (int fn = 0; fn < FN; ++fn)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int c = col0 + 8 * fn + 2 * t + e;
                            const double2 b = make_double2(bre[fm][fn][e], bim[fm][fn][e]), d = sh.dinv[c];
                            const double2 q = make_double2(b.x * d.x - b.y * d.y, b.x * d.y + b.y * d.x);
                            bt[c * E + r] = b;
                            lt[c * E + r] = q;
                            sum += (fabs(b.x) + fabs(b.y)) * (fabs(q.x) + fabs(q.y));  // |l|^2 |d|
                        }
                    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                    if (t == 0) atomicAdd(&sh.rowsum[r], sum);
                }
            }
            __syncthreads();
            if (tid < E) atomicAdd(&growth[ti * E + tid], sh.rowsum[tid]);
        }
        if (!joined) group_wait();
        if (sh.group > 1) {  // the column is complete
            group_arrive();
            group_wait();
        }
    }
    __syncthreads();
    if (sh.rank != 0) return;
    bool bad = sh.bad != 0;
    for (int i = tid; i < m; i += kBT)
        bad = bad || !(__ldcg(&growth[off + i]) <= kGrowthLimit * (fabs(R[i + i * ld]) + fabs(w * L[i + i * ld])));
    bad = __syncthreads_or(bad);
    if (tid == 0) status[sh.item.index] = bad ? -1 : 0;
}

template <int C>
__device__ __forceinline__ void solve_config(double2 *tiles, double *growth, double2 *dinv, double2 *smem,
                                             Shared &sh, double2 *z_all, int32_t *status) {
    solve_item<kBatchEdge[C], kBatchStage[C], kBatchBuffers[C]>(tiles, growth, dinv, smem, sh, z_all, status);
}

__global__ void __launch_bounds__(kBT, 2)
    batch_kernel(const BatchSys *__restrict__ systems, const BatchItem *__restrict__ items, int nitems, int grouped,
                 unsigned *counter, unsigned char *work, size_t slot_bytes, size_t tile_bytes, size_t growth_bytes,
                 int ctas, double2 *z_all, int32_t *status) {
    extern __shared__ __align__(16) unsigned char batch_smem[];
    __shared__ Shared sh;
    double2 *smem = reinterpret_cast<double2 *>(batch_smem);
    const int rank = (int)blockIdx.x % kBatchGroup;
    // the first `grouped` items by groups of CTAs (the clusters), then a CTA per item
    for (int phase = grouped > 0 ? 0 : 1; phase < 2; ++phase) {
        const int count = phase == 0 ? grouped : nitems - grouped;
        if (phase == 1 && (int)blockIdx.x >= ctas) return;  // no slot
        const size_t slot = blockIdx.x - (phase == 0 ? rank : 0);
        unsigned char *base = work + slot * slot_bytes;
        double2 *tiles = reinterpret_cast<double2 *>(base);
        double *growth = reinterpret_cast<double *>(base + tile_bytes);
        double2 *dinv = reinterpret_cast<double2 *>(base + tile_bytes + growth_bytes);
        if (threadIdx.x == 0) {
            sh.group = phase == 0 ? kBatchGroup : 1;
            sh.rank = phase == 0 ? rank : 0;
        }
        for (;;) {
            if (threadIdx.x == 0 && sh.rank == 0) sh.next = (int)atomicAdd(counter + phase, 1u);
            if (phase == 0) {
                group_arrive();
                group_wait();
                unsigned own = (unsigned)__cvta_generic_to_shared(&sh.next), first;
                int next;
                asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(first) : "r"(own));
                asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(next) : "r"(first) : "memory");
                group_arrive();  // the first CTA's `next` stays until all have read it
                group_wait();
                if (threadIdx.x == 0) sh.next = next;
            }
            if (threadIdx.x == 0 && sh.next < count) {
                sh.item = items[sh.next + (phase == 0 ? 0 : grouped)];
                sh.sys = systems[sh.item.sys];
            }
            __syncthreads();
            if (sh.next >= count) break;
            switch (sh.item.cfg) {
                case 0: solve_config<0>(tiles, growth, dinv, smem, sh, z_all, status); break;
                case 1: solve_config<1>(tiles, growth, dinv, smem, sh, z_all, status); break;
                case 2: solve_config<2>(tiles, growth, dinv, smem, sh, z_all, status); break;
                default: solve_config<3>(tiles, growth, dinv, smem, sh, z_all, status); break;
            }
            __syncthreads();
        }
        __syncthreads();  // before the next phase's `group` and `rank`
    }
}

// Bytes of the tiles, and the rows, of the larger tiling of either edge.
size_t tile_bytes(int64_t m, int64_t p, int64_t *rows) {
    size_t bytes = 0;
    *rows = 0;
    for (int c = 0; c < kBatchConfigs; ++c) {
        const int edge = kBatchEdge[c];
        // a system of fewer ports may be tiled the other way: at most this many tiles
        const int64_t side = ((m + edge - 1) / edge + (p + edge - 1) / edge) * edge;
        bytes = std::max(bytes, sizeof(double2) * (size_t)side * (size_t)side);
        *rows = std::max(*rows, side);
    }
    return bytes;
}

}  // namespace

size_t batch_smem_bytes() {
    size_t bytes = 0;
    for (int c = 0; c < kBatchConfigs; ++c)
        bytes = std::max(bytes, sizeof(double2) * 2 * kBatchStage[c] * kBatchBuffers[c] * (kBatchEdge[c] + 2));
    return bytes;
}

size_t batch_slot_bytes(int64_t mmax, int pmax) {
    int64_t rows = 0;
    const size_t bytes = tile_bytes(mmax, pmax, &rows) + sizeof(double) * (size_t)rows + sizeof(double2) * 64;
    return (bytes + 255) / 256 * 256;
}

namespace {

cudaLaunchConfig_t launch_config(int ctas, cudaLaunchAttribute *attr, cudaStream_t s) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)((ctas + kBatchGroup - 1) / kBatchGroup * kBatchGroup));
    c.blockDim = dim3(kBT);
    c.dynamicSmemBytes = batch_smem_bytes();
    c.stream = s;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = kBatchGroup;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    c.attrs = attr;
    c.numAttrs = 1;
    return c;
}

}  // namespace

int batch_resident_ctas() {
    int clusters = 0;
    cudaFuncSetAttribute(batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)batch_smem_bytes());
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t c = launch_config(kBatchGroup, &attr, nullptr);
    if (cudaOccupancyMaxActiveClusters(&clusters, batch_kernel, &c) != cudaSuccess) cudaGetLastError();
    return kBatchGroup * std::max(1, clusters);
}

fh_status batch_launch(const BatchSys *d_systems, const BatchItem *d_items, int nitems, int grouped,
                       unsigned *d_counter, void *d_work, size_t slot_bytes, int64_t mmax, int pmax, double2 *d_z,
                       int32_t *d_status, int ctas, cudaStream_t s, fh_error_info *err) {
    FHB_CUDA(cudaFuncSetAttribute(batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)batch_smem_bytes()));
    FHB_CUDA(cudaMemsetAsync(d_counter, 0, 2 * sizeof(unsigned), s));
    int64_t rows = 0;
    const size_t tb = tile_bytes(mmax, pmax, &rows);
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t c = launch_config(ctas, &attr, s);
    FHB_CUDA(cudaLaunchKernelEx(&c, batch_kernel, d_systems, d_items, nitems, grouped, d_counter,
                                static_cast<unsigned char *>(d_work), slot_bytes, tb, sizeof(double) * (size_t)rows,
                                ctas, d_z, d_status));
    return FH_OK;
}

}  // namespace fhb

using namespace fhb;

extern "C" fh_status fh_test_batch_solve(const double *r, const double *l, int64_t m, int64_t p, const double *omega,
                                         int32_t count, int32_t config, int32_t grouped, double *z,
                                         int32_t *failed, fh_error_info *err) {
    clear_error(err);
    if (!r || !l || !omega || !z || !failed || m < 0 || p < 1 || count < 1 || config < 0 || config >= kBatchConfigs ||
        grouped < 0 || grouped > count)
        return fail(err, FH_ERR_INVALID_ARGUMENT, "null argument, empty system or unknown configuration");
    fh_status st = ensure_device(err);
    if (st) return st;
    const size_t M = (size_t)(m + p), sym = 8 * M * M, zs = 16 * (size_t)(count * p * p);
    const int ctas = std::min<int>(batch_resident_ctas(), count);
    const size_t slot = batch_slot_bytes(m, (int)p);
    void *d[8] = {};
    struct Release {
        void **d;
        ~Release() {
            for (int k = 0; k < 8; ++k) cudaFree(d[k]);
        }
    } release{d};
    const size_t bytes[8] = {sym, sym, sizeof(BatchSys), sizeof(BatchItem) * (size_t)count, 2 * sizeof(unsigned),
                             slot * (size_t)ctas, zs, 4 * (size_t)count};
    for (int k = 0; k < 8; ++k) FHB_CUDA(cudaMalloc(&d[k], bytes[k]));
    BatchSys sys;
    sys.R = (double *)d[0], sys.L = (double *)d[1], sys.ld = (int64_t)M, sys.m = m, sys.p = p;
    std::vector<BatchItem> items((size_t)count);
    for (int32_t f = 0; f < count; ++f) {
        items[(size_t)f].cfg = config;
        items[(size_t)f].omega = omega[f];
        items[(size_t)f].z_offset = (int64_t)f * p * p;
        items[(size_t)f].index = f;
    }
    FHB_CUDA(cudaMemcpy(d[0], r, sym, cudaMemcpyHostToDevice));
    FHB_CUDA(cudaMemcpy(d[1], l, sym, cudaMemcpyHostToDevice));
    FHB_CUDA(cudaMemcpy(d[2], &sys, sizeof sys, cudaMemcpyHostToDevice));
    FHB_CUDA(cudaMemcpy(d[3], items.data(), bytes[3], cudaMemcpyHostToDevice));
    st = batch_launch((BatchSys *)d[2], (BatchItem *)d[3], count, grouped, (unsigned *)d[4], d[5], slot, m, (int)p,
                      (double2 *)d[6], (int32_t *)d[7], ctas, nullptr, err);
    if (st) return st;
    FHB_CUDA(cudaMemcpy(z, d[6], zs, cudaMemcpyDeviceToHost));
    FHB_CUDA(cudaMemcpy(failed, d[7], bytes[7], cudaMemcpyDeviceToHost));
    for (int32_t f = 0; f < count; ++f) failed[f] = failed[f] < 0;
    return FH_OK;
}

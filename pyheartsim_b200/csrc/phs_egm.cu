// Unipolar electrogram of the PyHeartSim B200 path: lead-field construction,
// FP64 contraction and normalisation.
//
// The reference (simulation/unipolar_electrogram_gpu.py:21-69) evaluates
//   egm[t,e] = sum_v c_v / l_ve^3 * sum_i (D_v grad V)_i * l_ve,i
// with one atomicAdd per (voxel, electrode, time).  Everything except V is
// independent of time, and the gradient is linear in V
// (simulation/unipolar_electrogram_equation_parts.py:60-103), so the sum is a
// matrix product egm = V M with a lead field M (n_v x n_e).  M is built once in
// FP64 (stored transposed, Mt[e][w], the K-major operand of the contraction)
// and the contraction runs as a GEMM.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <algorithm>
#include <vector>

#include "../../include/phs.h"
#include "phs_common.cuh"

namespace phs {

// Mt[e][w] = sum over incoming gradient terms (v, +-(d+1)) of
//            +-c_v / l^3 * (D_v^T l)_d / (2 Delta),  l = x_v - x_e, |l| clamped to >= 1.
// A thread keeps the first kLfTerms terms of its voxel (a lattice voxel has six
// at most) in registers and walks a chunk of electrodes, so a term costs its
// arithmetic only; that bounds the kernel (FP64), so 1 / l^3 comes from one
// rsqrt in place of a square root and a division.  91k voxels x 64 electrodes:
// 174 us with the terms read again for every electrode, now 99 us; the error of
// the electrogram against 64-bit reference sums is unchanged (1e-14).
constexpr int kLfTerms = 6, kLfElectrodes = 16;
template <bool TENSOR>
__global__ void __launch_bounds__(128) leadfield_kernel(int64_t n_v, int64_t n_e, const double* __restrict__ xyz,
                                                        const double* __restrict__ exyz, const double* __restrict__ c,
                                                        const double* __restrict__ D0,
                                                        const int32_t* __restrict__ in_ptr,
                                                        const int32_t* __restrict__ in_src,
                                                        const int8_t* __restrict__ in_dir, double inv2d,
                                                        double* __restrict__ Mt) {
    __shared__ double se[kLfElectrodes][3];
    const int64_t e0 = (int64_t)blockIdx.y * kLfElectrodes;
    const int ne = (int)((n_e - e0 < kLfElectrodes) ? n_e - e0 : kLfElectrodes);
    if ((int)threadIdx.x < 3 * ne) se[threadIdx.x / 3][threadIdx.x % 3] = exyz[3 * e0 + threadIdx.x];
    __syncthreads();
    for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n_v; w += (int64_t)gridDim.x * blockDim.x) {
        const int32_t b0 = in_ptr[w], b1 = in_ptr[w + 1];
        // a term: the source's position and the scaled row D_v^T e_d (identity: its
        // one component and which)
        auto load = [&](int32_t q, double (&x)[3], double (&p)[3], int& d) {
            const int32_t v = in_src[q];
            const int dd = in_dir[q];
            d = (dd > 0 ? dd : -dd) - 1;
#pragma unroll
            for (int i = 0; i < 3; ++i) x[i] = xyz[3 * (int64_t)v + i];
            const double s = (dd > 0) ? c[v] * inv2d : -(c[v] * inv2d);
            if (TENSOR) {
#pragma unroll
                for (int i = 0; i < 3; ++i) p[i] = s * D0[9 * (int64_t)v + 3 * i + d];
            } else {
                p[0] = s;
            }
        };
        auto value = [&](const double (&x)[3], const double (&p)[3], int d, const double* pe) {
            const double lx = x[0] - pe[0], ly = x[1] - pe[1], lz = x[2] - pe[2];
            const double l2 = lx * lx + ly * ly + lz * lz;
            const double r = (l2 < 1.0) ? 1.0 : rsqrt(l2);
            const double proj = TENSOR ? p[0] * lx + p[1] * ly + p[2] * lz : p[0] * (d == 0 ? lx : (d == 1 ? ly : lz));
            return proj * (r * r * r);
        };
        double x[kLfTerms][3], p[kLfTerms][3];
        int d[kLfTerms];
#pragma unroll
        for (int t = 0; t < kLfTerms; ++t)
            if (b0 + t < b1) load(b0 + t, x[t], p[t], d[t]);
        for (int e = 0; e < ne; ++e) {
            double acc = 0.0;
#pragma unroll
            for (int t = 0; t < kLfTerms; ++t)
                if (b0 + t < b1) acc += value(x[t], p[t], d[t], se[e]);
            for (int32_t q = b0 + kLfTerms; q < b1; ++q) {
                double xq[3], pq[3];
                int dq;
                load(q, xq, pq, dq);
                acc += value(xq, pq, dq, se[e]);
            }
            Mt[(e0 + e) * n_v + w] = acc;
        }
    }
}

// FP64 C[t][e] = sum_k A[t][k] * B[e][k] over one K-split; partials go to
// P[split][t][e].  128 x 64 output tile, K-steps of 16 staged through a ring of
// three shared-memory stages by cp.async, 8 warps of 32 x 32 each on the FP64
// matrix instruction (mma.m16n8k8; tcgen05 has no FP64 form).  The bound is the
// FP64 units: a warp's K-step of 8 costs 16 shared-memory loads for 128 clocks
// of matrix work.  Rows of 16 + 4 doubles keep those loads free of bank
// conflicts.  Copies are 16 bytes where both operands' rows start on such
// boundaries, else 8.  (64 x 64 tiles with 4 x 4 values per thread read shared
// memory once per two multiply-adds: 1000 x 64 x 91k took 1.25 ms = 9.4
// TFLOP/s, now 0.47 ms = 25 TFLOP/s.)
constexpr int DG_BM = 128, DG_BN = 64, DG_BK = 16, DG_STAGES = 3, DG_LD = DG_BK + 4;
constexpr size_t DG_SMEM = (size_t)DG_STAGES * (DG_BM + DG_BN) * DG_LD * sizeof(double);

template <int BYTES>
__device__ __forceinline__ void cp_async(double* dst, const double* src, int valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(valid) : "memory");
}

// D += A (16x8, row) * B (8x8, col): lane l holds a: rows l/4 and l/4 + 8, k l%4
// (a[0], a[1]) and l%4 + 4 (a[2], a[3]); b: column l/4, the same k; d: rows
// l/4 (d[0], d[1]) and l/4 + 8 (d[2], d[3]), columns 2 (l%4) and + 1.
__device__ __forceinline__ void mma_f64(double (&d)[4], const double (&a)[4], const double (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

template <int BYTES>
__global__ void __launch_bounds__(256, 2)
dgemm_tn_kernel(int64_t M, int64_t N, int64_t K, const double* __restrict__ A, int64_t lda,
                const double* __restrict__ B, int64_t ldb, double* __restrict__ P, int64_t kchunk) {
    extern __shared__ __align__(16) double dg_smem[];
    constexpr int STAGE = (DG_BM + DG_BN) * DG_LD;
    constexpr int VAL = BYTES / 8;                              // values per copy
    constexpr int PER_ROW = DG_BK / VAL;
    const int64_t m0 = (int64_t)blockIdx.x * DG_BM, n0 = (int64_t)blockIdx.y * DG_BN;
    const int64_t k_beg = (int64_t)blockIdx.z * kchunk;
    const int64_t k_end = (K < k_beg + kchunk) ? K : k_beg + kchunk;
    const int steps = (int)((k_end - k_beg + DG_BK - 1) / DG_BK);
    // rows past M or N and k past k_end are filled with zeros (nothing is read)
    auto stage_in = [&](int step) {
        double* st = dg_smem + (step % DG_STAGES) * STAGE;
        const int64_t k0 = k_beg + (int64_t)step * DG_BK;
#pragma unroll
        for (int i = 0; i < (DG_BM + DG_BN) * PER_ROW / 256; ++i) {
            const int q = i * 256 + threadIdx.x;
            const int row = q / PER_ROW, kk = (q % PER_ROW) * VAL;
            const bool is_a = row < DG_BM;
            const int64_t g = is_a ? m0 + row : n0 + (row - DG_BM);
            const int64_t left = k_end - (k0 + kk);
            int valid = (left >= VAL) ? BYTES : (left > 0 ? (int)left * 8 : 0);
            if (g >= (is_a ? M : N)) valid = 0;
            const double* src = is_a ? A : B;
            if (valid) src += g * (is_a ? lda : ldb) + k0 + kk;
            cp_async<BYTES>(st + row * DG_LD + kk, src, valid);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = (warp & 3) * 32, wn = (warp >> 2) * 32;
    const int g = lane >> 2, t = lane & 3;
    double acc[2][4][4] = {};
    for (int s = 0; s < DG_STAGES - 1; ++s) {
        if (s < steps) stage_in(s);
        else asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int s = 0; s < steps; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(DG_STAGES - 2) : "memory");
        __syncthreads();                       // stage s is in; stage s - 1 is no longer read
        if (s + DG_STAGES - 1 < steps) stage_in(s + DG_STAGES - 1);
        else asm volatile("cp.async.commit_group;" ::: "memory");
        const double* As = dg_smem + (s % DG_STAGES) * STAGE;
        const double* Bs = As + DG_BM * DG_LD;
#pragma unroll
        for (int kk = 0; kk < DG_BK; kk += 8) {
            double a[2][4], b[4][2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const double* p = As + (wm + 16 * i + g) * DG_LD + kk + t;
                a[i][0] = p[0];
                a[i][1] = p[8 * DG_LD];
                a[i][2] = p[4];
                a[i][3] = p[8 * DG_LD + 4];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const double* p = Bs + (wn + 8 * j + g) * DG_LD + kk + t;
                b[j][0] = p[0];
                b[j][1] = p[4];
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) mma_f64(acc[i][j], a[i], b[j]);
        }
    }
    double* Pz = P + (int64_t)blockIdx.z * M * N;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int64_t gm = m0 + wm + 16 * i + g + (r >> 1) * 8, gn = n0 + wn + 8 * j + 2 * t + (r & 1);
                if (gm < M && gn < N) Pz[gm * N + gn] = acc[i][j][r];
            }
}

// Sum split-K partials (deterministic): eight threads per value add an eighth of
// the splits each, in order, and the eighths are added in order.
template <typename TO>
__global__ void __launch_bounds__(256) splitk_reduce_kernel(int64_t MN, int splits, const double* __restrict__ P,
                                                            TO* __restrict__ C) {
    __shared__ double s[8][32];
    const int col = threadIdx.x & 31, part = threadIdx.x >> 5;
    const int per = (splits + 7) / 8;
    const int z0 = part * per, z1 = (z0 + per < splits) ? z0 + per : splits;
    for (int64_t i0 = (int64_t)blockIdx.x * 32; i0 < MN; i0 += (int64_t)gridDim.x * 32) {
        const int64_t i = i0 + col;
        double a = 0.0;
        if (i < MN) {
            for (int z = z0; z < z1; z += 8) {         // eight loads in flight, the last few too
                double v[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] = (z + q < z1) ? P[(int64_t)(z + q) * MN + i] : 0.0;
#pragma unroll
                for (int q = 0; q < 8; ++q) a += v[q];
            }
        }
        s[part][col] = a;
        __syncthreads();
        if (part == 0 && i < MN) {
            for (int q = 1; q < 8; ++q) a += s[q][col];
            C[i] = (TO)a;
        }
        __syncthreads();
    }
}

// ptp[e] = max_t egm[t][e] - min_t egm[t][e].  A CTA takes 32 adjacent
// electrodes (whole sectors of each time step's row) and deals the time steps to
// 32 groups of threads.  (A CTA per electrode read one value out of each sector:
// 118 us with scale_kernel for 1000 x 2048 FP32; now 30 us.)
constexpr int kPtpCols = 32, kPtpParts = 32;
template <typename T>
__global__ void __launch_bounds__(kPtpCols* kPtpParts) ptp_kernel(int64_t Tn, int64_t n_e, const T* __restrict__ egm,
                                                                  double* __restrict__ ptp) {
    __shared__ double smx[kPtpParts][kPtpCols], smn[kPtpParts][kPtpCols];
    const int col = threadIdx.x % kPtpCols, part = threadIdx.x / kPtpCols;
    const int64_t e = (int64_t)blockIdx.x * kPtpCols + col;
    double mx = -INFINITY, mn = INFINITY;
    if (e < n_e) {
        for (int64_t t = part; t < Tn; t += 8 * kPtpParts) {   // eight loads in flight
            T v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int64_t at = t + q * kPtpParts;
                v[q] = egm[(at < Tn ? at : t) * n_e + e];
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                mx = fmax(mx, (double)v[q]);
                mn = fmin(mn, (double)v[q]);
            }
        }
    }
    smx[part][col] = mx;
    smn[part][col] = mn;
    __syncthreads();
    if (part != 0 || e >= n_e) return;
    for (int q = 1; q < kPtpParts; ++q) {
        mx = fmax(mx, smx[q][col]);
        mn = fmin(mn, smn[q][col]);
    }
    ptp[e] = mx - mn;
}

// egm *= 1 / mean_e(ptp); every block recomputes the mean in the same order
// (threads over the electrodes, then a tree).
template <typename T>
__global__ void __launch_bounds__(256) scale_kernel(int64_t total, int64_t n_e, const double* __restrict__ ptp,
                                                    T* __restrict__ egm) {
    __shared__ double s[256];
    double a = 0.0;
    for (int64_t e = threadIdx.x; e < n_e; e += 256) a += ptp[e];
    s[threadIdx.x] = a;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
        __syncthreads();
    }
    const double sc = 1.0 / (s[0] / (double)n_e);
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x)
        egm[i] = (T)((double)egm[i] * sc);
}

// Split-K plan: about two CTAs per SM, at least 256 of K each, at most
// max_partials partial values.
static void contract_plan(int64_t T, int64_t n_v, int64_t n_e, int64_t max_partials, int64_t* splits, int64_t* kchunk) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t tiles = ((T + DG_BM - 1) / DG_BM) * ((n_e + DG_BN - 1) / DG_BN);
    const int64_t target = 2LL * sms;
    // whole waves of the chip: the splits that fit, not one more
    int64_t s = std::max<int64_t>(1, std::min<int64_t>(std::max<int64_t>(1, target / tiles), (n_v + 255) / 256));
    s = std::min<int64_t>(s, max_partials / (T * n_e));
    int64_t kc = (n_v + s - 1) / s;
    kc = ((kc + DG_BK - 1) / DG_BK) * DG_BK;
    *kchunk = kc;
    *splits = (n_v + kc - 1) / kc;
}

static cudaError_t contract_launch(int64_t T, int64_t n_v, int64_t n_e, const double* V, int64_t ldv, const double* Mt,
                                   double* egm, double* P, int64_t splits, int64_t kchunk, cudaStream_t stream) {
    const dim3 grid((unsigned)((T + DG_BM - 1) / DG_BM), (unsigned)((n_e + DG_BN - 1) / DG_BN), (unsigned)splits);
    const bool wide = (((uintptr_t)V | (uintptr_t)Mt) & 15) == 0 && ldv % 2 == 0 && n_v % 2 == 0;
    const auto fn = wide ? dgemm_tn_kernel<16> : dgemm_tn_kernel<8>;
    // both kernels' opt-in, whichever this call launches
    cudaError_t e = allow_dynamic_smem((const void*)dgemm_tn_kernel<16>, DG_SMEM);
    if (e == cudaSuccess) e = allow_dynamic_smem((const void*)dgemm_tn_kernel<8>, DG_SMEM);
    if (e != cudaSuccess) return e;
    fn<<<grid, 256, DG_SMEM, stream>>>(T, n_e, n_v, V, ldv, Mt, n_v, P, kchunk);
    const int64_t MN = T * n_e;
    splitk_reduce_kernel<double><<<(unsigned)std::min<int64_t>((MN + 31) / 32, 4736), 256, 0, stream>>>(MN, (int)splits,
                                                                                                       P, egm);
    return cudaGetLastError();
}

int contract_f64(int64_t T, int64_t n_v, int64_t n_e, const double* V, int64_t ldv, const double* Mt,
                 double* egm, cudaStream_t stream) {
    if (T <= 0 || n_v <= 0 || n_e <= 0 || ldv < n_v) return PHS_ERR_BAD_ARG;
    int64_t splits = 1, kchunk = 0;
    contract_plan(T, n_v, n_e, INT64_MAX, &splits, &kchunk);
    double* P = nullptr;
    PHS_CUDA_TRY(dev_alloc((void**)&P, (size_t)splits * T * n_e * sizeof(double), stream));
    cudaError_t e = contract_launch(T, n_v, n_e, V, ldv, Mt, egm, P, splits, kchunk, stream);
    dev_free(P, stream);
    if (e != cudaSuccess) { set_last_error("contract_f64", e); return PHS_ERR_CUDA; }
    return PHS_OK;
}

// Launch the split-K FP64 contraction into caller-provided partials
// P[splits][T][n_e] and reduce them into egm (used by the allocation-free entry
// point in phs_noalloc.cu).  `max_partials` bounds splits * T * n_e.
int contract_f64_into(int64_t T, int64_t n_v, int64_t n_e, const double* V, int64_t ldv, const double* Mt,
                      double* egm, double* P, int64_t max_partials, cudaStream_t stream) {
    if (T <= 0 || n_v <= 0 || n_e <= 0 || ldv < n_v || T * n_e > max_partials) return PHS_ERR_BAD_ARG;
    int64_t splits = 1, kchunk = 0;
    contract_plan(T, n_v, n_e, max_partials, &splits, &kchunk);
    cudaError_t e = contract_launch(T, n_v, n_e, V, ldv, Mt, egm, P, splits, kchunk, stream);
    if (e != cudaSuccess) { set_last_error("contract_f64_into", e); return PHS_ERR_CUDA; }
    return PHS_OK;
}

int normalize(int64_t T, int64_t n_e, void* egm, bool is_f64, cudaStream_t stream) {
    double* ptp = nullptr;
    PHS_CUDA_TRY(dev_alloc((void**)&ptp, (size_t)n_e * sizeof(double), stream));
    const int64_t total = T * n_e;
    const unsigned blocks = (unsigned)std::min<int64_t>((total + 255) / 256, 1184);
    const unsigned cols = (unsigned)((n_e + kPtpCols - 1) / kPtpCols);
    if (is_f64) {
        ptp_kernel<double><<<cols, kPtpCols * kPtpParts, 0, stream>>>(T, n_e, (const double*)egm, ptp);
        scale_kernel<double><<<blocks, 256, 0, stream>>>(total, n_e, ptp, (double*)egm);
    } else {
        ptp_kernel<float><<<cols, kPtpCols * kPtpParts, 0, stream>>>(T, n_e, (const float*)egm, ptp);
        scale_kernel<float><<<blocks, 256, 0, stream>>>(total, n_e, ptp, (float*)egm);
    }
    cudaError_t e = cudaGetLastError();
    dev_free(ptp, stream);
    if (e != cudaSuccess) { set_last_error("normalize", e); return PHS_ERR_CUDA; }
    return PHS_OK;
}

// defined in phs_egm_tc.cu
int contract_bf16x3(int64_t T, int64_t n_e, int64_t T_pad, int64_t n_e_pad, int64_t K_pad,
                    const uint16_t* Vhi, const uint16_t* Vlo, const uint16_t* Mhi, const uint16_t* Mlo,
                    float* egm, void* work, cudaStream_t stream, int config);
int bf16x3_config_count();
int64_t bf16x3_workspace(int64_t T_pad, int64_t n_e_pad, int64_t K_pad);
int bf16x3_status(const void* work, cudaStream_t stream);
int split_bf16(int64_t rows, int64_t cols, const void* src, int64_t ld, bool src_f64, uint16_t* hi,
               uint16_t* lo, int64_t rows_out, int64_t ld_out, cudaStream_t stream);

}  // namespace phs

using namespace phs;

extern "C" {

int phs_egm_leadfield_f64(int64_t n_v, int64_t n_e, const double* voxel_xyz, const double* electrode_xyz,
                          const double* c_voxel, const double* D0, const int32_t* in_ptr, const int32_t* in_src,
                          const int8_t* in_dir, double inv_two_delta, double* Mt, void* stream) {
    if (n_v <= 0 || n_e <= 0 || n_e > 65535 || !voxel_xyz || !electrode_xyz || !c_voxel || !in_ptr || !Mt)
        return PHS_ERR_BAD_ARG;
    const dim3 grid((unsigned)std::min<int64_t>((n_v + 127) / 128, 65535),
                    (unsigned)((n_e + kLfElectrodes - 1) / kLfElectrodes));
    if (D0)
        leadfield_kernel<true><<<grid, 128, 0, (cudaStream_t)stream>>>(n_v, n_e, voxel_xyz, electrode_xyz, c_voxel, D0,
                                                                      in_ptr, in_src, in_dir, inv_two_delta, Mt);
    else
        leadfield_kernel<false><<<grid, 128, 0, (cudaStream_t)stream>>>(n_v, n_e, voxel_xyz, electrode_xyz, c_voxel, D0,
                                                                       in_ptr, in_src, in_dir, inv_two_delta, Mt);
    PHS_CUDA_TRY(cudaGetLastError());
    return PHS_OK;
}

int phs_egm_contract_f64(int64_t T, int64_t n_v, int64_t n_e, const double* V, int64_t ldv, const double* Mt,
                         double* egm, void* stream) {
    if (!V || !Mt || !egm) return PHS_ERR_BAD_ARG;
    return contract_f64(T, n_v, n_e, V, ldv, Mt, egm, (cudaStream_t)stream);
}

int phs_egm_normalize(int64_t T, int64_t n_e, void* egm, int is_f64, void* stream) {
    if (T <= 0 || n_e <= 0 || !egm) return PHS_ERR_BAD_ARG;
    return normalize(T, n_e, egm, is_f64 != 0, (cudaStream_t)stream);
}

int phs_split_bf16(int64_t rows, int64_t cols, const void* src, int64_t ld, int src_is_f64, uint16_t* hi,
                   uint16_t* lo, int64_t rows_out, int64_t ld_out, void* stream) {
    if (rows <= 0 || cols <= 0 || ld < cols || rows_out < rows || ld_out < cols || !src || !hi || !lo)
        return PHS_ERR_BAD_ARG;
    return split_bf16(rows, cols, src, ld, src_is_f64 != 0, hi, lo, rows_out, ld_out, (cudaStream_t)stream);
}

int64_t phs_egm_bf16x3_workspace(int64_t T_pad, int64_t n_e_pad, int64_t K_pad) {
    return bf16x3_workspace(T_pad, n_e_pad, K_pad);
}

int phs_egm_contract_bf16x3(int64_t T, int64_t n_e, int64_t T_pad, int64_t n_e_pad, int64_t K_pad,
                            const uint16_t* Vhi, const uint16_t* Vlo, const uint16_t* Mhi, const uint16_t* Mlo,
                            float* egm, void* work, void* stream) {
    return contract_bf16x3(T, n_e, T_pad, n_e_pad, K_pad, Vhi, Vlo, Mhi, Mlo, egm, work, (cudaStream_t)stream, -1);
}

int phs_egm_contract_bf16x3_cfg(int64_t T, int64_t n_e, int64_t T_pad, int64_t n_e_pad, int64_t K_pad,
                                const uint16_t* Vhi, const uint16_t* Vlo, const uint16_t* Mhi, const uint16_t* Mlo,
                                float* egm, void* work, int config, void* stream) {
    if (config < 0) return PHS_ERR_BAD_ARG;
    return contract_bf16x3(T, n_e, T_pad, n_e_pad, K_pad, Vhi, Vlo, Mhi, Mlo, egm, work, (cudaStream_t)stream,
                           config);
}

int phs_egm_bf16x3_config_count(void) { return bf16x3_config_count(); }

int phs_egm_bf16x3_status(const void* work, void* stream) { return bf16x3_status(work, (cudaStream_t)stream); }

int phs_electrogram(int64_t T, int64_t n_v, int64_t n_e, const double* V, const double* voxel_xyz,
                    const double* electrode_xyz, const double* c_voxel, const double* D0, const int32_t* in_ptr,
                    const int32_t* in_src, const int8_t* in_dir, double delta, int mode, double* egm_out) {
    if (T <= 0 || n_v <= 0 || n_e <= 0 || !V || !voxel_xyz || !electrode_xyz || !c_voxel || !in_ptr ||
        !egm_out || !(delta > 0.0))
        return PHS_ERR_BAD_ARG;
    if (mode != PHS_EGM_F64 && mode != PHS_EGM_BF16X3) return PHS_ERR_BAD_ARG;
    const int32_t nnz = in_ptr[n_v];
    for (int64_t i = 0; i < nnz; ++i)
        if (in_src[i] < 0 || in_src[i] >= n_v || in_dir[i] == 0 || in_dir[i] > 3 || in_dir[i] < -3)
            return PHS_ERR_BAD_TABLE;
    cudaStream_t s = nullptr;
    std::vector<void*> bufs;
    auto alloc = [&](size_t bytes) -> void* {
        void* p = nullptr;
        if (dev_alloc(&p, std::max<size_t>(bytes, 16), s) != cudaSuccess) return nullptr;
        bufs.push_back(p);
        return p;
    };
    auto cleanup = [&](int rc) {
        for (void* p : bufs) dev_free(p, s);
        return rc;
    };
    double* dV = (double*)alloc((size_t)T * n_v * 8);
    double* dxyz = (double*)alloc((size_t)n_v * 24);
    double* dex = (double*)alloc((size_t)n_e * 24);
    double* dc = (double*)alloc((size_t)n_v * 8);
    double* dD = D0 ? (double*)alloc((size_t)n_v * 72) : nullptr;
    int32_t* dptr = (int32_t*)alloc((size_t)(n_v + 1) * 4);
    int32_t* dsrc = (int32_t*)alloc((size_t)nnz * 4);
    int8_t* ddir = (int8_t*)alloc((size_t)nnz);
    double* dMt = (double*)alloc((size_t)n_e * n_v * 8);
    double* degm = (double*)alloc((size_t)T * n_e * 8);
    if (!dV || !dxyz || !dex || !dc || (D0 && !dD) || !dptr || !dsrc || !ddir || !dMt || !degm)
        return cleanup(PHS_ERR_OOM);
    if (cudaMemcpy(dV, V, (size_t)T * n_v * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(dxyz, voxel_xyz, (size_t)n_v * 24, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(dex, electrode_xyz, (size_t)n_e * 24, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(dc, c_voxel, (size_t)n_v * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
        (D0 && cudaMemcpy(dD, D0, (size_t)n_v * 72, cudaMemcpyHostToDevice) != cudaSuccess) ||
        cudaMemcpy(dptr, in_ptr, (size_t)(n_v + 1) * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
        (nnz && cudaMemcpy(dsrc, in_src, (size_t)nnz * 4, cudaMemcpyHostToDevice) != cudaSuccess) ||
        (nnz && cudaMemcpy(ddir, in_dir, (size_t)nnz, cudaMemcpyHostToDevice) != cudaSuccess))
        return cleanup(PHS_ERR_CUDA);
    int rc = phs_egm_leadfield_f64(n_v, n_e, dxyz, dex, dc, dD, dptr, dsrc, ddir, 1.0 / (2.0 * delta), dMt, s);
    if (rc != PHS_OK) return cleanup(rc);
    if (mode == PHS_EGM_F64) {
        rc = contract_f64(T, n_v, n_e, dV, n_v, dMt, degm, s);
        if (rc != PHS_OK) return cleanup(rc);
        rc = normalize(T, n_e, degm, true, s);
    } else {
        const int64_t Tp = (T + 127) / 128 * 128, Ep = (n_e + 255) / 256 * 256, Kp = (n_v + 63) / 64 * 64;
        uint16_t* vh = (uint16_t*)alloc((size_t)Tp * Kp * 2);
        uint16_t* vl = (uint16_t*)alloc((size_t)Tp * Kp * 2);
        uint16_t* mh = (uint16_t*)alloc((size_t)Ep * Kp * 2);
        uint16_t* ml = (uint16_t*)alloc((size_t)Ep * Kp * 2);
        float* e32 = (float*)alloc((size_t)T * n_e * 4);
        void* work = alloc((size_t)std::max<int64_t>(bf16x3_workspace(Tp, Ep, Kp), 16));
        if (!vh || !vl || !mh || !ml || !e32 || !work) return cleanup(PHS_ERR_OOM);
        rc = split_bf16(T, n_v, dV, n_v, true, vh, vl, Tp, Kp, s);
        if (rc == PHS_OK) rc = split_bf16(n_e, n_v, dMt, n_v, true, mh, ml, Ep, Kp, s);
        if (rc == PHS_OK) rc = contract_bf16x3(T, n_e, Tp, Ep, Kp, vh, vl, mh, ml, e32, work, s, -1);
        if (rc == PHS_OK) rc = bf16x3_status(work, s);
        if (rc == PHS_OK) rc = normalize(T, n_e, e32, false, s);
        if (rc == PHS_OK) {
            const int64_t MN = T * n_e;
            // widen to the f64 output buffer
            std::vector<float> h32((size_t)MN);
            if (cudaMemcpy(h32.data(), e32, (size_t)MN * 4, cudaMemcpyDeviceToHost) != cudaSuccess)
                return cleanup(PHS_ERR_CUDA);
            for (int64_t i = 0; i < MN; ++i) egm_out[i] = (double)h32[(size_t)i];
            return cleanup(PHS_OK);
        }
        return cleanup(rc);
    }
    if (rc != PHS_OK) return cleanup(rc);
    cudaError_t ce = cudaMemcpy(egm_out, degm, (size_t)T * n_e * 8, cudaMemcpyDeviceToHost);
    if (ce != cudaSuccess) { set_last_error("phs_electrogram", ce); return cleanup(PHS_ERR_CUDA); }
    return cleanup(PHS_OK);
}

}  // extern "C"

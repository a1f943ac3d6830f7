// Pivoted incomplete Cholesky decomposition of the AO ERI matrix on the GPU,
// FP64 throughout: CholeskyERI::decompose (reference
// src/integrals/cholesky_eri.cc:40-149).
//
// E[(ij)][(kl)] = (ij|kl), composite index ij = i N + j.  Diagonal
// D_ij = (ij|ij); each step takes the first index of the largest D (:155-167),
// stops when it is below the threshold, forms
//   L_new[ij] = (E[ij][p] - sum_k L_k[ij] L_k[p]) / sqrt(D_p)   (:169-203)
// (no division when sqrt(D_p) <= 1e-12), then D -= L_new^2 clamped at 0
// (:108-109).  Products and differences are rounded separately, in the
// reference's order.  The vectors become the context's stored vectors.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "cd_common.cuh"
#include "cd_internal.h"
#include "sm100_ptx.cuh"
#include "../../include/mshqc_ao.h"

namespace mshqc_cd {
namespace {

// first index of the maximum of D (one CTA of 1024 threads)
__global__ void __launch_bounds__(1024) argmax_first_kernel(const double* __restrict__ D, int64_t n,
                                                            int64_t* __restrict__ pivot,
                                                            double* __restrict__ value) {
    __shared__ double sv[1024];
    __shared__ int64_t si[1024];
    double best = -INFINITY;
    int64_t bi = n;
    for (int64_t e = threadIdx.x; e < n; e += 1024)
        if (D[e] > best) {
            best = D[e];
            bi = e;
        }
    sv[threadIdx.x] = best;
    si[threadIdx.x] = bi;
    __syncthreads();
    for (int h = 512; h > 0; h >>= 1) {
        if (threadIdx.x < h) {
            const double v2 = sv[threadIdx.x + h];
            const int64_t i2 = si[threadIdx.x + h];
            if (v2 > sv[threadIdx.x] || (v2 == sv[threadIdx.x] && i2 < si[threadIdx.x])) {
                sv[threadIdx.x] = v2;
                si[threadIdx.x] = i2;
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        *pivot = si[0];
        *value = sv[0];
    }
}

// integral-direct variant: the column (e|p) arrives in out, is reduced in
// place in the order of src/integrals/cholesky_direct.cc:180-186 and divided
// by sqrt(D_p)
__global__ void chol_direct_column_kernel(const double* __restrict__ L, int m, int64_t n2, int64_t p, double Dp,
                                          double* __restrict__ out) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= n2) return;
    double val = out[e];
    for (int k = 0; k < m; ++k) val = __dsub_rn(val, __dmul_rn(L[(int64_t)k * n2 + e], L[(int64_t)k * n2 + p]));
    out[e] = val / sqrt(Dp);
}

// D -= L^2 with the direct variant's clamp: only small negatives (> -1e-10)
// become zero (src/integrals/cholesky_direct.cc:130-134)
__global__ void chol_direct_diag_update_kernel(double* __restrict__ D, const double* __restrict__ Lm, int64_t n2) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= n2) return;
    double d = __dsub_rn(D[e], __dmul_rn(Lm[e], Lm[e]));
    if (d < 0.0 && d > -1e-10) d = 0.0;
    D[e] = d;
}

// ---- the whole decomposition in one kernel -----------------------------------
// Each step needs the largest diagonal of all elements and the pivot's row of
// the vectors so far: a serial chain of steps, bound by latency.  With a launch
// per piece and a host round trip for the pivot a step took 44 us (N = 36);
// here the CTAs (all resident: cooperative launch) own a range of elements
// each, keep its diagonal and the first vectors of it in shared memory, and
// meet once per step: before the meeting every CTA publishes its own largest
// diagonal together with that element's row of the vectors, so whichever CTA
// holds the pivot, the others find everything they need after it.  The
// published copies alternate between two buffers: a CTA writes one again only
// after a meeting that its readers have reached.  N = 36, 180 vectors: 4.3 ms of
// kernels and 180 round trips before, about 5 us a step here.  The order of
// operations per element is that of the reference (see the file's head).
constexpr int CHOL_THREADS = 256, CHOL_PROW = 1024;   // pivot-row values staged at a time

struct CholArgs {
    const double* eri;
    int64_t n2;
    double threshold;
    double* L;
    double* cand_val;       // [2][gridDim.x]
    int64_t* cand_idx;      // [2][gridDim.x]
    double* rows;           // [2][gridDim.x][n2]
    unsigned* arrived;      // zeroed
    int* err;               // zeroed
    int64_t* n_out;
    int ep;                 // elements per CTA
    int ks;                 // vectors kept in shared memory
};

__global__ void __launch_bounds__(CHOL_THREADS) chol_decompose_kernel(CholArgs a) {
    extern __shared__ double csm[];
    double* Ls = csm;                               // [ks][ep]
    double* Ds = Ls + (size_t)a.ks * a.ep;          // [ep]
    double* Lp = Ds + a.ep;                         // [CHOL_PROW]
    __shared__ double wv[CHOL_THREADS / 32];
    __shared__ int64_t wi[CHOL_THREADS / 32];
    __shared__ double sval;
    __shared__ int64_t sidx;
    __shared__ int sstop;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, G = gridDim.x;
    const int64_t n2 = a.n2, e0 = (int64_t)blockIdx.x * a.ep;
    const int ne = (int)max((int64_t)0, min((int64_t)a.ep, n2 - e0));
    // larger value first, then the lower index
    auto better = [](double v, int64_t i, double bv, int64_t bi) { return v > bv || (v == bv && i < bi); };
    auto block_best = [&](double v, int64_t i) {
#pragma unroll
        for (int off = 16; off; off >>= 1) {
            const double ov = __shfl_xor_sync(0xffffffffu, v, off);
            const int64_t oi = __shfl_xor_sync(0xffffffffu, i, off);
            if (better(ov, oi, v, i)) {
                v = ov;
                i = oi;
            }
        }
        if (lane == 0) {
            wv[warp] = v;
            wi[warp] = i;
        }
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < CHOL_THREADS / 32; ++w)
                if (better(wv[w], wi[w], v, i)) {
                    v = wv[w];
                    i = wi[w];
                }
            sval = v;
            sidx = i;
        }
        __syncthreads();
    };
    for (int x = tid; x < ne; x += CHOL_THREADS) Ds[x] = a.eri[(e0 + x) * n2 + e0 + x];
    __syncthreads();
    int64_t m = 0;
    for (; m <= n2; ++m) {
        const int buf = (int)(m & 1);
        // publish this CTA's largest diagonal and that element's row
        double v = -INFINITY;
        int64_t idx = n2;
        for (int x = tid; x < ne; x += CHOL_THREADS)
            if (better(Ds[x], e0 + x, v, idx)) {
                v = Ds[x];
                idx = e0 + x;
            }
        block_best(v, idx);
        if (sidx < n2) {   // (none: no elements, or nothing but NaN, which is never a pivot)
            const int x = (int)(sidx - e0);
            double* row = a.rows + ((int64_t)buf * G + blockIdx.x) * n2;
            for (int64_t k = tid; k < m; k += CHOL_THREADS)
                row[k] = k < a.ks ? Ls[k * a.ep + x] : a.L[k * n2 + e0 + x];
        }
        if (tid == 0) {
            a.cand_val[buf * G + blockIdx.x] = sval;
            a.cand_idx[buf * G + blockIdx.x] = sidx;
        }
        // meet: everything published above is visible to all afterwards
        __threadfence();
        __syncthreads();
        if (tid == 0) {
            sstop = 0;
            atomicAdd(a.arrived, 1u);
            const unsigned target = (unsigned)G * (unsigned)(m + 1);
            const uint64_t t0 = sm100::globaltimer_ns();
            while (true) {
                unsigned seen;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(seen) : "l"(a.arrived) : "memory");
                if ((int)(seen - target) >= 0) break;
                if (sm100::globaltimer_ns() - t0 > 2000000000ull) {
                    atomicExch(a.err, 1);
                    sstop = 1;
                    break;
                }
            }
        }
        __syncthreads();
        if (sstop) return;
        // the pivot: every CTA finds it for itself
        v = -INFINITY;
        idx = n2;
        for (int g = tid; g < G; g += CHOL_THREADS) {
            const double cv = __ldcg(a.cand_val + buf * G + g);
            const int64_t ci = __ldcg(a.cand_idx + buf * G + g);
            if (better(cv, ci, v, idx)) {
                v = cv;
                idx = ci;
            }
        }
        block_best(v, idx);
        const double Dp = sval;
        const int64_t p = sidx;
        if (m == n2 || Dp < a.threshold) break;
        const double* prow = a.rows + ((int64_t)buf * G + p / a.ep) * n2;
        const double nf = sqrt(Dp);
        double* out = a.L + m * n2 + e0;
        for (int x0 = 0; x0 < a.ep; x0 += CHOL_THREADS) {
            const int x = x0 + tid;
            const bool live = x < ne;
            double val = live ? a.eri[(e0 + x) * n2 + p] : 0.0;
            for (int64_t k0 = 0; k0 < m; k0 += CHOL_PROW) {
                const int nk = (int)min((int64_t)CHOL_PROW, m - k0);
                for (int k = tid; k < nk; k += CHOL_THREADS) Lp[k] = __ldcg(prow + k0 + k);
                __syncthreads();
                if (live) {
                    int k = 0;
                    const int nsm = (int)max((int64_t)0, min((int64_t)nk, (int64_t)a.ks - k0));
                    const double* l = Ls + k0 * a.ep + x;
#pragma unroll 8
                    for (; k < nsm; ++k) val = __dsub_rn(val, __dmul_rn(l[(size_t)k * a.ep], Lp[k]));
                    const double* lg = a.L + k0 * n2 + e0 + x;
#pragma unroll 16
                    for (; k < nk; ++k) val = __dsub_rn(val, __dmul_rn(lg[k * n2], Lp[k]));
                }
                __syncthreads();
            }
            if (live) {
                const double l = nf > 1e-12 ? val / nf : val;
                out[x] = l;
                if (m < a.ks) Ls[m * a.ep + x] = l;
                const double d = __dsub_rn(Ds[x], __dmul_rn(l, l));
                Ds[x] = d < 0.0 ? 0.0 : d;
            }
        }
        __syncthreads();
    }
    if (blockIdx.x == 0 && tid == 0) *a.n_out = m;
}

}  // namespace
}  // namespace mshqc_cd

using namespace mshqc_cd;

extern "C" MSHQC_CD_API int mshqc_cd_cholesky_decompose(mshqc_cd_ctx* ctx, const double* eri, int64_t nbf,
                                                        double threshold, double* L_out, int64_t max_vectors,
                                                        int64_t* n_vectors, int* converged, int where) {
    if (!ctx) return set_error(MSHQC_CD_ERR_ARG, "null context");
    if (!eri || !n_vectors) return set_error(MSHQC_CD_ERR_ARG, "eri and n_vectors must be non-null");
    if (nbf <= 0) return set_error(MSHQC_CD_ERR_ARG, "nbf must be positive");
    if (!(threshold > 0.0)) return set_error(MSHQC_CD_ERR_ARG, "threshold must be positive");
    if (where != MSHQC_CD_HOST && where != MSHQC_CD_DEVICE)
        return set_error(MSHQC_CD_ERR_ARG, "unknown pointer location");
    DeviceGuard g(ctx->device);
    const int64_t n2 = nbf * nbf;
    ctx->invalidate_all();
    ctx->L_set = false;
    ctx->L_gen = false;
    CD_ALLOC(ctx->scratch, sizeof(double) * (size_t)(n2 * n2), false);
    double* dE = ctx->scratch.as<double>();
    if (where == MSHQC_CD_HOST) {
        CD_RC(upload(ctx, dE, eri, sizeof(double) * (size_t)(n2 * n2)));
    } else {
        CD_CUDA(cudaMemcpyAsync(dE, eri, sizeof(double) * (size_t)(n2 * n2), cudaMemcpyDeviceToDevice,
                                ctx->stream));
    }
    CD_RC(check_finite_device(ctx, dE, n2 * n2, "eri"));
    CD_ALLOC(ctx->L, sizeof(double) * (size_t)(n2 * n2), false);   // at most n^2 vectors
    double* L = ctx->L.as<double>();
    // elements per CTA: as few as fill the GPU, at least 32 (a warp)
    CholArgs k{};
    k.ep = (int)std::max<int64_t>(32, cdiv(n2, ctx->num_sms));
    const int G = (int)cdiv(n2, k.ep);
    const size_t smem_max = 200 * 1024;
    const size_t fixed = sizeof(double) * (size_t)(k.ep + CHOL_PROW);
    if (fixed > smem_max)
        return set_error(MSHQC_CD_ERR_UNSUPPORTED, "basis too large for the decomposition kernel");
    k.ks = (int)std::min<int64_t>(n2, (int64_t)((smem_max - fixed) / (sizeof(double) * k.ep)));
    const size_t smem = fixed + sizeof(double) * (size_t)k.ks * k.ep;
    // published candidates and rows, counters
    CD_ALLOC(ctx->partial, sizeof(double) * (size_t)(2 * G * n2 + 4 * G + 3), false);
    k.rows = ctx->partial.as<double>();
    k.cand_val = k.rows + 2 * (int64_t)G * n2;
    k.cand_idx = reinterpret_cast<int64_t*>(k.cand_val + 2 * G);
    k.n_out = k.cand_idx + 2 * G;
    k.arrived = reinterpret_cast<unsigned*>(k.n_out + 1);
    k.err = reinterpret_cast<int*>(k.n_out + 2);
    k.eri = dE;
    k.n2 = n2;
    k.threshold = threshold;
    k.L = L;
    CD_CUDA(cudaMemsetAsync(k.n_out, 0, 3 * sizeof(int64_t), ctx->stream));
    CD_CUDA(cudaFuncSetAttribute(chol_decompose_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    void* args[] = {&k};
    CD_CUDA(cudaLaunchCooperativeKernel((const void*)chol_decompose_kernel, dim3((unsigned)G), dim3(CHOL_THREADS), args,
                                        smem, ctx->stream));
    ctx->launches++;
    int64_t h[3];
    CD_CUDA(cudaMemcpyAsync(h, k.n_out, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
    CD_CUDA(cudaStreamSynchronize(ctx->stream));
    if ((int)h[2]) return set_error(MSHQC_CD_ERR_TIMEOUT, "decomposition kernel gave up waiting");
    const int64_t m = h[0];
    *n_vectors = m;
    if (converged) *converged = m < n2 ? 1 : 0;
    if (L_out) {
        if (m > max_vectors)
            return set_error(MSHQC_CD_ERR_ARG, "L_out holds " + std::to_string(max_vectors) + " vectors, " +
                                                   std::to_string(m) + " were produced");
        CD_RC(download(ctx, L_out, L, sizeof(double) * (size_t)(m * n2), where));
    }
    ctx->N = nbf;
    ctx->M = m;
    ctx->Mp = round_up(std::max<int64_t>(m, 1), 16);
    ctx->L_set = m > 0;
    CD_CUDA(cudaStreamSynchronize(ctx->stream));
    return MSHQC_CD_OK;
}

// Integral-direct pivoted Cholesky (reference src/integrals/cholesky_direct.cc:
// 32-187, DirectCholesky::compute): the ERI diagonal and, per vector, the one
// ERI column of the pivot come from the host AO engine (mshqc_ao_*), the
// pivot search, the column reduction and the diagonal update run on the
// device.  Stops when the largest diagonal is below the threshold or
// negative, or after N^2 / 2 vectors, as the reference does.
extern "C" MSHQC_CD_API int mshqc_cd_cholesky_direct(mshqc_cd_ctx* ctx, const mshqc_ao_basis* basis,
                                                     double threshold, double* L_out, int64_t max_vectors,
                                                     int64_t* n_vectors, int* converged, int where) {
    if (!ctx) return set_error(MSHQC_CD_ERR_ARG, "null context");
    if (!basis || !n_vectors) return set_error(MSHQC_CD_ERR_ARG, "basis and n_vectors must be non-null");
    if (!(threshold > 0.0)) return set_error(MSHQC_CD_ERR_ARG, "threshold must be positive");
    if (where != MSHQC_CD_HOST && where != MSHQC_CD_DEVICE)
        return set_error(MSHQC_CD_ERR_ARG, "unknown pointer location");
    int64_t nbf = 0;
    if (mshqc_ao_nbf(basis, &nbf) != MSHQC_AO_OK)
        return set_error(MSHQC_CD_ERR_ARG, std::string("basis: ") + mshqc_ao_last_error());
    DeviceGuard g(ctx->device);
    const int64_t n2 = nbf * nbf, vmax = n2 / 2 + 1;
    ctx->invalidate_all();
    ctx->L_set = false;
    ctx->L_gen = false;
    std::vector<double> hcol((size_t)n2);
    if (mshqc_ao_eri_diagonal(basis, hcol.data()) != MSHQC_AO_OK)
        return set_error(MSHQC_CD_ERR_ARG, std::string("ERI diagonal: ") + mshqc_ao_last_error());
    CD_ALLOC(ctx->scratch, sizeof(double) * (size_t)(n2 + 2), false);
    double* D = ctx->scratch.as<double>();
    double* pv = D + n2;
    CD_RC(upload(ctx, D, hcol.data(), sizeof(double) * (size_t)n2));
    CD_ALLOC(ctx->L, sizeof(double) * (size_t)(vmax * n2), false);
    double* L = ctx->L.as<double>();
    const unsigned blocks = (unsigned)cdiv(n2, 256);
    int64_t m = 0;
    bool conv = false;
    for (; m < vmax; ++m) {
        argmax_first_kernel<<<1, 1024, 0, ctx->stream>>>(D, n2, reinterpret_cast<int64_t*>(pv), pv + 1);
        CD_CUDA(cudaGetLastError());
        struct {
            int64_t p;
            double v;
        } h;
        CD_CUDA(cudaMemcpyAsync(&h, pv, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
        CD_CUDA(cudaStreamSynchronize(ctx->stream));
        if (h.v < threshold) {   // also a negative largest diagonal
            conv = h.v >= -1e-10;
            break;
        }
        if (mshqc_ao_eri_column(basis, h.p, hcol.data()) != MSHQC_AO_OK)
            return set_error(MSHQC_CD_ERR_ARG, std::string("ERI column: ") + mshqc_ao_last_error());
        CD_RC(upload(ctx, L + m * n2, hcol.data(), sizeof(double) * (size_t)n2));
        chol_direct_column_kernel<<<blocks, 256, 0, ctx->stream>>>(L, (int)m, n2, h.p, h.v, L + m * n2);
        chol_direct_diag_update_kernel<<<blocks, 256, 0, ctx->stream>>>(D, L + m * n2, n2);
        CD_CUDA(cudaGetLastError());
        ctx->launches += 3;
    }
    *n_vectors = m;
    if (converged) *converged = conv ? 1 : 0;
    if (L_out) {
        if (m > max_vectors)
            return set_error(MSHQC_CD_ERR_ARG, "L_out holds " + std::to_string(max_vectors) + " vectors, " +
                                                   std::to_string(m) + " were produced");
        CD_RC(download(ctx, L_out, L, sizeof(double) * (size_t)(m * n2), where));
    }
    ctx->N = nbf;
    ctx->M = m;
    ctx->Mp = round_up(std::max<int64_t>(m, 1), 16);
    ctx->L_set = m > 0;
    CD_CUDA(cudaStreamSynchronize(ctx->stream));
    return MSHQC_CD_OK;
}

// Batched FP64 GEMM on the FP64 tensor pipe (DMMA m8n8k4), sm_100a.
//
//   C(m, n) = alpha * sum_{h < kb} sum_k A_h(m, k) B_h(k, n) + beta * C(m, n)   per batch b
//
// A_h(m,k) lives at A + b*sA + h*skA + (A_K ? m*lda + k : k*lda + m)   (A_K: K contiguous)
// B_h(k,n) lives at B + b*sB + h*skB + (B_K ? n*ldb + k : k*ldb + n)   (B_K: K contiguous)
// C(m,n)   lives at C + b*sC + m*ldc + n
//
// T x T CTA tile (64, or 32 for small products), K step 16, 4 warps (2 x 2),
// three-stage cp.async ring with one barrier per K step.  Shared tiles keep
// the global orientation; the padded strides (20 for [row][k], T + 4 for
// [k][row]) make the 8-byte fragment reads of each half warp hit 16 distinct
// bank pairs.  Warps skip the 8-row fragments that lie outside the matrix,
// and odd CTAs swap the two warp rows, so that a product with few rows (the
// occupied orbitals) loads the four tensor pipes of an SM alike.
//
// Bound: the FP64 tensor pipe (37.0 TF/s, register-resident DMMAs).  One K
// step of a 64 x 64 tile is 970 cycles of it, so a product of few tiles and a
// long K leaves most SMs idle: gemm_run then splits the composite K range
// (h, k) over CTAs and adds the partials in a fixed order.
#pragma once

#include <algorithm>

#include "cd_common.cuh"
#include "cd_internal.h"

namespace mshqc_cd {

struct GemmF64Args {
    int M, N, K, batch;
    const double* A;
    int64_t lda, sA;
    const double* B;
    int64_t ldb, sB;
    double* C;
    int64_t ldc, sC;
    double alpha, beta;
    int kb;             // K batches (0 counts as 1)
    int64_t skA, skB;
    // tri > 0: rows and columns come in groups of tri (a multiple of 64), and
    // tiles of a column group before their row group are left out
    int tri;
    // sym != 0: A and B describe the same matrix; the tiles below the diagonal
    // are mirrored instead of computed (the launcher sets 2 when the kernel
    // itself writes the mirror images, 1 when the reduction of the splits does)
    int sym;
    // set by the launcher
    int S, per;         // K splits, K steps per split
};

namespace gemm_detail {
constexpr int BK = 16;
constexpr int STAGES = 3;
constexpr int SK = BK + 4;      // stride of a [row][k] tile
template <int T>
constexpr int tile_doubles() {  // doubles per operand per stage
    return T * SK > BK * (T + 4) ? T * SK : BK * (T + 4);
}
template <int T>
constexpr size_t smem_bytes() {
    return sizeof(double) * 2 * STAGES * tile_doubles<T>();
}

// One thread's share of an operand tile per K step: NC copies of VEC doubles.
//   KC = true : element (r, k) at base + r*ld + k  -> smem [r][k] (stride SK)
//   KC = false: element (r, k) at base + k*ld + r  -> smem [k][r] (stride T + 4)
// Rows, strides and validity of a thread's copies do not change between K
// steps, so a step costs one add per copy; a partial last step of a K batch
// takes the checked path.  (With every address and bound formed per copy the
// four warps of a CTA spent a third of a K step on it.)
template <bool KC, int VEC, int T>
struct TileLoader {
    static constexpr int CPR = KC ? BK / VEC : T / VEC;     // copies per tile line
    static constexpr int LPI = 128 / CPR;                   // lines per iteration of the 128 threads
    static constexpr int NC = (KC ? T : BK) / LPI;
    static constexpr int STRIDE = KC ? SK : T + 4;
    const double* ptr;      // source of copy 0 of the next step
    int64_t iline;          // between this thread's copies
    int64_t kadv;           // from one K step to the next
    uint32_t dst;           // shared address of copy 0 in stage 0
    uint32_t live;          // bit i: copy i has valid rows (KC); non-KC: bytes valid in every copy
    int line0, off;         // this thread's first line, element offset inside a line

    __device__ __forceinline__ void init(double* sm, int64_t ld, int r0, int nrows, int tid) {
        line0 = tid / CPR;
        off = (tid % CPR) * VEC;
        dst = smem_u32(sm + line0 * STRIDE + off);
        iline = (int64_t)LPI * ld;
        kadv = KC ? BK : (int64_t)BK * ld;
        if (KC) {
            live = 0;
#pragma unroll
            for (int i = 0; i < NC; ++i) live |= (r0 + line0 + i * LPI < nrows ? 1u : 0u) << i;
        } else {
            live = (uint32_t)max(0, min(VEC, nrows - (r0 + off))) * 8u;
        }
    }
    // source at K offset k0 of the K batch that starts at base
    __device__ __forceinline__ void seek(const double* base, int64_t ld, int r0, int k0) {
        ptr = KC ? base + (int64_t)(r0 + line0) * ld + k0 + off : base + (int64_t)(k0 + line0) * ld + r0 + off;
    }
    __device__ __forceinline__ void copy(uint32_t d, const double* src, int bytes) const {
        if constexpr (VEC == 2)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes));
        else
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(bytes));
    }
    // copies of one step into the stage at byte offset so; krem: valid K left
    // from this step's offset on; safe: any valid address (nothing is read
    // through it when no byte of a copy is valid)
    __device__ __forceinline__ void step(uint32_t so, int krem, const double* safe) {
        const uint32_t d = dst + so;
        if (krem >= BK) {
#pragma unroll
            for (int i = 0; i < NC; ++i) {
                const int bytes = KC ? (((live >> i) & 1u) ? VEC * 8 : 0) : (int)live;
                copy(d + i * (LPI * STRIDE * 8), bytes ? ptr + i * iline : safe, bytes);
            }
        } else {
#pragma unroll
            for (int i = 0; i < NC; ++i) {
                int bytes;
                if (KC)
                    bytes = ((live >> i) & 1u) ? max(0, min(VEC, krem - off)) * 8 : 0;
                else
                    bytes = line0 + i * LPI < krem ? (int)live : 0;
                copy(d + i * (LPI * STRIDE * 8), bytes ? ptr + i * iline : safe, bytes);
            }
        }
        ptr += kadv;
    }
};

template <bool KC, int T>
__device__ __forceinline__ double frag(const double* sm, int r, int k) {
    return KC ? sm[r * SK + k] : sm[k * (T + 4) + r];
}
}  // namespace gemm_detail

// One T x T tile of the product: rows m0.., columns n0.., batch b, K split `split`;
// swap: the warp rows change places
template <bool A_K, bool B_K, int VEC, int T>
__device__ __forceinline__ void gemm_tile(const GemmF64Args& p, int m0, int n0, int64_t b, int split, int swap) {
    using namespace gemm_detail;
    constexpr int TD = tile_doubles<T>();
    constexpr int WT = T / 2, NF = WT / 8;   // rows / columns per warp, 8-wide fragments
    extern __shared__ __align__(16) double gemm_smem[];
    double* smA = gemm_smem;
    double* smB = gemm_smem + STAGES * TD;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = (warp >> 1) ^ swap, wn = warp & 1;
    const double* A = p.A + b * p.sA;
    const double* B = p.B + b * p.sB;

    // this CTA's K steps: step t is K offset (t % nkb) * BK of K batch t / nkb
    const int nkb = (p.K + BK - 1) / BK;
    const int t0 = split * p.per, t1 = min(nkb * p.kb, t0 + p.per);
    const int nt = t1 - t0;
    int lh = t0 / nkb, lk = t0 % nkb;        // load cursor
    TileLoader<A_K, VEC, T> la;
    TileLoader<B_K, VEC, T> lb;
    la.init(smA, p.lda, m0, p.M, tid);
    lb.init(smB, p.ldb, n0, p.N, tid);
    la.seek(A + lh * p.skA, p.lda, m0, lk * BK);
    lb.seek(B + lh * p.skB, p.ldb, n0, lk * BK);
    auto load = [&](int stage) {
        const uint32_t so = (uint32_t)(stage * TD * 8);
        const int krem = p.K - lk * BK;
        la.step(so, krem, A);
        lb.step(so, krem, B);
        if (++lk == nkb) {
            lk = 0;
            ++lh;
            la.seek(A + lh * p.skA, p.lda, m0, 0);
            lb.seek(B + lh * p.skB, p.ldb, n0, 0);
        }
    };

    double acc[NF][NF][2];
#pragma unroll
    for (int i = 0; i < NF; ++i)
#pragma unroll
        for (int j = 0; j < NF; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    // fragments of this warp that hold rows / columns of the matrix
    const int fm = min(NF, max(0, (p.M - (m0 + wm * WT) + 7) / 8));
    const int fn = min(NF, max(0, (p.N - (n0 + wn * WT) + 7) / 8));

    int pre = 0;
#pragma unroll
    for (; pre < STAGES - 1; ++pre) {
        if (pre < nt) load(pre);
        cp_async_commit();
    }
    int stage = 0;
    for (int t = 0; t < nt; ++t) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();
        // the slot read in the previous step is free for step t + STAGES - 1
        if (t + STAGES - 1 < nt) load(stage == 0 ? STAGES - 1 : stage - 1);
        cp_async_commit();
        const double* sa = smA + stage * TD;
        const double* sb = smB + stage * TD;
        // fragments of 4 K at a time, the next ones loaded ahead of the DMMAs
        // of the current ones
        double af[2][NF], bf[2][NF];
        auto frags = [&](int h, int kk) {
#pragma unroll
            for (int i = 0; i < NF; ++i)
                af[h][i] = frag<A_K, T>(sa, wm * WT + i * 8 + (lane >> 2), kk + (lane & 3));
#pragma unroll
            for (int j = 0; j < NF; ++j)
                bf[h][j] = frag<B_K, T>(sb, wn * WT + j * 8 + (lane >> 2), kk + (lane & 3));
        };
        frags(0, 0);
        if (fm == NF && fn == NF) {
#pragma unroll
            for (int kk = 0; kk < BK; kk += 4) {
                const int h = (kk >> 2) & 1;
                if (kk + 4 < BK) frags(h ^ 1, kk + 4);
#pragma unroll
                for (int i = 0; i < NF; ++i)
#pragma unroll
                    for (int j = 0; j < NF; ++j) dmma_8x8x4(acc[i][j][0], acc[i][j][1], af[h][i], bf[h][j]);
            }
        } else {
#pragma unroll
            for (int kk = 0; kk < BK; kk += 4) {
                const int h = (kk >> 2) & 1;
                if (kk + 4 < BK) frags(h ^ 1, kk + 4);
#pragma unroll
                for (int i = 0; i < NF; ++i) {
                    if (i < fm) {
#pragma unroll
                        for (int j = 0; j < NF; ++j)
                            if (j < fn) dmma_8x8x4(acc[i][j][0], acc[i][j][1], af[h][i], bf[h][j]);
                    }
                }
            }
        }
        if (++stage == STAGES) stage = 0;
    }

    double* C = p.C + b * p.sC + (int64_t)split * p.M * p.ldc;   // split > 0: partial products only
#pragma unroll
    for (int i = 0; i < NF; ++i) {
        const int m = m0 + wm * WT + i * 8 + (lane >> 2);
        if (m >= p.M) continue;
#pragma unroll
        for (int j = 0; j < NF; ++j) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int n = n0 + wn * WT + j * 8 + 2 * (lane & 3) + e;
                if (n >= p.N) continue;
                double* cp = C + (int64_t)m * p.ldc + n;
                const double w = p.alpha * acc[i][j][e];
                double v = w;
                if (p.beta != 0.0) v += p.beta * (*cp);
                *cp = v;
                if (p.sym == 2 && m0 != n0) {   // 8 lanes write 64 contiguous bytes
                    cp = C + (int64_t)n * p.ldc + m;
                    v = w;
                    if (p.beta != 0.0) v += p.beta * (*cp);
                    *cp = v;
                }
            }
        }
    }
}

template <bool A_K, bool B_K, int VEC, int T>
__global__ void __launch_bounds__(128, T == 64 ? 3 : 6) gemm_f64_kernel(GemmF64Args p) {
    const int m0 = blockIdx.y * T, n0 = blockIdx.x * T;
    if (p.tri > 0 && n0 / p.tri < m0 / p.tri) return;
    if (p.sym && n0 < m0) return;
    gemm_tile<A_K, B_K, VEC, T>(p, m0, n0, blockIdx.z / p.S, (int)(blockIdx.z % p.S), (int)(blockIdx.x & 1));
}

// Tiles of a product that are done here after all: unit u of `list` (count of
// them) is batch b, row block mb (128) and column block nb (64) of the sliced
// product (ozaki_i8.cuh); trans: its rows are the columns here.
struct GemmListed {
    const int* count;
    const int* list;
    int nmb, nnb, group;
    int trans;
};
template <bool A_K, bool B_K, int VEC>
__global__ void __launch_bounds__(128, 3) gemm_f64_listed_kernel(GemmF64Args p, GemmListed l) {
    const int halves = 2 * *l.count;
    for (int t = blockIdx.x; t < halves; t += gridDim.x) {
        long long b;
        int mb, nb;
        tile_of_unit(l.list[t >> 1], l.nmb, l.nnb, l.group, b, mb, nb);
        const int r0 = mb * 128 + (t & 1) * 64, c0 = nb * 64;
        const int m0 = l.trans ? c0 : r0, n0 = l.trans ? r0 : c0;
        if (m0 >= p.M || n0 >= p.N) continue;
        gemm_tile<A_K, B_K, VEC, 64>(p, m0, n0, b, 0, t & 1);
        __syncthreads();   // the next tile loads into the stages read here
    }
}

// C = alpha * (sum of S partials, in a fixed order) + beta * C; partial s of
// batch b is the M x N matrix at ws + (b * S + s) * M * N.  64 elements x 4
// partial lanes per CTA.  symT > 0: only the tiles on and above the diagonal
// (edge symT) were computed, the others are their mirror images.
static __global__ void __launch_bounds__(256) gemm_reduce_kernel(const double* __restrict__ ws, int S, int M, int N,
                                                                 double alpha, double beta, double* __restrict__ C,
                                                                 int64_t ldc, int64_t sC, int symT) {
    __shared__ double red[4][64];
    const int64_t MN = (int64_t)M * N;
    const int64_t e = blockIdx.x * 64LL + (threadIdx.x & 63);
    const int g = threadIdx.x >> 6;
    const int64_t m = e / N, n = e % N;
    double s0 = 0.0, s1 = 0.0;
    if (e < MN) {
        const int64_t src = (symT > 0 && n / symT < m / symT) ? n * N + m : e;
        const double* w = ws + (int64_t)blockIdx.y * S * MN + src;
        int s = g;
        for (; s + 4 < S; s += 8) {
            s0 += w[(int64_t)s * MN];
            s1 += w[(int64_t)(s + 4) * MN];
        }
        if (s < S) s0 += w[(int64_t)s * MN];
    }
    red[g][threadIdx.x & 63] = s0 + s1;
    __syncthreads();
    if (g == 0 && e < MN) {
        const int t = threadIdx.x;
        double* c = C + blockIdx.y * sC + m * ldc + n;
        double v = alpha * ((red[0][t] + red[1][t]) + (red[2][t] + red[3][t]));
        if (beta != 0.0) v += beta * (*c);
        *c = v;
    }
}

template <bool A_K, bool B_K, int VEC, int T>
inline cudaError_t gemm_f64_launch(const GemmF64Args& a, cudaStream_t st) {
    constexpr size_t smem = gemm_detail::smem_bytes<T>();
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f64_kernel<A_K, B_K, VEC, T>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    dim3 grid((unsigned)cdiv(a.N, T), (unsigned)cdiv(a.M, T), (unsigned)(a.batch * a.S));
    gemm_f64_kernel<A_K, B_K, VEC, T><<<grid, 128, smem, st>>>(a);
    return cudaGetLastError();
}

// every operand row is 16-byte aligned
inline bool gemm_aligned16(const GemmF64Args& a) {
    auto al16 = [](const void* ptr, int64_t ld, int64_t s, int64_t sk) {
        return (reinterpret_cast<uintptr_t>(ptr) % 16 == 0) && (ld % 2 == 0) && (s % 2 == 0) && (sk % 2 == 0);
    };
    return al16(a.A, a.lda, a.sA, a.skA) && al16(a.B, a.ldb, a.sB, a.skB);
}

// One kernel with the tile T and the K splits a.S x a.per already chosen;
// picks 16-byte copies when every operand row is 16-byte aligned.
template <int T>
inline cudaError_t gemm_f64_tiled(const GemmF64Args& a, bool a_k, bool b_k, cudaStream_t st) {
    const bool v16 = gemm_aligned16(a);
    if (a_k && b_k) return v16 ? gemm_f64_launch<true, true, 2, T>(a, st) : gemm_f64_launch<true, true, 1, T>(a, st);
    if (a_k) return v16 ? gemm_f64_launch<true, false, 2, T>(a, st) : gemm_f64_launch<true, false, 1, T>(a, st);
    if (b_k) return v16 ? gemm_f64_launch<false, true, 2, T>(a, st) : gemm_f64_launch<false, true, 1, T>(a, st);
    return v16 ? gemm_f64_launch<false, false, 2, T>(a, st) : gemm_f64_launch<false, false, 1, T>(a, st);
}

// The listed tiles of a product (a.S = 1, a.per = all K steps): as many CTAs as
// fit, which leave at once when the list is empty (about 3 us).
template <bool A_K, bool B_K, int VEC>
inline cudaError_t gemm_f64_listed_launch(const GemmF64Args& a, const GemmListed& l, int num_sms, cudaStream_t st) {
    constexpr size_t smem = gemm_detail::smem_bytes<64>();
    cudaError_t e = cudaFuncSetAttribute(gemm_f64_listed_kernel<A_K, B_K, VEC>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    gemm_f64_listed_kernel<A_K, B_K, VEC><<<3 * num_sms, 128, smem, st>>>(a, l);
    return cudaGetLastError();
}
inline cudaError_t gemm_f64_listed(GemmF64Args a, bool a_k, bool b_k, const GemmListed& l, int num_sms,
                                   cudaStream_t st) {
    a.kb = 1;
    a.S = 1;
    a.per = (int)cdiv(a.K, gemm_detail::BK);
    const bool v16 = gemm_aligned16(a);
    if (a_k && b_k)
        return v16 ? gemm_f64_listed_launch<true, true, 2>(a, l, num_sms, st)
                   : gemm_f64_listed_launch<true, true, 1>(a, l, num_sms, st);
    if (a_k)
        return v16 ? gemm_f64_listed_launch<true, false, 2>(a, l, num_sms, st)
                   : gemm_f64_listed_launch<true, false, 1>(a, l, num_sms, st);
    if (b_k)
        return v16 ? gemm_f64_listed_launch<false, true, 2>(a, l, num_sms, st)
                   : gemm_f64_listed_launch<false, true, 1>(a, l, num_sms, st);
    return v16 ? gemm_f64_listed_launch<false, false, 2>(a, l, num_sms, st)
               : gemm_f64_listed_launch<false, false, 1>(a, l, num_sms, st);
}

// The product with the tile and the K split chosen by shape, on the context's
// stream; split partials go to ctx->gemm_ws.
//  * 32 x 32 tiles where a side is at most 32, where they pad less than 64 x 64
//    tiles (which run at 35.1 of the pipe's 37.0 TF/s, 32 x 32 at 32.5: 8192 x
//    8192 x 2400), and where 64 x 64 tiles would leave SMs idle and K is too
//    short to split (a K step of a 32 x 32 tile is 243 cycles of the tensor
//    pipe against 970).
//  * K is split when the tiles do not fill the resident CTAs (3 per SM with
//    64 x 64 tiles, 6 with 32 x 32) and each split keeps at least 8 (16) K
//    steps: fewer are not worth the reduction's launch.  A split product takes
//    at most 256 K steps per partial while the partials stay small, which
//    bounds the length of the rounding chain of one accumulator.
inline int gemm_run(mshqc_cd_ctx* ctx, GemmF64Args a, bool a_k, bool b_k) {
    using namespace gemm_detail;
    if (a.M <= 0 || a.N <= 0 || a.batch <= 0) return MSHQC_CD_OK;
    if (a.kb <= 0) a.kb = 1;
    const int64_t steps = cdiv(a.K, BK) * a.kb;
    auto tiles = [&](int T) { return cdiv(a.M, T) * cdiv(a.N, T) * a.batch; };
    const int64_t sms = ctx->num_sms;
    const bool small = a.tri == 0 && (a.M <= 32 || a.N <= 32 || (tiles(64) < sms && steps < 16) ||
                                      1.06 * 1024.0 * tiles(32) < 4096.0 * tiles(64));
    const int T = small ? 32 : 64;
    const int64_t slots = (small ? 6 : 3) * sms, min_steps = small ? 16 : 8;
    const int64_t nt = a.sym ? (tiles(T) + cdiv(a.M, T) * a.batch) / 2 : tiles(T);
    const int64_t MN = (int64_t)a.M * a.N;
    int64_t S = std::max<int64_t>(1, std::min<int64_t>(slots / std::max<int64_t>(nt, 1), steps / min_steps));
    if (S > 1 && steps / S > 256)
        S = std::max(S, std::min<int64_t>(cdiv(steps, 256), (int64_t(1) << 25) / (MN * a.batch)));
    S = std::max<int64_t>(1, std::min<int64_t>(S, 65535 / a.batch));
    a.per = (int)std::max<int64_t>(1, cdiv(steps, S));
    a.S = (int)std::max<int64_t>(1, cdiv(steps, a.per));
    if (a.S > 1) {
        const size_t bytes = sizeof(double) * (size_t)(MN * a.S * a.batch);
        cudaError_t e = ctx->gemm_ws.reserve(bytes, false, ctx->stream);
        if (e == cudaErrorMemoryAllocation && ctx->release_slices()) e = ctx->gemm_ws.reserve(bytes, false, ctx->stream);
        if (e == cudaErrorMemoryAllocation) {   // no room for the partials: no split
            a.S = 1;
            a.per = (int)steps;
        } else {
            CD_CUDA(e);
        }
    }
    if (a.S == 1) {
        if (a.sym) a.sym = 2;
        CD_CUDA(T == 32 ? gemm_f64_tiled<32>(a, a_k, b_k, ctx->stream) : gemm_f64_tiled<64>(a, a_k, b_k, ctx->stream));
        ctx->launches++;
        return MSHQC_CD_OK;
    }
    GemmF64Args w = a;
    w.C = ctx->gemm_ws.as<double>();
    w.ldc = a.N;
    w.sC = MN * a.S;
    w.alpha = 1.0;
    w.beta = 0.0;
    w.sym = a.sym ? 1 : 0;
    CD_CUDA(T == 32 ? gemm_f64_tiled<32>(w, a_k, b_k, ctx->stream) : gemm_f64_tiled<64>(w, a_k, b_k, ctx->stream));
    dim3 grid((unsigned)cdiv(MN, 64), (unsigned)a.batch);
    gemm_reduce_kernel<<<grid, 256, 0, ctx->stream>>>(ctx->gemm_ws.as<double>(), a.S, a.M, a.N, a.alpha, a.beta, a.C,
                                                      a.ldc, a.sC, a.sym ? T : 0);
    CD_CUDA(cudaGetLastError());
    ctx->launches += 2;
    return MSHQC_CD_OK;
}

}  // namespace mshqc_cd

// Orchestration of the Cholesky-MP2 kernels: half transforms, pair energies,
// reductions.  Called from the C ABI (cd_abi.cu) with the device selected.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "cd_common.cuh"
#include "cd_internal.h"
#include "gemm_f64.cuh"
#include "pair_energy_f64.cuh"
#include "pair_energy_s.cuh"
#include "pair_energy_tc.cuh"
#include "split_bf16.cuh"
#include "gamma_tc.cuh"
#include "vtile_tc.cuh"
#include "amp_elem.cuh"
#include "ozaki_i8.cuh"
#include "slice_guard.cuh"

namespace mshqc_cd {


namespace {

// Partitioned backward: whether the next unit (block pair, or occupied block
// of an FP64 pass) belongs to this context's share.  Units beyond the plan
// (which a mismatch between plan_partition and the passes would produce)
// belong to nobody; run_gradient checks the count afterwards.
bool owns_next(mshqc_cd_ctx* ctx) {
    const int64_t k = ctx->part_next++;
    if (!ctx->part_active) return true;
    return k < (int64_t)ctx->part_owned.size() && ctx->part_owned[(size_t)k] != 0;
}

// ---------------------------------------------------------------------------
// occupied block sizes of the backward passes
// ---------------------------------------------------------------------------
// Unpartitioned, a block is as large as a share of the free device memory
// allows (fewer, larger launches).  Partitioned, the block sizes are a
// function of the problem dimensions and the number of ranks only, so that
// every rank enumerates the same units whatever memory its GPU has free: at
// most the staging these fixed budgets hold, and small enough that there are
// about 32 units per rank for the cost-balanced plan (4 per rank in the
// opposite-spin passes, whose units are blocks of rows against all columns).
// MSHQC_CD_BWD_BLOCK (occupied orbitals per block) overrides both rules in
// every pass.
constexpr size_t kPartTcBudget = size_t(16) << 30;
constexpr size_t kPartF64Budget = size_t(8) << 30;

// Wave pacing of the persistent tile kernels (WavePacer in sm100_ptx.cuh):
// copies per epoch and epochs of slack.  On by default for Gamma (its K runs
// to 57600 and unpaced CTAs drift apart: 7x the DRAM traffic), off for the
// integral tiles (K = M; pacing them changed nothing at N=2000).
// MSHQC_CD_PACE (Gamma) and MSHQC_CD_PACE_TILES (integral tiles) = off
// disables it, = <every>,<slack> enables it with those values.
void pace_params(int* every, int* slack, const char* var, bool on_by_default) {
    *every = on_by_default ? 16 : 0;
    *slack = 2;
    const char* env = std::getenv(var);
    if (!env) return;
    if (std::strcmp(env, "off") == 0) {
        *every = 0;
        return;
    }
    int e = 0, s = 0;
    if (std::sscanf(env, "%d,%d", &e, &s) == 2 && e > 0 && s >= 0) {
        *every = e;
        *slack = s;
    }
}

int64_t env_block() {
    const char* env = std::getenv("MSHQC_CD_BWD_BLOCK");
    if (!env) return 0;
    const long long b = std::atoll(env);
    return b > 0 ? (int64_t)b : 0;
}

// block sizes (rows bI, columns bJ) of a tensor-core pass; staging per (i, j)
// of S (FP32, VS columns) and the four BF16 amplitude operands
void tc_block_sizes(const mshqc_cd_ctx* ctx, int64_t ox, int64_t oy, int64_t VRx, int64_t VRy, int64_t VSy,
                    bool sym, size_t free_budget, int64_t* bI, int64_t* bJ) {
    const bool part = ctx->part_active;
    const size_t budget = part ? kPartTcBudget : free_budget;
    if (sym) {
        const double per_b2 = (double)VRx * (4.0 * VSy + 8.0 * VRy);
        *bI = std::max<int64_t>(1, std::min<int64_t>(ox, (int64_t)std::sqrt((double)budget / per_b2)));
        if (part) {
            // nb blocks give nb (nb + 1) / 2 block pairs: about 32 per rank
            const int64_t nb = (int64_t)std::ceil(std::sqrt(64.0 * ctx->part_size));
            *bI = std::min<int64_t>(*bI, std::max<int64_t>(1, cdiv(ox, nb)));
        }
    } else {
        const double per_i = (double)VRx * oy * (4.0 * VSy + 8.0 * VRy);
        *bI = std::max<int64_t>(1, std::min<int64_t>(ox, (int64_t)((double)budget / per_i)));
        if (part) *bI = std::min<int64_t>(*bI, std::max<int64_t>(1, cdiv(ox, 4 * (int64_t)ctx->part_size)));
    }
    if (const int64_t b = env_block()) *bI = std::min<int64_t>(ox, b);
    *bJ = sym ? *bI : oy;
}

// block sizes (rows bI, columns bJ) of an FP64 pass: staging of S and of the
// amplitudes, both FP64, per (i, j)
void f64_block_sizes(const mshqc_cd_ctx* ctx, int64_t ox, int64_t oy, int64_t vpx, int64_t vpy, bool sym,
                     size_t free_budget, int64_t* bI, int64_t* bJ) {
    const bool part = ctx->part_active;
    const double budget = (double)(part ? kPartF64Budget : free_budget);
    const double per_ij = 2.0 * sizeof(double) * (double)vpx * (double)vpy;
    if (sym) {
        *bI = std::max<int64_t>(1, std::min<int64_t>(ox, (int64_t)std::sqrt(budget / per_ij)));
        if (part) {
            const int64_t nb = (int64_t)std::ceil(std::sqrt(64.0 * ctx->part_size));
            *bI = std::min<int64_t>(*bI, std::max<int64_t>(1, cdiv(ox, nb)));
        }
    } else {
        *bI = std::max<int64_t>(1, std::min<int64_t>(ox, (int64_t)(budget / (per_ij * oy))));
        if (part) *bI = std::min<int64_t>(*bI, std::max<int64_t>(1, cdiv(ox, 4 * (int64_t)ctx->part_size)));
    }
    if (const int64_t b = env_block()) *bI = std::min<int64_t>(ox, b);
    *bJ = sym ? *bI : oy;
}

int require_inputs(mshqc_cd_ctx* ctx, int spin) {
    if (!ctx->L_set) return set_error(MSHQC_CD_ERR_STATE, "Cholesky vectors not set");
    if (!ctx->spin[spin].set)
        return set_error(MSHQC_CD_ERR_STATE,
                         spin == 0 ? "alpha orbitals not set" : "beta orbitals not set");
    return MSHQC_CD_OK;
}

// ---------------------------------------------------------------------------
// transforms shared over occupied orbitals (partition + host collectives)
// ---------------------------------------------------------------------------
// Rank r of R owns the occupied orbitals [r p, min(o, (r + 1) p)),
// p = ceil(o / R); per-orbital buffers (B, Gamma) then hold R p rows so that
// every rank's chunk has the same size for the collectives.
bool sharded(const mshqc_cd_ctx* ctx) { return ctx->part_active && ctx->coll_set && ctx->part_size > 1; }
int64_t shard_p(const mshqc_cd_ctx* ctx, int64_t o) { return cdiv(o, ctx->part_size); }
void shard_range(const mshqc_cd_ctx* ctx, int64_t o, int64_t* lo, int64_t* hi) {
    if (!sharded(ctx)) {
        *lo = 0;
        *hi = o;
        return;
    }
    const int64_t p = shard_p(ctx, o);
    *lo = std::min(o, (int64_t)ctx->part_rank * p);
    *hi = std::min(o, *lo + p);
}
int64_t b_rows(const mshqc_cd_ctx* ctx, int64_t o) { return sharded(ctx) ? shard_p(ctx, o) * ctx->part_size : o; }

int run_collective(mshqc_cd_ctx* ctx, bool gather, double* buf, int64_t count) {
    int (*fn)(double*, int64_t, void*, void*) = gather ? ctx->coll.allgather : ctx->coll.reduce_scatter;
    const int rc = fn(buf, count, (void*)ctx->stream, ctx->coll.user);
    if (rc != 0)
        return set_error(MSHQC_CD_ERR_STATE, std::string(gather ? "allgather" : "reduce_scatter") +
                                                 " callback failed with " + std::to_string(rc));
    return MSHQC_CD_OK;
}

// Bytes of int8 slices one product operand may hold (bounds the vectors
// sub-chunks of the first product and the orbital batches of the second).
constexpr size_t kSliceBytes = size_t(2) << 30;

// ---------------------------------------------------------------------------
// products of int8 slices (ozaki_i8.cuh)
// ---------------------------------------------------------------------------
// out[b](x, y) = alpha sum_k X(x, k) Y(y, k) + beta out at out + b cb + x ldc + y.
// The 128-row operand is the one that pads the tiles less: X, or (sw) Y with
// the result stored transposed.
template <class C>
bool oz_swap(int64_t x, int64_t y) {
    const double straight = (double)round_up(x, ozaki::BM) * round_up(y, C::BN);
    const double swapped = (double)round_up(y, ozaki::BM) * round_up(x, C::BN);
    return swapped < straight;
}
template <class C>
OzakiOperand oz_operand(int64_t rows, int64_t K, bool as_a, int64_t batch) {
    return ozaki_operand(rows, K, as_a ? ozaki::BM : C::BN, (int)batch);
}
// an operand's digits and, behind them, the squares that the guard samples
template <class C>
size_t oz_bytes(const OzakiOperand& op) {
    return (ozaki::operand_bytes<C>(op.Rp, op.Kp) +
            (C::GUARD ? sizeof(uint32_t) * ozaki::SAMPLE_WORDS * (size_t)op.Rp : 0)) * (size_t)op.batch;
}
int* slice_err(mshqc_cd_ctx* ctx) { return ctx->status.as<CallStatus>()->slice_err; }
// One sliced product; A has the 128-row blocks.  With C::GUARD its accuracy is
// that of an FP64 chain or better: tiles whose rows say otherwise (slice_guard.cuh)
// are left out and computed by the FP64 product from the operands' sources.
// N = 400, o = 40, vectors of two fragments with couplings of 10^-6: FP64 energy
// 15.7 ms without slices, 11.7 with, gradient 37.8 and 40.3 (nearly every tile
// left out); rows of one kind 15.8 and 5.9, 37.8 and 17.6, the guards 0.2 and
// 0.5 of them.  Reserves what it needs before it writes a result.
template <class C>
int oz_gemm(mshqc_cd_ctx* ctx, const OzakiOperand& A, const OzakiOperand& B, double* out, int64_t ldc, int64_t cb,
            double alpha, double beta, OzakiOpts o) {
    const int64_t nmb = A.Rp / ozaki::BM, nnb = B.Rp / C::BN;
    GemmListed l{};
    if (C::GUARD) {
        const int64_t units = nmb * nnb * (o.a_shared ? B.batch : A.batch);
        CD_ALLOC(ctx->oz_tiles, (size_t)(sizeof(int) * (units + 1) + units), false);
        int* count = ctx->oz_tiles.as<int>();
        uint8_t* left_out = reinterpret_cast<uint8_t*>(count + 1 + units);
        CD_CUDA(guard_slices(A, B, o, left_out, count, count + 1, ctx->stream));
        o.left_out = left_out;
        l.count = count;
        l.list = count + 1;
        l.nmb = (int)nmb;  l.nnb = (int)nnb;  l.group = ozaki::GROUP;
        l.trans = o.trans ? 1 : 0;
    }
    CD_CUDA(ozaki_gemm<C>(A, B, out, ldc, cb, alpha, beta, o, slice_err(ctx), ctx->num_sms, ctx->stream));
    ctx->launches++;
    if (C::GUARD) {
        const OzakiOperand& X = o.trans ? B : A;   // rows of the result, and its columns
        const OzakiOperand& Y = o.trans ? A : B;
        const bool xs = o.trans ? o.b_shared : o.a_shared, ys = o.trans ? o.a_shared : o.b_shared;
        GemmF64Args g{};
        g.M = (int)X.R;  g.N = (int)Y.R;  g.K = (int)X.K;  g.batch = X.batch;
        g.A = X.src;  g.lda = X.ld;  g.sA = xs ? 0 : X.sb;
        g.B = Y.src;  g.ldb = Y.ld;  g.sB = ys ? 0 : Y.sb;
        g.C = out;  g.ldc = ldc;  g.sC = cb;
        g.alpha = alpha;  g.beta = beta;
        CD_CUDA(gemm_f64_listed(g, !X.t, !Y.t, l, ctx->num_sms, ctx->stream));
        ctx->launches += 2;
    }
    return MSHQC_CD_OK;
}
template <class C>
int oz_mul(mshqc_cd_ctx* ctx, const OzakiOperand& X, bool x_shared, const OzakiOperand& Y, bool y_shared, bool sw,
           double* out, int64_t ldc, int64_t cb, double alpha, double beta) {
    OzakiOpts o;
    o.a_shared = sw ? y_shared : x_shared;
    o.b_shared = sw ? x_shared : y_shared;
    o.trans = sw;
    return oz_gemm<C>(ctx, sw ? Y : X, sw ? X : Y, out, ldc, cb, alpha, beta, o);
}
// reserves an operand's digits and what goes with its rows
template <class C>
int oz_reserve(mshqc_cd_ctx* ctx, DevBuf& q, DevBuf& e, size_t bytes, OzakiOperand& op) {
    CD_ALLOC(q, bytes, false);
    CD_ALLOC(e, op.row_bytes(C::GUARD), false);
    op.q = q.as<int8_t>();
    op.e = e.as<int>();
    if (C::GUARD)
        op.smp = reinterpret_cast<uint32_t*>(op.q + ozaki::operand_bytes<C>(op.Rp, op.Kp) * (size_t)op.batch);
    return MSHQC_CD_OK;
}
// the rows of Y that hold a spin's half-transformed vectors
double* y_rows(mshqc_cd_ctx* ctx, int spin) {
    return ctx->Y.as<double>() + ctx->Yr[spin].row * ctx->M * ctx->N;
}

// Second half of the forward transform from the spin's rows of Y [i - lo][Q][nu]:
// B[i][a][Q] = sum_nu C[nu, o+a] Y[i][Q][nu], a batch of orbitals i at a time
template <class C>
int second_half_sliced(mshqc_cd_ctx* ctx, int spin, int64_t lo, int64_t hi) {
    SpinState& s = ctx->spin[spin];
    const int64_t N = ctx->N, M = ctx->M, Mp = ctx->Mp, o = s.nocc, v = N - o, ni = hi - lo, vp = s.vp;
    const bool sw = oz_swap<C>(v, M);
    OzakiOperand Av = oz_operand<C>(v, N, !sw, 1);
    CD_RC(oz_reserve<C>(ctx, ctx->oz_a, ctx->oz_ea, oz_bytes<C>(Av), Av));
    CD_CUDA(ozaki_slice<C>(s.C.as<double>() + o * N, N, 0, Av, ctx->num_sms, ctx->stream));
    ctx->launches++;
    const int64_t per_i = (int64_t)oz_bytes<C>(oz_operand<C>(M, N, sw, 1));
    const int64_t ib = std::max<int64_t>(1, std::min<int64_t>(ni, (int64_t)kSliceBytes / per_i));
    for (int64_t i0 = lo; i0 < hi; i0 += ib) {
        const int64_t nb = std::min(ib, hi - i0);
        OzakiOperand By = oz_operand<C>(M, N, sw, nb);
        CD_RC(oz_reserve<C>(ctx, ctx->oz_b, ctx->oz_eb, (size_t)(per_i * nb), By));
        CD_CUDA(ozaki_slice<C>(y_rows(ctx, spin) + (i0 - lo) * M * N, N, M * N, By, ctx->num_sms, ctx->stream));
        ctx->launches++;
        CD_RC(oz_mul<C>(ctx, Av, true, By, false, sw, s.B64.as<double>() + i0 * vp * Mp, Mp, vp * Mp, 1.0, 0.0));
    }
    return MSHQC_CD_OK;
}

// FP64 products of at least this many operations run as int8 slices of full
// accuracy (ozaki::Full) where each sliced element takes part in at least
// kSlicedMinReuse multiply-adds: slicing costs about 6 ps an element (HBM),
// the DMMA products 0.06 ps an operation, the sliced ones 0.03.  Second half
// transforms and virtual products of the gradient at M = 4 N, o = N / 10, DMMA
// and sliced (stage times, ms): N = 203 (1.3e9 operations, v = 183) 0.17 and 0.18,
// 0.26 and 0.37; N = 300 (9.7e9, v = 270) 0.50 and 0.48, 0.84 and 0.84; N = 360
// 1.18 and 1.10, 1.88 and 1.77; N = 400 1.56 and 1.49, 2.35 and 2.17.
// MSHQC_CD_FP64_SLICES=off keeps every FP64 product on the DMMA pipe, =on slices
// at every size.
constexpr double kSlicedMinFlops = 4e9;
constexpr int64_t kSlicedMinReuse = 256;
bool fp64_slices(const mshqc_cd_ctx* ctx, double flops, double min_flops, int64_t reuse) {
    if (ctx->slices_refused) return false;
    if (const char* env = std::getenv("MSHQC_CD_FP64_SLICES")) {
        if (std::strcmp(env, "off") == 0) return false;
        if (std::strcmp(env, "on") == 0) return true;
    }
    return flops >= min_flops && reuse >= kSlicedMinReuse;
}

// The sliced FP64 products hold their slices next to the operands.  Each of the
// functions below reserves them before it writes a result, so where the memory
// does not hold them the FP64 products run instead, for the rest of the call (each
// attempt frees buffers, which waits for the device).
bool no_room(mshqc_cd_ctx* ctx, int rc) {
    if (rc != MSHQC_CD_ERR_ALLOC) return false;
    ctx->release_slices();
    ctx->slices_refused = true;
    return true;
}

bool int8_transform_enabled(const mshqc_cd_ctx* ctx) {
    if (ctx->N > ozaki::Mixed::MAXK) return false;
    const char* env = std::getenv("MSHQC_CD_TRANSFORM");
    return !(env && std::strcmp(env, "f64") == 0);
}

// The forward half transform of a mixed request runs on the int8 tensor cores
// from N = 512 on; below, the FP64 products (DMMA, full slices) take the same
// time and their B is exact (forward transform of the gradient step: N = 400
// 1.34 ms FP64, 1.38 int8; N = 520 4.3 DMMA, 3.2 int8; N = 600 7.1 and 4.7).
// The transposed transforms keep the int8 products at every size (N = 400 2.3 ms
// either way, N = 600 10.6 DMMA, 6.7 int8, open shell 23.2 and 10.9).
// MSHQC_CD_TRANSFORM=i8 forces the int8 products, =f64 the FP64 ones.
constexpr int64_t kInt8ForwardMinN = 512;
bool int8_forward_enabled(const mshqc_cd_ctx* ctx) {
    if (!int8_transform_enabled(ctx)) return false;
    const char* env = std::getenv("MSHQC_CD_TRANSFORM");
    if (env && std::strcmp(env, "i8") == 0) return true;
    return ctx->N >= kInt8ForwardMinN;
}

// First half of the forward transform for the occupied orbitals [lo, hi) of the
// given spins: Y[row of i][(Q,nu)] = sum_mu C[mu,i] L[Q][nu*N + mu], one chunk of
// vectors at a time.  Two spins are one product over both spins' orbitals, so
// the vectors are read (and sliced) once: unrestricted N = 600, 60 + 58
// orbitals, 10.5 -> 7.1 ms with the second halves.  i8: int8 slices of the mixed
// accuracy, else FP64 on the DMMA pipe (every vector element meets few
// orbitals: full slices would cost more than the products).
int first_half(mshqc_cd_ctx* ctx, int nsp, const int* spins, const int64_t* lo, const int64_t* hi, bool i8) {
    const int64_t N = ctx->N, M = ctx->M;
    int64_t rows = 0;
    ctx->Yr[0].ok = ctx->Yr[1].ok = false;
    ctx->both_used |= nsp == 2;
    for (int k = 0; k < nsp; ++k) rows += std::max<int64_t>(0, hi[k] - lo[k]);
    CD_ALLOC_FIRST(ctx->Y, sizeof(double) * (size_t)std::max<int64_t>(1, rows) * M * N, false);
    int64_t r = 0;
    for (int k = 0; k < nsp; ++k) {
        auto& y = ctx->Yr[spins[k]];
        y.i8 = i8;
        y.row = r;
        y.lo = lo[k];
        y.hi = hi[k];
        r += std::max<int64_t>(0, hi[k] - lo[k]);
    }
    // the rows are valid once every product that fills them is queued
    auto filled = [&]() {
        for (int k = 0; k < nsp; ++k) ctx->Yr[spins[k]].ok = true;
        return MSHQC_CD_OK;
    };
    if (rows == 0) return filled();
    // the orbitals as contiguous rows
    const double* C = ctx->spin[spins[0]].C.as<double>() + lo[0] * N;
    if (nsp == 2) {
        CD_ALLOC(ctx->cpack, sizeof(double) * (size_t)(rows * N), false);
        r = 0;
        for (int k = 0; k < nsp; ++k) {
            const int64_t ni = std::max<int64_t>(0, hi[k] - lo[k]);
            CD_CUDA(cudaMemcpyAsync(ctx->cpack.as<double>() + r * N, ctx->spin[spins[k]].C.as<double>() + lo[k] * N,
                                    sizeof(double) * (size_t)(ni * N), cudaMemcpyDeviceToDevice, ctx->stream));
            r += ni;
        }
        C = ctx->cpack.as<double>();
    }
    using Cfg = ozaki::Mixed;
    const bool sw = round_up(rows, Cfg::BN) < round_up(rows, ozaki::BM);
    OzakiOperand Ao = oz_operand<Cfg>(rows, N, !sw, 1);
    if (i8) {
        CD_RC(oz_reserve<Cfg>(ctx, ctx->oz_a, ctx->oz_ea, oz_bytes<Cfg>(Ao), Ao));
        CD_CUDA(ozaki_slice<Cfg>(C, N, 0, Ao, ctx->num_sms, ctx->stream));
        ctx->launches++;
    }
    const int64_t per_q = (int64_t)ozaki::operand_bytes<Cfg>(round_up(N, ozaki::BM), ozaki::padded_k(N));
    const int64_t qs = i8 ? std::max<int64_t>(1, (int64_t)kSliceBytes / per_q) : M;
    const int64_t qc = vectors_chunk_size(ctx);
    for (int64_t Q0 = 0; Q0 < M; Q0 += qc) {
        const int64_t mc = std::min(qc, M - Q0);
        const double* Lc = nullptr;
        CD_RC(vectors_chunk(ctx, Q0, mc, &Lc));
        for (int64_t q0 = 0; q0 < mc; q0 += qs) {
            const int64_t ms = std::min(qs, mc - q0);
            const double* L = Lc + q0 * N * N;
            double* Y = ctx->Y.as<double>() + (Q0 + q0) * N;
            if (i8) {
                OzakiOperand Bl = oz_operand<Cfg>(ms * N, N, sw, 1);
                CD_RC(oz_reserve<Cfg>(ctx, ctx->oz_b, ctx->oz_eb, oz_bytes<Cfg>(Bl), Bl));
                CD_CUDA(ozaki_slice<Cfg>(L, N, 0, Bl, ctx->num_sms, ctx->stream));
                ctx->launches++;
                CD_RC(oz_mul<Cfg>(ctx, Ao, true, Bl, false, sw, Y, M * N, 0, 1.0, 0.0));
            } else {
                GemmF64Args g{};
                g.M = (int)rows;  g.N = (int)(ms * N);  g.K = (int)N;  g.batch = 1;
                g.A = C;  g.lda = N;
                g.B = L;  g.ldb = N;
                g.C = Y;  g.ldc = M * N;
                g.alpha = 1.0;  g.beta = 0.0;
                CD_RC(gemm_run(ctx, g, true, true));
            }
        }
    }
    return filled();
}

// Forward half transforms of the given spins into the padded [i][a][Q] layout,
// for this rank's occupied orbitals (B rows outside stay zero).  FP64, or with
// i8 both products on the int8 tensor cores at the mixed accuracy (about 2^-33
// of the row maxima per term), which only the mixed-precision path uses.
int transform(mshqc_cd_ctx* ctx, int nsp, const int* spins, bool i8) {
    const int64_t N = ctx->N, M = ctx->M, Mp = ctx->Mp;
    int64_t lo[2], hi[2];
    for (int k = 0; k < nsp; ++k) {
        SpinState& s = ctx->spin[spins[k]];
        shard_range(ctx, s.nocc, &lo[k], &hi[k]);
        s.vp = round_up(N - s.nocc, 64);
        s.invalidate();   // run_transforms marks B valid, with its last launch queued
        CD_ALLOC_FIRST(s.B64, sizeof(double) * (size_t)b_rows(ctx, s.nocc) * s.vp * Mp, true);
        s.B64_prec = i8 ? MSHQC_CD_FP16X3 : MSHQC_CD_FP64;
    }
    CD_RC(first_half(ctx, nsp, spins, lo, hi, i8));
    for (int k = 0; k < nsp; ++k) {
        SpinState& s = ctx->spin[spins[k]];
        const int64_t o = s.nocc, v = N - o, ni = hi[k] - lo[k];
        if (ni <= 0) continue;
        if (i8) {
            CD_RC(second_half_sliced<ozaki::Mixed>(ctx, spins[k], lo[k], hi[k]));
            continue;
        }
        const char* tenv = std::getenv("MSHQC_CD_TRANSFORM");   // f64: DMMA for both halves
        if (!(tenv && std::strcmp(tenv, "f64") == 0) && fp64_slices(ctx, 2.0 * v * M * N * ni, kSlicedMinFlops, v)) {
            const int rc = second_half_sliced<ozaki::Full>(ctx, spins[k], lo[k], hi[k]);
            if (!no_room(ctx, rc)) {
                CD_RC(rc);
                continue;
            }
        }
        // B[i][a][Q] = sum_nu C[nu, o+a] Y[i][Q][nu]
        GemmF64Args g{};
        g.M = (int)v;  g.N = (int)M;  g.K = (int)N;  g.batch = (int)ni;
        g.A = s.C.as<double>() + o * N;  g.lda = N;  g.sA = 0;
        g.B = y_rows(ctx, spins[k]);  g.ldb = N;  g.sB = M * N;
        g.C = s.B64.as<double>() + lo[k] * s.vp * Mp;  g.ldc = Mp;  g.sC = s.vp * Mp;
        g.alpha = 1.0;  g.beta = 0.0;
        CD_RC(gemm_run(ctx, g, true, true));
    }
    return MSHQC_CD_OK;
}

// Whether the half-transformed vectors of both spins may be held at once: the
// buffer already has the room, or it is at most a quarter of the free memory (an
// eighth where an earlier call ran out of memory or this one cannot be done again,
// one_spin_retry: the buffers formed after it are about three times its size, and
// the staging needs its part).
int both_spins_fit(mshqc_cd_ctx* ctx, bool* yes) {
    *yes = false;
    if (ctx->one_spin) return MSHQC_CD_OK;
    int64_t rows = 0;
    for (int s = 0; s < 2; ++s) {
        int64_t lo, hi;
        shard_range(ctx, ctx->spin[s].nocc, &lo, &hi);
        rows += hi - lo;
    }
    const size_t need = sizeof(double) * (size_t)(rows * ctx->M * ctx->N);
    *yes = need <= ctx->Y.bytes;
    if (*yes) return MSHQC_CD_OK;
    size_t free_b = 0, total_b = 0;
    CD_CUDA(cudaMemGetInfo(&free_b, &total_b));
    *yes = need <= (free_b + ctx->Y.bytes) / (sharded(ctx) || ctx->cautious ? 8 : 4);
    return MSHQC_CD_OK;
}

// Whether the FP64 integral and Gamma products of blocks of `rows` x `cols`
// composite virtual rows run as int8 slices of full accuracy.  Whole calls at
// M = 4 N, o = N / 10, DMMA and sliced (energy; gradient, ms): N = 128 (2.4e9
// operations) 0.28 and 0.32; 0.69 and 0.87.  N = 161 (1.2e10) 0.55 and 0.44; 1.50
// and 1.22.  N = 180 (2.1e10) 0.66 and 0.51; 1.73 and 1.44.  N = 245 2.03 and 1.05;
// 5.05 and 3.06.  N = 161 with M = 403, o = 17 (8.9e9): equal.  So the two cross
// between 2.4e9 and 1.2e10; the line lies above, on the DMMA side.
constexpr double kSlicedPairFlops = 1.6e10;
bool sliced_pairs(const mshqc_cd_ctx* ctx, int64_t rows, int64_t cols) {
    return fp64_slices(ctx, 2.0 * rows * cols * ctx->Mp, kSlicedPairFlops, ctx->Mp);
}

// S[(i,a)][(j,b)] = sum_Q X[(i,a)][Q] Y[(j,b)][Q] of a block pair from int8
// slices (row length of S: nJ vpy); tri: column orbitals j >= i only
int sliced_integrals(mshqc_cd_ctx* ctx, const SpinState& X, const SpinState& Y, int64_t I0, int64_t nI, int64_t J0,
                     int64_t nJ, bool tri, double* S) {
    using Cfg = ozaki::Full;
    const int64_t Mp = ctx->Mp;
    OzakiOperand A = oz_operand<Cfg>(nI * X.vp, Mp, true, 1), B = oz_operand<Cfg>(nJ * Y.vp, Mp, false, 1);
    CD_RC(oz_reserve<Cfg>(ctx, ctx->oz_a, ctx->oz_ea, oz_bytes<Cfg>(A), A));
    CD_RC(oz_reserve<Cfg>(ctx, ctx->oz_b, ctx->oz_eb, oz_bytes<Cfg>(B), B));
    CD_CUDA(ozaki_slice<Cfg>(X.B64.as<double>() + I0 * X.vp * Mp, Mp, 0, A, ctx->num_sms, ctx->stream));
    CD_CUDA(ozaki_slice<Cfg>(Y.B64.as<double>() + J0 * Y.vp * Mp, Mp, 0, B, ctx->num_sms, ctx->stream));
    OzakiOpts o;
    o.tri = tri ? (int)X.vp : 0;
    ctx->launches += 2;
    return oz_gemm<Cfg>(ctx, A, B, S, nJ * Y.vp, 0, 1.0, 0.0, o);
}

// gamma[r][Q] += sum_k A(r, k) B[k][Q] over `rows` amplitude rows and K columns
// (transposed: A(r, k) = A[k * lda + r]); the amplitudes' slices go to `work`
int sliced_gamma(mshqc_cd_ctx* ctx, const double* A, int64_t lda, bool transposed, int64_t rows, int64_t K,
                 const double* B, double* gamma, DevBuf& work) {
    using Cfg = ozaki::Full;
    const int64_t Mp = ctx->Mp;
    OzakiOperand Ta = oz_operand<Cfg>(rows, K, true, 1), Tb = oz_operand<Cfg>(Mp, K, false, 1);
    CD_RC(oz_reserve<Cfg>(ctx, work, ctx->oz_ea, oz_bytes<Cfg>(Ta), Ta));
    CD_RC(oz_reserve<Cfg>(ctx, ctx->oz_b, ctx->oz_eb, oz_bytes<Cfg>(Tb), Tb));
    if (transposed)
        CD_CUDA(ozaki_slice_t<Cfg>(A, lda, 0, Ta, ctx->stream));
    else
        CD_CUDA(ozaki_slice<Cfg>(A, lda, 0, Ta, ctx->num_sms, ctx->stream));
    CD_CUDA(ozaki_slice_t<Cfg>(B, Mp, 0, Tb, ctx->stream));
    OzakiOpts o;
    if (K > 4096) {
        // long K: CTAs that share operand slabs are kept together
        CD_ALLOC(ctx->pace, sizeof(int) * (size_t)ctx->num_sms, false);
        o.pace = ctx->pace.as<int>();
    }
    ctx->launches += transposed ? 4 : 3;
    return oz_gemm<Cfg>(ctx, Ta, Tb, gamma, Mp, 0, 1.0, 1.0, o);
}

// One pair-energy pass: spins, where its pair sums go (ctx->pair_sum, doubles:
// npairs sums, for the restricted mode npairs opposite-spin sums after them) and
// its totals (CallStatus::totals).
struct PairPass {
    int mode, sx, sy;
    int npairs, ox, oy;
    int64_t off;
    int total;
};

// Deterministic reductions of per-unit partials (ctx->partial, the opposite-spin
// part of the restricted mode after them) into the pass's sums and totals.
int reduce_units(mshqc_cd_ctx* ctx, const PairPass& p, int nblocks) {
    const unsigned planes = p.mode == PAIR_RESTRICTED ? 2 : 1;
    double* sums = ctx->pair_sum.as<double>() + p.off;
    reduce_pairs_kernel<<<dim3((unsigned)cdiv(p.npairs, 128), planes), 128, 0, ctx->stream>>>(
        ctx->partial.as<double>(), p.npairs, nblocks, sums);
    CD_CUDA(cudaGetLastError());
    reduce_total_kernel<<<planes, 256, 0, ctx->stream>>>(sums, p.npairs, ctx->status.as<CallStatus>()->totals + p.total);
    CD_CUDA(cudaGetLastError());
    ctx->launches += 2;
    return MSHQC_CD_OK;
}

// The ordered pair-energy matrix (row-major ox * oy) from a pass's pair sums.
void fill_pairs(const PairPass& p, const double* ps, std::vector<double>& m) {
    const int ox = p.ox, oy = p.oy;
    m.assign((size_t)ox * oy, 0.0);
    if (p.mode == PAIR_OPPOSITE_SPIN) {
        std::memcpy(m.data(), ps, sizeof(double) * m.size());
        return;
    }
    for (int i = 0; i < ox; ++i)
        for (int j = p.mode == PAIR_RESTRICTED ? i : i + 1; j < ox; ++j) {
            const double e = *ps++;
            m[(size_t)i * ox + j] = i == j ? e : 0.5 * e;
            m[(size_t)j * ox + i] = i == j ? e : 0.5 * e;
        }
}

template <int MODE>
int pair_pass_f64_staged(mshqc_cd_ctx* ctx, const PairPass& pp);

// One FP64 pair-energy pass.
int pair_pass_f64(mshqc_cd_ctx* ctx, const PairPass& pp) {
    const SpinState& X = ctx->spin[pp.sx];
    const SpinState& Y = ctx->spin[pp.sy];
    const int mode = pp.mode, ox = pp.ox, oy = pp.oy;
    const int vx = (int)(ctx->N - ox), vy = (int)(ctx->N - oy);
    const int nbx = (int)(X.vp / 64), nby = (int)(Y.vp / 64);
    if (sliced_pairs(ctx, ox * X.vp, oy * Y.vp)) {
        const int rc = mode == PAIR_RESTRICTED  ? pair_pass_f64_staged<PAIR_RESTRICTED>(ctx, pp)
                       : mode == PAIR_SAME_SPIN ? pair_pass_f64_staged<PAIR_SAME_SPIN>(ctx, pp)
                                                : pair_pass_f64_staged<PAIR_OPPOSITE_SPIN>(ctx, pp);
        if (!no_room(ctx, rc)) return rc;
        ctx->W.release();
    }
    const int npairs = pp.npairs, nblocks = (int)block_count(mode, nbx, nby);
    const int64_t units = (int64_t)npairs * nblocks;
    CD_ALLOC_FIRST(ctx->partial, sizeof(double) * units * 2, false);
    PairF64Args a{};
    a.X = X.B64.as<double>();
    a.Y = Y.B64.as<double>();
    a.vx = vx;  a.vy = vy;
    a.vpx = (int)X.vp;  a.vpy = (int)Y.vp;
    a.Mp = (int)ctx->Mp;
    a.eox = X.eps.as<double>();  a.evx = a.eox + ox;
    a.eoy = Y.eps.as<double>();  a.evy = a.eoy + oy;
    a.ox = ox;  a.oy = oy;  a.nbx = nbx;  a.nby = nby;
    a.nblocks = nblocks;
    a.partial = ctx->partial.as<double>();
    a.partial2 = ctx->partial.as<double>() + units;
    const size_t smem = pair_f64_detail::SMEM_BYTES;
    begin_stage(ctx, ST_PAIR);
    if (mode == PAIR_RESTRICTED) {
        CD_CUDA(cudaFuncSetAttribute(pair_energy_f64_kernel<PAIR_RESTRICTED>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        pair_energy_f64_kernel<PAIR_RESTRICTED><<<(unsigned)units, 256, smem, ctx->stream>>>(a);
    } else if (mode == PAIR_SAME_SPIN) {
        CD_CUDA(cudaFuncSetAttribute(pair_energy_f64_kernel<PAIR_SAME_SPIN>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        pair_energy_f64_kernel<PAIR_SAME_SPIN><<<(unsigned)units, 256, smem, ctx->stream>>>(a);
    } else {
        CD_CUDA(cudaFuncSetAttribute(pair_energy_f64_kernel<PAIR_OPPOSITE_SPIN>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        pair_energy_f64_kernel<PAIR_OPPOSITE_SPIN><<<(unsigned)units, 256, smem, ctx->stream>>>(a);
    }
    end_stage(ctx);
    CD_CUDA(cudaGetLastError());
    ctx->launches++;
    return reduce_units(ctx, pp, nblocks);
}


// The FP64 pair-energy pass of larger systems: integrals of block pairs into a
// staging block (int8 slices of full accuracy), energies from there.
template <int MODE>
int pair_pass_f64_staged(mshqc_cd_ctx* ctx, const PairPass& pp) {
    constexpr bool kSym = MODE != PAIR_OPPOSITE_SPIN;
    const SpinState& X = ctx->spin[pp.sx];
    const SpinState& Y = ctx->spin[pp.sy];
    const int64_t ox = X.nocc, oy = Y.nocc;
    const int npairs = pp.npairs;
    size_t free_b = 0, total_b = 0;
    CD_CUDA(cudaMemGetInfo(&free_b, &total_b));
    const size_t budget = std::min<size_t>((free_b + ctx->W.bytes) / 3, size_t(40) << 30);
    const int64_t per_row = (int64_t)sizeof(double) * X.vp * Y.vp;   // per (i, j)
    const int64_t bI = kSym ? std::max<int64_t>(1, std::min<int64_t>(ox, (int64_t)std::sqrt((double)budget / per_row)))
                            : std::max<int64_t>(1, std::min<int64_t>(ox, (int64_t)(budget / (per_row * oy))));
    const int64_t bJ = kSym ? bI : oy;
    // 4 CTAs a pair where the pairs alone do not fill the GPU several times
    const int nch = npairs < 32 * ctx->num_sms ? 4 : 1;
    const int64_t units = (int64_t)npairs * nch;
    CD_ALLOC_FIRST(ctx->W, (size_t)(bI * bJ * per_row), false);
    CD_ALLOC_FIRST(ctx->partial, sizeof(double) * (size_t)units * 2, false);
    begin_stage(ctx, ST_PAIR);
    for (int64_t I0 = 0; I0 < ox; I0 += bI) {
        const int64_t nI = std::min(bI, ox - I0);
        for (int64_t J0 = kSym ? I0 : 0; J0 < oy; J0 += bJ) {
            const int64_t nJ = std::min(bJ, oy - J0);
            const int rc = sliced_integrals(ctx, X, Y, I0, nI, J0, nJ, kSym && I0 == J0, ctx->W.as<double>());
            if (rc != MSHQC_CD_OK) {
                end_stage(ctx);
                return rc;
            }
            PairStagedArgs p{};
            p.S = ctx->W.as<double>();
            p.ldS = nJ * Y.vp;
            p.vpx = (int)X.vp;  p.vpy = (int)Y.vp;
            p.vx = (int)(ctx->N - ox);  p.vy = (int)(ctx->N - oy);
            p.ox = (int)ox;  p.oy = (int)oy;
            p.i0 = (int)I0;  p.nbi = (int)nI;  p.j0 = (int)J0;  p.nbj = (int)nJ;
            p.nchunk = nch;
            p.eox = X.eps.as<double>();  p.evx = p.eox + ox;
            p.eoy = Y.eps.as<double>();  p.evy = p.eoy + oy;
            p.partial = ctx->partial.as<double>();
            p.partial2 = p.partial + units;
            pair_energy_staged_kernel<MODE><<<(unsigned)(nI * nJ * nch), 256, 0, ctx->stream>>>(p);
            CD_CUDA(cudaGetLastError());
            ctx->launches++;
        }
    }
    end_stage(ctx);
    return reduce_units(ctx, pp, nch);
}

// ---------------------------------------------------------------------------
// FP16x3 tensor-core path
// ---------------------------------------------------------------------------
int64_t tc_rows(int64_t v) { return 128 * round_up(cdiv(v, 128), 2); }

// fixed-point hi/lo split of one spin's FP64 MO vectors into the blocked layout,
// with the per-row exponents, exact diagonal integrals and hi/lo row norms
int split_fixed(mshqc_cd_ctx* ctx, int spin, int layout) {
    SpinState& s = ctx->spin[spin];
    const int64_t o = s.nocc, v = ctx->N - s.nocc, M = ctx->M, Mp = ctx->Mp;
    const bool pair_layout = layout == 1;
    // rows per orbital; the integral-tile layout packs them across orbitals
    const int64_t rows = pair_layout ? tc_rows(v) : round_up(v, 32), nqc = Mp / 16;
    const int64_t total = round_up(o * rows, 256);
    const size_t n = (size_t)(nqc * total * 16);   // elements of hi, as many of lo
    CD_ALLOC_FIRST(s.B16, 2 * n * sizeof(uint16_t), false);
    CD_ALLOC_FIRST(s.expo, sizeof(int) * o * rows, true);
    CD_ALLOC_FIRST(s.diag, sizeof(double) * o * rows, true);
    // (a spin is split once per call: its slots in the status are zero)
    unsigned long long* norms = ctx->status.as<CallStatus>()->norms[spin];
    s.vp16 = rows;
    s.Mp16 = Mp;
    {
        const int64_t warps = o * rows;
        const int blocks = (int)std::min<int64_t>(cdiv(warps * 32, 256), (int64_t)ctx->num_sms * 32);
        row_scale_kernel<<<blocks, 256, 0, ctx->stream>>>(
            s.B64.as<double>(), s.vp, Mp, (int)v, (int)M, o, rows, s.expo.as<int>(),
            s.diag.as<double>(), nullptr, 0, 0, 0, nullptr, norms);
        CD_CUDA(cudaGetLastError());
        ctx->launches++;
    }
    {
        const int64_t threads = (int64_t)(n / 8);
        const int blocks = (int)std::min<int64_t>(cdiv(threads, 256), (int64_t)ctx->num_sms * 16);
        split_fixed_blocked_kernel<<<blocks, 256, 0, ctx->stream>>>(
            s.B64.as<double>(), s.vp, Mp, (int)v, (int)M, o, nqc, rows, total / 8, s.expo.as<int>(),
            s.B16.as<uint16_t>());
        CD_CUDA(cudaGetLastError());
        ctx->launches++;
    }
    // largest row norms (the Cauchy-Schwarz bound of the integer accumulators):
    // with the call's status
    s.norms_pending = true;
    s.B16_valid = true;
    s.B16_layout = layout;
    return MSHQC_CD_OK;
}

// exact sum_Q B_alpha[i][a][Q] B_beta[i][a][Q] for the opposite-spin diagonal
int opposite_spin_diag(mshqc_cd_ctx* ctx) {
    if (ctx->diag_os_valid) return MSHQC_CD_OK;
    SpinState& A = ctx->spin[0];
    SpinState& B = ctx->spin[1];
    const int64_t oa = A.nocc, va = ctx->N - A.nocc, rows = A.vp16;
    const int o2 = (int)std::min(A.nocc, B.nocc);
    const int v2 = (int)std::min(ctx->N - A.nocc, ctx->N - B.nocc);
    CD_ALLOC_FIRST(ctx->diag_os, sizeof(double) * std::max<int64_t>(1, (int64_t)o2 * rows), true);
    CD_ALLOC_FIRST(ctx->scratch, sizeof(double) * (size_t)(oa * rows * 2), false);
    double* tmp = ctx->scratch.as<double>();
    int* etmp = reinterpret_cast<int*>(tmp + oa * rows);
    const int64_t warps = oa * rows;
    const int blocks = (int)std::min<int64_t>(cdiv(warps * 32, 256), (int64_t)ctx->num_sms * 32);
    row_scale_kernel<<<blocks, 256, 0, ctx->stream>>>(
        A.B64.as<double>(), A.vp, ctx->Mp, (int)va, (int)ctx->M, oa, rows, etmp, tmp, B.B64.as<double>(), B.vp, o2,
        v2, ctx->diag_os.as<double>(), nullptr);
    CD_CUDA(cudaGetLastError());
    ctx->launches++;
    ctx->diag_os_valid = true;
    return MSHQC_CD_OK;
}

template <int MODE>
cudaError_t launch_tc(const PairTcArgs& a, int grid, cudaStream_t st) {
    const size_t smem = pair_tc::SMEM_BYTES;
    cudaError_t e = cudaFuncSetAttribute(pair_energy_tc_kernel<MODE>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    pair_energy_tc_kernel<MODE><<<grid, pair_tc::THREADS, smem, st>>>(a);
    return cudaGetLastError();
}

// The integer accumulators of a pass are exact when every partial sum stays
// below 2^24: |sum hi hi'| <= sqrt(max sum hi^2 * max sum hi'^2), likewise for
// the cross terms (Cauchy-Schwarz over the Q index).
bool pass_exact(const mshqc_cd_ctx* ctx, const PairPass& pp) {
    const SpinState& X = ctx->spin[pp.sx];
    const SpinState& Y = ctx->spin[pp.sy];
    const double lim = 16777216.0;
    const double bhh = std::sqrt(X.max_norm_hi * Y.max_norm_hi);
    const double bx = std::sqrt(X.max_norm_hi * Y.max_norm_lo) + std::sqrt(X.max_norm_lo * Y.max_norm_hi);
    return bhh < lim && bx < lim;
}

int pair_pass_tc(mshqc_cd_ctx* ctx, const PairPass& pp) {
    const SpinState& X = ctx->spin[pp.sx];
    const SpinState& Y = ctx->spin[pp.sy];
    const int mode = pp.mode, ox = pp.ox, oy = pp.oy;
    const int vx = (int)(ctx->N - ox), vy = (int)(ctx->N - oy);
    const int nbx = (int)cdiv(vx, 128), nby = (int)cdiv(vy, 128);
    const int npairs = pp.npairs, nblocks = (int)block_count(mode, nbx, nby);
    const int64_t units = (int64_t)npairs * nblocks;
    CD_ALLOC_FIRST(ctx->partial, sizeof(double) * units * 2, false);
    if (mode == PAIR_OPPOSITE_SPIN) {
        begin_stage(ctx, ST_SPLIT);
        CD_RC(opposite_spin_diag(ctx));
        end_stage(ctx);
    }
    if (X.B16_layout != 1 || Y.B16_layout != 1)
        return set_error(MSHQC_CD_ERR_STATE, "fixed-point operands not in the pair layout");
    PairTcArgs a{};
    a.Xp = X.B16.as<uint16_t>();
    a.Yp = Y.B16.as<uint16_t>();
    a.ex = X.expo.as<int>();  a.ey = Y.expo.as<int>();
    if (mode == PAIR_OPPOSITE_SPIN) {
        a.diag = ctx->diag_os.as<double>();
        a.diag_o = (int)std::min(X.nocc, Y.nocc);
        a.diag_v = std::min(vx, vy);
    } else {
        a.diag = X.diag.as<double>();
        a.diag_o = ox;
        a.diag_v = vx;
    }
    a.rows_x = (int)X.vp16;  a.rows_y = (int)Y.vp16;
    a.nqc = (int)(ctx->Mp / 16);
    a.vx = vx;  a.vy = vy;
    a.eox = X.eps.as<double>();  a.evx = a.eox + ox;
    a.eoy = Y.eps.as<double>();  a.evy = a.eoy + oy;
    a.ox = ox;  a.oy = oy;  a.nbx = nbx;  a.nby = nby;
    a.nblocks = nblocks;
    a.units = units;
    a.partial = ctx->partial.as<double>();
    a.partial2 = ctx->partial.as<double>() + units;
    a.err = ctx->status.as<CallStatus>()->tile_err;
    const int grid = (int)std::min<int64_t>(units, ctx->num_sms);
    cudaError_t e;
    begin_stage(ctx, ST_PAIR);
    if (mode == PAIR_RESTRICTED)
        e = launch_tc<PAIR_RESTRICTED>(a, grid, ctx->stream);
    else if (mode == PAIR_SAME_SPIN)
        e = launch_tc<PAIR_SAME_SPIN>(a, grid, ctx->stream);
    else
        e = launch_tc<PAIR_OPPOSITE_SPIN>(a, grid, ctx->stream);
    end_stage(ctx);
    if (e != cudaSuccess) return cuda_error(e, "pair_energy_tc_kernel launch");
    ctx->launches++;
    return reduce_units(ctx, pp, nblocks);
}

}  // namespace

int invalidate_spin(mshqc_cd_ctx* ctx, int spin) {
    ctx->spin[spin].invalidate();
    ctx->diag_os_valid = false;
    ctx->Yr[spin].ok = false;
    return MSHQC_CD_OK;
}

namespace {

// an FP64 request never reuses int8-slice products; a mixed one reuses either
bool transform_needed(const mshqc_cd_ctx* ctx, int spin, int precision) {
    const SpinState& s = ctx->spin[spin];
    return !s.B64_valid || (precision == MSHQC_CD_FP64 && s.B64_prec != MSHQC_CD_FP64);
}

int run_transforms(mshqc_cd_ctx* ctx, int nsp, const int* spins, int precision) {
    begin_stage(ctx, ST_TRANSFORM);
    CD_RC(transform(ctx, nsp, spins, precision == MSHQC_CD_FP16X3 && int8_forward_enabled(ctx)));
    for (int k = 0; k < nsp; ++k) {
        SpinState& s = ctx->spin[spins[k]];
        // shared over ranks: this rank's orbitals so far, now all of them
        if (sharded(ctx))
            CD_RC(run_collective(ctx, true, s.B64.as<double>(), shard_p(ctx, s.nocc) * s.vp * ctx->Mp));
        s.B64_valid = true;
    }
    end_stage(ctx);
    return MSHQC_CD_OK;
}

}  // namespace

int ensure_transform(mshqc_cd_ctx* ctx, int spin, int precision, int layout) {
    CD_RC(require_inputs(ctx, spin));
    SpinState& s = ctx->spin[spin];
    if (precision != MSHQC_CD_FP64 && precision != MSHQC_CD_FP16X3)
        return set_error(MSHQC_CD_ERR_ARG, "unknown precision");
    if (transform_needed(ctx, spin, precision)) CD_RC(run_transforms(ctx, 1, &spin, precision));
    if (precision == MSHQC_CD_FP16X3 && (!s.B16_valid || s.B16_layout != layout)) {
        begin_stage(ctx, ST_SPLIT);
        CD_RC(split_fixed(ctx, spin, layout));
        end_stage(ctx);
    }
    return MSHQC_CD_OK;
}

// Both spins: in one pass over the vectors where both need it and fit.
int ensure_transforms(mshqc_cd_ctx* ctx, int precision, int layout) {
    CD_RC(require_inputs(ctx, 0));
    CD_RC(require_inputs(ctx, 1));
    if ((precision == MSHQC_CD_FP64 || precision == MSHQC_CD_FP16X3) && transform_needed(ctx, 0, precision) &&
        transform_needed(ctx, 1, precision)) {
        bool fit = false;
        CD_RC(both_spins_fit(ctx, &fit));
        const int spins[2] = {0, 1};
        if (fit) CD_RC(run_transforms(ctx, 2, spins, precision));
    }
    for (int s = 0; s < 2; ++s) CD_RC(ensure_transform(ctx, s, precision, layout));
    return MSHQC_CD_OK;
}

int run_energy(mshqc_cd_ctx* ctx, int kind, int precision, mshqc_cd_energy* out) {
    std::memset(out, 0, sizeof(*out));
    ctx->fixed_point_exact = 1;
    reset_stages(ctx);
    CD_RC(require_inputs(ctx, 0));
    if (kind == MSHQC_CD_UNRESTRICTED) CD_RC(require_inputs(ctx, 1));
    cudaEvent_t e0 = ctx->ev[0], e1 = ctx->ev[1], e2 = ctx->ev[2];
    CD_RC(begin_call(ctx));
    CD_CUDA(cudaEventRecord(e0, ctx->stream));
    if (kind == MSHQC_CD_UNRESTRICTED)
        CD_RC(ensure_transforms(ctx, precision, 1));
    else
        CD_RC(ensure_transform(ctx, 0, precision, 1));
    CD_CUDA(cudaEventRecord(e1, ctx->stream));
    for (auto& p : ctx->pair_energy) p.clear();
    // the passes, their sums one after the other: one copy back at the end
    PairPass pass[3];
    int np = 0;
    int64_t copied = 0, sums = 0;
    auto add = [&](int mode, int sx, int sy) {
        PairPass& p = pass[np];
        p.mode = mode;
        p.sx = sx;
        p.sy = sy;
        p.ox = (int)ctx->spin[sx].nocc;
        p.oy = (int)ctx->spin[sy].nocc;
        p.npairs = (int)pair_count(mode, p.ox, p.oy);
        p.off = copied;
        p.total = np++;
        copied += p.npairs;
        sums = copied + (mode == PAIR_RESTRICTED ? p.npairs : 0);
    };
    if (kind == MSHQC_CD_RESTRICTED) {
        add(PAIR_RESTRICTED, 0, 0);
    } else {
        add(PAIR_SAME_SPIN, 0, 0);
        add(PAIR_SAME_SPIN, 1, 1);
        add(PAIR_OPPOSITE_SPIN, 0, 1);
    }
    CD_ALLOC(ctx->pair_sum, sizeof(double) * (size_t)std::max<int64_t>(1, sums), false);
    for (int k = 0; k < np; ++k)
        if (pass[k].npairs > 0)   // (no same-spin pair with one electron)
            CD_RC(precision == MSHQC_CD_FP16X3 ? pair_pass_tc(ctx, pass[k]) : pair_pass_f64(ctx, pass[k]));
    CD_CUDA(cudaEventRecord(e2, ctx->stream));
    CallStatus st;
    const void* hs = nullptr;
    CD_RC(finish_call(ctx, &st, ctx->pair_sum.p, sizeof(double) * (size_t)copied, &hs));
    collect_stages(ctx);
    for (int k = 0; k < np; ++k) {
        fill_pairs(pass[k], static_cast<const double*>(hs) + pass[k].off, ctx->pair_energy[k]);
        if (precision == MSHQC_CD_FP16X3 && pass[k].npairs > 0 && !pass_exact(ctx, pass[k])) ctx->fixed_point_exact = 0;
    }
    if (kind == MSHQC_CD_RESTRICTED) {
        out->total = st.totals[0];
        out->os = st.totals[1];
        out->ss_aa = out->ss_bb = 0.5 * (out->total - out->os);
    } else {
        out->ss_aa = st.totals[0];
        out->ss_bb = st.totals[1];
        out->os = st.totals[2];
        out->total = out->ss_aa + out->ss_bb + out->os;
    }
    float t01 = 0, t12 = 0;
    CD_CUDA(cudaEventElapsedTime(&t01, e0, e1));
    CD_CUDA(cudaEventElapsedTime(&t12, e1, e2));
    out->ms_transform = t01;
    out->ms_energy = t12;
    out->ms_total = t01 + t12;
    return MSHQC_CD_OK;
}

// ---------------------------------------------------------------------------
// backward
// ---------------------------------------------------------------------------
namespace {

// out[k] = (accumulate ? out[k] : 0) + alpha * sum_b parts[b * stride + k].
// HBM bound: 32 elements x 8 lanes of batches per CTA (lane g takes b = g, g + 8,
// ...; the lanes are added in order).  One thread per element walking all 1600
// batches of a 40 x 400 product left most SMs idle (190 us, now 20; N = 400, o = 40
// mixed transposed transforms 2.51 -> 2.34 ms).
__global__ void __launch_bounds__(256) sum_batches_kernel(const double* __restrict__ parts, int nb, int64_t stride,
                                                          int64_t n, double alpha, int accumulate,
                                                          double* __restrict__ out) {
    __shared__ double red[8][32];
    const int c = threadIdx.x & 31, g = threadIdx.x >> 5;
    const int64_t k = blockIdx.x * (int64_t)32 + c;
    double acc = 0.0;
    if (k < n) {
#pragma unroll 8
        for (int b = g; b < nb; b += 8) acc += parts[(int64_t)b * stride + k];
    }
    red[g][c] = acc;
    __syncthreads();
    if (g || k >= n) return;
    for (int h = 1; h < 8; ++h) acc += red[h][c];
    out[k] = accumulate ? out[k] + alpha * acc : alpha * acc;
}

int sum_batches(mshqc_cd_ctx* ctx, const double* parts, int nb, int64_t stride, int64_t n, double alpha,
                bool accumulate, double* out) {
    if (n <= 0) return MSHQC_CD_OK;
    sum_batches_kernel<<<(unsigned)cdiv(n, 32), 256, 0, ctx->stream>>>(parts, nb, stride, n, alpha,
                                                                         accumulate ? 1 : 0, out);
    CD_CUDA(cudaGetLastError());
    ctx->launches++;
    return MSHQC_CD_OK;
}

// dE/dC from Gamma (ctx->gam[spin], [o][vp][Mp] FP64) with dE/dB = scale * Gamma
// (4 restricted, 2 unrestricted):
//   dC[nu, o+a] = sum_{i,Q} dE/dB[i][a][Q] Y[i][Q][nu],
//   W[i][Q][nu] = sum_a dE/dB[i][a][Q] C[nu, o+a]      (into the rows of Y),
//   dC[mu, i]   = sum_{Q,nu} L[Q][nu][mu] W[i][Q][nu].
// The first two per spin here, the last for all spins at once in occupied_part.
// The transforms shared over ranks: rank r's Gamma rows [lo, hi) are completed
// by the reduce-scatter, and its transposed transforms cover those orbitals
// only (dC's other occupied columns zero); unshared: [0, o).
int virtual_part_f64(mshqc_cd_ctx* ctx, int spin, double scale, double* dC) {
    const SpinState& s = ctx->spin[spin];
    const int64_t N = ctx->N, M = ctx->M, Mp = ctx->Mp, o = s.nocc, v = N - o, vp = s.vp;
    const int64_t lo = ctx->Yr[spin].lo, ni = ctx->Yr[spin].hi - lo;
    const double* Gm = ctx->gam[spin].as<double>() + lo * vp * Mp;
    double* Y = y_rows(ctx, spin);
    ctx->Yr[spin].ok = false;   // W goes there
    // dC[nu, o+a] (row-major [a][nu] == column-major dC): one product over the
    // composite K = (i, Q); v x N output tiles alone leave most SMs idle at
    // small v
    GemmF64Args g{};
    g.M = (int)v;  g.N = (int)N;  g.K = (int)M;  g.batch = 1;
    g.kb = (int)ni;
    g.A = Gm;  g.lda = Mp;  g.skA = vp * Mp;
    g.B = Y;  g.ldb = N;  g.skB = M * N;
    g.C = dC + o * N;  g.ldc = N;  g.sC = 0;
    g.alpha = scale;  g.beta = 0.0;
    CD_RC(gemm_run(ctx, g, true, false));
    GemmF64Args w{};
    w.M = (int)M;  w.N = (int)N;  w.K = (int)v;  w.batch = (int)ni;
    w.A = Gm;  w.lda = Mp;  w.sA = vp * Mp;
    w.B = s.C.as<double>() + o * N;  w.ldb = N;  w.sB = 0;
    w.C = Y;  w.ldc = N;  w.sC = M * N;
    w.alpha = 1.0;  w.beta = 0.0;
    return gemm_run(ctx, w, false, false);
}

// The same on the int8 tensor cores, batched over orbitals i so that every
// product has K = M or v; the partial dC of the batches are summed in order.
template <class Cfg>
int virtual_part_i8(mshqc_cd_ctx* ctx, int spin, double scale, double* dC) {
    const SpinState& s = ctx->spin[spin];
    const int64_t N = ctx->N, M = ctx->M, Mp = ctx->Mp, o = s.nocc, v = N - o, vp = s.vp;
    const int64_t lo = ctx->Yr[spin].lo, hi = ctx->Yr[spin].hi, ni = hi - lo;
    const double* C = s.C.as<double>();
    const double* Gm = ctx->gam[spin].as<double>();
    double* Y = y_rows(ctx, spin);
    ctx->Yr[spin].ok = false;   // W goes there
    // dC[nu, o+a]: Gamma_i (rows a, K = Q) against Y_i^T (rows nu, K = Q, strided by N)
    {
        const bool sw = oz_swap<Cfg>(v, N);
        const size_t pa = oz_bytes<Cfg>(oz_operand<Cfg>(v, M, !sw, 1));
        const size_t pb = oz_bytes<Cfg>(oz_operand<Cfg>(N, M, sw, 1));
        const size_t pp = sizeof(double) * (size_t)(v * N);
        const int64_t ib = std::max<int64_t>(1, std::min<int64_t>(ni, (int64_t)(2 * kSliceBytes / (pa + pb + pp))));
        CD_ALLOC(ctx->oz_p, pp * ib, false);
        for (int64_t i0 = lo; i0 < hi; i0 += ib) {
            const int64_t nb = std::min(ib, hi - i0);
            OzakiOperand A = oz_operand<Cfg>(v, M, !sw, nb), B = oz_operand<Cfg>(N, M, sw, nb);
            CD_RC(oz_reserve<Cfg>(ctx, ctx->oz_a, ctx->oz_ea, pa * nb, A));
            CD_RC(oz_reserve<Cfg>(ctx, ctx->oz_b, ctx->oz_eb, pb * nb, B));
            CD_CUDA(ozaki_slice<Cfg>(Gm + i0 * vp * Mp, Mp, vp * Mp, A, ctx->num_sms, ctx->stream));
            CD_CUDA(ozaki_slice_t<Cfg>(Y + (i0 - lo) * M * N, N, M * N, B, ctx->stream));
            ctx->launches += 3;
            CD_RC(oz_mul<Cfg>(ctx, A, false, B, false, sw, ctx->oz_p.as<double>(), N, v * N, 1.0, 0.0));
            CD_RC(sum_batches(ctx, ctx->oz_p.as<double>(), (int)nb, v * N, v * N, scale, i0 > lo, dC + o * N));
        }
    }
    // W[i][Q][nu] into Y: Gamma_i^T (rows Q, K = a, strided by Mp) against
    // C_vir^T (rows nu, K = a, strided by N), shared
    {
        const bool sw = oz_swap<Cfg>(M, N);
        const size_t pa = oz_bytes<Cfg>(oz_operand<Cfg>(M, v, !sw, 1));
        const int64_t ib = std::max<int64_t>(1, std::min<int64_t>(ni, (int64_t)(kSliceBytes / pa)));
        OzakiOperand B = oz_operand<Cfg>(N, v, sw, 1);
        CD_RC(oz_reserve<Cfg>(ctx, ctx->oz_b, ctx->oz_eb, oz_bytes<Cfg>(B), B));
        CD_CUDA(ozaki_slice_t<Cfg>(C + o * N, N, 0, B, ctx->stream));
        ctx->launches += 2;
        for (int64_t i0 = lo; i0 < hi; i0 += ib) {
            const int64_t nb = std::min(ib, hi - i0);
            OzakiOperand A = oz_operand<Cfg>(M, v, !sw, nb);
            CD_RC(oz_reserve<Cfg>(ctx, ctx->oz_a, ctx->oz_ea, pa * nb, A));
            CD_CUDA(ozaki_slice_t<Cfg>(Gm + i0 * vp * Mp, Mp, vp * Mp, A, ctx->stream));
            ctx->launches += 2;
            CD_RC(oz_mul<Cfg>(ctx, A, false, B, true, sw, Y + (i0 - lo) * M * N, N, M * N, 1.0, 0.0));
        }
    }
    return MSHQC_CD_OK;
}

int virtual_part(mshqc_cd_ctx* ctx, int spin, double scale, double* dC, bool i8) {
    if (i8) return virtual_part_i8<ozaki::Mixed>(ctx, spin, scale, dC);
    const auto& y = ctx->Yr[spin];
    const int64_t v = ctx->N - ctx->spin[spin].nocc;
    const bool full = int8_transform_enabled(ctx) &&
                      fp64_slices(ctx, 2.0 * v * ctx->M * ctx->N * (y.hi - y.lo), kSlicedMinFlops, v);
    if (full) {   // N = 600, o = 60: the transposed transforms 12.8 -> 8.8 ms; N = 400, o = 40: 2.3 -> 1.9
        const int rc = virtual_part_i8<ozaki::Full>(ctx, spin, scale, dC);
        if (!no_room(ctx, rc)) return rc;
    }
    return virtual_part_f64(ctx, spin, scale, dC);
}

// dC[mu, i] = scale sum_{Q,nu} W[i][Q][nu] L[Q][nu][mu] for the W rows of the
// given spins (consecutive rows of Y, both spins in one product): over chunks of
// vectors, FP64 with K = (Q, nu), or per vector on the int8 tensor cores
// (W_Q rows i against L_Q rows mu, K = nu) with the partials summed in order.
// The rows of L_Q are contiguous when the vectors are symmetric (the same
// digits either way); otherwise they are sliced from the strided columns.
int occupied_part(mshqc_cd_ctx* ctx, int nsp, const int* spins, double scale, double* const* dC, bool i8) {
    using Cfg = ozaki::Mixed;
    const int64_t N = ctx->N, M = ctx->M;
    int64_t rows = 0, off[2] = {0, 0}, ni[2] = {0, 0};
    for (int k = 0; k < nsp; ++k) {
        const auto& y = ctx->Yr[spins[k]];
        off[k] = rows;
        ni[k] = y.hi - y.lo;
        rows += ni[k];
    }
    if (rows <= 0) return MSHQC_CD_OK;
    const double* W = y_rows(ctx, spins[0]);
    const int64_t qc = vectors_chunk_size(ctx);
    if (!i8) {
        double* out = dC[0] + ctx->Yr[spins[0]].lo * N;
        if (nsp == 2) {
            CD_ALLOC_FIRST(ctx->occ_parts, sizeof(double) * (size_t)(rows * N), false);
            out = ctx->occ_parts.as<double>();
        }
        for (int64_t Q0 = 0; Q0 < M; Q0 += qc) {
            const int64_t mc = std::min(qc, M - Q0);
            const double* Lc = nullptr;
            CD_RC(vectors_chunk(ctx, Q0, mc, &Lc));
            // only `rows` rows: K is what fills the GPU
            GemmF64Args g{};
            g.M = (int)rows;  g.N = (int)N;  g.K = (int)(mc * N);  g.batch = 1;
            g.A = W + Q0 * N;  g.lda = M * N;  g.sA = 0;
            g.B = Lc;  g.ldb = N;  g.sB = 0;
            g.C = out;  g.ldc = N;  g.sC = 0;
            g.alpha = scale;  g.beta = Q0 == 0 ? 0.0 : 1.0;
            CD_RC(gemm_run(ctx, g, true, false));
        }
        for (int k = 0; k < nsp && nsp == 2; ++k)
            if (ni[k] > 0)
                CD_CUDA(cudaMemcpyAsync(dC[k] + ctx->Yr[spins[k]].lo * N, out + off[k] * N,
                                        sizeof(double) * (size_t)(ni[k] * N), cudaMemcpyDeviceToDevice, ctx->stream));
        return MSHQC_CD_OK;
    }
    bool sym = false;
    CD_RC(vectors_symmetric(ctx, &sym));
    const bool sw = oz_swap<Cfg>(rows, N);
    const size_t pa = oz_bytes<Cfg>(oz_operand<Cfg>(rows, N, !sw, 1));
    const size_t pb = oz_bytes<Cfg>(oz_operand<Cfg>(N, N, sw, 1));
    const size_t pp = sizeof(double) * (size_t)(rows * N);
    const int64_t nq_max = std::max<int64_t>(1, (int64_t)(2 * kSliceBytes / (pa + pb + pp)));
    // (batches are a grid dimension of the slicing kernels)
    const int64_t nq = std::min<int64_t>(std::min(nq_max, qc), 65535);
    CD_ALLOC(ctx->oz_p, pp * nq, false);
    for (int64_t Q0 = 0; Q0 < M; Q0 += qc) {
        const int64_t mc = std::min(qc, M - Q0);
        const double* Lc = nullptr;
        CD_RC(vectors_chunk(ctx, Q0, mc, &Lc));
        for (int64_t q0 = 0; q0 < mc; q0 += nq) {
            const int64_t nb = std::min(nq, mc - q0);
            OzakiOperand A = oz_operand<Cfg>(rows, N, !sw, nb), B = oz_operand<Cfg>(N, N, sw, nb);
            CD_RC(oz_reserve<Cfg>(ctx, ctx->oz_a, ctx->oz_ea, pa * nb, A));
            CD_RC(oz_reserve<Cfg>(ctx, ctx->oz_b, ctx->oz_eb, pb * nb, B));
            CD_CUDA(ozaki_slice<Cfg>(W + (Q0 + q0) * N, M * N, N, A, ctx->num_sms, ctx->stream));
            if (sym)
                CD_CUDA(ozaki_slice<Cfg>(Lc + q0 * N * N, N, N * N, B, ctx->num_sms, ctx->stream));
            else
                CD_CUDA(ozaki_slice_t<Cfg>(Lc + q0 * N * N, N, N * N, B, ctx->stream));
            ctx->launches += sym ? 2 : 3;
            CD_RC(oz_mul<Cfg>(ctx, A, false, B, false, sw, ctx->oz_p.as<double>(), N, rows * N, 1.0, 0.0));
            for (int k = 0; k < nsp; ++k)
                CD_RC(sum_batches(ctx, ctx->oz_p.as<double>() + off[k] * N, (int)nb, rows * N, ni[k] * N, scale,
                                  Q0 + q0 > 0, dC[k] + ctx->Yr[spins[k]].lo * N));
        }
    }
    return MSHQC_CD_OK;
}

// The transposed transforms of the given spins.  Y of the orbitals is reused
// where the forward transforms left it; the open-shell int8 products take it
// from int8 slices always (the sizes whose forward transform is FP64 form it
// again).
int transposed_transforms(mshqc_cd_ctx* ctx, int nsp, const int* spins, double scale, double* const* dC, bool i8) {
    int64_t lo[2], hi[2];
    bool have = true;
    for (int k = 0; k < nsp; ++k) {
        const SpinState& s = ctx->spin[spins[k]];
        shard_range(ctx, s.nocc, &lo[k], &hi[k]);
        if (sharded(ctx))
            CD_RC(run_collective(ctx, false, ctx->gam[spins[k]].as<double>(),
                                 shard_p(ctx, s.nocc) * s.vp * ctx->Mp));
        if (hi[k] - lo[k] < s.nocc)
            CD_CUDA(cudaMemsetAsync(dC[k], 0, sizeof(double) * (size_t)(s.nocc * ctx->N), ctx->stream));
        if (hi[k] <= lo[k])
            CD_CUDA(cudaMemsetAsync(dC[k] + s.nocc * ctx->N, 0,
                                    sizeof(double) * (size_t)((ctx->N - s.nocc) * ctx->N), ctx->stream));
        const auto& y = ctx->Yr[spins[k]];
        have = have && y.ok && y.lo == lo[k] && y.hi == hi[k] && !(nsp == 2 && i8 && !y.i8);
    }
    if (!have) {
        bool fit = nsp == 1;
        if (nsp == 2) CD_RC(both_spins_fit(ctx, &fit));
        if (!fit) {   // one spin after the other
            for (int k = 0; k < nsp; ++k) {
                CD_RC(first_half(ctx, 1, &spins[k], &lo[k], &hi[k], i8));
                if (hi[k] <= lo[k]) continue;
                CD_RC(virtual_part(ctx, spins[k], scale, dC[k], i8));
                CD_RC(occupied_part(ctx, 1, &spins[k], scale, &dC[k], i8));
            }
            return MSHQC_CD_OK;
        }
        CD_RC(first_half(ctx, nsp, spins, lo, hi, i8));
    }
    for (int k = 0; k < nsp; ++k) {
        if (hi[k] <= lo[k]) continue;
        CD_RC(virtual_part(ctx, spins[k], scale, dC[k], i8));
    }
    return occupied_part(ctx, nsp, spins, scale, dC, i8);
}

// the int8 products for the mixed path (unless switched off), FP64 otherwise
int transposed_dispatch(mshqc_cd_ctx* ctx, int nsp, const int* spins, double scale, double* const* dC, int precision) {
    const bool i8 = precision == MSHQC_CD_FP16X3 && int8_transform_enabled(ctx);
    return transposed_transforms(ctx, nsp, spins, scale, dC, i8);
}

// ---------------------------------------------------------------------------
// backward building blocks (tensor-core and FP64 unrestricted passes)
// ---------------------------------------------------------------------------
struct BwdDims {
    int64_t o, v, vp;       // occupied, virtual, FP64 padding (64)
    int64_t RS;             // tensor-core staging and amplitude rows per orbital (32)
    int64_t VR;             // amplitude K per orbital (128)
    int64_t VS;             // columns per orbital the block sizes are reckoned with (256)
};

BwdDims bwd_dims(const mshqc_cd_ctx* ctx, int spin) {
    BwdDims d;
    d.o = ctx->spin[spin].nocc;
    d.v = ctx->N - d.o;
    d.vp = ctx->spin[spin].vp;
    d.RS = round_up(d.v, 32);
    d.VR = round_up(d.v, 128);
    d.VS = round_up(d.VR, 256);
    return d;
}

// Bytes a backward pass may stage: a third of the free memory (the staging it
// already holds included), at most 40 GB.  A pass of a small system whose
// staging is held already does not ask the driver (20 us).
int staging_budget(mshqc_cd_ctx* ctx, size_t held, double whole, size_t* budget) {
    *budget = size_t(40) << 30;
    if (whole <= (double)std::min<size_t>(held, size_t(256) << 20)) return MSHQC_CD_OK;
    size_t free_b = 0, total_b = 0;
    CD_CUDA(cudaMemGetInfo(&free_b, &total_b));
    *budget = std::min<size_t>((free_b + held) / 3, *budget);
    return MSHQC_CD_OK;
}

// BF16 hi/lo copy of one spin's MO vectors transposed to rows Q (RQ rows),
// K = (j, b) with b padded to VR: the B operand of the Gamma GEMM.
int make_bt(mshqc_cd_ctx* ctx, int spin, DevBuf& buf, int64_t RQ, const uint16_t** bt) {
    SpinState& s = ctx->spin[spin];
    const BwdDims d = bwd_dims(ctx, spin);
    const size_t nbt = (size_t)RQ * d.o * d.VR;
    CD_ALLOC_FIRST(buf, 2 * nbt * sizeof(uint16_t), false);
    const int64_t threads = (d.o * d.VR / 16) * RQ * 2;
    const int blocks = (int)std::min<int64_t>(cdiv(threads, 256), (int64_t)ctx->num_sms * 16);
    begin_stage(ctx, ST_SPLIT);
    bt_split_kernel<<<blocks, 256, 0, ctx->stream>>>(s.B64.as<double>(), s.vp, ctx->Mp, (int)d.v, (int)ctx->M,
                                                     d.o, d.VR, RQ, buf.as<uint16_t>());
    end_stage(ctx);
    CD_CUDA(cudaGetLastError());
    ctx->launches++;
    *bt = buf.as<uint16_t>();
    return MSHQC_CD_OK;
}

// gamma[(i0 + R / RS, R % RS)][Q] (+)= sum_K A[R][K] BT[Q][K] for R < rows;
// K in orbital groups of VRk (vk of them valid); a_rbs / b_rbs: K chunks per row
// block of A (128 rows) and of BT (256 rows), bt pointing at the first K chunk
// used
int launch_gamma(mshqc_cd_ctx* ctx, const uint16_t* amp, int64_t a_rbs, const uint16_t* bt, int64_t b_rbs, int64_t RQ,
                 int64_t K, int64_t VRk, int64_t vk, int64_t rows, int64_t RS, int64_t v, int64_t vp, int i0,
                 double* gamma, int accumulate) {
    GammaTcArgs g{};
    g.A = amp;  g.B = bt;
    g.a_rbs = a_rbs;  g.b_rbs = b_rbs;
    g.nk = (int)(K / 16);
    g.KP = 32;
    g.kg = (int)(VRk / 16);
    g.kv = (int)cdiv(vk, 16);
    g.nrb = (int)cdiv(rows, 128);
    g.nqb = (int)(RQ / 256);
    g.rows = rows;
    g.RS = (int)RS;  g.v = (int)v;  g.vp = (int)vp;  g.Mp = (int)ctx->Mp;  g.i0 = i0;
    g.gamma = gamma;
    g.err = ctx->status.as<CallStatus>()->gamma_err;
    g.accumulate = accumulate;
    const size_t gsm = gamma_tc::SMEM_BYTES;
    CD_CUDA(cudaFuncSetAttribute(gamma_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gsm));
    const int grid = (int)std::min<int64_t>((int64_t)g.nrb * g.nqb, ctx->num_sms);
    g.group = 16;
    if (const char* env = std::getenv("MSHQC_CD_GAMMA_GROUP")) g.group = std::max(1, std::atoi(env));
    pace_params(&g.pace_every, &g.pace_slack, "MSHQC_CD_PACE", true);
    if (g.pace_every > 0) {
        CD_ALLOC(ctx->pace, sizeof(int) * (size_t)grid, true);
        g.pace = ctx->pace.as<int>();
    }
    begin_stage(ctx, ST_GAMMA);
    gamma_tc_kernel<<<grid, gamma_tc::THREADS, gsm, ctx->stream>>>(g);
    end_stage(ctx);
    CD_CUDA(cudaGetLastError());
    ctx->launches++;
    return MSHQC_CD_OK;
}

// dE/de of one backward pass from its per-pair sums (amp_elem.cuh)
int reduce_deps(mshqc_cd_ctx* ctx, const double* prow, const double* pcol, const double* pocc, int64_t ox,
                int64_t oy, int64_t rsx, int64_t csy, int64_t vx, int64_t vy, double* deps_x, double* deps_y) {
    const int64_t npairs = ox * oy;
    if (prow) {   // (the symmetric modes keep row and column sums together)
        deps_rows_kernel<<<(unsigned)cdiv(vx, 16), 1024, 0, ctx->stream>>>(prow, npairs, (int)rsx, (int)vx,
                                                                           deps_x + ox);
        ctx->launches++;
    }
    deps_rows_kernel<<<(unsigned)cdiv(vy, 16), 1024, 0, ctx->stream>>>(pcol, npairs, (int)csy, (int)vy,
                                                                       deps_y + oy);
    deps_occ_kernel<<<(unsigned)cdiv(std::max(ox, oy), 128), 128, 0, ctx->stream>>>(pocc, (int)ox, (int)oy,
                                                                                    deps_x, deps_y);
    CD_CUDA(cudaGetLastError());
    ctx->launches += 2;
    return MSHQC_CD_OK;
}

// One mixed-precision backward pass over block pairs (I, J): rows i in I of
// spin sx, columns j in J of spin sy.  Per block pair: (ia|jb) tiles on the
// tensor cores (exact fixed point, FP32 staging), the element-wise amplitude
// pass, Gamma_sx[I] += amplitudes x B_sy[J] and, when `mirror`, the transposed
// amplitudes update Gamma_sy[J] += amplitudes^T x B_sx[I].
//  * same spin / restricted: blocks of b orbitals, I <= J only.  The amplitude
//    of pair (j, i) is the transpose of that of (i, j) (t^{ji}_{ba} =
//    t^{ij}_{ab}), so off-diagonal pairs are computed once and count twice;
//    this halves the integral tiles and the element-wise pass.
//  * opposite spin: row blocks I against all beta columns (no symmetry).
// Energies go to `partial` (ox * oy, one per ordered pair, zero where a
// mirrored pair stands in), dE/de to deps_x / deps_y.
template <int MODE>
int tc_backward_pass(mshqc_cd_ctx* ctx, int sx, int sy, const uint16_t* btx, const uint16_t* bty, int64_t RQ,
                     double* deps_x, double* deps_y, double* partial) {
    constexpr bool kSym = MODE != AMP_OPPOSITE_SPIN;
    SpinState& X = ctx->spin[sx];
    SpinState& Y = ctx->spin[sy];
    const BwdDims dx = bwd_dims(ctx, sx), dy = bwd_dims(ctx, sy);
    const int64_t Mp = ctx->Mp;
    // the staging this pass reuses counts as available, so that the block size
    // of a repeated call does not shrink because the previous call holds it
    size_t budget = 0;
    CD_RC(staging_budget(ctx, ctx->amp.bytes + ctx->ampT.bytes + ctx->W.bytes,
                         (double)(dx.o * dx.VR) * (double)dy.o * (4.0 * dy.VS + 8.0 * dy.VR), &budget));
    // block sizes: rows bI, columns bJ (all of them for the opposite spin)
    int64_t bI, bJ;
    tc_block_sizes(ctx, dx.o, dy.o, dx.VR, dy.VR, dy.VS, kSym, budget, &bI, &bJ);
    const size_t n_amp = sizeof(uint16_t) * (size_t)(bI * dx.VR) * (size_t)(bJ * dy.VR);
    CD_ALLOC_FIRST(ctx->amp, 2 * n_amp, false);   // hi and lo
    CD_ALLOC_FIRST(ctx->ampT, 2 * n_amp, false);
    // (the size the block sizes are reckoned with; the packed rows take less of it)
    CD_ALLOC_FIRST(ctx->W, sizeof(float) * (size_t)(bI * dx.VR) * (size_t)(bJ * dy.VS), false);
    const int64_t npairs = dx.o * dy.o;
    // (zero where a mirrored pair stands in)
    const int64_t nrow = kSym ? 0 : dx.RS;
    CD_ALLOC_FIRST(ctx->dsum, sizeof(double) * (size_t)(npairs * (nrow + dy.RS + 1)), true);
    CD_CUDA(cudaMemsetAsync(partial, 0, sizeof(double) * (size_t)npairs, ctx->stream));
    double* pcol = ctx->dsum.as<double>();
    double* pocc = pcol + npairs * dy.RS;
    double* prow = kSym ? nullptr : pocc + npairs;
    if (X.B16_layout != 0 || Y.B16_layout != 0)
        return set_error(MSHQC_CD_ERR_STATE, "fixed-point operands not in the integral-tile layout");
    const size_t vsm = vtile_tc::SMEM_BYTES;
    CD_CUDA(cudaFuncSetAttribute(vtile_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)vsm));
    for (int64_t I0 = 0; I0 < dx.o; I0 += bI) {
        const int nI = (int)std::min<int64_t>(bI, dx.o - I0);
        for (int64_t J0 = kSym ? I0 : 0; J0 < dy.o; J0 += bJ) {
            if (!owns_next(ctx)) continue;
            const int nJ = (int)std::min<int64_t>(bJ, dy.o - J0);
            const bool mirror = !kSym || J0 != I0;
            // a diagonal block pair computes its pairs i <= j only; the
            // element-wise pass writes the (j, i) amplitudes as transposes
            const bool tri = kSym && J0 == I0;
            const int npl = tri ? nI * (nI + 1) / 2 : nI * nJ;
            VtileArgs a{};
            a.X = X.B16.as<uint16_t>();
            a.Y = Y.B16.as<uint16_t>();
            a.ex = X.expo.as<int>();  a.ey = Y.expo.as<int>();
            a.diag = sx == sy ? X.diag.as<double>() : nullptr;
            a.RSx = (int)dx.RS;  a.RSy = (int)dy.RS;
            a.nqc = (int)(Mp / 16);
            a.vx = (int)dx.v;  a.vy = (int)dy.v;
            a.r0 = I0 * dx.RS;  a.r1 = (I0 + nI) * dx.RS;
            a.c0 = J0 * dy.RS;  a.c1 = (J0 + nJ) * dy.RS;
            a.ldS = nJ * dy.RS;
            a.rb0 = (int)(a.r0 / 128);  a.nrb = (int)cdiv(a.r1, 128) - a.rb0;
            a.cb0 = (int)(a.c0 / 256);  a.ncb = (int)cdiv(a.c1, 256) - a.cb0;
            a.group = 12;
            a.S = ctx->W.as<float>();
            a.err = ctx->status.as<CallStatus>()->tile_err;
            a.tri = tri ? 1 : 0;
            const int64_t vunits = (int64_t)a.nrb * a.ncb;
            const int vgrid = (int)std::min<int64_t>(vunits, ctx->num_sms);
            pace_params(&a.pace_every, &a.pace_slack, "MSHQC_CD_PACE_TILES", false);
            if (a.pace_every > 0) {
                CD_ALLOC(ctx->pace, sizeof(int) * (size_t)vgrid, true);
                a.pace = ctx->pace.as<int>();
            }
            begin_stage(ctx, ST_AMPLITUDE);
            vtile_tc_kernel<<<vgrid, vtile_tc::THREADS, vsm, ctx->stream>>>(a);
            end_stage(ctx);
            CD_CUDA(cudaGetLastError());
            ctx->launches++;
            AmpElemArgs e{};
            e.S = ctx->W.as<float>();
            e.ldS = (long long)nJ * dy.RS;
            e.rsx = (int)dx.RS;  e.csy = (int)dy.RS;  e.ksy = (int)dy.VR;  e.ksx = (int)dx.VR;
            e.ox = (int)dx.o;  e.oy = (int)dy.o;  e.vx = (int)dx.v;  e.vy = (int)dy.v;
            e.i0 = (int)I0;  e.nbi = nI;  e.j0 = (int)J0;  e.nbj = nJ;
            e.wgt = (kSym && mirror) ? 2.0 : 1.0;
            e.eox = X.eps.as<double>();  e.evx = e.eox + dx.o;
            e.eoy = Y.eps.as<double>();  e.evy = e.eoy + dy.o;
            e.A16 = ctx->amp.as<uint16_t>();
            e.nkA = (long long)nJ * dy.VR / 16;
            if (mirror) {
                e.T16 = ctx->ampT.as<uint16_t>();
                e.nkT = (long long)nI * dx.VR / 16;
            } else if (tri) {
                e.T16 = e.A16;  e.nkT = e.nkA;
                e.tri = 1;
            }
            e.partial = partial;
            e.prow = prow;  e.pcol = pcol;  e.pocc = pocc;
            // split each pair's row tiles over several CTAs when the block
            // pair alone does not fill the GPU several times over
            const int ta = (int)(dx.RS / 32) * (kSym ? (int)(dx.RS / 32) + 1 : 2) / 2;   // tile pairs, or tile rows
            int nch = 1;
            while (nch < 16 && 2 * nch <= ta && (int64_t)npl * nch < 8LL * ctx->num_sms) nch *= 2;
            e.nchunk = nch;
            if (nch > 1) {
                const size_t per = (size_t)npl * nch;
                CD_ALLOC_FIRST(ctx->amp_chunks, sizeof(double) * per * ((size_t)dy.RS + 2), false);
                e.cpcol = ctx->amp_chunks.as<double>();
                e.cpart = e.cpcol + per * dy.RS;
                e.cpocc = e.cpart + per;
            }
            begin_stage(ctx, ST_AMP_ELEM);
            launch_amp<MODE, true>(e, npl * nch, ctx->stream);
            CD_CUDA(cudaGetLastError());
            ctx->launches++;
            if (nch > 1) {
                amp_chunks_combine_kernel<<<(unsigned)cdiv((int64_t)npl * dy.RS, 256), 256, 0, ctx->stream>>>(e, npl);
                CD_CUDA(cudaGetLastError());
                ctx->launches++;
            }
            end_stage(ctx);
            // Gamma_sx[I] += A x B_sy[J]  (K range of J inside the transposed B of spin sy)
            // first K chunk of block J (I) inside a 256-row block of BT
            const size_t kJ = (size_t)J0 * dy.VR / 16 * 8192, kI = (size_t)I0 * dx.VR / 16 * 8192;
            const int64_t nkBy = dy.o * dy.VR / 16, nkBx = dx.o * dx.VR / 16;
            CD_RC(launch_gamma(ctx, e.A16, e.nkA, bty + kJ, nkBy, RQ, (int64_t)nJ * dy.VR, dy.VR,
                               dy.v, (int64_t)nI * dx.RS, dx.RS, dx.v, dx.vp, (int)I0, ctx->gam[sx].as<double>(), 1));
            if (mirror) {
                // Gamma_sy[J] += A^T x B_sx[I]
                CD_RC(launch_gamma(ctx, e.T16, e.nkT, btx + kI, nkBx, RQ,
                                   (int64_t)nI * dx.VR, dx.VR, dx.v, (int64_t)nJ * dy.RS, dy.RS, dy.v, dy.vp, (int)J0,
                                   ctx->gam[sy].as<double>(), 1));
            }
        }
    }
    CD_RC(reduce_deps(ctx, prow, pcol, pocc, dx.o, dy.o, dx.RS, dy.RS, dx.v, dy.v, deps_x, deps_y));
    return MSHQC_CD_OK;
}

// The FP64 counterpart of tc_backward_pass, over the same block pairs: S =
// B_x[I] B_y[J]^T and the Gamma products around the element-wise pass, as int8
// slices of full accuracy (larger block pairs) or FP64 DMMA GEMMs.  A diagonal block pair of the symmetric modes forms S
// for j >= i only (GemmF64Args::tri), and the element-wise pass completes the
// amplitude block with the transposes.
template <int MODE>
int f64_backward_pass(mshqc_cd_ctx* ctx, int sx, int sy, double* deps_x, double* deps_y, double* partial) {
    constexpr bool kSym = MODE != AMP_OPPOSITE_SPIN;
    SpinState& X = ctx->spin[sx];
    SpinState& Y = ctx->spin[sy];
    const BwdDims dx = bwd_dims(ctx, sx), dy = bwd_dims(ctx, sy);
    const int64_t Mp = ctx->Mp;
    size_t budget = 0;
    CD_RC(staging_budget(ctx, ctx->amp.bytes + ctx->W.bytes,
                         2.0 * sizeof(double) * (double)(dx.o * dx.vp) * (double)(dy.o * dy.vp), &budget));
    int64_t bI, bJ;
    f64_block_sizes(ctx, dx.o, dy.o, dx.vp, dy.vp, kSym, budget, &bI, &bJ);
    const size_t n_stage = sizeof(double) * (size_t)(bI * dx.vp) * (size_t)(bJ * dy.vp);
    CD_ALLOC_FIRST(ctx->W, n_stage, false);
    CD_ALLOC_FIRST(ctx->amp, n_stage, false);
    const int64_t npairs = dx.o * dy.o;
    // (zero where a mirrored pair stands in)
    const int64_t nrow = kSym ? 0 : dx.vp;
    CD_ALLOC_FIRST(ctx->dsum, sizeof(double) * (size_t)(npairs * (nrow + dy.vp + 1)), true);
    CD_CUDA(cudaMemsetAsync(partial, 0, sizeof(double) * (size_t)npairs, ctx->stream));
    double* pcol = ctx->dsum.as<double>();
    double* pocc = pcol + npairs * dy.vp;
    double* prow = kSym ? nullptr : pocc + npairs;
    double* S = ctx->W.as<double>();
    double* A = ctx->amp.as<double>();
    for (int64_t I0 = 0; I0 < dx.o; I0 += bI) {
        const int nI = (int)std::min<int64_t>(bI, dx.o - I0);
        const double* XI = X.B64.as<double>() + I0 * dx.vp * Mp;
        for (int64_t J0 = kSym ? I0 : 0; J0 < dy.o; J0 += bJ) {
            if (!owns_next(ctx)) continue;
            const int nJ = (int)std::min<int64_t>(bJ, dy.o - J0);
            const bool mirror = !kSym || J0 != I0;
            const bool tri = kSym && J0 == I0;
            const int npl = tri ? nI * (nI + 1) / 2 : nI * nJ;
            const int64_t ldS = (int64_t)nJ * dy.vp;
            const double* YJ = Y.B64.as<double>() + J0 * dy.vp * Mp;
            // S[(i,a)][(j,b)] = sum_Q X[(i,a)][Q] Y[(j,b)][Q]
            bool sliced = sliced_pairs(ctx, nI * dx.vp, ldS);
            begin_stage(ctx, ST_AMPLITUDE);
            if (sliced) {
                const int rc = sliced_integrals(ctx, X, Y, I0, nI, J0, nJ, tri, S);
                sliced = !no_room(ctx, rc);
                if (sliced) CD_RC(rc);
            }
            if (!sliced) {
                GemmF64Args g{};
                g.M = (int)(nI * dx.vp);  g.N = (int)ldS;  g.K = (int)Mp;  g.batch = 1;
                g.A = XI;  g.lda = Mp;  g.sA = 0;
                g.B = YJ;  g.ldb = Mp;  g.sB = 0;
                g.C = S;  g.ldc = ldS;  g.sC = 0;
                g.alpha = 1.0;  g.beta = 0.0;
                g.tri = tri ? (int)dx.vp : 0;
                CD_RC(gemm_run(ctx, g, true, true));
            }
            end_stage(ctx);
            AmpElemArgs e{};
            e.S = S;
            e.ldS = ldS;
            e.rsx = (int)dx.vp;  e.csy = (int)dy.vp;  e.ksy = (int)dy.vp;  e.ksx = (int)dx.vp;
            e.ox = (int)dx.o;  e.oy = (int)dy.o;  e.vx = (int)dx.v;  e.vy = (int)dy.v;
            e.i0 = (int)I0;  e.nbi = nI;  e.j0 = (int)J0;  e.nbj = nJ;
            e.wgt = (kSym && mirror) ? 2.0 : 1.0;
            e.tri = tri ? 1 : 0;
            e.eox = X.eps.as<double>();  e.evx = e.eox + dx.o;
            e.eoy = Y.eps.as<double>();  e.evy = e.eoy + dy.o;
            e.A64 = A;  e.ldA = ldS;
            e.partial = partial;
            e.prow = prow;  e.pcol = pcol;  e.pocc = pocc;
            const int ta = (int)(dx.vp / 32) * (kSym ? (int)(dx.vp / 32) + 1 : 2) / 2;   // tile pairs, or tile rows
            int nch = 1;
            while (nch < 16 && 2 * nch <= ta && (int64_t)npl * nch < 8LL * ctx->num_sms) nch *= 2;
            e.nchunk = nch;
            if (nch > 1) {
                const size_t per = (size_t)npl * nch;
                CD_ALLOC_FIRST(ctx->amp_chunks, sizeof(double) * per * ((size_t)dy.vp + 2), false);
                e.cpcol = ctx->amp_chunks.as<double>();
                e.cpart = e.cpcol + per * dy.vp;
                e.cpocc = e.cpart + per;
            }
            begin_stage(ctx, ST_AMP_ELEM);
            launch_amp<MODE, false>(e, npl * nch, ctx->stream);
            CD_CUDA(cudaGetLastError());
            ctx->launches++;
            if (nch > 1) {
                amp_chunks_combine_kernel<<<(unsigned)cdiv((int64_t)npl * dy.vp, 256), 256, 0, ctx->stream>>>(e, npl);
                CD_CUDA(cudaGetLastError());
                ctx->launches++;
            }
            end_stage(ctx);
            begin_stage(ctx, ST_GAMMA);
            double* gx = ctx->gam[sx].as<double>() + I0 * dx.vp * Mp;
            double* gy = ctx->gam[sy].as<double>() + J0 * dy.vp * Mp;
            // the staged integrals are used up: their block takes the slices
            bool todo_x = true, todo_y = mirror;
            if (sliced) {
                int rc = sliced_gamma(ctx, A, ldS, false, nI * dx.vp, ldS, YJ, gx, ctx->W);
                todo_x = no_room(ctx, rc);
                if (!todo_x) CD_RC(rc);
                if (mirror && !todo_x) {
                    rc = sliced_gamma(ctx, A, ldS, true, ldS, nI * dx.vp, XI, gy, ctx->W);
                    todo_y = no_room(ctx, rc);
                    if (!todo_y) CD_RC(rc);
                }
                CD_ALLOC_FIRST(ctx->W, n_stage, false);
                S = ctx->W.as<double>();
            }
            if (todo_x) {
                // Gamma_x[(i,a)][Q] += sum_{(j,b) in J} t[(i,a)][(j,b)] Y[(j,b)][Q]
                GemmF64Args h{};
                h.M = (int)(nI * dx.vp);  h.N = (int)Mp;  h.K = (int)ldS;  h.batch = 1;
                h.A = A;  h.lda = ldS;  h.sA = 0;
                h.B = YJ;  h.ldb = Mp;  h.sB = 0;
                h.C = gx;  h.ldc = Mp;  h.sC = 0;
                h.alpha = 1.0;  h.beta = 1.0;
                CD_RC(gemm_run(ctx, h, true, false));
            }
            if (todo_y) {
                // Gamma_y[(j,b)][Q] += sum_{(i,a) in I} t[(i,a)][(j,b)] X[(i,a)][Q]
                GemmF64Args k{};
                k.M = (int)ldS;  k.N = (int)Mp;  k.K = (int)(nI * dx.vp);  k.batch = 1;
                k.A = A;  k.lda = ldS;  k.sA = 0;
                k.B = XI;  k.ldb = Mp;  k.sB = 0;
                k.C = gy;  k.ldc = Mp;  k.sC = 0;
                k.alpha = 1.0;  k.beta = 1.0;
                CD_RC(gemm_run(ctx, k, false, false));
            }
            end_stage(ctx);
        }
    }
    CD_RC(reduce_deps(ctx, prow, pcol, pocc, dx.o, dy.o, dx.vp, dy.vp, dx.v, dy.v, deps_x, deps_y));
    return MSHQC_CD_OK;
}

// The gradients below only queue work: energies and error flags come back with
// the call's status.  One total per pass from its per-pair energies:
int queue_total(mshqc_cd_ctx* ctx, const double* pairs, int64_t n, int k) {
    reduce_total_kernel<<<1, 256, 0, ctx->stream>>>(pairs, (int)n, ctx->status.as<CallStatus>()->totals + k);
    CD_CUDA(cudaGetLastError());
    ctx->launches++;
    return MSHQC_CD_OK;
}

// Restricted gradient: one pass over block pairs (FP64 or tensor cores), then
// the transposed half transforms with dE/dB = 4 Gamma.
int gradient_restricted(mshqc_cd_ctx* ctx, int precision, double* dC, double* deps) {
    SpinState& s = ctx->spin[0];
    const int64_t N = ctx->N, Mp = ctx->Mp, RQ = round_up(ctx->M, 256), o = s.nocc;
    const bool tc = precision == MSHQC_CD_FP16X3;
    const uint16_t* bt = nullptr;
    if (tc) CD_RC(make_bt(ctx, 0, ctx->BT, RQ, &bt));
    CD_ALLOC_FIRST(ctx->gam[0], sizeof(double) * (size_t)b_rows(ctx, o) * s.vp * Mp, true);
    CD_CUDA(cudaMemsetAsync(deps, 0, sizeof(double) * N, ctx->stream));
    CD_ALLOC_FIRST(ctx->partial, sizeof(double) * (size_t)(o * o), false);   // one energy per pair (i, j)
    double* part = ctx->partial.as<double>();
    if (tc)
        CD_RC(tc_backward_pass<AMP_RESTRICTED>(ctx, 0, 0, bt, bt, RQ, deps, deps, part));
    else
        CD_RC(f64_backward_pass<AMP_RESTRICTED>(ctx, 0, 0, deps, deps, part));
    CD_RC(queue_total(ctx, part, o * o, 0));
    begin_stage(ctx, ST_TRANSPOSED);
    const int spins[1] = {0};
    CD_RC(transposed_dispatch(ctx, 1, spins, 4.0, &dC, precision));
    end_stage(ctx);
    return MSHQC_CD_OK;
}

// Unrestricted gradient (CD-UMP2 energy, the OMP2 step): same-spin passes for
// alpha and beta and one opposite-spin pass, Gamma accumulated per spin, then
// the transposed transforms with dE/dB = 2 Gamma.  Totals: ss_aa, ss_bb, os.
int gradient_unrestricted(mshqc_cd_ctx* ctx, int precision, double* const dC[2], double* const deps[2]) {
    const BwdDims da = bwd_dims(ctx, 0), db = bwd_dims(ctx, 1);
    const int64_t N = ctx->N, Mp = ctx->Mp, RQ = round_up(ctx->M, 256);
    const bool tc = precision == MSHQC_CD_FP16X3;
    const uint16_t *bta = nullptr, *btb = nullptr;
    if (tc) {
        CD_RC(make_bt(ctx, 0, ctx->BT, RQ, &bta));
        CD_RC(make_bt(ctx, 1, ctx->BT_b, RQ, &btb));
    }
    CD_ALLOC_FIRST(ctx->gam[0], sizeof(double) * (size_t)b_rows(ctx, da.o) * da.vp * Mp, true);
    CD_ALLOC_FIRST(ctx->gam[1], sizeof(double) * (size_t)b_rows(ctx, db.o) * db.vp * Mp, true);
    for (int s = 0; s < 2; ++s) CD_CUDA(cudaMemsetAsync(deps[s], 0, sizeof(double) * N, ctx->stream));
    const int64_t n0 = da.o * da.o, n1 = db.o * db.o, n2 = da.o * db.o;   // one energy per pair
    CD_ALLOC_FIRST(ctx->partial, sizeof(double) * (size_t)(n0 + n1 + n2), false);
    double* part = ctx->partial.as<double>();
    if (tc) {
        CD_RC(tc_backward_pass<AMP_SAME_SPIN>(ctx, 0, 0, bta, bta, RQ, deps[0], deps[0], part));
        CD_RC(tc_backward_pass<AMP_SAME_SPIN>(ctx, 1, 1, btb, btb, RQ, deps[1], deps[1], part + n0));
        CD_RC(tc_backward_pass<AMP_OPPOSITE_SPIN>(ctx, 0, 1, bta, btb, RQ, deps[0], deps[1], part + n0 + n1));
    } else {
        CD_RC(f64_backward_pass<AMP_SAME_SPIN>(ctx, 0, 0, deps[0], deps[0], part));
        CD_RC(f64_backward_pass<AMP_SAME_SPIN>(ctx, 1, 1, deps[1], deps[1], part + n0));
        CD_RC(f64_backward_pass<AMP_OPPOSITE_SPIN>(ctx, 0, 1, deps[0], deps[1], part + n0 + n1));
    }
    CD_RC(queue_total(ctx, part, n0, 0));
    CD_RC(queue_total(ctx, part + n0, n1, 1));
    CD_RC(queue_total(ctx, part + n0 + n1, n2, 2));
    begin_stage(ctx, ST_TRANSPOSED);
    const int spins[2] = {0, 1};
    CD_RC(transposed_dispatch(ctx, 2, spins, 2.0, dC, precision));
    end_stage(ctx);
    return MSHQC_CD_OK;
}

// The shares of a partitioned gradient call.  Enumerates the backward's units
// in the order the passes visit them, with the partitioned block sizes (a
// function of the dimensions and the rank count only), weighs each by its
// tensor-core or DMMA work (integral tiles + Gamma products, in (i, j) pair
// units: a diagonal block pair has no mirrored Gamma product), and deals them
// out longest first to the least-loaded rank (ties to the lower rank).  Every
// rank computes the same plan and keeps its own units.
int plan_partition(mshqc_cd_ctx* ctx, int kind, int precision) {
    std::vector<double> cost;
    const bool unres = kind == MSHQC_CD_UNRESTRICTED;
    auto tc_pass = [&](int sx, int sy, bool sym) {
        const BwdDims dx = bwd_dims(ctx, sx), dy = bwd_dims(ctx, sy);
        int64_t bI, bJ;
        tc_block_sizes(ctx, dx.o, dy.o, dx.VR, dy.VR, dy.VS, sym, 0, &bI, &bJ);
        for (int64_t I0 = 0; I0 < dx.o; I0 += bI) {
            const int64_t nI = std::min(bI, dx.o - I0);
            for (int64_t J0 = sym ? I0 : 0; J0 < dy.o; J0 += bJ) {
                const int64_t nJ = std::min(bJ, dy.o - J0);
                // integral tiles of the pairs computed + Gamma products
                if (sym && J0 == I0)
                    cost.push_back(0.5 * (double)nI * (nI + 1) + (double)nI * nI);
                else
                    cost.push_back(3.0 * nI * nJ);
            }
        }
    };
    // the FP64 passes visit the same kind of units; per block pair: S GEMM
    // (half of it on a diagonal block pair) + Gamma products
    auto f64_pass = [&](int sx, int sy, bool sym) {
        const BwdDims dx = bwd_dims(ctx, sx), dy = bwd_dims(ctx, sy);
        int64_t bI, bJ;
        f64_block_sizes(ctx, dx.o, dy.o, dx.vp, dy.vp, sym, 0, &bI, &bJ);
        for (int64_t I0 = 0; I0 < dx.o; I0 += bI) {
            const int64_t nI = std::min(bI, dx.o - I0);
            for (int64_t J0 = sym ? I0 : 0; J0 < dy.o; J0 += bJ) {
                const int64_t nJ = std::min(bJ, dy.o - J0);
                if (sym && J0 == I0)
                    cost.push_back(0.5 * (double)nI * (nI + 1) + (double)nI * nI);
                else
                    cost.push_back(3.0 * nI * nJ);
            }
        }
    };
    if (!unres && precision == MSHQC_CD_FP64) {
        f64_pass(0, 0, true);
    } else if (!unres) {
        tc_pass(0, 0, true);
    } else if (precision == MSHQC_CD_FP16X3) {
        tc_pass(0, 0, true);
        tc_pass(1, 1, true);
        tc_pass(0, 1, false);
    } else {
        f64_pass(0, 0, true);
        f64_pass(1, 1, true);
        f64_pass(0, 1, false);
    }
    std::vector<size_t> order(cost.size());
    for (size_t k = 0; k < order.size(); ++k) order[k] = k;
    std::stable_sort(order.begin(), order.end(), [&](size_t a, size_t b) { return cost[a] > cost[b]; });
    std::vector<double> load((size_t)ctx->part_size, 0.0);
    ctx->part_owned.assign(cost.size(), 0);
    for (size_t k : order) {
        const size_t r = (size_t)(std::min_element(load.begin(), load.end()) - load.begin());
        load[r] += cost[k];
        if ((int)r == ctx->part_rank) ctx->part_owned[k] = 1;
    }
    return MSHQC_CD_OK;
}

}  // namespace

int run_gradient(mshqc_cd_ctx* ctx, int kind, int precision, mshqc_cd_energy* e_out, double* dC_a,
                 double* dC_b, double* deps_a, double* deps_b, int where) {
    if (kind != MSHQC_CD_RESTRICTED && kind != MSHQC_CD_UNRESTRICTED)
        return set_error(MSHQC_CD_ERR_ARG, "unknown kind");
    const bool unres = kind == MSHQC_CD_UNRESTRICTED;
    CD_RC(require_inputs(ctx, 0));
    if (unres) CD_RC(require_inputs(ctx, 1));
    const int64_t N = ctx->N;
    // the partition applies to this call's backward only
    struct PartitionScope {
        mshqc_cd_ctx* c;
        explicit PartitionScope(mshqc_cd_ctx* x) : c(x) { c->part_active = c->part_size > 1; c->part_next = 0; }
        ~PartitionScope() { c->part_active = false; }
    } part_scope(ctx);
    cudaEvent_t e0 = ctx->ev[0], e1 = ctx->ev[1], e2 = ctx->ev[2];
    reset_stages(ctx);
    CD_RC(begin_call(ctx));
    CD_CUDA(cudaEventRecord(e0, ctx->stream));
    if (unres)
        CD_RC(ensure_transforms(ctx, precision));
    else
        CD_RC(ensure_transform(ctx, 0, precision));
    CD_CUDA(cudaEventRecord(e1, ctx->stream));
    if (ctx->part_active) CD_RC(plan_partition(ctx, kind, precision));
    double* dC[2] = {nullptr, nullptr};
    double* de[2] = {nullptr, nullptr};
    for (int s = 0; s < (unres ? 2 : 1); ++s) {
        CD_ALLOC_FIRST(ctx->grad[s], sizeof(double) * (size_t)(N * N + N), false);
        dC[s] = ctx->grad[s].as<double>();
        de[s] = dC[s] + N * N;
    }
    ctx->fixed_point_exact = 1;
    CD_RC(unres ? gradient_unrestricted(ctx, precision, dC, de) : gradient_restricted(ctx, precision, dC[0], de[0]));
    if (ctx->part_active && ctx->part_next != (int64_t)ctx->part_owned.size())
        return set_error(MSHQC_CD_ERR_STATE, "partition plan covers " + std::to_string(ctx->part_owned.size()) +
                                                 " units, the backward visited " + std::to_string(ctx->part_next));
    CD_CUDA(cudaEventRecord(e2, ctx->stream));
    const cudaMemcpyKind dir = where == MSHQC_CD_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
    double* out_c[2] = {dC_a, dC_b};
    double* out_e[2] = {deps_a, deps_b};
    for (int s = 0; s < (unres ? 2 : 1); ++s) {
        if (out_c[s]) CD_CUDA(cudaMemcpyAsync(out_c[s], dC[s], sizeof(double) * N * N, dir, ctx->stream));
        if (out_e[s]) CD_CUDA(cudaMemcpyAsync(out_e[s], de[s], sizeof(double) * N, dir, ctx->stream));
    }
    CallStatus st;
    CD_RC(finish_call(ctx, &st));
    collect_stages(ctx);
    if (st.tile_err[1]) ctx->fixed_point_exact = 0;
    if (e_out) {
        std::memset(e_out, 0, sizeof(*e_out));
        e_out->total = unres ? st.totals[0] + st.totals[1] + st.totals[2] : st.totals[0];
        if (unres) {
            e_out->ss_aa = st.totals[0];
            e_out->ss_bb = st.totals[1];
            e_out->os = st.totals[2];
        }
        float t01 = 0, t12 = 0;
        CD_CUDA(cudaEventElapsedTime(&t01, e0, e1));
        CD_CUDA(cudaEventElapsedTime(&t12, e1, e2));
        e_out->ms_transform = t01;
        e_out->ms_energy = t12;
        e_out->ms_total = t01 + t12;
    }
    return MSHQC_CD_OK;
}

}  // namespace mshqc_cd

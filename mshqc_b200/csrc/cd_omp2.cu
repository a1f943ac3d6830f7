// CD-OMP2 on the GPU: one gradient evaluation of CholeskyOMP2::compute
// (reference src/mp2/cholesky_omp2.cc:442-466) and its orbital-rotation loop
// (:375-424, :427-512), FP64 throughout.
//
// Amplitudes: the same-spin t = ((ia|jb) - (ib|ja))/D and opposite-spin
// t = (ia|jb)/D of the reference (:94-183) are formed block by block (rows i
// of one block, every j) by an FP64 GEMM and the element-wise pass of
// amp_elem.cuh; nothing of size o^2 v^2 is ever held.  Each amplitude block
// A[(i,a)][(j,b)] feeds the one-particle density (:232-326) through two
// contractions:
//   column Gram  Gvv_x[a][b] += c * sum_i sum_(j,c) A[(i,a)][(j,c)] A[(i,b)][(j,c)]
//   row Gram     Goo_y[i][j] += c * sum_(k,a) sum_b A[(k,a)][(i,b)] A[(k,a)][(j,b)]
// Same-spin blocks give both blocks of their own spin (c = +1/2, -1/2, using
// t[i,k,a,b] = t[k,i,b,a]).  An opposite-spin block that holds every alpha row
// gives all four blocks (the other two Grams contract its columns); when
// memory splits the rows, a second pass with beta rows gives Gvv_beta and
// Goo_alpha.  Each Gram is one product over a composite K (a batch index and a
// contiguous index, GemmF64Args::kb) with the tiles below the diagonal
// mirrored: few output tiles and a K of 10^4 .. 10^6, so the split of K over
// CTAs is what fills the GPU.  At N = 180, o = 18 the earlier form (one GEMM
// per occupied orbital, 9 CTAs each) took 14 ms per iteration for the column
// Grams, this one 0.5 ms.
// The generalized Fock matrix (:331-369) uses the Cholesky J and K:
//   J = sum_Q <L^Q, P_tot> L^Q,   K_s = sum_Q L^Q P_s L^Q,
// with Z^Q = P_s L^Q for all Q as one batched GEMM and K_s as one GEMM over
// the composite index (Q, nu); F_mo = C^T (H + J - K_s) C.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "amp_elem.cuh"
#include "cd_common.cuh"
#include "cd_internal.h"
#include "gemm_f64.cuh"
#include "pair_energy_f64.cuh"

namespace mshqc_cd {
namespace {

// out[q] = sum_k L[q * n + k] P[k] (one CTA per q, fixed-order tree)
__global__ void dot_rows_kernel(const double* __restrict__ L, int64_t n, const double* __restrict__ P,
                                double* __restrict__ out) {
    __shared__ double red[256];
    const double* row = L + (int64_t)blockIdx.x * n;
    double s = 0.0;
    for (int64_t k = threadIdx.x; k < n; k += 256) s = fma(row[k], P[k], s);
    red[threadIdx.x] = s;
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
        if (threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x] = red[0];
}

// parts[s][k] = sum over the s-th share of the vectors of coef[q] L[q * n + k]:
// the Coulomb matrix of one pass over the vectors.  HBM bound (8 bytes per
// multiply-add), so one thread per element and, when n alone does not fill
// the GPU, the vectors split over blockIdx.y; gemm_reduce_kernel adds the
// shares in order.  N = 400, M = 1600: 1.02 ms as a GEMM with one row, 0.37 ms
// here (5.5 TB/s).
__global__ void __launch_bounds__(256) coulomb_kernel(const double* __restrict__ L, int64_t n, int M, int per,
                                                      const double* __restrict__ coef, double* __restrict__ parts) {
    const int64_t k = blockIdx.x * 256LL + threadIdx.x;
    if (k >= n) return;
    const int q0 = blockIdx.y * per, q1 = min(M, q0 + per);
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int q = q0;
    for (; q + 4 <= q1; q += 4) {
        const double* l = L + (int64_t)q * n + k;
        s0 = fma(coef[q], l[0], s0);
        s1 = fma(coef[q + 1], l[n], s1);
        s2 = fma(coef[q + 2], l[2 * n], s2);
        s3 = fma(coef[q + 3], l[3 * n], s3);
    }
    for (; q < q1; ++q) s0 = fma(coef[q], L[(int64_t)q * n + k], s0);
    parts[(int64_t)blockIdx.y * n + k] = (s0 + s1) + (s2 + s3);
}

// G (N x N) = blockdiag(Goo (o x o), Gvv (v x v, row stride vp)), zero elsewhere
__global__ void blockdiag_kernel(const double* __restrict__ Goo, const double* __restrict__ Gvv, int64_t N,
                                 int64_t o, int64_t vp, double* __restrict__ G) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= N * N) return;
    const int64_t r = t / N, c = t % N;
    double x = 0.0;
    if (r < o && c < o) x = Goo[r * o + c];
    else if (r >= o && c >= o) x = Gvv[(r - o) * vp + (c - o)];
    G[t] = x;
}

// out = a + s * b (elementwise)
__global__ void axpy_kernel(const double* __restrict__ a, double s, const double* __restrict__ b, int64_t n,
                            double* __restrict__ out) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t < n) out[t] = a[t] + s * b[t];
}

unsigned blocks_for(int64_t n, int threads = 256) { return (unsigned)cdiv(n, threads); }

// J = beta * J + sum_q coef[q] L[q] over mc vectors of n elements
int coulomb(mshqc_cd_ctx* ctx, const double* L, int64_t n, int64_t mc, const double* coef, double beta, double* J) {
    const int64_t want = std::max<int64_t>(1, 8LL * ctx->num_sms / cdiv(n, 256));
    const int per = (int)std::max<int64_t>(4, cdiv(mc, want));
    const int S = (int)cdiv(mc, per);
    CD_ALLOC_FIRST(ctx->gemm_ws, sizeof(double) * (size_t)(S * n), false);
    coulomb_kernel<<<dim3(blocks_for(n), (unsigned)S), 256, 0, ctx->stream>>>(L, n, (int)mc, per, coef,
                                                                              ctx->gemm_ws.as<double>());
    CD_CUDA(cudaGetLastError());
    gemm_reduce_kernel<<<dim3((unsigned)cdiv(n, 64), 1), 256, 0, ctx->stream>>>(ctx->gemm_ws.as<double>(), S, 1, (int)n,
                                                                                1.0, beta, J, n, 0, 0);
    CD_CUDA(cudaGetLastError());
    ctx->launches += 2;
    return MSHQC_CD_OK;
}

struct OpdmOut {
    double* Goo[2];   // o_s x o_s
    double* Gvv[2];   // vp_s x vp_s (padded)
};

// G (+)= coef * sum_h sum_k A_h[m][k] A_h[n][k]  (n x n, symmetric)
int gram(mshqc_cd_ctx* ctx, const double* A, bool a_k, int64_t n, int64_t K, int64_t ld, int64_t kb, int64_t skb,
         double coef, double* G, int64_t ldg) {
    GemmF64Args g{};
    g.M = g.N = (int)n;  g.K = (int)K;  g.batch = 1;
    g.A = g.B = A;  g.lda = g.ldb = ld;
    g.kb = (int)kb;  g.skA = g.skB = skb;
    g.C = G;  g.ldc = ldg;
    g.alpha = coef;  g.beta = 1.0;
    g.sym = 1;
    return gemm_run(ctx, g, a_k, a_k);
}

// One amplitude pass: rows i of spin sx (blocks), columns every j of spin sy.
// Gvv_sx += col_coef * column Gram, Goo_sy += row_coef * row Gram; pair
// energies to `partial` when it is not null.  With `both` (opposite spin) and
// all rows in one block, Gvv_sy and Goo_sx are added too and *both is set.
template <int MODE>
int opdm_pass(mshqc_cd_ctx* ctx, int sx, int sy, double col_coef, double row_coef, const OpdmOut& out,
              double* partial, bool* both) {
    SpinState& X = ctx->spin[sx];
    SpinState& Y = ctx->spin[sy];
    const int64_t N = ctx->N, Mp = ctx->Mp;
    const int64_t ox = X.nocc, vx = N - ox, vpx = X.vp;
    const int64_t oy = Y.nocc, vy = N - oy, vpy = Y.vp;
    const int64_t ldS = oy * vpy;
    size_t free_b = 0, total_b = 0;
    CD_CUDA(cudaMemGetInfo(&free_b, &total_b));
    const size_t per_i = 2 * sizeof(double) * (size_t)vpx * ldS;
    const size_t held = ctx->W.bytes + ctx->amp.bytes;
    const size_t budget = std::max<size_t>(per_i, std::min<size_t>((free_b + held) / 4, size_t(24) << 30));
    const int bi = (int)std::max<int64_t>(1, std::min<int64_t>(ox, (int64_t)(budget / per_i)));
    CD_ALLOC_FIRST(ctx->W, per_i / 2 * bi, false);
    CD_ALLOC_FIRST(ctx->amp, per_i / 2 * bi, false);
    if (!partial) {
        // energies of this pass are not needed: throw-away slots, one per pair
        CD_ALLOC(ctx->pair_sum, sizeof(double) * (size_t)(ox * oy), false);
        partial = ctx->pair_sum.as<double>();
    }
    const double* A = ctx->amp.as<double>();
    for (int i0 = 0; i0 < ox; i0 += bi) {
        const int nbi = (int)std::min<int64_t>(bi, ox - i0);
        const int64_t R = (int64_t)nbi * vpx;
        // S[(i,a)][(j,b)] = sum_Q X[(i,a)][Q] Y[(j,b)][Q]; a same-spin block of
        // all rows is symmetric
        GemmF64Args g{};
        g.M = (int)R;  g.N = (int)ldS;  g.K = (int)Mp;  g.batch = 1;
        g.A = X.B64.as<double>() + (int64_t)i0 * vpx * Mp;  g.lda = Mp;  g.sA = 0;
        g.B = Y.B64.as<double>();  g.ldb = Mp;  g.sB = 0;
        g.C = ctx->W.as<double>();  g.ldc = ldS;  g.sC = 0;
        g.alpha = 1.0;  g.beta = 0.0;
        g.sym = sx == sy && nbi == ox ? 1 : 0;
        CD_RC(gemm_run(ctx, g, true, true));
        AmpElemArgs e{};
        e.S = ctx->W.as<double>();
        e.ldS = ldS;
        e.rsx = (int)vpx;  e.csy = (int)vpy;  e.ksy = (int)vpy;
        e.ox = (int)ox;  e.oy = (int)oy;  e.vx = (int)vx;  e.vy = (int)vy;
        e.i0 = i0;  e.nbi = nbi;  e.j0 = 0;  e.nbj = (int)oy;  e.wgt = 1.0;
        e.eox = X.eps.as<double>();  e.evx = e.eox + ox;
        e.eoy = Y.eps.as<double>();  e.evy = e.eoy + oy;
        e.A64 = ctx->amp.as<double>();  e.ldA = ldS;
        e.partial = partial;   // no dE/de here: prow, pcol, pocc stay null
        launch_amp<MODE, false>(e, nbi * oy, ctx->stream);
        CD_CUDA(cudaGetLastError());
        ctx->launches++;
        // column Gram: K batches i, K = (j, c)
        CD_RC(gram(ctx, A, true, vpx, ldS, ldS, nbi, vpx * ldS, col_coef, out.Gvv[sx], vpx));
        // row Gram: K batches (k, a), K = b
        CD_RC(gram(ctx, A, true, oy, vpy, vpy, R, ldS, row_coef, out.Goo[sy], oy));
        if (both && nbi == ox) {
            // the same amplitudes as rows of spin sy: K batches j, K = (i, a)
            CD_RC(gram(ctx, A, false, vpy, R, ldS, oy, vpy, col_coef, out.Gvv[sy], vpy));
            // and K batches a, K = (j, b)
            CD_RC(gram(ctx, A, true, ox, ldS, vpx * ldS, vpx, ldS, row_coef, out.Goo[sx], ox));
            *both = true;
        }
    }
    return MSHQC_CD_OK;
}

// Device layout of ctx->opdm (doubles): Goo_a, Goo_b, Gvv_a (vp_a^2), Gvv_b,
// then per spin P, F (N^2 each), then G, T, J, K, Fao (N^2 each), coef (M).
struct Omp2Buffers {
    double* Goo[2];
    double* Gvv[2];
    double* P[2];
    double* F[2];
    double *G, *T, *J, *K, *Fao, *coef, *deps;
};

int omp2_buffers(mshqc_cd_ctx* ctx, Omp2Buffers& b) {
    const int64_t N = ctx->N, M = ctx->M;
    const int64_t o0 = ctx->spin[0].nocc, o1 = ctx->spin[1].nocc;
    const int64_t vp0 = round_up(N - o0, 64), vp1 = round_up(N - o1, 64);
    // the blocks before the matrices padded to an even count: 16-byte rows for even N
    const int64_t noo = round_up(o0 * o0 + o1 * o1, 2);
    const int64_t n = noo + vp0 * vp0 + vp1 * vp1 + 9 * N * N + M + 2 * N;
    CD_ALLOC_FIRST(ctx->opdm, sizeof(double) * (size_t)n, false);
    double* p = ctx->opdm.as<double>();
    b.Goo[0] = p;  p += o0 * o0;
    b.Goo[1] = p;  p += noo - o0 * o0;
    b.Gvv[0] = p;  p += vp0 * vp0;
    b.Gvv[1] = p;  p += vp1 * vp1;
    b.P[0] = p;  p += N * N;
    b.P[1] = p;  p += N * N;
    b.F[0] = p;  p += N * N;
    b.F[1] = p;  p += N * N;
    b.G = p;  p += N * N;
    b.T = p;  p += N * N;
    b.J = p;  p += N * N;
    b.K = p;  p += N * N;
    b.Fao = p;  p += N * N;
    b.coef = p;  p += M;
    b.deps = p;
    return MSHQC_CD_OK;
}

// P = C[:, :o] C[:, :o]^T (C column-major)
int occupied_density(mshqc_cd_ctx* ctx, const double* C, int64_t o, double* P) {
    const int64_t N = ctx->N;
    GemmF64Args g{};
    g.M = (int)N;  g.N = (int)N;  g.K = (int)o;  g.batch = 1;
    g.A = C;  g.lda = N;  g.sA = 0;
    g.B = C;  g.ldb = N;  g.sB = 0;
    g.C = P;  g.ldc = N;  g.sC = 0;
    g.alpha = 1.0;  g.beta = 0.0;
    CD_RC(gemm_run(ctx, g, false, false));
    return MSHQC_CD_OK;
}

// The gradient evaluation at the context's current orbitals.  Pref[s]: the
// reference density of spin s (device, N*N).  Outputs stay in the buffers;
// *e_mp2 receives the OMP2 energy (same-spin + opposite-spin).
int omp2_pieces_device(mshqc_cd_ctx* ctx, const double* const Pref[2], Omp2Buffers& b, double* e_mp2) {
    const int64_t N = ctx->N, M = ctx->M, NN = N * N;
    CD_RC(begin_call(ctx));
    CD_RC(ensure_transforms(ctx, MSHQC_CD_FP64));
    CD_RC(omp2_buffers(ctx, b));
    const int64_t o0 = ctx->spin[0].nocc, o1 = ctx->spin[1].nocc;
    const int64_t vp0 = ctx->spin[0].vp, vp1 = ctx->spin[1].vp;
    // OPDM blocks start at zero
    CD_CUDA(cudaMemsetAsync(b.Goo[0], 0, sizeof(double) * (size_t)(round_up(o0 * o0 + o1 * o1, 2) + vp0 * vp0 + vp1 * vp1),
                            ctx->stream));
    const int64_t n0 = o0 * o0, n1 = o1 * o1, n2 = o0 * o1;   // one energy per pair
    CD_ALLOC_FIRST(ctx->partial, sizeof(double) * (size_t)(n0 + n1 + n2), false);
    double* part = ctx->partial.as<double>();
    OpdmOut out{{b.Goo[0], b.Goo[1]}, {b.Gvv[0], b.Gvv[1]}};
    begin_stage(ctx, ST_AMPLITUDE);
    CD_RC(opdm_pass<AMP_SAME_SPIN>(ctx, 0, 0, 0.5, -0.5, out, part, nullptr));
    CD_RC(opdm_pass<AMP_SAME_SPIN>(ctx, 1, 1, 0.5, -0.5, out, part + n0, nullptr));
    bool both = false;
    CD_RC(opdm_pass<AMP_OPPOSITE_SPIN>(ctx, 0, 1, 1.0, -1.0, out, part + n0 + n1, &both));
    if (!both) CD_RC(opdm_pass<AMP_OPPOSITE_SPIN>(ctx, 1, 0, 1.0, -1.0, out, nullptr, nullptr));
    end_stage(ctx);
    const int64_t offs[3] = {0, n0, n0 + n1}, cnt[3] = {n0, n1, n2};
    for (int k = 0; k < 3; ++k) {
        reduce_total_kernel<<<1, 256, 0, ctx->stream>>>(part + offs[k], (int)cnt[k],
                                                        ctx->status.as<CallStatus>()->totals + k);
        CD_CUDA(cudaGetLastError());
        ctx->launches++;
    }

    begin_stage(ctx, ST_OTHER);
    // P_s = Pref_s + C_s blockdiag(Goo_s, Gvv_s) C_s^T
    for (int s = 0; s < 2; ++s) {
        const SpinState& sp = ctx->spin[s];
        const double* C = sp.C.as<double>();
        blockdiag_kernel<<<blocks_for(NN), 256, 0, ctx->stream>>>(b.Goo[s], b.Gvv[s], N, sp.nocc, sp.vp, b.G);
        CD_CUDA(cudaGetLastError());
        // T = C G  (T[r][c] = sum_k C(r,k) G(k,c))
        GemmF64Args g{};
        g.M = (int)N;  g.N = (int)N;  g.K = (int)N;  g.batch = 1;
        g.A = C;  g.lda = N;  g.B = b.G;  g.ldb = N;  g.C = b.T;  g.ldc = N;
        g.alpha = 1.0;  g.beta = 0.0;
        CD_RC(gemm_run(ctx, g, false, false));
        // P = T C^T + Pref
        CD_CUDA(cudaMemcpyAsync(b.P[s], Pref[s], sizeof(double) * NN, cudaMemcpyDeviceToDevice, ctx->stream));
        GemmF64Args h{};
        h.M = (int)N;  h.N = (int)N;  h.K = (int)N;  h.batch = 1;
        h.A = b.T;  h.lda = N;  h.B = C;  h.ldb = N;  h.C = b.P[s];  h.ldc = N;
        h.alpha = 1.0;  h.beta = 1.0;
        CD_RC(gemm_run(ctx, h, true, false));
        ctx->launches++;
    }
    // J = sum_Q <L^Q, P_a + P_b> L^Q
    axpy_kernel<<<blocks_for(NN), 256, 0, ctx->stream>>>(b.P[0], 1.0, b.P[1], NN, b.G);
    dot_rows_kernel<<<(unsigned)M, 256, 0, ctx->stream>>>(ctx->L.as<double>(), NN, b.G, b.coef);
    CD_CUDA(cudaGetLastError());
    ctx->launches += 2;
    CD_RC(coulomb(ctx, ctx->L.as<double>(), NN, M, b.coef, 0.0, b.J));
    CD_ALLOC_FIRST(ctx->Zt, sizeof(double) * (size_t)(M * NN), false);
    for (int s = 0; s < 2; ++s) {
        const double* C = ctx->spin[s].C.as<double>();
        // Z^Q = P_s L^Q for every Q (batched)
        GemmF64Args z{};
        z.M = (int)N;  z.N = (int)N;  z.K = (int)N;  z.batch = (int)M;
        z.A = b.P[s];  z.lda = N;  z.sA = 0;
        z.B = ctx->L.as<double>();  z.ldb = N;  z.sB = NN;
        z.C = ctx->Zt.as<double>();  z.ldc = N;  z.sC = NN;
        z.alpha = 1.0;  z.beta = 0.0;
        CD_RC(gemm_run(ctx, z, true, false));
        // K[mu][lam] = sum_{(Q,nu)} L^Q(mu,nu) Z^Q(nu,lam)
        GemmF64Args k{};
        k.M = (int)N;  k.N = (int)N;  k.K = (int)(M * N);  k.batch = 1;
        k.A = ctx->L.as<double>();  k.lda = N;
        k.B = ctx->Zt.as<double>();  k.ldb = N;
        k.C = b.K;  k.ldc = N;
        k.alpha = 1.0;  k.beta = 0.0;
        CD_RC(gemm_run(ctx, k, false, false));
        // F_ao = H + J - K
        axpy_kernel<<<blocks_for(NN), 256, 0, ctx->stream>>>(ctx->Hcore.as<double>(), 1.0, b.J, NN, b.Fao);
        axpy_kernel<<<blocks_for(NN), 256, 0, ctx->stream>>>(b.Fao, -1.0, b.K, NN, b.Fao);
        CD_CUDA(cudaGetLastError());
        // T = F_ao C, then F_mo (column-major): out[c][r] = sum_mu T(mu,c) C(mu,r)
        GemmF64Args t{};
        t.M = (int)N;  t.N = (int)N;  t.K = (int)N;  t.batch = 1;
        t.A = b.Fao;  t.lda = N;  t.B = C;  t.ldb = N;  t.C = b.T;  t.ldc = N;
        t.alpha = 1.0;  t.beta = 0.0;
        CD_RC(gemm_run(ctx, t, true, true));
        GemmF64Args f{};
        f.M = (int)N;  f.N = (int)N;  f.K = (int)N;  f.batch = 1;
        f.A = b.T;  f.lda = N;  f.B = C;  f.ldb = N;  f.C = b.F[s];  f.ldc = N;
        f.alpha = 1.0;  f.beta = 0.0;
        CD_RC(gemm_run(ctx, f, false, true));
        ctx->launches += 2;
    }
    end_stage(ctx);
    CallStatus st;
    CD_RC(finish_call(ctx, &st));
    *e_mp2 = st.totals[0] + st.totals[1] + st.totals[2];
    return MSHQC_CD_OK;
}

// W = c0 I + c1 A + c2 A2 + c3 A3 (N x N)
__global__ void poly3_kernel(const double* __restrict__ A, const double* __restrict__ A2,
                             const double* __restrict__ A3, int64_t N, double c0, double c1, double c2, double c3,
                             double* __restrict__ W) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t < N * N) W[t] = fma(c3, A3[t], fma(c2, A2[t], fma(c1, A[t], t / N == t % N ? c0 : 0.0)));
}

// exp(A) for a real N x N matrix (row-major) of 1-norm norm1, by scaling and
// squaring with the degree-19 Taylor polynomial: with ||A / 2^s||_1 <= 1/2 the
// truncation error is below 1e-24.  The polynomial in four-term groups of
// powers of A^4 (Paterson and Stockmeyer) takes 7 products where Horner's form
// in A takes 19; each is a latency-bound chain of small tiles.  E, W and
// pw (3 N^2: the powers) are work matrices; *result points at whichever of E
// and W holds exp(A).
int expm_device(mshqc_cd_ctx* ctx, double* A, double norm1, double* E, double* W, double* pw,
                const double** result) {
    const int64_t N = ctx->N, NN = N * N;
    int s = 0;
    while (norm1 > 0.5 && s < 60) {
        norm1 *= 0.5;
        ++s;
    }
    const double scale = std::ldexp(1.0, -s);
    // Z = alpha X Y + beta Z
    auto mul = [&](const double* X, const double* Y, double alpha, double beta, double* Z) {
        GemmF64Args g{};
        g.M = (int)N;  g.N = (int)N;  g.K = (int)N;  g.batch = 1;
        g.A = X;  g.lda = N;  g.B = Y;  g.ldb = N;  g.C = Z;  g.ldc = N;
        g.alpha = alpha;  g.beta = beta;
        return gemm_run(ctx, g, true, false);
    };
    double *A2 = pw, *A3 = pw + NN, *A4 = pw + 2 * NN;   // powers of scale * A
    CD_RC(mul(A, A, scale * scale, 0.0, A2));
    CD_RC(mul(A, A2, scale, 0.0, A3));
    CD_RC(mul(A2, A2, 1.0, 0.0, A4));
    double c[20];
    c[0] = 1.0;
    for (int k = 1; k < 20; ++k) c[k] = c[k - 1] / k;
    for (int h = 4; h >= 0; --h) {
        // W = B_h + A4 E, E the higher groups
        poly3_kernel<<<blocks_for(NN), 256, 0, ctx->stream>>>(A, A2, A3, N, c[4 * h], c[4 * h + 1] * scale,
                                                              c[4 * h + 2], c[4 * h + 3], W);
        CD_CUDA(cudaGetLastError());
        ctx->launches++;
        if (h < 4) CD_RC(mul(A4, E, 1.0, 1.0, W));
        std::swap(E, W);
    }
    for (int q = 0; q < s; ++q) {
        CD_RC(mul(E, E, 1.0, 0.0, W));
        std::swap(E, W);
    }
    *result = E;
    return MSHQC_CD_OK;
}

// C_s <- C_s exp(-kappa), kappa from w (v x o, column-major w(a,i)) and the
// MO Fock diagonal exactly as reference src/mp2/cholesky_omp2.cc:375-400
// (damping 0.5, level shift 0.2, |denominator| >= 1e-2), then the new
// orbitals replace the context's.  F_host: F_mo column-major N x N.
int rotate_spin(mshqc_cd_ctx* ctx, int spin, const std::vector<double>& F_host) {
    const int64_t N = ctx->N, NN = N * N, o = ctx->spin[spin].nocc, v = N - o;
    std::vector<double> A(NN, 0.0);   // row-major A = -kappa
    for (int64_t a = 0; a < v; ++a)
        for (int64_t i = 0; i < o; ++i) {
            double diff = F_host[(o + a) * N + (o + a)] - F_host[i * N + i] + 0.2;
            if (std::abs(diff) < 1e-2) diff = diff >= 0 ? 1e-2 : -1e-2;
            const double w = 2.0 * F_host[i * N + (o + a)];   // w(a,i) = 2 F(o+a, i)
            const double val = (w / diff) * 0.5;
            A[(o + a) * N + i] = -val;    // -kappa(o+a, i)
            A[i * N + (o + a)] = val;     // -kappa(i, o+a)
        }
    double norm1 = 0.0;
    for (int64_t c = 0; c < N; ++c) {
        double col = 0.0;
        for (int64_t r = 0; r < N; ++r) col += std::abs(A[r * N + c]);
        norm1 = std::max(norm1, col);
    }
    CD_ALLOC_FIRST(ctx->omp2_ws, sizeof(double) * (size_t)(7 * NN), false);
    double* dA = ctx->omp2_ws.as<double>();
    double* E0 = dA + NN;
    double* E1 = E0 + NN;
    double* Cn = E1 + NN;
    double* pw = Cn + NN;
    CD_CUDA(cudaMemcpyAsync(dA, A.data(), sizeof(double) * NN, cudaMemcpyHostToDevice, ctx->stream));
    const double* E = nullptr;
    CD_RC(expm_device(ctx, dA, norm1, E0, E1, pw, &E));
    // column-major C_new = C E: as row-major arrays C_new^T = E^T C^T
    double* C = ctx->spin[spin].C.as<double>();
    GemmF64Args g{};
    g.M = (int)N;  g.N = (int)N;  g.K = (int)N;  g.batch = 1;
    g.A = E;  g.lda = N;  g.B = C;  g.ldb = N;  g.C = Cn;  g.ldc = N;
    g.alpha = 1.0;  g.beta = 0.0;
    CD_RC(gemm_run(ctx, g, false, false));
    CD_CUDA(cudaMemcpyAsync(C, Cn, sizeof(double) * NN, cudaMemcpyDeviceToDevice, ctx->stream));
    return invalidate_spin(ctx, spin);
}

int require_omp2_inputs(mshqc_cd_ctx* ctx) {
    if (!ctx->L_set) return set_error(MSHQC_CD_ERR_STATE, "Cholesky vectors not set");
    if (!ctx->spin[0].set || !ctx->spin[1].set)
        return set_error(MSHQC_CD_ERR_STATE, "OMP2 needs alpha and beta orbitals (set both; equal for RHF)");
    if (!ctx->H_set) return set_error(MSHQC_CD_ERR_STATE, "core Hamiltonian not set");
    if (ctx->L_gen)
        return set_error(MSHQC_CD_ERR_UNSUPPORTED,
                         "OMP2 needs stored Cholesky vectors (mshqc_cd_set_vectors), not generated ones");
    return MSHQC_CD_OK;
}

// reference densities: caller's (host or device) or C_occ C_occ^T
int reference_densities(mshqc_cd_ctx* ctx, const double* Pa, const double* Pb, int where, double* dst[2]) {
    const int64_t N = ctx->N, NN = N * N;
    const double* in[2] = {Pa, Pb};
    for (int s = 0; s < 2; ++s) {
        if (in[s]) {
            if (where == MSHQC_CD_HOST)
                CD_RC(upload(ctx, dst[s], in[s], sizeof(double) * NN));
            else
                CD_CUDA(cudaMemcpyAsync(dst[s], in[s], sizeof(double) * NN, cudaMemcpyDeviceToDevice,
                                        ctx->stream));
        } else {
            CD_RC(occupied_density(ctx, ctx->spin[s].C.as<double>(), ctx->spin[s].nocc, dst[s]));
        }
    }
    return MSHQC_CD_OK;
}

// norm2[q] = sum_k L[q * n + k]^2 (one CTA per q, fixed-order tree)
__global__ void row_norm2_kernel(const double* __restrict__ L, int64_t n, double* __restrict__ norm2) {
    __shared__ double red[256];
    const double* row = L + (int64_t)blockIdx.x * n;
    double s = 0.0;
    for (int64_t k = threadIdx.x; k < n; k += 256) s = fma(row[k], row[k], s);
    red[threadIdx.x] = s;
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
        if (threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) norm2[blockIdx.x] = red[0];
}

// Z^q = 0 for the vectors whose Frobenius norm is at most `thr` (the
// exchange screening of src/scf/cholesky_rhf.cc:120-126); norm2[q] = |L^q|^2.
// Row z of vector q: N elements at Z + q * sq + z * ldz (grid: N, vectors, rows)
__global__ void screen_slabs_kernel(double* __restrict__ Z, const double* __restrict__ norm2, int64_t N, int64_t sq,
                                    int64_t ldz, double thr) {
    if (norm2[blockIdx.y] > thr * thr) return;
    double* z = Z + (int64_t)blockIdx.y * sq + (int64_t)blockIdx.z * ldz;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < N; t += (int64_t)gridDim.x * blockDim.x)
        z[t] = 0.0;
}

// Pivoted Cholesky factor of a density matrix P (N x N) for the exchange
// build: X[k][n], k < rank, with P ~ sum_k X[k] X[k]^T.  One CTA; step k takes
// the largest remaining diagonal, forms the column left-looking (thread per
// row, X[k] contiguous in n) and updates the diagonal.  Stops when the largest
// remaining diagonal is at rounding level of the first one, or after rmax
// vectors.  Latency bound: about 3 us a step at N = 400.  D is N doubles of
// work; out: [0] rank.
__global__ void __launch_bounds__(1024) density_factor_kernel(const double* __restrict__ P, int64_t N, int rmax,
                                                              double* __restrict__ X, double* __restrict__ D,
                                                              int* __restrict__ rank) {
    __shared__ double sv[32];
    __shared__ int si[32];
    __shared__ double best_v;
    __shared__ int best_i;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int64_t n = tid; n < N; n += 1024) D[n] = P[n * N + n];
    double first = 0.0;
    int k = 0;
    for (; k < rmax; ++k) {
        __syncthreads();
        double v = -1.0;
        int idx = 0;
        for (int64_t n = tid; n < N; n += 1024)
            if (D[n] > v) {
                v = D[n];
                idx = (int)n;
            }
#pragma unroll
        for (int off = 16; off; off >>= 1) {
            const double ov = __shfl_xor_sync(0xffffffffu, v, off);
            const int oi = __shfl_xor_sync(0xffffffffu, idx, off);
            if (ov > v || (ov == v && oi < idx)) {
                v = ov;
                idx = oi;
            }
        }
        if (lane == 0) {
            sv[warp] = v;
            si[warp] = idx;
        }
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < 32; ++w)
                if (sv[w] > v || (sv[w] == v && si[w] < idx)) {
                    v = sv[w];
                    idx = si[w];
                }
            best_v = v;
            best_i = idx;
        }
        __syncthreads();
        const double dp = best_v;
        const int64_t p = best_i;
        if (k == 0) first = dp;
        if (!(dp > 0x1p-50 * first)) break;
        const double inv = 1.0 / sqrt(dp);
        for (int64_t n = tid; n < N; n += 1024) {
            double a0 = P[p * N + n], a1 = 0.0, a2 = 0.0, a3 = 0.0;
            int h = 0;
            for (; h + 4 <= k; h += 4) {
                const double* x = X + (int64_t)h * N;
                a0 = fma(-x[n], x[p], a0);
                a1 = fma(-x[N + n], x[N + p], a1);
                a2 = fma(-x[2 * N + n], x[2 * N + p], a2);
                a3 = fma(-x[3 * N + n], x[3 * N + p], a3);
            }
            for (; h < k; ++h) a0 = fma(-X[(int64_t)h * N + n], X[(int64_t)h * N + p], a0);
            const double x = ((a0 + a1) + (a2 + a3)) * inv;
            X[(int64_t)k * N + n] = x;
            D[n] = n == p ? 0.0 : fma(-x, x, D[n]);
        }
    }
    if (tid == 0) *rank = k;
}

// *bad = 1 when the factor misses P: in some 32 x 32 tile of it,
//   max |P - sum_k X[k] X[k]^T| > (8 + r / 4) 2^-52 max sum_k |X[k]| |X[k]^T|.
// Tiles are held to their own size, so parts of P far below the rest keep their
// relative accuracy (against the largest element of P alone, a block 10^-16 of
// it was left out); the allowance is below the N 2^-53 of the chains of P L^Q
// for r <= N / 4, and twice what densities formed in FP64 need (0.4 ... 0.8 of
// (4 + r / 8) 2^-52, N = 96 ... 500).  Grid: tiles.  A NaN compares as a miss.
__global__ void __launch_bounds__(256) density_residual_kernel(const double* __restrict__ P, int64_t N,
                                                               const double* __restrict__ X,
                                                               const int* __restrict__ rank,
                                                               unsigned long long* __restrict__ bad) {
    __shared__ double sr[8], ss[8];
    const int r = *rank, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    // columns and rows beyond N repeat the last ones
    const int64_t j = min((int64_t)blockIdx.x * 32 + tx, N - 1);
    int64_t i[4];
    double d[4], sum[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        i[c] = min((int64_t)blockIdx.y * 32 + ty + 8 * c, N - 1);
        d[c] = P[i[c] * N + j];
        sum[c] = 0.0;
    }
    for (int k = 0; k < r; ++k) {
        const double* x = X + (int64_t)k * N;
        const double y = x[j];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const double z = x[i[c]];
            d[c] = fma(-z, y, d[c]);
            sum[c] = fma(fabs(z), fabs(y), sum[c]);
        }
    }
    double mr = 0.0, ms = 0.0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        if (!(mr >= fabs(d[c]))) mr = mr != mr ? mr : fabs(d[c]);   // (a NaN is taken and kept)
        ms = fmax(ms, sum[c]);
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        const double o = __shfl_xor_sync(0xffffffffu, mr, off);
        if (!(mr >= o)) mr = mr != mr ? mr : o;
        ms = fmax(ms, __shfl_xor_sync(0xffffffffu, ms, off));
    }
    if (tx == 0) {
        sr[ty] = mr;
        ss[ty] = ms;
    }
    __syncthreads();
    if (threadIdx.x) return;
    for (int w = 1; w < 8; ++w) {
        if (!(mr >= sr[w])) mr = mr != mr ? mr : sr[w];
        ms = fmax(ms, ss[w]);
    }
    if (!(mr <= (8.0 + r / 4.0) * 0x1p-52 * ms)) *bad = 1;
}

// Factors of the densities of an exchange build in ctx->dens_x (X[s] there,
// rank[s] vectors each, the two spins' one after the other), or rank[s] = 0
// where P[s] is not represented by at most N / 4 vectors to rounding
// (density_residual_kernel looks at every element, so an indefinite or
// unsymmetric P is refused too).  The exchange then takes 4 M N^2 r operations
// instead of 4 M N^3.
// UHF builds of N / 10 electrons, whole calls: N = 96 0.38 ms with factors, 0.55
// without, N = 64 0.32 without, nearly all of it the host's copies.  A density of
// full rank pays for N / 4 steps in vain: 1.1 of 34.7 ms at N = 400.
constexpr int64_t kDensityFactorMinN = 96;
int density_factors(mshqc_cd_ctx* ctx, int nspin, const double* const P[2], const double* X[2], int rank[2]) {
    const int64_t N = ctx->N;
    const int rmax = (int)(N / 4);
    rank[0] = rank[1] = 0;
    X[0] = X[1] = nullptr;
    if (N < kDensityFactorMinN) return MSHQC_CD_OK;
    CD_ALLOC_FIRST(ctx->dens_x, sizeof(double) * (size_t)((2 * (rmax + 1) + rmax) * N + 8), false);
    double* base = ctx->dens_x.as<double>();
    unsigned long long* tail = reinterpret_cast<unsigned long long*>(base + 2 * (rmax + 1) * N);   // [spin][bad, unused, rank]
    CD_CUDA(cudaMemsetAsync(tail, 0, 6 * sizeof(unsigned long long), ctx->stream));
    for (int s = 0; s < nspin; ++s) {
        double* x = base + (int64_t)s * (rmax + 1) * N;
        int* rk = reinterpret_cast<int*>(tail + 3 * s + 2);
        density_factor_kernel<<<1, 1024, 0, ctx->stream>>>(P[s], N, rmax, x, x + (int64_t)rmax * N, rk);
        CD_CUDA(cudaGetLastError());
        const unsigned nt = (unsigned)cdiv(N, 32);
        density_residual_kernel<<<dim3(nt, nt), 256, 0, ctx->stream>>>(P[s], N, x, rk, tail + 3 * s);
        CD_CUDA(cudaGetLastError());
        ctx->launches += 2;
        X[s] = x;
    }
    unsigned long long h[6];
    CD_CUDA(cudaMemcpyAsync(h, tail, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
    CD_CUDA(cudaStreamSynchronize(ctx->stream));
    for (int s = 0; s < nspin; ++s) {
        if (h[3 * s] == 0) rank[s] = (int)(h[3 * s + 2] & 0xffffffffull);
    }
    if (rank[0] > 0 && rank[1] > 0) {
        // the second spin's rows right after the first's (never overlapping: rank <= N / 4)
        double* x1 = base + rank[0] * N;
        CD_CUDA(cudaMemcpyAsync(ctx->dens_x.as<double>() + 2 * (rmax + 1) * N + 8, X[1],
                                sizeof(double) * (size_t)(rank[1] * N), cudaMemcpyDeviceToDevice, ctx->stream));
        CD_CUDA(cudaMemcpyAsync(x1, ctx->dens_x.as<double>() + 2 * (rmax + 1) * N + 8,
                                sizeof(double) * (size_t)(rank[1] * N), cudaMemcpyDeviceToDevice, ctx->stream));
        X[1] = x1;
    }
    return MSHQC_CD_OK;
}

// Cholesky Coulomb and exchange matrices of the SCF Fock builds,
//   J = sum_Q <L^Q, P_tot> L^Q,   K_s = sum_Q L^Q P_s L^Q,
// P_tot = P[0] (nspin 1) or P[0] + P[1] (nspin 2), over chunks of vectors
// (stored or generated): per chunk the coefficients <L^Q, P_tot> (one dot
// product per vector) and J += coef . L.  Exchange of a density of low rank
// (an SCF density has the rank of its occupied orbitals): V_k^Q = L^Q X_k and
// K_s += V V^T over the composite index (k, Q), of which the tiles on and above
// the diagonal are computed; otherwise Z^Q = P_s L^Q as one batched GEMM and
// K_s += L . Z over the composite index (Q, nu).  All matrices are N x N and
// symmetric; device pointers on the context stream.  UHF, N = 400, M = 1600,
// 40 and 38 electrons: 85.9 ms before (the K product ran on 49 CTAs), 27 ms
// with the full products and K split, 3.6 ms with the factors.
int cholesky_jk_device(mshqc_cd_ctx* ctx, int nspin, const double* const P[2], bool screen, double* J,
                       double* const K[2], double* work) {
    const int64_t N = ctx->N, NN = N * N, M = ctx->M;
    const double* Ptot = P[0];
    if (nspin == 2) {
        axpy_kernel<<<blocks_for(NN), 256, 0, ctx->stream>>>(P[0], 1.0, P[1], NN, work);
        CD_CUDA(cudaGetLastError());
        ctx->launches++;
        Ptot = work;
    }
    const double* X[2];
    int rank[2];
    CD_RC(density_factors(ctx, nspin, P, X, rank));
    CD_CUDA(cudaMemsetAsync(J, 0, sizeof(double) * NN, ctx->stream));
    for (int s = 0; s < nspin; ++s) CD_CUDA(cudaMemsetAsync(K[s], 0, sizeof(double) * NN, ctx->stream));
    // factored spins first: their V in one product over all factor rows
    const int rtot = rank[0] + rank[1];
    const double* Xall = rank[0] > 0 ? X[0] : X[1];
    bool dense = false;
    for (int s = 0; s < nspin; ++s) dense = dense || rank[s] == 0;
    // vectors per chunk: the generator's chunk, and at most 2 GB of Z (or V)
    const int64_t per_q = std::max<int64_t>((int64_t)rtot * N, dense ? NN : 1);
    const int64_t mc_max = std::max<int64_t>(
        1, std::min<int64_t>({vectors_chunk_size(ctx), (int64_t)((size_t(2) << 30) / (sizeof(double) * per_q)),
                              (int64_t)65535}));
    CD_ALLOC_FIRST(ctx->Zt, sizeof(double) * (size_t)(mc_max * per_q), false);
    CD_ALLOC_FIRST(ctx->omp2_ws, sizeof(double) * (size_t)(2 * mc_max), false);
    double* coef = ctx->omp2_ws.as<double>();
    double* norm2 = coef + mc_max;
    double* Z = ctx->Zt.as<double>();
    for (int64_t Q0 = 0; Q0 < M; Q0 += mc_max) {
        const int64_t mc = std::min<int64_t>(mc_max, M - Q0);
        const double* Lc = nullptr;
        CD_RC(vectors_chunk(ctx, Q0, mc, &Lc));
        dot_rows_kernel<<<(unsigned)mc, 256, 0, ctx->stream>>>(Lc, NN, Ptot, coef);
        CD_CUDA(cudaGetLastError());
        ctx->launches++;
        CD_RC(coulomb(ctx, Lc, NN, mc, coef, 1.0, J));
        if (screen) {
            row_norm2_kernel<<<(unsigned)mc, 256, 0, ctx->stream>>>(Lc, NN, norm2);
            CD_CUDA(cudaGetLastError());
            ctx->launches++;
        }
        // Z (rows x [Q][N], row stride ldz between factor rows or N): A_rows L^Q per vector
        auto left_product = [&](const double* A, int64_t rows, int64_t ldz, int64_t sz) -> int {
            GemmF64Args z{};
            z.M = (int)rows;  z.N = (int)N;  z.K = (int)N;  z.batch = (int)mc;
            z.A = A;  z.lda = N;  z.sA = 0;
            z.B = Lc;  z.ldb = N;  z.sB = NN;
            z.C = Z;  z.ldc = ldz;  z.sC = sz;
            z.alpha = 1.0;  z.beta = 0.0;
            CD_RC(gemm_run(ctx, z, true, false));
            if (screen) {
                dim3 grid((unsigned)std::min<int64_t>(cdiv(N, 256), 1024), (unsigned)mc, (unsigned)rows);
                screen_slabs_kernel<<<grid, 256, 0, ctx->stream>>>(Z, norm2, N, sz, ldz, 1e-8);
                CD_CUDA(cudaGetLastError());
                ctx->launches++;
            }
            return MSHQC_CD_OK;
        };
        if (rtot > 0) {
            // V[k][Q][mu]; K_s[mu][lam] += sum_{(k,Q)} V V
            CD_RC(left_product(Xall, rtot, mc * N, N));
            int64_t k0 = 0;
            for (int s = 0; s < nspin; ++s) {
                if (rank[s] == 0) continue;
                GemmF64Args k{};
                k.M = k.N = (int)N;  k.K = (int)(rank[s] * mc);  k.batch = 1;
                k.A = k.B = Z + k0 * mc * N;  k.lda = k.ldb = N;
                k.C = K[s];  k.ldc = N;
                k.alpha = 1.0;  k.beta = 1.0;
                k.sym = 1;
                CD_RC(gemm_run(ctx, k, false, false));
                k0 += rank[s];
            }
        }
        for (int s = 0; s < nspin; ++s) {
            if (rank[s] > 0) continue;
            CD_RC(left_product(P[s], N, N, NN));
            GemmF64Args k{};
            k.M = (int)N;  k.N = (int)N;  k.K = (int)(mc * N);  k.batch = 1;
            k.A = Lc;  k.lda = N;
            k.B = Z;  k.ldb = N;
            k.C = K[s];  k.ldc = N;
            k.alpha = 1.0;  k.beta = 1.0;
            CD_RC(gemm_run(ctx, k, false, false));
        }
    }
    return MSHQC_CD_OK;
}

}  // namespace
}  // namespace mshqc_cd

using namespace mshqc_cd;

extern "C" {

MSHQC_CD_API int mshqc_cd_set_core_hamiltonian(mshqc_cd_ctx* ctx, const double* H, int where) {
    if (!ctx) return set_error(MSHQC_CD_ERR_ARG, "null context");
    if (!H) return set_error(MSHQC_CD_ERR_ARG, "H is null");
    if (!ctx->L_set) return set_error(MSHQC_CD_ERR_STATE, "set_vectors must precede set_core_hamiltonian");
    DeviceGuard g(ctx->device);
    const int64_t NN = ctx->N * ctx->N;
    CD_ALLOC(ctx->Hcore, sizeof(double) * (size_t)NN, false);
    if (where == MSHQC_CD_HOST) {
        CD_RC(upload(ctx, ctx->Hcore.p, H, sizeof(double) * NN));
    } else {
        CD_CUDA(cudaMemcpyAsync(ctx->Hcore.p, H, sizeof(double) * NN, cudaMemcpyDeviceToDevice, ctx->stream));
    }
    CD_RC(check_finite_device(ctx, ctx->Hcore.as<double>(), NN, "H"));
    ctx->H_set = true;
    CD_CUDA(cudaStreamSynchronize(ctx->stream));
    return MSHQC_CD_OK;
}

MSHQC_CD_API int mshqc_cd_get_orbitals(mshqc_cd_ctx* ctx, int spin, double* C, int where) {
    if (!ctx) return set_error(MSHQC_CD_ERR_ARG, "null context");
    if (spin != MSHQC_CD_ALPHA && spin != MSHQC_CD_BETA)
        return set_error(MSHQC_CD_ERR_ARG, "spin must be 0 (alpha) or 1 (beta)");
    if (!ctx->spin[spin].set) return set_error(MSHQC_CD_ERR_STATE, "orbitals of this spin not set");
    DeviceGuard g(ctx->device);
    CD_RC(download(ctx, C, ctx->spin[spin].C.p, sizeof(double) * ctx->N * ctx->N, where));
    return MSHQC_CD_OK;
}

MSHQC_CD_API int mshqc_cd_omp2_pieces(mshqc_cd_ctx* ctx, const double* P_a, const double* P_b, double* e_mp2,
                                      double* Goo_a, double* Gvv_a, double* Goo_b, double* Gvv_b, double* F_a,
                                      double* F_b, int where) {
    if (!ctx) return set_error(MSHQC_CD_ERR_ARG, "null context");
    CD_RC(require_omp2_inputs(ctx));
    DeviceGuard g(ctx->device);
    reset_stages(ctx);
    const int64_t N = ctx->N, NN = N * N;
    // reference densities (ctx->scratch is not used by the FP64 passes)
    CD_ALLOC(ctx->scratch, sizeof(double) * (size_t)(2 * NN), false);
    double* pr[2] = {ctx->scratch.as<double>(), ctx->scratch.as<double>() + NN};
    CD_RC(reference_densities(ctx, P_a, P_b, where, pr));
    Omp2Buffers b{};
    double e = 0.0;
    const double* prc[2] = {pr[0], pr[1]};
    CD_RC(one_spin_retry(ctx, [&] { return omp2_pieces_device(ctx, prc, b, &e); }));
    collect_stages(ctx);
    if (e_mp2) *e_mp2 = e;
    // OPDM blocks out without the padding
    for (int s = 0; s < 2; ++s) {
        const int64_t o = ctx->spin[s].nocc, v = N - o, vp = ctx->spin[s].vp;
        double* goo = s == 0 ? Goo_a : Goo_b;
        double* gvv = s == 0 ? Gvv_a : Gvv_b;
        double* f = s == 0 ? F_a : F_b;
        if (goo) CD_RC(download(ctx, goo, b.Goo[s], sizeof(double) * o * o, where));
        if (gvv) {
            if (where == MSHQC_CD_HOST) {
                std::vector<double> tmp((size_t)(vp * vp));
                CD_RC(download(ctx, tmp.data(), b.Gvv[s], sizeof(double) * vp * vp, MSHQC_CD_HOST));
                for (int64_t a = 0; a < v; ++a)
                    std::memcpy(gvv + a * v, tmp.data() + a * vp, sizeof(double) * v);
            } else {
                CD_CUDA(cudaMemcpy2DAsync(gvv, sizeof(double) * v, b.Gvv[s], sizeof(double) * vp,
                                          sizeof(double) * v, v, cudaMemcpyDeviceToDevice, ctx->stream));
                CD_CUDA(cudaStreamSynchronize(ctx->stream));
            }
        }
        if (f) CD_RC(download(ctx, f, b.F[s], sizeof(double) * NN, where));
    }
    return MSHQC_CD_OK;
}

MSHQC_CD_API int mshqc_cd_omp2(mshqc_cd_ctx* ctx, const mshqc_cd_omp2_config* cfg, const double* P_a,
                               const double* P_b, int where, mshqc_cd_omp2_result* res) {
    if (!ctx) return set_error(MSHQC_CD_ERR_ARG, "null context");
    if (!cfg || !res) return set_error(MSHQC_CD_ERR_ARG, "cfg and res must be non-null");
    if (cfg->max_iterations < 0) return set_error(MSHQC_CD_ERR_ARG, "max_iterations must be >= 0");
    CD_RC(require_omp2_inputs(ctx));
    DeviceGuard g(ctx->device);
    const int64_t N = ctx->N, NN = N * N;
    const int64_t na = ctx->spin[0].nocc, nb = ctx->spin[1].nocc;
    std::memset(res, 0, sizeof(*res));
    cudaEvent_t e0 = ctx->ev[0], e1 = ctx->ev[1];
    CD_CUDA(cudaEventRecord(e0, ctx->stream));
    reset_stages(ctx);
    // reference densities live in ctx->scratch for the whole loop
    CD_ALLOC(ctx->scratch, sizeof(double) * (size_t)(2 * NN), false);
    double* pref[2] = {ctx->scratch.as<double>(), ctx->scratch.as<double>() + NN};
    CD_RC(reference_densities(ctx, P_a, P_b, where, pref));
    const double* prc[2] = {pref[0], pref[1]};
    double e_prev = cfg->e_scf, e_corr = 0.0;
    int iter = 0, converged = 0;
    std::vector<double> Fa((size_t)NN), Fb((size_t)NN);
    while (iter < cfg->max_iterations) {
        ++iter;
        Omp2Buffers b{};
        CD_RC(one_spin_retry(ctx, [&] { return omp2_pieces_device(ctx, prc, b, &e_corr); }));
        CD_CUDA(cudaMemcpyAsync(Fa.data(), b.F[0], sizeof(double) * NN, cudaMemcpyDeviceToHost, ctx->stream));
        CD_CUDA(cudaMemcpyAsync(Fb.data(), b.F[1], sizeof(double) * NN, cudaMemcpyDeviceToHost, ctx->stream));
        CD_CUDA(cudaStreamSynchronize(ctx->stream));
        const double e_cur = cfg->e_scf + e_corr;
        double g2 = 0.0;
        for (int s = 0; s < 2; ++s) {
            const std::vector<double>& F = s == 0 ? Fa : Fb;
            const int64_t o = s == 0 ? na : nb;
            for (int64_t i = 0; i < o; ++i)
                for (int64_t a = o; a < N; ++a) {
                    const double w = 2.0 * F[i * N + a];
                    g2 += w * w;
                }
        }
        const double g_norm = std::sqrt(g2);
        if (g_norm < cfg->gradient_threshold && std::abs(e_cur - e_prev) < cfg->energy_threshold) {
            converged = 1;
            break;
        }
        CD_RC(rotate_spin(ctx, 0, Fa));
        CD_RC(occupied_density(ctx, ctx->spin[0].C.as<double>(), na, pref[0]));
        if (na != nb) {
            CD_RC(rotate_spin(ctx, 1, Fb));
            CD_RC(occupied_density(ctx, ctx->spin[1].C.as<double>(), nb, pref[1]));
        } else {
            // closed-shell count: beta follows alpha (reference :481-484)
            CD_CUDA(cudaMemcpyAsync(ctx->spin[1].C.p, ctx->spin[0].C.p, sizeof(double) * NN,
                                    cudaMemcpyDeviceToDevice, ctx->stream));
            CD_RC(invalidate_spin(ctx, 1));
            CD_CUDA(cudaMemcpyAsync(pref[1], pref[0], sizeof(double) * NN, cudaMemcpyDeviceToDevice,
                                    ctx->stream));
        }
        e_prev = e_cur;
    }
    CD_CUDA(cudaEventRecord(e1, ctx->stream));
    CD_CUDA(cudaEventSynchronize(e1));
    collect_stages(ctx);
    float ms = 0.0f;
    CD_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    res->energy_scf = cfg->e_scf;
    res->energy_mp2_corr = e_corr;
    res->energy_total = e_prev;   // the reference reports the previous iterate's total
    res->iterations = iter;
    res->converged = converged;
    res->ms_total = ms;
    return MSHQC_CD_OK;
}

MSHQC_CD_API int mshqc_cd_cholesky_fock(mshqc_cd_ctx* ctx, int nspin, const double* P_a, const double* P_b,
                                        const double* H, int screen_exchange, double* F_a, double* F_b,
                                        double* J, double* K_a, double* K_b, int where) {
    if (!ctx) return set_error(MSHQC_CD_ERR_ARG, "null context");
    if (nspin != 1 && nspin != 2) return set_error(MSHQC_CD_ERR_ARG, "nspin must be 1 (RHF) or 2 (UHF)");
    if (!P_a || (nspin == 2 && !P_b)) return set_error(MSHQC_CD_ERR_ARG, "density missing");
    if ((F_a || (nspin == 2 && F_b)) && !H) return set_error(MSHQC_CD_ERR_ARG, "a Fock matrix needs H");
    if (where != MSHQC_CD_HOST && where != MSHQC_CD_DEVICE) return set_error(MSHQC_CD_ERR_ARG, "bad where");
    if (!ctx->L_set) return set_error(MSHQC_CD_ERR_STATE, "set_vectors (or gen_vectors) must come first");
    DeviceGuard g(ctx->device);
    reset_stages(ctx);
    const int64_t NN = ctx->N * ctx->N;
    // P_a P_b H | J K_a K_b | F work
    CD_ALLOC_FIRST(ctx->opdm, sizeof(double) * (size_t)(8 * NN), false);
    double* base = ctx->opdm.as<double>();
    double* P[2] = {base, base + NN};
    double* Hd = base + 2 * NN;
    double* Jd = base + 3 * NN;
    double* Kd[2] = {base + 4 * NN, base + 5 * NN};
    double* Fd = base + 6 * NN;
    double* work = base + 7 * NN;
    const double* in[3] = {P_a, nspin == 2 ? P_b : nullptr, H};
    double* dst[3] = {P[0], P[1], Hd};
    for (int k = 0; k < 3; ++k) {
        if (!in[k]) continue;
        if (where == MSHQC_CD_HOST)
            CD_RC(upload(ctx, dst[k], in[k], sizeof(double) * NN));
        else
            CD_CUDA(cudaMemcpyAsync(dst[k], in[k], sizeof(double) * NN, cudaMemcpyDeviceToDevice, ctx->stream));
    }
    const double* Pc[2] = {P[0], P[1]};
    begin_stage(ctx, ST_OTHER);
    CD_RC(cholesky_jk_device(ctx, nspin, Pc, nspin == 1 && screen_exchange != 0, Jd, Kd, work));
    end_stage(ctx);
    if (J) CD_RC(download(ctx, J, Jd, sizeof(double) * NN, where));
    double* Kout[2] = {K_a, K_b};
    double* Fout[2] = {F_a, F_b};
    // RHF (src/scf/cholesky_rhf.cc:136): F = H + J - K/2 with the total density;
    // UHF (src/scf/cholesky_uhf.cc:90-98): F_s = H + J - K_s
    const double kf = nspin == 1 ? -0.5 : -1.0;
    for (int s = 0; s < nspin; ++s) {
        if (Kout[s]) CD_RC(download(ctx, Kout[s], Kd[s], sizeof(double) * NN, where));
        if (Fout[s]) {
            axpy_kernel<<<blocks_for(NN), 256, 0, ctx->stream>>>(Hd, 1.0, Jd, NN, Fd);
            axpy_kernel<<<blocks_for(NN), 256, 0, ctx->stream>>>(Fd, kf, Kd[s], NN, Fd);
            CD_CUDA(cudaGetLastError());
            ctx->launches += 2;
            CD_RC(download(ctx, Fout[s], Fd, sizeof(double) * NN, where));
        }
    }
    CD_CUDA(cudaStreamSynchronize(ctx->stream));
    collect_stages(ctx);
    return MSHQC_CD_OK;
}

}  // extern "C"

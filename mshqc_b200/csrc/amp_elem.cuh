// Element-wise amplitude pass of the MP2 backward.
//
// Input: a staging block of integrals S[(i - i0, a)][(j, b)] = (ia|jb) for
// the occupied rows i of one block and every j (FP32 from vtile_tc.cuh, or
// FP64 from the FP64 GEMM), 32 x 32 tiles with D = e_i + e_j - e_a - e_b
// (|D| < 1e-12 skipped, reference src/mp2/cholesky_rmp2.cc:139):
//
//   RESTRICTED     V = (ia|jb), W = (ib|ja); t = V/D, amplitude tt = (2V - W)/D,
//                  energy V tt, r = t tt          (dE/dB = 4 Gamma)
//   SAME_SPIN      g = V - W, amplitude t = g/D, energy g t / 4, r = t^2 / 4
//                                                  (dE/dB = 2 Gamma)
//   OPPOSITE_SPIN  X alpha, Y beta; amplitude t = V/D, energy V t, r = t^2
//                  (dE/dB_alpha = 2 Gamma_alpha, dE/dB_beta = 2 Gamma_beta)
//
// The energies are those of reference src/mp2/cholesky_rmp2.cc:135-151 and
// src/mp2/cholesky_ump2.cc:316-346, :436-453 summed over ordered pairs.
// Gamma = amplitude x B is formed afterwards by a GEMM with K = (j, b); this
// pass writes the amplitude operand of that GEMM: BF16 hi/lo in the blocked
// K-major layout of the tensor-core Gamma kernel (SPLIT), or FP64 row-major
// [(i - i0, a)][(j, b)] for the FP64 GEMM.  With SPLIT it can also write the
// transposed operand [(j, b)][(i - i0, a)]: Gamma_beta of the opposite-spin
// pass, or, for the symmetric modes (t^{ji}_{ba} = t^{ij}_{ab}), the rows j of
// a block pair (I, J) whose mirror (J, I) is not computed.
// Symmetric modes (amp_sym_kernel): the tiles (A, B) and (B, A) of a pair go
// together, so an integral is read once (it is V of one element and W of the
// other), and the two elements share D and 1/D.  Row and column sums land in the
// same place (dE/de of one spin), so one vector per pair holds both.
// Opposite spin (amp_os_kernel): one tile at a time, row sums per a and column
// sums per b.  A CTA of 256 threads takes a pair, or a share of its tiles, and
// loads the next tile while it works on the current one; per-pair sums are
// written by one thread each, and deps_*_kernel turn them into dE/de (+r on a
// and b, -r on i and j) in a fixed order.
// Bound by HBM traffic and, next to it, by FP64 arithmetic and conversions: the
// mixed path reads 4 bytes of S and writes 4 of hi/lo per amplitude and operand.
// An amplitude is split into hi and lo once, in registers, and the operands'
// 16-byte rows are gathered from the packed words; with mirrored tiles apart
// (every integral read twice, every 1/D taken twice) and one split per operand
// the pass took 32.3 ms of the N = 1000, o = 100 restricted mixed backward and
// 12.9 ms of the N = 600 unrestricted one, now 20.0 and 9.6 (4.1 TB/s at
// N = 1000); FP64, N = 600, o = 60: 4.8 -> 3.7 ms.  The CTAs per SM
// do not matter: 20.7, 21.3, 19.9, 21.9 ms with 3, 4, 5, 6 (mixed, N = 1000), the
// spread of one setting.
#pragma once

#include <cuda_bf16.h>

#include <type_traits>

#include "cd_common.cuh"
#include "sm100_ptx.cuh"

namespace mshqc_cd {

enum AmpMode { AMP_RESTRICTED = 0, AMP_SAME_SPIN = 1, AMP_OPPOSITE_SPIN = 2 };

struct AmpElemArgs {
    const void* S;          // float (SPLIT) or double
    long long ldS;          // row length of S
    int rsx;                // rows per occupied i in S and in the output (multiple of 32)
    int csy;                // columns per occupied j in S, rows of the transposed output (multiple of 32)
    int ksy;                // output K per occupied j (multiple of 32, >= csy)
    int ksx;                // K per occupied i of the transposed output (multiple of 32, >= rsx)
    int ox, oy, vx, vy, i0, nbi;   // oy: all column orbitals (pair index i * oy + j)
    int j0, nbj;            // the column orbitals of this block: j0 .. j0 + nbj - 1
    double wgt;             // weight of the pair sums (2 when the mirror block (J, I) is skipped)
    const double* eox; const double* evx;   // energies of the row spin
    const double* eoy; const double* evy;   // of the column spin
    uint16_t* A16; long long nkA;   // SPLIT: hi / lo operand, rows R = ii*rsx + a, K = jj*ksy + b (nkA = K / 16)
    uint16_t* T16; long long nkT;   // SPLIT, optional transpose: rows jj*csy + b, K = ii*ksx + a
    double* A64; long long ldA;                   // FP64: [R][K], K = jj*ksy + b
    double* partial;        // [ox * oy] energy of each pair (i, j), i over all row orbitals
    double* prow;           // opposite spin: [ox * oy][rsx] sum_b r per pair and row a (or null)
    double* pcol;           // [ox * oy][csy] sum_a r per pair and column b; symmetric modes: row and
                            // column sums of a pair together (or null)
    double* pocc;           // [ox * oy] sum_ab r per pair (or null)
    // nchunk > 1: each pair's row tiles are split over nchunk CTAs (CTA
    // lp * nchunk + c takes chunk c of local pair lp = ii * nbj + jj); their
    // column sums, energies and totals go to cpcol [lp][c][csy], cpart and
    // cpocc [lp][c], and amp_chunks_combine_kernel adds the chunks in order
    int nchunk;
    double* cpcol; double* cpart; double* cpocc;
    // tri: a diagonal block pair of the symmetric modes with only its pairs
    // ii <= jj (nbi == nbj, local pairs in the order of vtile_pair): an
    // off-diagonal pair stands for (i, j) and (j, i) -- weight 2 -- and its
    // transposed amplitudes go into the same operand (T16 = A16)
    int tri;
};

namespace amp_detail {
// local pair lp -> (ii, jj), row-major or the upper triangle (see tri)
__device__ __forceinline__ void local_pair(const AmpElemArgs& p, int lp, int& ii, int& jj) {
    if (!p.tri) {
        ii = lp / p.nbj;
        jj = lp % p.nbj;
        return;
    }
    int r = lp, i = 0;
    while (r >= p.nbi - i) {
        r -= p.nbi - i;
        ++i;
    }
    ii = i;
    jj = i + r;
}
}  // namespace amp_detail

namespace amp_detail {
// blocked K-major element offset of hi of (row R, column k) in the operand
// layout of the Gamma kernel (lo: + 2048): 128-row blocks, each holding its nkc
// 16-wide K chunks one after the other (so consecutive K chunks of a tile are
// one copy), the hi slab and then the lo slab in a chunk, 8 x 8 core matrices
// inside a slab
__device__ __forceinline__ long long blocked_offset(long long R, long long k, long long nkc) {
    return ((R >> 7) * nkc + (k >> 4)) * 4096 + (((R & 127) >> 3) * 16 + ((k & 15) >> 3) * 8 + (R & 7)) * 8 +
           (k & 7);
}

// amplitude -> BF16 hi (low half word) and lo (high half word)
__device__ __forceinline__ uint32_t split_amp(double t) {
    const __nv_bfloat16 h = __double2bfloat16(t);
    const __nv_bfloat16 l = __double2bfloat16(t - (double)__bfloat162float(h));
    return (uint32_t)__bfloat16_as_ushort(h) | ((uint32_t)__bfloat16_as_ushort(l) << 16);
}

// 32 x 32 amplitude tile T (rows R0.., columns k0..; transposed: the tile's
// transpose) -> hi/lo operand: job = 0 .. 127 writes 8 consecutive k of one row,
// 16 bytes of hi and 16 of lo; a warp fills four 128-byte lines of each
__device__ __forceinline__ void store_tile(const uint32_t (*T)[33], bool transposed, int job, long long R0,
                                           long long k0, long long nk, uint16_t* dst) {
    const int r = job >> 2, g = job & 3;
    const uint32_t* t = transposed ? &T[g * 8][r] : &T[r][g * 8];
    const int step = transposed ? 33 : 1;
    uint32_t w[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) w[e] = t[e * step];
    uint16_t* d = dst + blocked_offset(R0 + r, k0 + g * 8, nk);
    *reinterpret_cast<uint4*>(d) = make_uint4(__byte_perm(w[0], w[1], 0x5410), __byte_perm(w[2], w[3], 0x5410),
                                              __byte_perm(w[4], w[5], 0x5410), __byte_perm(w[6], w[7], 0x5410));
    *reinterpret_cast<uint4*>(d + 2048) =
        make_uint4(__byte_perm(w[0], w[1], 0x7632), __byte_perm(w[2], w[3], 0x7632),
                   __byte_perm(w[4], w[5], 0x7632), __byte_perm(w[6], w[7], 0x7632));
}
}  // namespace amp_detail

template <bool SPLIT>
__global__ void __launch_bounds__(256, SPLIT ? 5 : 4) amp_os_kernel(AmpElemArgs p) {
    using TS = typename std::conditional<SPLIT, float, double>::type;
    __shared__ TS Vt[32][33];
    __shared__ uint32_t T[SPLIT ? 32 : 1][33];   // amplitudes as BF16 hi and lo
    __shared__ double colpart[8][33];
    __shared__ double red_e[8], red_r[8];
    const TS* S = static_cast<const TS*>(p.S);
    const int ta = p.rsx / 32, tb = p.csy / 32;
    const int R = p.nchunk > 1 ? p.nchunk : 1;
    const int lp = (int)(blockIdx.x / R), ch = (int)(blockIdx.x % R);
    const int ii = lp / p.nbj, jj = lp % p.nbj;
    const double wgt = p.wgt;
    const bool write_t = p.T16 != nullptr;
    const int xb0 = ch * ta / R, xb1 = (ch + 1) * ta / R;   // this CTA's row tiles
    const int i = p.i0 + ii, j = p.j0 + jj;
    const long long pair = (long long)i * p.oy + j;          // over all occupied rows
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;   // 32 x 8
    const double eij = p.eox[i] + p.eoy[j];
    double* prow = p.prow ? p.prow + pair * p.rsx : nullptr;
    double* pcol = !p.pcol ? nullptr
                   : R == 1 ? p.pcol + pair * p.csy
                            : p.cpcol + ((long long)lp * R + ch) * p.csy;
    const TS* Srow = S + (long long)ii * p.rsx * p.ldS + (long long)jj * p.csy;
    // this thread's four elements of tile (a0, b0): rows ty + 8k, column tx
    auto load_tile = [&](int a0, int b0, TS (&v)[4]) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = ty + 8 * k;
            // streaming loads: the staging is read here and never again
            v[k] = __ldcs(Srow + (long long)(a0 + r) * p.ldS + b0 + tx);
        }
    };
    TS vn[4];
    if (xb0 < xb1) load_tile(xb0 * 32, 0, vn);
    double esum = 0.0, rtot = 0.0;
    // row blocks outer, column blocks inner: a thread's rows stay fixed over
    // the inner loop, so their sums over b stay in registers; the column sums
    // of a tile are reduced across the warps and added to pcol in xb order
    for (int xb = xb0; xb < xb1; ++xb) {
        const int a0 = xb * 32;
        double rsum[4] = {0.0, 0.0, 0.0, 0.0};
        for (int yb = 0; yb < tb; ++yb) {
            const int b0 = yb * 32;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                Vt[ty + 8 * k][tx] = vn[k];
            }
            // the next tile's loads overlap this tile's arithmetic and stores
            if (yb + 1 < tb)
                load_tile(a0, b0 + 32, vn);
            else if (xb + 1 < xb1)
                load_tile(a0 + 32, 0, vn);
            __syncthreads();
            double cp = 0.0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int r = ty * 4 + k;
                const int a = a0 + r, b = b0 + tx;
                double amp = 0.0, rr = 0.0;
                if (a < p.vx && b < p.vy) {
                    const double D = eij - p.evx[a] - p.evy[b];
                    if (fabs(D) >= kDenomSkip) {
                        const double V = (double)Vt[r][tx];
                        const double rD = SPLIT ? sm100::recip_nr(D) : 1.0 / D;
                        amp = V * rD;
                        rr = amp * amp;
                        esum = fma(V, amp, esum);
                    }
                }
                rsum[k] += rr;
                cp += rr;
                if (SPLIT)
                    T[r][tx] = amp_detail::split_amp(amp);
                else
                    p.A64[((long long)ii * p.rsx + a) * p.ldA + (long long)jj * p.ksy + b] = amp;
            }
            rtot += cp;
            colpart[ty][tx] = cp;
            __syncthreads();
            if (SPLIT) {
                if (threadIdx.x < 128)
                    amp_detail::store_tile(T, false, threadIdx.x, (long long)ii * p.rsx + a0,
                                           (long long)jj * p.ksy + b0, p.nkA, p.A16);
                else if (write_t)
                    amp_detail::store_tile(T, true, threadIdx.x - 128, (long long)jj * p.csy + b0,
                                           (long long)ii * p.ksx + a0, p.nkT, p.T16);
            }
            if (pcol && ty == 0) {
                double c = 0.0;
#pragma unroll
                for (int w = 0; w < 8; ++w) c += colpart[w][tx];
                pcol[b0 + tx] = (xb == xb0 ? 0.0 : pcol[b0 + tx]) + wgt * c;
            }
            __syncthreads();   // Vt, T, colpart are refilled by the next tile
        }
        if (prow) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                double rs = rsum[k];
#pragma unroll
                for (int off = 16; off; off >>= 1) rs += __shfl_xor_sync(0xffffffffu, rs, off);
                if (tx == 0) prow[a0 + ty * 4 + k] = wgt * rs;
            }
        }
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        esum += __shfl_xor_sync(0xffffffffu, esum, off);
        rtot += __shfl_xor_sync(0xffffffffu, rtot, off);
    }
    if (tx == 0) {
        red_e[ty] = esum;
        red_r[ty] = rtot;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double e = 0.0, r = 0.0;
        for (int w = 0; w < 8; ++w) {
            e += red_e[w];
            r += red_r[w];
        }
        if (R == 1) {
            p.partial[pair] = wgt * e;
            if (p.pocc) p.pocc[pair] = wgt * r;
        } else {
            p.cpart[(long long)lp * R + ch] = wgt * e;
            if (p.pocc) p.cpocc[(long long)lp * R + ch] = wgt * r;
        }
    }
}

template <int MODE, bool SPLIT>
__global__ void __launch_bounds__(256, SPLIT ? 5 : 3) amp_sym_kernel(AmpElemArgs p) {
    static_assert(MODE != AMP_OPPOSITE_SPIN, "symmetric modes");
    using TS = typename std::conditional<SPLIT, float, double>::type;
    __shared__ TS Vs[32][33], Ws[32][33];
    // amplitudes (a, b) and (b, a), with SPLIT as BF16 hi and lo: split once, however
    // many operands take them
    using TA = typename std::conditional<SPLIT, uint32_t, double>::type;
    __shared__ TA T1[32][33], T2[32][33];
    __shared__ double colpart[8][33];
    __shared__ double rowbuf[32];
    __shared__ double red_e[8], red_r[8];
    const TS* S = static_cast<const TS*>(p.S);
    const int nt = p.rsx / 32, ntp = nt * (nt + 1) / 2;   // tiles a side, tile pairs A <= B
    const int R = p.nchunk > 1 ? p.nchunk : 1;
    const int lp = (int)(blockIdx.x / R), ch = (int)(blockIdx.x % R);
    int ii, jj;
    amp_detail::local_pair(p, lp, ii, jj);
    const double wgt = p.tri ? (ii < jj ? 2.0 : 1.0) : p.wgt;
    const bool write_t = p.T16 != nullptr && !(p.tri && ii == jj);
    // FP64 operand of a diagonal block pair: the (j, i) amplitudes go into A64
    // as the transposes of the (i, j) ones
    const bool write_t64 = !SPLIT && p.tri && ii != jj;
    const int i = p.i0 + ii, j = p.j0 + jj;
    const long long pair = (long long)i * p.oy + j;          // over all occupied rows
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;   // 32 x 8
    const double eij = p.eox[i] + p.eoy[j];
    double* psum = !p.pcol ? nullptr
                   : R == 1 ? p.pcol + pair * p.csy
                            : p.cpcol + ((long long)lp * R + ch) * p.csy;
    // lane tx of warp 0 alone touches the elements of psum that are tx mod 32
    if (psum && ty == 0)
        for (int b = tx; b < p.csy; b += 32) psum[b] = 0.0;
    const TS* Srow = S + (long long)ii * p.rsx * p.ldS + (long long)jj * p.csy;
    const int t0 = (int)((long long)ch * ntp / R), t1 = (int)((long long)(ch + 1) * ntp / R);
    int A = 0, B = t0;
    while (B >= nt - A) {
        B -= nt - A;
        ++A;
    }
    B += A;
    TS vn[4], wn[4];
    auto load = [&](int a0, int b0) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = ty + 8 * k;
            // streaming loads: the staging is read here and never again
            vn[k] = __ldcs(Srow + (long long)(a0 + r) * p.ldS + b0 + tx);
            if (a0 != b0) wn[k] = __ldcs(Srow + (long long)(b0 + r) * p.ldS + a0 + tx);
        }
    };
    if (t0 < t1) load(A * 32, B * 32);
    double esum = 0.0, rtot = 0.0;
    double rsum[4] = {0.0, 0.0, 0.0, 0.0};
    for (int t = t0; t < t1; ++t) {
        const int a0 = A * 32, b0 = B * 32;
        const bool diag = a0 == b0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            Vs[ty + 8 * k][tx] = vn[k];
            Ws[ty + 8 * k][tx] = diag ? vn[k] : wn[k];
        }
        const bool row_end = B + 1 == nt || t + 1 == t1;   // last tile of this row block here
        if (++B == nt) {
            ++A;
            B = A;
        }
        // the next tile's loads overlap this tile's arithmetic and stores
        if (t + 1 < t1) load(A * 32, B * 32);
        __syncthreads();
        double cp = 0.0;
        const int b = b0 + tx;
        const double eb = b < p.vy ? eij - p.evy[b] : 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = ty * 4 + k, a = a0 + r;
            double amp1 = 0.0, amp2 = 0.0, rr = 0.0;
            if (a < p.vx && b < p.vy) {
                const double D = eb - p.evx[a];
                if (fabs(D) >= kDenomSkip) {
                    const double V = (double)Vs[r][tx], W = (double)Ws[tx][r];
                    const double rD = SPLIT ? sm100::recip_nr(D) : 1.0 / D;
                    if (MODE == AMP_RESTRICTED) {
                        amp1 = (2.0 * V - W) * rD;
                        rr = V * rD * amp1;
                        esum = fma(V, amp1, esum);
                        if (!diag) {
                            amp2 = (2.0 * W - V) * rD;
                            rr = fma(W * rD, amp2, rr);
                            esum = fma(W, amp2, esum);
                        }
                    } else {
                        const double g = V - W;
                        amp1 = g * rD;
                        rr = 0.25 * amp1 * amp1;
                        double e = 0.25 * g * amp1;
                        if (!diag) {
                            amp2 = -amp1;
                            rr += rr;
                            e += e;
                        }
                        esum += e;
                    }
                }
            }
            rsum[k] += rr;
            cp += rr;
            if constexpr (SPLIT) {
                T1[r][tx] = amp_detail::split_amp(amp1);
                if (!diag) T2[tx][r] = amp_detail::split_amp(amp2);
            } else {
                T1[r][tx] = amp1;
                if (!diag) T2[tx][r] = amp2;
                p.A64[((long long)ii * p.rsx + a) * p.ldA + (long long)jj * p.ksy + b] = amp1;
            }
        }
        rtot += cp;
        if (psum) {
            colpart[ty][tx] = cp;
            if (row_end) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    double rs = rsum[k];
#pragma unroll
                    for (int off = 16; off; off >>= 1) rs += __shfl_xor_sync(0xffffffffu, rs, off);
                    if (tx == 0) rowbuf[ty * 4 + k] = rs;
                    rsum[k] = 0.0;
                }
            }
        }
        __syncthreads();
        if constexpr (SPLIT) {
            // up to four operand tiles of 128 jobs: A (a, b), T of it, and their mirrors
            const int ntile = (diag ? 1 : 2) * (write_t ? 2 : 1);
            for (int job = threadIdx.x; job < 128 * ntile; job += 256) {
                const int which = job >> 7;
                const bool second = diag ? false : (which & 1) != 0;      // the tile (b, a)
                const bool trans = diag ? which == 1 : which >= 2;
                const uint32_t(*T)[33] = second ? T2 : T1;
                const int ra = second ? b0 : a0, rb = second ? a0 : b0;   // its row and column virtuals
                if (!trans)
                    amp_detail::store_tile(T, false, job & 127, (long long)ii * p.rsx + ra,
                                           (long long)jj * p.ksy + rb, p.nkA, p.A16);
                else
                    amp_detail::store_tile(T, true, job & 127, (long long)jj * p.csy + rb,
                                           (long long)ii * p.ksx + ra, p.nkT, p.T16);
            }
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int r = ty + 8 * k;
                if (!diag)
                    p.A64[((long long)ii * p.rsx + b0 + r) * p.ldA + (long long)jj * p.ksy + a0 + tx] = T2[r][tx];
                if (write_t64) {   // rows (j, b) of the operand, columns (i, a), and the mirror
                    p.A64[((long long)jj * p.ksy + b0 + r) * p.ldA + (long long)ii * p.rsx + a0 + tx] = T1[tx][r];
                    if (!diag)
                        p.A64[((long long)jj * p.ksy + a0 + r) * p.ldA + (long long)ii * p.rsx + b0 + tx] = T2[tx][r];
                }
            }
        }
        if (psum && ty == 0) {
            double c = 0.0;
#pragma unroll
            for (int w = 0; w < 8; ++w) c += colpart[w][tx];
            psum[b0 + tx] += wgt * c;
            if (row_end) psum[a0 + tx] += wgt * rowbuf[tx];
        }
        __syncthreads();   // the shared tiles are refilled by the next tile pair
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        esum += __shfl_xor_sync(0xffffffffu, esum, off);
        rtot += __shfl_xor_sync(0xffffffffu, rtot, off);
    }
    if (tx == 0) {
        red_e[ty] = esum;
        red_r[ty] = rtot;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double e = 0.0, r = 0.0;
        for (int w = 0; w < 8; ++w) {
            e += red_e[w];
            r += red_r[w];
        }
        if (R == 1) {
            p.partial[pair] = wgt * e;
            if (p.pocc) p.pocc[pair] = wgt * r;
        } else {
            p.cpart[(long long)lp * R + ch] = wgt * e;
            if (p.pocc) p.cpocc[(long long)lp * R + ch] = wgt * r;
        }
    }
}

// The chunk partials of the kernels above (nchunk > 1) of the nbi x nbj local
// pairs added in chunk order into the per-pair outputs: one thread per
// (local pair, column b); the b == 0 thread also does energy and total.
static __global__ void amp_chunks_combine_kernel(AmpElemArgs p, int npl) {
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (idx >= (long long)npl * p.csy) return;
    const int lp = (int)(idx / p.csy), b = (int)(idx % p.csy);
    const int R = p.nchunk;
    int ii, jj;
    amp_detail::local_pair(p, lp, ii, jj);
    const long long pair = (long long)(p.i0 + ii) * p.oy + p.j0 + jj;
    if (p.pcol) {
        double sc = 0.0;
        for (int c = 0; c < R; ++c) sc += p.cpcol[((long long)lp * R + c) * p.csy + b];
        p.pcol[pair * p.csy + b] = sc;
    }
    if (b == 0) {
        double e = 0.0, r = 0.0;
        for (int c = 0; c < R; ++c) {
            e += p.cpart[(long long)lp * R + c];
            if (p.pocc) r += p.cpocc[(long long)lp * R + c];
        }
        p.partial[pair] = e;
        if (p.pocc) p.pocc[pair] = r;
    }
}

template <int MODE, bool SPLIT>
inline void launch_amp(const AmpElemArgs& e, int64_t ctas, cudaStream_t st) {
    if constexpr (MODE == AMP_OPPOSITE_SPIN)
        amp_os_kernel<SPLIT><<<(unsigned)ctas, 256, 0, st>>>(e);
    else
        amp_sym_kernel<MODE, SPLIT><<<(unsigned)ctas, 256, 0, st>>>(e);
}

// dE/de from the per-pair sums, in a fixed order (no atomics):
// deps_x[ox + a] += sum_pairs prow, deps_y[oy + b] += sum_pairs pcol,
// deps_x[i] -= sum_j pocc[i][j], deps_y[j] -= sum_i pocc[i][j]
// 16 columns x 64 pair lanes per CTA: one thread per column walked every pair
// alone and took 2.1 ms (N = 600, six calls) of latency; here 0.1 ms.
static __global__ void __launch_bounds__(1024) deps_rows_kernel(const double* __restrict__ prow, long long npairs,
                                                                int rsx, int v, double* __restrict__ dvir) {
    __shared__ double red[64][17];
    const int c = threadIdx.x & 15, g = threadIdx.x >> 4;
    const int a = blockIdx.x * 16 + c;
    double s0 = 0.0, s1 = 0.0;
    if (a < v) {
        long long q = g;
        for (; q + 64 < npairs; q += 128) {
            s0 += prow[q * rsx + a];
            s1 += prow[(q + 64) * rsx + a];
        }
        if (q < npairs) s0 += prow[q * rsx + a];
    }
    red[g][c] = s0 + s1;
    __syncthreads();
    for (int h = 32; h > 0; h >>= 1) {
        if (g < h) red[g][c] += red[g + h][c];
        __syncthreads();
    }
    if (g == 0 && a < v) dvir[a] += red[0][c];
}

// (dx and dy may be the same array: thread t touches only element t of each)
static __global__ void deps_occ_kernel(const double* __restrict__ pocc, int ox, int oy, double* __restrict__ dx,
                                       double* __restrict__ dy) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < ox) {
        double s = 0.0;
        for (int j = 0; j < oy; ++j) s += pocc[(long long)t * oy + j];
        dx[t] -= s;
    }
    if (t < oy) {
        double s = 0.0;
        for (int i = 0; i < ox; ++i) s += pocc[(long long)i * oy + t];
        dy[t] -= s;
    }
}

}  // namespace mshqc_cd

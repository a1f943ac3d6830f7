// Pair energies from staged FP64 integrals (the FP64 energy path of larger
// systems).
//
// Input: a block S[(i - i0, a)][(j - j0, b)] = (ia|jb), rows of vpx and columns
// of vpy per occupied orbital (multiples of 64), from the int8-slice products
// of full accuracy (ozaki_i8.cuh).  One CTA takes a share of the 32 x 32 tiles
// of one pair (i, j); in the symmetric modes a tile (A, B), A <= B, comes with
// its mirror tile, so V = (ia|jb) and W = (ib|ja) are both at hand and the
// formulas and weights are those of pair_energy_f64.cuh.  The share's
// compensated sum goes to partial[pair * nchunk + chunk], the pairs numbered as
// in the tables of the fused kernels.
//
// HBM bound: 8 bytes per integral, read once.  N = 400, o = 40: 0.25 ms; the
// fused DMMA kernel it stands in for took 14.4 ms (24 TF/s), the products into
// the staging block take 3.6 ms.
#pragma once

#include "cd_common.cuh"
#include "pair_energy_f64.cuh"

namespace mshqc_cd {

struct PairStagedArgs {
    const double* S;
    long long ldS;
    int vpx, vpy, vx, vy;
    int ox, oy;             // all occupied orbitals of the two spins
    int i0, nbi, j0, nbj;   // the block's orbitals
    int nchunk;
    const double* eox; const double* evx;
    const double* eoy; const double* evy;
    double* partial;
    double* partial2;       // RESTRICTED: opposite-spin part
};

template <int MODE>
__global__ void __launch_bounds__(256, 4) pair_energy_staged_kernel(PairStagedArgs p) {
    constexpr bool kSym = MODE != PAIR_OPPOSITE_SPIN;
    __shared__ double Wt[2][kSym ? 32 : 1][33];
    __shared__ double red_s[2][8], red_c[2][8];
    const int ch = (int)(blockIdx.x % p.nchunk), lp = (int)(blockIdx.x / p.nchunk);
    const int ii = lp / p.nbj, jj = lp % p.nbj;
    const int i = p.i0 + ii, j = p.j0 + jj;
    if (kSym && (j < i || (MODE == PAIR_SAME_SPIN && j == i))) return;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int ta = p.vpx / 32, tb = p.vpy / 32;
    const int nt = kSym ? ta * (ta + 1) / 2 : ta * tb;
    const int t0 = (int)((long long)ch * nt / p.nchunk), t1 = (int)((long long)(ch + 1) * nt / p.nchunk);
    // tile t0 of the row-major (upper-triangular) order
    int A = 0, B = 0;
    if (kSym) {
        int r = t0;
        while (r >= ta - A) {
            r -= ta - A;
            ++A;
        }
        B = A + r;
    } else {
        A = t0 / tb;
        B = t0 % tb;
    }
    const double* Sp = p.S + (long long)ii * p.vpx * p.ldS + (long long)jj * p.vpy;
    const double eij = p.eox[i] + p.eoy[j];
    KSum sum, sum2;
    sum.init();
    sum2.init();
    double v[4], w[4];
    auto load = [&](int a0, int b0) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = ty + 8 * k;
            v[k] = __ldcs(Sp + (long long)(a0 + r) * p.ldS + b0 + tx);
            if (kSym) w[k] = __ldcs(Sp + (long long)(b0 + r) * p.ldS + a0 + tx);
        }
    };
    if (t0 < t1) load(A * 32, B * 32);
    for (int t = t0; t < t1; ++t) {
        const int a0 = A * 32, b0 = B * 32;
        double cv[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            cv[k] = v[k];
            if (kSym) Wt[t & 1][ty + 8 * k][tx] = w[k];
        }
        if (++B == tb) {
            ++A;
            B = kSym ? A : 0;
        }
        if (t + 1 < t1) load(A * 32, B * 32);
        if (kSym) __syncthreads();   // the other buffer is written before the next barrier
        const int b = b0 + tx;
        const double weight = !kSym ? 1.0 : MODE == PAIR_RESTRICTED ? (a0 == b0 ? 1.0 : 2.0) : (a0 == b0 ? 0.5 : 1.0);
        if (b < p.vy) {
            const double eb = eij - p.evy[b];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int a = a0 + ty + 8 * k;
                if (a >= p.vx) continue;
                const double D = eb - p.evx[a];
                if (fabs(D) < kDenomSkip) continue;
                const double V = cv[k];
                if (MODE == PAIR_RESTRICTED) {
                    const double W = Wt[t & 1][tx][ty + 8 * k];
                    const double rD = weight * (1.0 / D);
                    sum.add((V * V + W * W - V * W) * rD);
                    sum2.add((V * V + W * W) * rD);
                } else if (MODE == PAIR_SAME_SPIN) {
                    const double g = V - Wt[t & 1][tx][ty + 8 * k];
                    sum.add(weight * (g * g / D));
                } else {
                    sum.add(V * V / D);
                }
            }
        }
    }
    if (MODE == PAIR_RESTRICTED) {
        // pair weight; the opposite-spin part counts V_ab^2 once per (a, b)
        const double w2 = i < j ? 2.0 : 1.0;
        sum.s *= w2;
        sum.c *= w2;
        sum2.s *= 0.5 * w2;
        sum2.c *= 0.5 * w2;
    }
    warp_reduce_ksum(sum);
    if (MODE == PAIR_RESTRICTED) warp_reduce_ksum(sum2);
    if (tx == 0) {
        red_s[0][ty] = sum.s;
        red_c[0][ty] = sum.c;
        red_s[1][ty] = sum2.s;
        red_c[1][ty] = sum2.c;
    }
    __syncthreads();
    if (threadIdx.x < (MODE == PAIR_RESTRICTED ? 2 : 1)) {
        KSum t;
        t.init();
        for (int k = 0; k < 8; ++k) {
            t.add(red_s[threadIdx.x][k]);
            t.c += red_c[threadIdx.x][k];
        }
        const long long pair = MODE == PAIR_RESTRICTED  ? (long long)i * p.ox - (long long)i * (i - 1) / 2 + (j - i)
                               : MODE == PAIR_SAME_SPIN ? (long long)i * (p.ox - 1) - (long long)i * (i - 1) / 2 + (j - i - 1)
                                                        : (long long)i * p.oy + j;
        (threadIdx.x == 0 ? p.partial : p.partial2)[pair * p.nchunk + ch] = t.value();
    }
}

}  // namespace mshqc_cd

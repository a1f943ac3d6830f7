// Which tiles of a sliced FP64 product (ozaki_i8.cuh, Full) the FP64 product has
// to compute.
//
// A slice holds an element to a multiple of 2^{e-54}, 2^e just above its row's
// maximum, so its rounding error does not shrink with the element.  An FP64
// chain errs relative to the terms x_k y_k themselves.  Where two rows are
// large in different places (orbitals far apart, graded rows) the terms are far
// below 2^{e_x + e_y} and the sliced result would be the worse one: with two
// rows of 400 elements that are 10^-6 of their maxima where the other is large,
// 10^5 times.  Rounding errors taken as independent and uniform, in units of
// 2^{e_x + e_y} and with q = (x / 2^{e_x})^2:
//   chain of K terms   2^-54.7 sqrt(K sum_k q_x q_y)
//   slices             2^-55.8 sqrt(sum_k q_x + sum_k q_y)
// so the slices are the better ones where G = sum_k q_x q_y exceeds
// 0.22 (mean q_x + mean q_y).  A tile is taken when every output of it has
// G >= 0.25 (mean q_x + mean q_y).  Restated against exact sums for Gaussian,
// graded, same-sign and heavy-tailed rows and for pairs of fragments, K = 60 ...
// 1600: the two errors meet at 0.2 ... 0.25.
//
// The means come with the slices (squares of the leading digits), and so do the
// squares of the first and the middle 32 elements of each row: G grows with
// every term, so a tile is decided as soon as all its outputs have passed, and
// rows of one kind mostly pass with these 64.  The other tiles go on with
// squares formed from the FP64 rows, 32 K at a time and scattered over K: taken
// in order, the core orbitals' columns of the amplitudes, small for every row,
// kept the Gamma tiles of N = 600 undecided for 2300 terms (6.9 ms of a 27 ms
// product).  A tile that has not passed after 8 such steps, or a sixteenth of K,
// is left out: deciding it over all of K takes half as long as its FP64 product
// (two fragments, N = 400, FP64 gradient: 59.9 ms, with the limit 40.3).  BF16
// squares, FP32 sums (positive terms: relative error below 2%), m16n8k16 MMAs; 8
// warps of 32 x 32 outputs, 4 CTAs per SM (N = 400 integrals: 163, 137, 116, 204
// us with 2, 3, 4, 5).
#pragma once

#include <cuda_bf16.h>

#include <algorithm>
#include <numeric>

#include "cd_common.cuh"
#include "ozaki_i8.cuh"

namespace mshqc_cd {

struct SliceGuardArgs {
    struct Side {
        const double* src;      // element (r, k): src + batch * sb + r * ld + k, or (t) + k * ld + r
        long long ld, sb;
        const int* e;           // raw row exponents, sums of the leading digits' squares, sampled squares
        const unsigned* sq;
        const uint32_t* sample;
        long long eb;           // rows per batch of both
        int R, t;
    } a, b;                     // 128-row and 64-row operand
    int K;
    int stride;                 // from one scattered K step to the next
    int limit;                  // scattered steps at most
    int nmb, nnb, group, tri;   // as in OzakiArgs
    uint8_t* left_out;          // per unit
    int* count;                 // units left out (zeroed) ...
    int* list;                  // ... and which
};

namespace slice_guard {
constexpr int KS = 32, LW = 36;     // K per step, 32-bit words per shared row (16, or 32 of the sample)

// least G of an output: the row's and the column's share add up
__device__ __forceinline__ float share(const SliceGuardArgs::Side& s, long long i, int r, int K) {
    if (r >= s.R) return -INFINITY;
    const int e = s.e[i];
    if (e == ozaki::kNoExponent) return -INFINITY;   // zeros: exact
    if (e == ozaki::kBadExponent || e < ozaki::kTinyExponent) return INFINITY;   // NaN, infinity; sliced as zero
    return 0.25f / 4096.0f * ((float)s.sq[i] / (float)K + 0.25f);
}

__device__ __forceinline__ int high(const double* x) { return __ldg(reinterpret_cast<const int*>(x) + 1); }

// one K step of ROWS rows from r0 on into shared rows of 32 BF16 squares; a
// thread takes pairs of consecutive k
template <int ROWS>
__device__ __forceinline__ void load(const SliceGuardArgs::Side& s, const double* src, const int* base, int r0, int k0,
                                     int K, uint32_t* sm) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int NJ = ROWS / 16;       // pairs per thread
    int x[NJ][2];
    if (!s.t) {   // two rows a warp, 16 lanes each
        const int r1 = warp * 2 + (lane >> 4), kp = lane & 15, k = k0 + 2 * kp;
        const double* q = src + (r0 + r1) * s.ld + k;
        const bool k0in = k < K, k1in = k + 1 < K;
#pragma unroll
        for (int j = 0; j < NJ; ++j, q += 16 * s.ld) {
            const bool in = r0 + r1 + 16 * j < s.R;
            x[j][0] = in && k0in ? high(q) : 0;
            x[j][1] = in && k1in ? high(q + 1) : 0;
        }
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const int r = r1 + 16 * j;
            sm[r * LW + kp] = ozaki::square_pair(x[j][0], x[j][1], base[r]);
        }
    } else {      // a warp per 32 rows and K pair
        constexpr int G = ROWS / 32;
        const int r1 = (warp % G) * 32 + lane, kp1 = warp / G, r = r0 + r1;
        const double* q = src + (k0 + 2 * kp1) * s.ld + r;
        const bool in = r < s.R;
#pragma unroll
        for (int j = 0; j < NJ; ++j, q += 2 * (8 / G) * s.ld) {
            const int k = k0 + 2 * (kp1 + j * (8 / G));
            x[j][0] = in && k < K ? high(q) : 0;
            x[j][1] = in && k + 1 < K ? high(q + s.ld) : 0;
        }
        const int b = base[r1];
#pragma unroll
        for (int j = 0; j < NJ; ++j) sm[r1 * LW + kp1 + j * (8 / G)] = ozaki::square_pair(x[j][0], x[j][1], b);
    }
}

// the sampled squares of ROWS rows: both chunks, 128 bytes a row
template <int ROWS>
__device__ __forceinline__ void load_sample(const uint32_t* sample, uint32_t* sm) {
#pragma unroll
    for (int j = 0; j < ROWS / 32; ++j) {
        const int x = threadIdx.x + 256 * j, r = x >> 3, w = (x & 7) * 4;
        *reinterpret_cast<uint4*>(sm + r * LW + w) =
            __ldg(reinterpret_cast<const uint4*>(sample + (long long)r * ozaki::SAMPLE_WORDS + w));
    }
}

// four 8 x 8 matrices of 16-bit elements; lane l gives the address of row l % 8
// of matrix l / 8
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const uint32_t* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(smem_u32(p)));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
}  // namespace slice_guard

// one CTA per unit (128 x 64 outputs)
static __global__ void __launch_bounds__(256, 4) slice_guard_kernel(SliceGuardArgs p) {
    using namespace slice_guard;
    constexpr int BM = 128, BN = 64;
    __shared__ __align__(16) uint32_t sa[BM * LW], sb[BN * LW];
    __shared__ float ta[BM], tb[BN];
    __shared__ int xa[BM], xb[BN];
    const long long u = blockIdx.x;
    long long b;
    int mb, nb;
    tile_of_unit(u, p.nmb, p.nnb, p.group, b, mb, nb);
    if (p.tri > 0 && nb * BN / p.tri < mb * BM / p.tri) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = mb * BM, c0 = nb * BN;
    load_sample<BM>(p.a.sample + (b * p.a.eb + r0) * ozaki::SAMPLE_WORDS, sa);
    load_sample<BN>(p.b.sample + (b * p.b.eb + c0) * ozaki::SAMPLE_WORDS, sb);
    if (tid < BM) {
        const long long i = b * p.a.eb + r0 + tid;
        ta[tid] = share(p.a, i, r0 + tid, p.K);
        xa[tid] = ozaki::square_base(p.a.e[i]);
    } else if (tid < BM + BN) {
        const int c = tid - BM;
        const long long i = b * p.b.eb + c0 + c;
        tb[c] = share(p.b, i, c0 + c, p.K);
        xb[c] = ozaki::square_base(p.b.e[i]);
    }
    __syncthreads();
    const double* A = p.a.src + b * p.a.sb;
    const double* B = p.b.src + b * p.b.sb;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32, g = lane >> 2, t = lane & 3;
    // sums that start at minus what they have to reach
    float acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float need = ta[wm + 16 * i + g + 8 * (q >> 1)] + tb[wn + 8 * j + 2 * t + (q & 1)];
                acc[i][j][q] = need == need ? -need : -INFINITY;   // (zeros against a NaN row: not taken)
            }
    // fragments: rows and 16-byte halves of a 16-wide K half that this lane addresses
    const uint32_t* fa = sa + (wm + (lane & 15)) * LW + (lane >> 4) * 4;
    const uint32_t* fb = sb + (wn + (lane & 7) + (lane >> 4) * 8) * LW + ((lane >> 3) & 1) * 4;
    auto multiply = [&](int halves) {   // 16-wide halves of a step
#pragma unroll 2
        for (int h = 0; h < halves; ++h) {
            uint32_t a0[4], a1[4], b0[4], b1[4];
            ldmatrix4(a0, fa + 8 * h);
            ldmatrix4(a1, fa + 16 * LW + 8 * h);
            ldmatrix4(b0, fb + 8 * h);              // columns 0 .. 7: k 0 .. 7, 8 .. 15; columns 8 .. 15
            ldmatrix4(b1, fb + 16 * LW + 8 * h);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                mma_bf16(acc[0][j], a0, b0[2 * j], b0[2 * j + 1]);
                mma_bf16(acc[1][j], a1, b0[2 * j], b0[2 * j + 1]);
                mma_bf16(acc[0][2 + j], a0, b1[2 * j], b1[2 * j + 1]);
                mma_bf16(acc[1][2 + j], a1, b1[2 * j], b1[2 * j + 1]);
            }
        }
        float least = INFINITY;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int q = 0; q < 4; ++q) least = fminf(least, acc[i][j][q]);
        return __syncthreads_and(least >= 0.0f) != 0;   // (also: the shared rows are read)
    };
    const int steps = (p.K + KS - 1) / KS, mid = ozaki::sample_chunk(steps), rest = steps - 2;
    bool passed = multiply(steps > 1 ? 4 : 2);
    // the other steps, scattered: stride, 2 stride, ... mod their number, coprime to it
    for (int n = 0, at = 0; n < p.limit && !passed; ++n) {
        const int k0 = (at + 1 < mid ? at + 1 : at + 2) * KS;
        if ((at += p.stride) >= rest) at -= rest;
        load<BM>(p.a, A, xa, r0, k0, p.K, sa);
        load<BN>(p.b, B, xb, c0, k0, p.K, sb);
        __syncthreads();
        passed = multiply(2);
    }
    if (tid == 0) {
        p.left_out[u] = passed ? 0 : 1;
        if (!passed) p.list[atomicAdd(p.count, 1)] = (int)u;
    }
}

// Decides every unit of the product of A (128-row operand) and B.
inline cudaError_t guard_slices(const OzakiOperand& A, const OzakiOperand& B, const OzakiOpts& o, uint8_t* left_out,
                               int* count, int* list, cudaStream_t st) {
    SliceGuardArgs p{};
    auto side = [](const OzakiOperand& x, bool shared) {
        SliceGuardArgs::Side s{};
        s.src = x.src;  s.ld = x.ld;  s.sb = shared ? 0 : x.sb;
        s.e = x.e;  s.sq = x.sq();  s.sample = x.smp;
        s.eb = shared ? 0 : x.Rp;
        s.R = (int)x.R;  s.t = x.t ? 1 : 0;
        return s;
    };
    p.a = side(A, o.a_shared);
    p.b = side(B, o.b_shared);
    p.K = (int)A.K;
    // about 0.62 of the scattered steps, coprime to their number
    const int steps = (p.K + slice_guard::KS - 1) / slice_guard::KS, rest = std::max(1, steps - 2);
    p.limit = std::min(std::max(0, steps - 2), std::max(8, steps / 16));
    p.stride = std::max(1, (int)(0.618 * rest));
    while (std::gcd(p.stride, rest) != 1) ++p.stride;
    p.nmb = (int)(A.Rp / 128);  p.nnb = (int)(B.Rp / 64);
    p.group = ozaki::GROUP;
    p.tri = o.tri;
    p.left_out = left_out;  p.count = count;  p.list = list;
    cudaError_t e = cudaMemsetAsync(count, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    const long long units = (long long)p.nmb * p.nnb * (o.a_shared ? B.batch : A.batch);
    slice_guard_kernel<<<(unsigned)units, 256, 0, st>>>(p);
    return cudaGetLastError();
}

}  // namespace mshqc_cd

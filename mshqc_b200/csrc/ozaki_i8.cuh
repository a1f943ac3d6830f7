// FP64 matrix products on the 8-bit integer tensor cores (tcgen05 kind::i8)
// by slicing, after Ozaki, Ogita, Oishi and Rump (error-free splitting of
// floating-point matrix products) in the integer form of Ootomo, Ozaki and
// Yokota ("DGEMM on integer matrix multiplication unit", 2024).
//
// Every row r of an operand is scaled by its own power of two 2^e_r with
// max_k |x_rk| < 2^e_r, rounded to a multiple of a fixed fraction of 2^e_r and
// cut into S signed 8-bit digits.  A row x times a row y is then a sum over
// digit pairs (s, t) of exact 32-bit integer tensor-core products; the pairs of
// equal s + t share an accumulator, and the epilogue combines the W
// accumulators (s + t < W) in 64-bit integers and rounds to FP64.
//
//  * Mixed (S = 5, W = 5): 35-bit integers, base-128 digits with the sign of
//    the number, the 15 pairs s + t < 5.  The error per term is below about
//    2^-32 2^{e_x + e_y}: for the mixed path, whose fixed-point splitting keeps
//    19 bits.  |sum| <= 5 127^2 K < 2^31 for K <= 26624.
//  * Full (S = 7, W = 8): multiples of 2^{e-54} (elements within a binade of
//    the row maximum are exact), base-256 digits in [-128, 127] (the bytes of
//    (m + c) ^ c with c = 128 in every byte), the 34 pairs s + t < 8.  Dropped
//    pairs are below 2^-59 2^{e_x + e_y} per term, the representation error
//    below 2^-55 2^e per element, and nothing is rounded during the
//    accumulation: against 80-bit sums of Gaussian rows the relative error is
//    9e-17 at K = 60 and 1.3e-16 at K = 6000, where a chain of FP64 FMAs has
//    2.5e-16 and 2.4e-15.  For the FP64 path, where both rows of a product are
//    large in the same places: the errors are relative to the row maxima, not
//    to the terms, and slice_guard.cuh leaves the other tiles to the FP64
//    product.  K <= 21760 per accumulation; longer K runs in segments that are
//    added in FP64.
//
// Operand storage: blocks of BR rows (128 for A, the tile's column count for
// B), each holding its 32-wide K chunks one after the other, each chunk the S
// digit slabs one after the other, each slab in the UMMA core-matrix K-major
// layout:
//   (rb * nkc + k / 32) * S * BR * 32 + s * BR * 32
//     + ((r % BR / 8) * 2 + (k % 32) / 16) * 128 + (r % 8) * 16 + k % 16
// so a K chunk of a tile is one bulk copy per operand (a bulk copy costs its
// issuing thread about 70 cycles whatever its size).
#pragma once

#include <cuda_bf16.h>

#include <algorithm>

#include "cd_common.cuh"
#include "pair_energy_tc.cuh"
#include "sm100_ptx.cuh"

namespace mshqc_cd {

namespace ozaki {
constexpr int BM = 128, KB = 32;           // tile rows (A), K bytes per chunk
constexpr uint32_t TMEM_COLS = 512;        // W accumulators of BN columns
constexpr uint64_t kWaitLimitNs = 2000000000ull;
constexpr uint64_t kPaceLimitNs = 200000ull;
constexpr int kBadExponent = 1 << 14;      // row with an infinity or NaN: its products are NaN
constexpr int kNoExponent = (int)0x80808080;   // row of zeros (byte pattern 0x80: memset)
constexpr int kTinyExponent = -890;        // rows below 2^-890 are sliced as zero
constexpr int GROUP = 16;                  // row blocks per tile group (tile_of_unit)
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 64 + 32 * EPI_WARPS;

struct Mixed {
    static constexpr int S = 5, W = 5, BN = 96, STAGES = 6;
    static constexpr int FIXED = 35;       // integer = x 2^{FIXED - e}
    static constexpr int SHIFT = 42;       // product = T 2^{e_x + e_y - SHIFT}
    static constexpr long long MAXK = 26624;
    static constexpr bool GUARD = false;   // (the caller chose this accuracy)
};
struct Full {
    static constexpr int S = 7, W = 8, BN = 64, STAGES = 5;
    static constexpr int FIXED = 54;
    static constexpr int SHIFT = 68;
    static constexpr long long MAXK = 21760;
    static constexpr bool GUARD = true;    // tiles below FP64 accuracy go to the FP64 product
};
static_assert(5LL * 127 * 127 * Mixed::MAXK < 2147483648LL, "int32 accumulation not exact");
// Full: the leading digit is at most 65, so the largest accumulators are the
// 7 pairs with two leading digits and the 6 pairs without
static_assert((2LL * 65 * 128 + 5LL * 128 * 128) * Full::MAXK < 2147483648LL, "int32 accumulation not exact");
static_assert(6LL * 128 * 128 * Full::MAXK < 2147483648LL, "int32 accumulation not exact");

template <class C>
struct Dims {
    static constexpr uint32_t SLAB_A = BM * KB, SLAB_B = C::BN * KB;
    static constexpr uint32_t OFF_B = C::S * SLAB_A;
    static constexpr uint32_t STAGE_BYTES = C::S * (SLAB_A + SLAB_B);
    static constexpr uint32_t SMEM_DATA = C::STAGES * STAGE_BYTES;
    static constexpr size_t SMEM_BYTES = SMEM_DATA + 1024 + 256;
    static_assert(C::W * C::BN <= (int)TMEM_COLS, "accumulators exceed TMEM");
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");
};

inline long long padded_rows(long long rows, int tile) { return (rows + tile - 1) / tile * tile; }
inline long long padded_k(long long k) { return (k + KB - 1) / KB * KB; }
// bytes of one sliced operand (all slices, one batch)
template <class C>
inline size_t operand_bytes(long long Rp, long long Kp) { return (size_t)C::S * (size_t)Rp * (size_t)Kp; }

// The S digits of x 2^{FIXED - e} as bytes: byte j of (lo, hi) is digit S - 1 - j.
template <class C>
__device__ __forceinline__ void digits(double xs, uint32_t& lo, uint32_t& hi) {
    const long long m = __double2ll_rn(xs);
    if constexpr (C::S == 7) {
        constexpr long long c = 0x0080808080808080LL;
        const unsigned long long u = (unsigned long long)((m + c) ^ c);
        lo = (uint32_t)u;
        hi = (uint32_t)(u >> 32);
    } else {
        const bool neg = m < 0;
        const unsigned long long am = (unsigned long long)min(neg ? -m : m, (1LL << C::FIXED) - 1);
        const uint32_t a = (uint32_t)am;
        // 7-bit fields to bytes, then all bytes negated (each is at most 127)
        uint32_t w = (a & 0x7Fu) | ((a & 0x3F80u) << 1) | ((a & 0x1FC000u) << 2) | ((a & 0xFE00000u) << 3);
        uint32_t h = (uint32_t)(am >> 28);
        if (neg) {
            w = (0x80808080u - w) ^ 0x80808080u;
            h = 0u - h;
        }
        lo = w;
        hi = h & 0xFFu;
    }
}

// bytes of four words gathered per byte position: out[j] = byte j of w0..w3
__device__ __forceinline__ void transpose_bytes(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3,
                                                uint32_t (&out)[4]) {
    const uint32_t t0 = __byte_perm(w0, w1, 0x5140), t1 = __byte_perm(w2, w3, 0x5140);
    const uint32_t t2 = __byte_perm(w0, w1, 0x7362), t3 = __byte_perm(w2, w3, 0x7362);
    out[0] = __byte_perm(t0, t1, 0x5410);
    out[1] = __byte_perm(t0, t1, 0x7632);
    out[2] = __byte_perm(t2, t3, 0x5410);
    out[3] = __byte_perm(t2, t3, 0x7632);
}

// four consecutive elements -> word[s] = their digits s
template <class C>
__device__ __forceinline__ void digit_words(const double (&xs)[4], uint32_t (&word)[C::S]) {
    uint32_t lo[4], hi[4], t[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) digits<C>(xs[c], lo[c], hi[c]);
    transpose_bytes(lo[0], lo[1], lo[2], lo[3], t);
#pragma unroll
    for (int j = 0; j < 4; ++j) word[C::S - 1 - j] = t[j];
    transpose_bytes(hi[0], hi[1], hi[2], hi[3], t);
#pragma unroll
    for (int j = 4; j < C::S; ++j) word[C::S - 1 - j] = t[j - 4];
}

// |x| as an ordered integer: infinities and NaN come out largest
__device__ __forceinline__ unsigned long long abs_bits(double x) {
    return (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
}
// exponent e with |x| < 2^e of the largest |x| of a row
__device__ __forceinline__ int row_exponent(unsigned long long mx) {
    const int ef = (int)(mx >> 52);
    return ef == 2047 ? kBadExponent : ef - 1022;
}
// the exponent used: 0 for zero or tiny rows
__host__ __device__ inline int fixed_exponent(int e) { return e < kTinyExponent ? 0 : e; }
// Squares of x / 2^e for the guard (slice_guard.cuh), from the high word of x;
// square_base is what brings the row's exponents to FP32 (rows of zeros, NaN or
// infinity: all squares 0).
__device__ __forceinline__ int square_base(int e) {
    return e == kNoExponent || e == kBadExponent ? 0x7fffffff : (e + 896) << 20;
}
__device__ __forceinline__ float square(int xhi, int base) {
    const float f = __int_as_float(max((xhi & 0x7fffffff) - base, 0) << 3);
    return f * f;
}
__device__ __forceinline__ uint32_t square_pair(int x0hi, int x1hi, int base) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(square(x0hi, base), square(x1hi, base));
    return *reinterpret_cast<const uint32_t*>(&v);
}
// The two 32-wide K chunks whose squares are kept with the slices: the first one
// (graded rows are largest there) and the middle one.  Words per row.
constexpr int SAMPLE_WORDS = 32;
__host__ __device__ inline int sample_chunk(int nkc) { return nkc / 2; }
// 2^{FIXED - e}, or 0 for rows whose digits are all zero
template <class C>
__device__ __forceinline__ double to_fixed(int e) {
    return e == kBadExponent ? 0.0 : pow2d(C::FIXED - e);   // e >= kTinyExponent: in range
}
}  // namespace ozaki

// Slices of the rows of row-major FP64 matrices (batch b: rows r < R at
// src + b * src_batch + r * ld, K elements each).  One CTA per group of 8
// padded rows, a warp per 32-wide K chunk: lane = (row, 8 consecutive K), so
// that the loads are 256 contiguous bytes per row and every store of a slice
// is 256 contiguous bytes.  HELD: chunks a warp keeps in registers between
// the row-maximum pass and the slicing pass (K <= 256 HELD); 0: the rows are
// read twice.  HBM bound: 8 bytes read (16 for HELD = 0) and S written per
// element.  N = 600 vectors (6.9 GB): 1 warp per 8 rows with 16-element lanes
// took 18.4 ms per 30 calls, this form 5.5.
// dst as in the header comment (blocks of BR rows); [batch][Rp] each: e the raw
// exponents (kNoExponent: a row of zeros) and, with C::GUARD, sq the sums of the
// leading digits' squares, sample the squares of two K chunks.
template <class C, int BR, int HELD, bool V2>
static __global__ void __launch_bounds__(256) ozaki_slice_kernel(const double* __restrict__ src, long long ld,
                                                                 long long src_batch, int R, int K, int Rp, int Kp,
                                                                 int8_t* __restrict__ dst, int* __restrict__ e,
                                                                 unsigned* __restrict__ sq,
                                                                 uint32_t* __restrict__ sample) {
    using namespace ozaki;
    __shared__ unsigned long long smx[8][8];
    __shared__ int ssq[8][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rr = lane & 7, qd = lane >> 3;
    const int nkc = Kp / KB;
    const long long b = blockIdx.y;
    auto load8 = [&](const double* row, bool live, int kc, double (&x)[8]) {
        const int k = kc * KB + qd * 8;
        if (V2 && live && k + 8 <= K) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const double2 v = *reinterpret_cast<const double2*>(row + k + 2 * j);
                x[2 * j] = v.x;
                x[2 * j + 1] = v.y;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = (live && k + j < K) ? row[k + j] : 0.0;
        }
    };
    for (int g = blockIdx.x; g < Rp / 8; g += gridDim.x) {
        const int r0 = g * 8, r = r0 + rr;
        const bool live = r < R;
        const double* row = src + b * src_batch + (live ? r : 0) * ld;
        unsigned long long mx = 0;
        double held[HELD > 0 ? HELD : 1][8];
        if (HELD > 0) {
#pragma unroll
            for (int h = 0; h < HELD; ++h) {
                if (warp + 8 * h < nkc) load8(row, live, warp + 8 * h, held[h]);
            }
#pragma unroll
            for (int h = 0; h < HELD; ++h)
                if (warp + 8 * h < nkc)
#pragma unroll
                    for (int j = 0; j < 8; ++j) mx = max(mx, abs_bits(held[h][j]));
        } else {
            for (int kc = warp; kc < nkc; kc += 8) {
                double x[8];
                load8(row, live, kc, x);
#pragma unroll
                for (int j = 0; j < 8; ++j) mx = max(mx, abs_bits(x[j]));
            }
        }
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        if (lane < 8) smx[warp][lane] = mx;
        __syncthreads();
        mx = smx[0][rr];
#pragma unroll
        for (int w = 1; w < 8; ++w) mx = max(mx, smx[w][rr]);
        __syncthreads();   // smx is rewritten by the next group
        const int er = mx == 0 ? kNoExponent : row_exponent(mx);
        if (threadIdx.x < 8) e[b * Rp + r] = er;
        const double f = to_fixed<C>(fixed_exponent(er));
        int squares = 0;   // of the leading digits
        const bool zero = f == 0.0;   // 0 * infinity would not be 0
        int8_t* out = dst + b * ((long long)C::S * Kp * Rp) + (long long)(r0 / BR) * nkc * (C::S * BR * KB) +
                      (r0 % BR) / 8 * 256 + (qd >> 1) * 128 + rr * 16 + (qd & 1) * 8;
        auto emit = [&](int kc, const double (&x)[8]) {
            uint32_t w0[C::S], w1[C::S];
            const double a[4] = {zero ? 0.0 : x[0] * f, zero ? 0.0 : x[1] * f, zero ? 0.0 : x[2] * f,
                                 zero ? 0.0 : x[3] * f};
            const double c[4] = {zero ? 0.0 : x[4] * f, zero ? 0.0 : x[5] * f, zero ? 0.0 : x[6] * f,
                                 zero ? 0.0 : x[7] * f};
            digit_words<C>(a, w0);
            digit_words<C>(c, w1);
            if (C::GUARD) {
                squares = __dp4a((int)w1[0], (int)w1[0], __dp4a((int)w0[0], (int)w0[0], squares));
                if (kc == 0 || kc == sample_chunk(nkc)) {
                    const int base = square_base(er);
                    uint32_t w[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        w[j] = square_pair(__double2hiint(x[2 * j]), __double2hiint(x[2 * j + 1]), base);
                    *reinterpret_cast<uint4*>(sample + (b * Rp + r) * SAMPLE_WORDS + (kc ? 16 : 0) + qd * 4) =
                        make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
            int8_t* o = out + (long long)kc * (C::S * BR * KB);
#pragma unroll
            for (int s = 0; s < C::S; ++s) *reinterpret_cast<uint2*>(o + s * BR * KB) = make_uint2(w0[s], w1[s]);
        };
        if (HELD > 0) {
#pragma unroll
            for (int h = 0; h < HELD; ++h)
                if (warp + 8 * h < nkc) emit(warp + 8 * h, held[h]);
        } else {
            for (int kc = warp; kc < nkc; kc += 8) {
                double x[8];
                load8(row, live, kc, x);
                emit(kc, x);
            }
        }
        if (C::GUARD) {
            squares += __shfl_xor_sync(0xffffffffu, squares, 8);
            squares += __shfl_xor_sync(0xffffffffu, squares, 16);
            if (lane < 8) ssq[warp][lane] = squares;
            __syncthreads();
            if (threadIdx.x < 8) {
                unsigned n = 0;
                for (int w = 0; w < 8; ++w) n += (unsigned)ssq[w][lane];
                sq[b * Rp + r] = n;
            }
            // (ssq is written again after the next group's barriers)
        }
    }
}

// Slices of the rows of matrices stored with the rows contiguous and K
// strided (batch b: element (r, k) at src + b * src_batch + k * ld + r), in
// two passes: row maxima over K splits (atomicMax of the exponent into e,
// which starts at kNoExponent), then one thread per (row, 16-wide K group)
// writing the S digits (and, with C::GUARD, the squares as above; sq starts at
// 0).
namespace ozaki {
constexpr int kRowmaxSpan = 512;               // K elements per row-maximum thread
}  // namespace ozaki

static __global__ void __launch_bounds__(256) ozaki_rowmax_t_kernel(const double* __restrict__ src, long long ld,
                                                                    long long src_batch, long long R, long long K,
                                                                    long long Rp, int* __restrict__ e) {
    using namespace ozaki;
    const long long r = blockIdx.x * 256LL + threadIdx.x;
    const long long b = blockIdx.z;
    if (r >= R) return;
    const long long k0 = (long long)blockIdx.y * kRowmaxSpan, k1 = std::min<long long>(K, k0 + kRowmaxSpan);
    const double* col = src + b * src_batch + r;
    unsigned long long mx = 0;
    long long k = k0;
    for (; k + 8 <= k1; k += 8) {
        double x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = col[(k + j) * ld];
#pragma unroll
        for (int j = 0; j < 8; ++j) mx = max(mx, abs_bits(x[j]));
    }
    for (; k < k1; ++k) mx = max(mx, abs_bits(col[k * ld]));
    if (mx > 0) atomicMax(e + b * Rp + r, row_exponent(mx));
}

// grid (Rp / 32, ceil(Kp / 128), batch), 256 threads: lane -> row, warp -> 16-wide K group
template <class C, int BR>
static __global__ void __launch_bounds__(256) ozaki_slice_t_kernel(const double* __restrict__ src, long long ld,
                                                                   long long src_batch, int R, int K, int Rp, int Kp,
                                                                   const int* __restrict__ e,
                                                                   int8_t* __restrict__ dst,
                                                                   unsigned* __restrict__ sq,
                                                                   uint32_t* __restrict__ sample) {
    using namespace ozaki;
    const int lane = threadIdx.x & 31;
    const int r = blockIdx.x * 32 + lane;
    const int k0 = (blockIdx.y * 8 + (threadIdx.x >> 5)) * 16;
    const long long b = blockIdx.z;
    if (k0 >= Kp) return;
    const bool live = r < R;
    const int er = e[b * Rp + r];
    const double f = to_fixed<C>(fixed_exponent(er));
    const double* col = src + b * src_batch + r + k0 * ld;
    const int kv = live && f != 0.0 ? K - k0 : 0;   // valid K of this thread
    double x[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = j < kv ? col[j * ld] : 0.0;
    if (C::GUARD && (k0 < KB || (k0 >> 5) == sample_chunk(Kp / KB))) {
        const int base = square_base(er);
        uint32_t w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            w[j] = square_pair(__double2hiint(x[2 * j]), __double2hiint(x[2 * j + 1]), base);
        uint4* d = reinterpret_cast<uint4*>(sample + (b * Rp + r) * SAMPLE_WORDS + (k0 < KB ? 0 : 16) +
                                            ((k0 & 31) >> 1));
        d[0] = make_uint4(w[0], w[1], w[2], w[3]);
        d[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] *= f;
    uint32_t word[4][C::S];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const double a[4] = {x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]};
        digit_words<C>(a, word[q]);
    }
    if (C::GUARD) {
        int squares = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) squares = __dp4a((int)word[q][0], (int)word[q][0], squares);
        if (squares > 0) atomicAdd(sq + b * Rp + r, (unsigned)squares);
    }
    int8_t* out = dst + b * ((long long)C::S * Kp * Rp) + ((long long)(r / BR) * (Kp / KB) + (k0 >> 5)) * (C::S * BR * KB) +
                  (((r % BR >> 3) * 2 + ((k0 & 31) >> 4)) << 7) + ((r & 7) << 4);
#pragma unroll
    for (int s = 0; s < C::S; ++s)
        *reinterpret_cast<uint4*>(out + s * BR * KB) = make_uint4(word[0][s], word[1][s], word[2][s], word[3][s]);
}

struct OzakiArgs {
    const int8_t* A; long long a_batch; const int* eA; long long ea_batch;
    const int8_t* B; long long b_batch; const int* eB; long long eb_batch;
    int nkc;                   // K chunks of the operands
    int kc0, kc1;              // chunks of this product
    int M, N;                  // valid output rows and columns
    int nmb, nnb, batch;       // row blocks (128), column blocks (BN), batches
    int group;                 // row blocks per tile group (tile_of_unit)
    int tri;                   // > 0: rows and columns in groups of tri; column groups before the row group skipped
    double* C; long long ldc, c_batch;
    int trans;                 // 1: C(m, n) at C + n * ldc + m
    double alpha, beta;
    int vec;                   // rows of C 32-byte aligned: 256-bit accesses
    int* pace; int pace_every, pace_slack;
    const uint8_t* left_out;   // per unit: 1 if the FP64 product computes the tile (C::GUARD)
    int* err;
};

namespace ozaki {
// 256-bit accesses of 4 doubles (32-byte aligned)
__device__ __forceinline__ void st4(double* p, double a, double b, double c, double d) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};\n" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}
__device__ __forceinline__ void ld4(const double* p, double (&x)[4]) {
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];\n"
                 : "=d"(x[0]), "=d"(x[1]), "=d"(x[2]), "=d"(x[3])
                 : "l"(p)
                 : "memory");
}
}  // namespace ozaki

// C = alpha * A B^T + beta * C per batch (A: M x K rows, B: N x K rows, both
// sliced).  Warp 0 producer (one bulk copy per operand and 32-wide K chunk),
// warp 1 MMA issuer and TMEM owner, warps 2..9 epilogue (exact 64-bit
// combination, one or two roundings to FP64, 64 contiguous bytes of C per
// thread or 256 per warp when transposed).
//
// The MMAs of a chunk: A slice s against the stacked B slices 0 .. min(S, W-s)-1,
// in parts of at most 256 columns; B slice t lands in accumulator s + t.  An
// MMA with 128 rows takes N / 2 cycles (at least about 48), so what counts is
// the total of columns: 1440 per chunk of a 128 x 96 tile (Mixed), 2176 of a
// 128 x 64 tile (Full).  Waits are bounded.
template <class C>
static __global__ void __launch_bounds__(ozaki::THREADS, 1) ozaki_gemm_kernel(OzakiArgs p) {
    using namespace ozaki;
    using namespace sm100;
    using D = Dims<C>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + D::SMEM_DATA);
    uint64_t* empty = full + C::STAGES;
    uint64_t* tmem_full = empty + C::STAGES;
    uint64_t* tmem_empty = tmem_full + 1;
    uint64_t* drain = tmem_empty + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(tmem_full, 1);
        mbar_init(tmem_empty, EPI_WARPS);
        mbar_init(drain, 1);
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    const long long units = (long long)p.nmb * p.nnb * p.batch;
    const long long first = blockIdx.x, step = gridDim.x;
    const int nk = p.kc1 - p.kc0;
    auto skipped = [&](long long u, int mb, int nb) {
        return (p.tri > 0 && nb * C::BN / p.tri < mb * BM / p.tri) || (C::GUARD && p.left_out[u]);
    };

    if (warp == 0) {
        // producer: lane 0 issues the copies, the whole warp paces
        WavePacer pacer;
        pacer.init(p.pace, (int)gridDim.x, p.pace_every, p.pace_slack);
        uint32_t stage = 0, phase = 0, fill_phase = 0, filled = 0;
        bool stop = false;
        for (long long u = first; u < units && !stop; u += step) {
            long long b;
            int mb, nb;
            tile_of_unit(u, p.nmb, p.nnb, p.group, b, mb, nb);
            if (skipped(u, mb, nb)) continue;
            const int8_t* a0 = p.A + b * p.a_batch + ((long long)mb * p.nkc + p.kc0) * (C::S * (long long)D::SLAB_A);
            const int8_t* b0 = p.B + b * p.b_batch + ((long long)nb * p.nkc + p.kc0) * (C::S * (long long)D::SLAB_B);
            for (int kc = 0; kc < nk; ++kc) {
                pacer.step(lane, kPaceLimitNs);
                int ok = 1;
                if (lane == 0) {
                    if (*abort_flag) {
                        ok = 0;
                    } else if (!mbar_wait_bounded(&empty[stage], phase ^ 1, kWaitLimitNs)) {
                        atomicExch(p.err, 31);
                        *abort_flag = 1;
                        ok = 0;
                    } else {
                        uint8_t* sb = smem + stage * D::STAGE_BYTES;
                        mbar_arrive_expect_tx(&full[stage], D::STAGE_BYTES);
                        bulk_g2s(sb, a0, C::S * D::SLAB_A, &full[stage]);
                        bulk_g2s(sb + D::OFF_B, b0, C::S * D::SLAB_B, &full[stage]);
                        a0 += C::S * D::SLAB_A;
                        b0 += C::S * D::SLAB_B;
                    }
                }
                if (!__shfl_sync(0xffffffffu, ok, 0)) {
                    stop = true;
                    break;
                }
                fill_phase = (fill_phase & ~(1u << stage)) | (phase << stage);
                filled |= 1u << stage;
                if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
            }
        }
        pacer.finish(lane);
        if (lane == 0) {
            if (!*abort_flag) {
                for (int s = 0; s < C::STAGES; ++s) {
                    if (!mbar_wait_bounded(&empty[stage], phase ^ 1, kWaitLimitNs)) {
                        atomicExch(p.err, 35);
                        break;
                    }
                    if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
                }
            } else {
                for (int s = 0; s < C::STAGES; ++s)
                    if ((filled >> s) & 1u) mbar_wait_bounded(&full[s], (fill_phase >> s) & 1u, kWaitLimitNs);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            uint32_t stage = 0, phase = 0, acc_phase = 0;
            // descriptors of the operands at stage 0; a byte offset adds to the
            // low word in units of 16 bytes
            const uint64_t da0 = smem_desc_kmajor(smem_addr(smem), 128, 256);
            const uint64_t db0 = smem_desc_kmajor(smem_addr(smem) + D::OFF_B, 128, 256);
            for (long long u = first; u < units && !*abort_flag; u += step) {
                long long b;
                int mb, nb;
                tile_of_unit(u, p.nmb, p.nnb, p.group, b, mb, nb);
                if (skipped(u, mb, nb)) continue;
                if (!mbar_wait_bounded(tmem_empty, acc_phase ^ 1, kWaitLimitNs)) {
                    atomicExch(p.err, 32);
                    *abort_flag = 1;
                    break;
                }
                acc_phase ^= 1;
                tc_fence_after();
                for (int kc = 0; kc < nk; ++kc) {
                    if (!mbar_wait_bounded(&full[stage], phase, kWaitLimitNs)) {
                        atomicExch(p.err, 33);
                        *abort_flag = 1;
                        break;
                    }
                    tc_fence_after();
                    const uint64_t so = (uint64_t)(stage * (D::STAGE_BYTES >> 4));
                    const uint32_t more = kc > 0 ? 1u : 0u;
                    // products of A slice s with B slices t0 .. t0 + n - 1 as one MMA
                    auto mma = [&](int s, int t0, int cols, uint32_t acc) {
                        mma_i8(tmem + (uint32_t)((s + t0) * C::BN), da0 + so + (uint64_t)(s * (D::SLAB_A >> 4)),
                               db0 + so + (uint64_t)(t0 * (D::SLAB_B >> 4)), idesc_s8_s32(BM, cols), acc);
                    };
                    auto mma_half = [&](int s, int row0, int cols, uint32_t acc) {   // from stacked B row row0 on
                        mma_i8(tmem + (uint32_t)(s * C::BN + row0), da0 + so + (uint64_t)(s * (D::SLAB_A >> 4)),
                               db0 + so + (uint64_t)(row0 * (KB >> 4)), idesc_s8_s32(BM, cols), acc);
                    };
                    if constexpr (C::S == 5) {
                        // 480, 384, 288, 192, 96 columns; the s = 0 products of the
                        // first chunk start every accumulator
                        mma_half(0, 0, 240, more);
                        mma_half(0, 240, 240, more);
                        mma_half(1, 0, 192, 1u);
                        mma_half(1, 192, 192, 1u);
                        mma_half(2, 0, 144, 1u);
                        mma_half(2, 144, 144, 1u);
                        mma(3, 0, 192, 1u);
                        mma(4, 0, 96, 1u);
                    } else {
                        // 448, 448, 384, 320, 256, 192, 128 columns; accumulator 7 is
                        // started by (s, t) = (1, 6)
                        mma_half(0, 0, 224, more);
                        mma_half(0, 224, 224, more);
                        mma(1, 0, 192, 1u);
                        mma(1, 3, 192, 1u);
                        mma(1, 6, 64, more);
                        mma(2, 0, 192, 1u);
                        mma(2, 3, 192, 1u);
                        mma_half(3, 0, 160, 1u);
                        mma_half(3, 160, 160, 1u);
                        mma(4, 0, 256, 1u);
                        mma(5, 0, 192, 1u);
                        mma(6, 0, 128, 1u);
                    }
                    mma_commit(&empty[stage]);
                    if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
                }
                if (*abort_flag) break;
                mma_commit(tmem_full);
            }
            mma_commit(drain);
            if (!mbar_wait_bounded(drain, 0, kWaitLimitNs)) atomicExch(p.err, 36);
        }
    } else {
        const int q = warp & 3, half = (warp - 2) >> 2;   // TMEM lane quadrant, half of the columns
        constexpr int HC = C::BN / 2;
        const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
        uint32_t acc_phase = 0;
        for (long long u = first; u < units; u += step) {
            if (*abort_flag) break;
            long long b;
            int mb, nb;
            tile_of_unit(u, p.nmb, p.nnb, p.group, b, mb, nb);
            if (skipped(u, mb, nb)) continue;
            const int m = mb * BM + q * 32 + lane;   // this thread's TMEM row
            const bool mrow = m < p.M;
            const int ea = mrow ? fixed_exponent(p.eA[b * p.ea_batch + m]) : 0;
            double* Cb = p.C + b * p.c_batch;
            const int* eb = p.eB + b * p.eb_batch;
            if (!mbar_wait_bounded(tmem_full, acc_phase, kWaitLimitNs)) {
                atomicExch(p.err, 34);
                *abort_flag = 1;
                break;
            }
            acc_phase ^= 1;
            tc_fence_after();
#pragma unroll 1
            for (int c0 = half * HC; c0 < half * HC + HC; c0 += 8) {
                uint32_t acc[C::W][8];
#pragma unroll
                for (int w = 0; w < C::W; ++w) tmem_ld8(lane_base + (uint32_t)(w * C::BN + c0), acc[w]);
                tmem_ld_wait();
                const int n0 = nb * C::BN + c0;
                double v[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    double t;
                    if constexpr (C::S == 5) {
                        // sum_w acc_w 2^(7(4-w)) exactly in 64 bits (|T| < 2^60), one rounding
                        long long T = (long long)(int)acc[0][k];
#pragma unroll
                        for (int w = 1; w < C::W; ++w) T = T * 128 + (long long)(int)acc[w][k];
                        t = (double)T;
                    } else {
                        // sum_w acc_w 2^(8(7-w)) as two exact halves (|.| < 2^56)
                        long long h = (long long)(int)acc[0][k], l = (long long)(int)acc[4][k];
#pragma unroll
                        for (int w = 1; w < 4; ++w) {
                            h = h * 256 + (long long)(int)acc[w][k];
                            l = l * 256 + (long long)(int)acc[w + 4][k];
                        }
                        t = fma((double)h, 0x1p32, (double)l);
                    }
                    const int n = n0 + k;
                    const int en = n < p.N ? fixed_exponent(eb[n]) : 0;
                    // the scale in two powers of two: no overflow or underflow on the way
                    const int es = ea + en - C::SHIFT, e1 = es >> 1;
                    v[k] = ea == kBadExponent || en == kBadExponent
                               ? __longlong_as_double(0x7FF8000000000000LL)
                               : p.alpha * (t * pow2d(e1) * pow2d(es - e1));
                }
                if (mrow) {
                    if (p.trans) {
#pragma unroll
                        for (int k = 0; k < 8; ++k)
                            if (n0 + k < p.N) {
                                double* c = Cb + (long long)(n0 + k) * p.ldc + m;
                                *c = p.beta != 0.0 ? fma(p.beta, *c, v[k]) : v[k];
                            }
                    } else {
                        double* c = Cb + (long long)m * p.ldc + n0;
                        if (p.vec && n0 + 8 <= p.N) {
                            if (p.beta != 0.0) {
                                double x[4], y[4];
                                ld4(c, x);
                                ld4(c + 4, y);
#pragma unroll
                                for (int k = 0; k < 4; ++k) {
                                    v[k] = fma(p.beta, x[k], v[k]);
                                    v[4 + k] = fma(p.beta, y[k], v[4 + k]);
                                }
                            }
                            st4(c, v[0], v[1], v[2], v[3]);
                            st4(c + 4, v[4], v[5], v[6], v[7]);
                        } else {
#pragma unroll
                            for (int k = 0; k < 8; ++k)
                                if (n0 + k < p.N) c[k] = p.beta != 0.0 ? fma(p.beta, c[k], v[k]) : v[k];
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tmem_empty);
        }
    }

    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, TMEM_COLS);
    }
}

// ---- host side ---------------------------------------------------------------

// One sliced operand: rows R (padded to Rp, a multiple of the block BR), K
// (padded to Kp), `batch` copies.
struct OzakiOperand {
    int8_t* q = nullptr;
    int* e = nullptr;           // row exponents and, behind them, the digits' squares (row_bytes)
    uint32_t* smp = nullptr;    // sampled squares, SAMPLE_WORDS a row (C::GUARD)
    long long R = 0, Rp = 0, K = 0, Kp = 0;
    int BR = 0;
    int batch = 1;
    // the matrices it was sliced from: element (r, k) of batch b at
    // src + b * sb + r * ld + k, or (t) src + b * sb + k * ld + r
    const double* src = nullptr;
    long long ld = 0, sb = 0;
    bool t = false;
    unsigned* sq() const { return reinterpret_cast<unsigned*>(e + Rp * batch); }
    size_t row_bytes(bool guard) const { return sizeof(int) * (size_t)(Rp * batch) * (guard ? 2 : 1); }
};

inline OzakiOperand ozaki_operand(long long R, long long K, int tile, int batch) {
    OzakiOperand op;
    op.R = R;
    op.BR = tile;
    op.Rp = ozaki::padded_rows(R, tile);
    op.K = K;
    op.Kp = ozaki::padded_k(K);
    op.batch = batch;
    return op;
}

template <class C, int BR>
inline cudaError_t ozaki_slice_br(const double* src, long long ld, long long src_batch, const OzakiOperand& op,
                                  int num_sms, cudaStream_t st) {
    const bool v2 = reinterpret_cast<uintptr_t>(src) % 16 == 0 && ld % 2 == 0 && src_batch % 2 == 0;
    // enough CTAs for every SM; each walks its row groups
    const long long want = std::max<long long>(1, 16LL * num_sms / op.batch);
    const dim3 grid((unsigned)std::min<long long>(op.Rp / 8, want), (unsigned)op.batch);
    const long long nkc = op.Kp / ozaki::KB;
#define MSHQC_SLICE(H)                                                                                              \
    do {                                                                                                            \
        if (v2)                                                                                                     \
            ozaki_slice_kernel<C, BR, H, true><<<grid, 256, 0, st>>>(src, ld, src_batch, (int)op.R, (int)op.K,      \
                                                                     (int)op.Rp, (int)op.Kp, op.q, op.e, op.sq(),   \
                                                                     op.smp);                                  \
        else                                                                                                        \
            ozaki_slice_kernel<C, BR, H, false><<<grid, 256, 0, st>>>(src, ld, src_batch, (int)op.R, (int)op.K,     \
                                                                      (int)op.Rp, (int)op.Kp, op.q, op.e, op.sq(),  \
                                                                      op.smp);                                 \
    } while (0)
    if (nkc <= 16)
        MSHQC_SLICE(2);
    else if (nkc <= 32)
        MSHQC_SLICE(4);
    else if (nkc <= 64)
        MSHQC_SLICE(8);
    else
        MSHQC_SLICE(0);
#undef MSHQC_SLICE
    return cudaGetLastError();
}
template <class C>
inline cudaError_t ozaki_slice(const double* src, long long ld, long long src_batch, OzakiOperand& op, int num_sms,
                               cudaStream_t st) {
    op.src = src;  op.ld = ld;  op.sb = src_batch;  op.t = false;
    if (op.Rp <= 0 || op.batch <= 0) return cudaSuccess;
    return op.BR == ozaki::BM ? ozaki_slice_br<C, ozaki::BM>(src, ld, src_batch, op, num_sms, st)
                              : ozaki_slice_br<C, C::BN>(src, ld, src_batch, op, num_sms, st);
}

// Transposed source: element (r, k) of batch b at src + b * src_batch + k * ld + r.
template <class C>
inline cudaError_t ozaki_slice_t(const double* src, long long ld, long long src_batch, OzakiOperand& op,
                                 cudaStream_t st) {
    using namespace ozaki;
    op.src = src;  op.ld = ld;  op.sb = src_batch;  op.t = true;
    cudaError_t err = cudaMemsetAsync(op.e, 0x80, sizeof(int) * (size_t)(op.Rp * op.batch), st);
    if (err != cudaSuccess) return err;
    if (C::GUARD) {
        err = cudaMemsetAsync(op.sq(), 0, sizeof(unsigned) * (size_t)(op.Rp * op.batch), st);
        if (err != cudaSuccess) return err;
    }
    if (op.R > 0 && op.K > 0) {
        dim3 g1((unsigned)((op.R + 255) / 256), (unsigned)((op.K + kRowmaxSpan - 1) / kRowmaxSpan),
                (unsigned)op.batch);
        ozaki_rowmax_t_kernel<<<g1, 256, 0, st>>>(src, ld, src_batch, op.R, op.K, op.Rp, op.e);
        err = cudaGetLastError();
        if (err != cudaSuccess) return err;
    }
    dim3 g2((unsigned)(op.Rp / 32), (unsigned)((op.Kp + 127) / 128), (unsigned)op.batch);
    if (op.BR == BM)
        ozaki_slice_t_kernel<C, BM><<<g2, 256, 0, st>>>(src, ld, src_batch, (int)op.R, (int)op.K, (int)op.Rp,
                                                        (int)op.Kp, op.e, op.q, op.sq(), op.smp);
    else
        ozaki_slice_t_kernel<C, C::BN><<<g2, 256, 0, st>>>(src, ld, src_batch, (int)op.R, (int)op.K, (int)op.Rp,
                                                           (int)op.Kp, op.e, op.q, op.sq(), op.smp);
    return cudaGetLastError();
}

// Options of a sliced product: a shared operand (a_shared / b_shared) is one
// matrix used by every batch; trans and tri as in OzakiArgs; pace: progress
// counters for CTAs with a long K (num_sms ints, zeroed here), or null.
struct OzakiOpts {
    bool a_shared = false, b_shared = false;
    bool trans = false;
    int tri = 0;
    int* pace = nullptr;
    const uint8_t* left_out = nullptr;
};

// C[b] = alpha * A[b] B[b]^T + beta * C[b] over the batches.  K beyond what one
// exact accumulation holds runs in segments that add up in C.
template <class C>
inline cudaError_t ozaki_gemm(const OzakiOperand& A, const OzakiOperand& B, double* Cp, long long ldc,
                              long long c_batch, double alpha, double beta, const OzakiOpts& o, int* err,
                              int num_sms, cudaStream_t st) {
    using namespace ozaki;
    cudaError_t e = cudaFuncSetAttribute(ozaki_gemm_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)Dims<C>::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    const int batch = o.a_shared ? B.batch : A.batch;
    if (A.Kp != B.Kp || A.Kp <= 0 || A.BR != BM || B.BR != C::BN || A.Rp % BM != 0 || B.Rp % C::BN != 0 ||
        (C::GUARD && !o.left_out) || (!o.a_shared && !o.b_shared && A.batch != B.batch) || (o.a_shared && o.b_shared && batch != 1))
        return cudaErrorInvalidValue;
    OzakiArgs p{};
    p.A = A.q;  p.a_batch = o.a_shared ? 0 : (long long)operand_bytes<C>(A.Rp, A.Kp);
    p.eA = A.e;  p.ea_batch = o.a_shared ? 0 : A.Rp;
    p.B = B.q;  p.b_batch = o.b_shared ? 0 : (long long)operand_bytes<C>(B.Rp, B.Kp);
    p.eB = B.e;  p.eb_batch = o.b_shared ? 0 : B.Rp;
    p.nkc = (int)(A.Kp / KB);
    p.M = (int)A.R;  p.N = (int)B.R;
    p.nmb = (int)(A.Rp / BM);  p.nnb = (int)(B.Rp / C::BN);  p.batch = batch;
    p.group = GROUP;
    p.left_out = o.left_out;
    p.tri = o.tri;
    p.C = Cp;  p.ldc = ldc;  p.c_batch = c_batch;
    p.trans = o.trans ? 1 : 0;
    p.alpha = alpha;
    p.vec = reinterpret_cast<uintptr_t>(Cp) % 32 == 0 && ldc % 4 == 0 && c_batch % 4 == 0 ? 1 : 0;
    p.err = err;
    const long long units = (long long)p.nmb * p.nnb * p.batch;
    const unsigned grid = (unsigned)std::max<long long>(1, std::min<long long>(units, num_sms));
    const int max_chunks = (int)(C::MAXK / KB), segs = (p.nkc + max_chunks - 1) / max_chunks;
    for (int s = 0; s < segs; ++s) {
        p.kc0 = (int)((long long)p.nkc * s / segs);
        p.kc1 = (int)((long long)p.nkc * (s + 1) / segs);
        p.beta = s == 0 ? beta : 1.0;
        if (o.pace) {
            e = cudaMemsetAsync(o.pace, 0, sizeof(int) * (size_t)num_sms, st);
            if (e != cudaSuccess) return e;
            p.pace = o.pace;
            p.pace_every = 16;
            p.pace_slack = 2;
        }
        ozaki_gemm_kernel<C><<<grid, THREADS, Dims<C>::SMEM_BYTES, st>>>(p);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace mshqc_cd

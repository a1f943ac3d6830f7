// Integral tiles of the MP2 backward on the tensor cores (tcgen05):
//
//   S[(i - i0, a)][(j, b)] = (ia|jb) = sum_Q X^Q_ia Y^Q_jb     (FP32)
//
// for the occupied rows i of one block and the columns j of another (or all
// j), every tile computed once;
// X and Y are the MO vectors of one spin (restricted, same spin) or of the
// two spins (opposite spin: X alpha, Y beta).
// Operands are the exact fixed-point hi/lo of split_bf16.cuh in its blocked
// layout (128-row blocks) over the composite rows (i, a) and (j, b), packed at v rounded
// to 32 per orbital, so a tile runs across orbitals (padding every orbital's
// rows to 128 and columns to 256 took 1.66 times the tiles at v = 540).  Tiles
// lie on the grid of the composite rows; the edge tiles of a block store only
// the block's rows and columns.  A stage holds KS = 2 Q steps of three 128-row
// blocks with both halves, one 16 KB copy each: the tile's rows (A) and its two
// column blocks (B0, B1); each step's [hi; lo] of a column block is one 256-row
// operand.  Per 16-wide Q step
//   A hi . [B0 hi; B0 lo] -> hh in columns [0,128), hi*lo' in [128,256)
//   A lo . B0 hi          -> += [128,256)           and the same for B1 in [256,512)
// (384 cycles as with three 128x256 products, but three copies a stage instead of
// six, which took longer to issue than the MMAs).  The integers accumulate
// exactly, and the epilogue recovers
//   (ia|jb) = u_ia u_jb (hh + x / 256)
// in FP64, substitutes the exact (ia|ia) for i = j, a = b when X = Y, and
// stores it rounded to FP32 into the row-major staging matrix S (row length
// nbj * RSy).  amp_elem.cuh turns S into amplitudes.
//
// Warp roles (576 threads): warp 0 producer, warp 1 MMA issuer and TMEM
// owner, warps 2..17 epilogue (TMEM lane quadrant warp % 4, column quarter
// (warp - 2) / 4): the two accumulators fill TMEM, so a tile's MMAs wait for
// the epilogue of the one before it, and four warps took as long over it as the
// MMAs of 100 Q steps.  Waits are bounded as in pair_energy_tc.cuh.
#pragma once

#include "cd_common.cuh"
#include "pair_energy_tc.cuh"
#include "sm100_ptx.cuh"
#include "split_bf16.cuh"

namespace mshqc_cd {

struct VtileArgs {
    const uint16_t* X; const uint16_t* Y;       // blocked fixed-point operands (rows i, a; columns j, b)
    const int* ex; const int* ey;               // row exponents of the composite rows
    const double* diag;                         // exact (ia|ia) per composite row when X = Y, else null
    int RSx, RSy;           // composite rows per orbital
    int nqc;                // 16-wide Q chunks
    int vx, vy;
    long long r0, r1, c0, c1;   // the block's composite rows and columns
    int rb0, nrb, cb0, ncb;     // its row blocks (128) and column blocks (256)
    int group;              // row blocks per tile group, see vtile_unit
    float* S;               // staging [r1 - r0][ldS]
    long long ldS;
    int* err;
    int tri;                // 1: a diagonal block of X = Y: tiles with a pair i <= j only
    int* pace;              // gridDim.x zeroed progress counters (WavePacer), or null
    int pace_every, pace_slack;
};

// Unit u -> (row block, column block), in groups of `group` row blocks with all
// column blocks, column-block-major inside a group: a wave of 148 tiles then
// reads about 12 row blocks and 12 column blocks.  False: no pair i <= j in the
// tile (tri).
__device__ __forceinline__ bool vtile_unit(const VtileArgs& p, int u, int& rb, int& cb) {
    const int pg = p.group * p.ncb, grp = u / pg, g0 = grp * p.group;
    const int gsz = min(p.nrb - g0, p.group), x = u - grp * pg;
    cb = x / gsz;
    rb = p.rb0 + g0 + x - cb * gsz;
    cb += p.cb0;
    return !p.tri || (cb * 256 + 255) / p.RSy >= rb * 128 / p.RSx;
}

namespace vtile_tc {
constexpr int BM = 128, BN = 256, KC = 16, KS = 2, STAGES = 4, EPI_WARPS = 16, THREADS = 64 + 32 * EPI_WARPS;
constexpr uint32_t SLAB = 128 * KC * 2;      // 4 KB: 128 rows of a Q step, hi or lo
constexpr uint32_t CHUNK = 2 * SLAB;         // hi and lo
constexpr uint32_t PIECE = KS * CHUNK;       // a 128-row block's part of a stage (16 KB)
constexpr uint32_t STAGE_BYTES = 3 * PIECE;  // A, B0, B1: 48 KB
constexpr uint32_t SMEM_DATA = STAGES * STAGE_BYTES;           // 192 KB
constexpr size_t SMEM_BYTES = SMEM_DATA + 1024 + 256 + BN * 8;
constexpr uint64_t kWaitLimitNs = 2000000000ull;
constexpr uint64_t kPaceLimitNs = 200000ull;   // a pacing wait longer than this turns pacing off
constexpr uint32_t TMEM_COLS = 512;
}  // namespace vtile_tc

__global__ void __launch_bounds__(vtile_tc::THREADS, 1) vtile_tc_kernel(VtileArgs p) {
    using namespace vtile_tc;
    using namespace sm100;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + SMEM_DATA);
    uint64_t* empty = full + STAGES;
    uint64_t* tmem_full = empty + STAGES;
    uint64_t* tmem_empty = tmem_full + 1;
    uint64_t* drain = tmem_empty + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    double* cs_s = reinterpret_cast<double*>(smem + SMEM_DATA + 256);   // BN column scales

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
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

    const int units = p.nrb * p.ncb;
    const int first = blockIdx.x, step = gridDim.x;
    const int nk = p.nqc;

    if (warp == 0) {
        // producer: lane 0 issues the copies, the whole warp paces
        WavePacer pacer;
        pacer.init(p.pace, (int)gridDim.x, p.pace_every, p.pace_slack);
        uint32_t stage = 0, phase = 0, fill_phase = 0, filled = 0;
        bool stop = false;
        for (int u = first; u < units && !stop; u += step) {
            int rb, cb;
            if (!vtile_unit(p, u, rb, cb)) continue;
            // 128-row blocks at Q step 0 (nqc steps of 4096 elements each)
            const size_t nq = (size_t)p.nqc * 4096;
            const uint16_t* a0 = p.X + (size_t)rb * nq;
            const uint16_t* b0 = p.Y + (size_t)(2 * cb) * nq;
            for (int kq = 0; kq < nk; kq += KS) {
                pacer.step(lane, kPaceLimitNs);
                int ok = 1;
                if (lane == 0) {
                    if (*abort_flag) {
                        ok = 0;
                    } else if (!mbar_wait_bounded(&empty[stage], phase ^ 1, kWaitLimitNs)) {
                        atomicExch(p.err, 21);
                        *abort_flag = 1;
                        ok = 0;
                    } else {
                        const uint32_t bytes = (uint32_t)min(KS, nk - kq) * CHUNK;
                        uint8_t* sb = smem + stage * STAGE_BYTES;
                        mbar_arrive_expect_tx(&full[stage], 3 * bytes);
                        const size_t kk = (size_t)kq * 4096;
                        bulk_g2s(sb, a0 + kk, bytes, &full[stage]);
                        bulk_g2s(sb + PIECE, b0 + kk, bytes, &full[stage]);
                        bulk_g2s(sb + 2 * PIECE, b0 + nq + kk, bytes, &full[stage]);
                    }
                }
                if (!__shfl_sync(0xffffffffu, ok, 0)) {
                    stop = true;
                    break;
                }
                fill_phase = (fill_phase & ~(1u << stage)) | (phase << stage);
                filled |= 1u << stage;
                if (++stage == STAGES) { stage = 0; phase ^= 1; }
            }
        }
        pacer.finish(lane);
        if (lane == 0) {
            if (!*abort_flag) {
                for (int s = 0; s < STAGES; ++s) {
                    if (!mbar_wait_bounded(&empty[stage], phase ^ 1, kWaitLimitNs)) {
                        atomicExch(p.err, 25);
                        break;
                    }
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
            } else {
                for (int s = 0; s < STAGES; ++s)
                    if ((filled >> s) & 1u) mbar_wait_bounded(&full[s], (fill_phase >> s) & 1u, kWaitLimitNs);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t IDESC = idesc_f16_f32(BM, 128), IDESC2 = idesc_f16_f32(BM, 256);
            uint32_t stage = 0, phase = 0, acc_phase = 0;
            // descriptors at stage 0; a byte offset adds to the low word in units of 16
            const uint32_t sbase = smem_addr(smem);
            const uint64_t da = smem_desc_kmajor(sbase, 128, 256);
            const uint64_t d0 = smem_desc_kmajor(sbase + PIECE, 128, 256);
            const uint64_t d1 = smem_desc_kmajor(sbase + 2 * PIECE, 128, 256);
            constexpr uint64_t LO = SLAB >> 4;   // the lo slab after the hi slab
            for (int u = first; u < units && !*abort_flag; u += step) {
                int rb, cb;
                if (!vtile_unit(p, u, rb, cb)) continue;
                if (!mbar_wait_bounded(tmem_empty, acc_phase ^ 1, kWaitLimitNs)) {
                    atomicExch(p.err, 22);
                    *abort_flag = 1;
                    break;
                }
                acc_phase ^= 1;
                tc_fence_after();
                for (int kq = 0; kq < nk; kq += KS) {
                    if (!mbar_wait_bounded(&full[stage], phase, kWaitLimitNs)) {
                        atomicExch(p.err, 23);
                        *abort_flag = 1;
                        break;
                    }
                    tc_fence_after();
#pragma unroll
                    for (int c = 0; c < KS; ++c) {
                        if (kq + c < nk) {
                            const uint64_t so = (uint64_t)(stage * (STAGE_BYTES >> 4)) + c * (CHUNK >> 4);
                            const uint32_t more = c > 0 || kq > 0 ? 1u : 0u;
                            mma_f16(tmem, da + so, d0 + so, IDESC2, more);
                            mma_f16(tmem + 128, da + so + LO, d0 + so, IDESC, 1u);
                            mma_f16(tmem + 256, da + so, d1 + so, IDESC2, more);
                            mma_f16(tmem + 384, da + so + LO, d1 + so, IDESC, 1u);
                        }
                    }
                    mma_commit(&empty[stage]);
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
                if (*abort_flag) break;
                mma_commit(tmem_full);
            }
            mma_commit(drain);
            if (!mbar_wait_bounded(drain, 0, kWaitLimitNs)) atomicExch(p.err, 26);
        }
    } else {
        const int q = warp & 3, part = (warp - 2) >> 2;
        const int row = q * 32 + lane;
        const int etid = threadIdx.x - 64;
        uint32_t acc_phase = 0;
        for (int u = first; u < units; u += step) {
            int rb, cb;
            if (!vtile_unit(p, u, rb, cb)) continue;
            const long long r = (long long)rb * BM + row, h0 = (long long)cb * BN;   // composite row, first column
            for (int c = etid; c < BN; c += 32 * EPI_WARPS) {
                const long long h = h0 + c;
                cs_s[c] = h < p.c1 && h % p.RSy < p.vy ? pow2d(p.ey[h] - kFixedHiBits) : 0.0;
            }
            // the epilogue warps leave together (a named barrier must
            // never wait for a warp that already left the loop)
            if (bar_any(1, 32 * EPI_WARPS, *abort_flag != 0)) break;
            const bool got = mbar_wait_bounded(tmem_full, acc_phase, kWaitLimitNs);
            if (bar_any(1, 32 * EPI_WARPS, !got)) {
                if (!got) atomicExch(p.err, 24);
                *abort_flag = 1;
                break;
            }
            acc_phase ^= 1;
            tc_fence_after();
            const bool rin = r >= p.r0 && r < p.r1;   // a row of the block
            const bool arow = rin && r % p.RSx < p.vx;
            const double rs = arow ? pow2d(p.ex[r] - kFixedHiBits) : 0.0;
            const int dcol = p.diag && arow && r >= h0 && r < h0 + BN ? (int)(r - h0) : -1;
            const double dg = dcol >= 0 ? p.diag[r] : 0.0;
            float* dst = p.S + (r - p.r0) * p.ldS + (h0 - p.c0);
            const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
            float amax = 0.0f;   // integer accumulators stay exact below 2^24
#pragma unroll 1
            for (int c0 = part * (BN / 4); c0 < (part + 1) * (BN / 4); c0 += 16) {
                uint32_t h[16], xx[16];
                // column c of block c / 128: hh at 256 (c / 128) + c % 128, x 128 further
                const uint32_t col = (uint32_t)((c0 >> 7) * 256 + (c0 & 127));
                tmem_ld16(lane_base + col, h);
                tmem_ld16(lane_base + 128 + col, xx);
                tmem_ld_wait();
                float out[16];
#pragma unroll
                for (int k = 0; k < 16; ++k) {
                    amax = fmaxf(amax, fmaxf(fabsf(__uint_as_float(h[k])), fabsf(__uint_as_float(xx[k]))));
                    double V = fma((double)__uint_as_float(xx[k]), 1.0 / kFixedLoScale,
                                   (double)__uint_as_float(h[k])) * (rs * cs_s[c0 + k]);
                    if (c0 + k == dcol) V = dg;
                    out[k] = arow ? (float)V : 0.0f;
                }
                // (the block's ends are multiples of 32 columns)
                if (rin && h0 + c0 >= p.c0 && h0 + c0 < p.c1) {
                    // streaming stores (evict first): the staging is read once
                    // by the element-wise pass, and must not push the
                    // operands that other CTAs still read out of L2
                    float4* d4 = reinterpret_cast<float4*>(dst + c0);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        __stcs(d4 + k, make_float4(out[4 * k], out[4 * k + 1], out[4 * k + 2], out[4 * k + 3]));
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tmem_empty);
            if (amax >= 16777216.0f) atomicOr(p.err + 1, 1);
            asm volatile("bar.sync 1, %0;\n" ::"n"(32 * EPI_WARPS) : "memory");   // cs_s reused by the next unit
        }
    }

    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, TMEM_COLS);
    }
}

}  // namespace mshqc_cd

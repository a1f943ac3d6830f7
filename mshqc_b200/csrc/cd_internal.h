// Internal state of a libmshqc_cuda context (not part of the C ABI).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "../../include/mshqc_cd.h"

namespace mshqc_cd {

// Grow-only device allocation: a context allocates on the first call at a
// given size and reuses the memory afterwards.
struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
    cudaError_t reserve(size_t nbytes, bool zero, cudaStream_t st);
    void release();
    template <class T>
    T* as() const { return static_cast<T*>(p); }
};

struct DeviceGuard {
    int prev = 0, target = 0;
    explicit DeviceGuard(int dev);
    ~DeviceGuard();
};

struct SpinState {
    DevBuf C, eps;          // N*N column-major, N
    int64_t nocc = 0;
    bool set = false;
    // FP64 MO vectors [i][a][Q] (a padded to vp, Q to Mp)
    DevBuf B64;
    int64_t vp = 0;
    bool B64_valid = false;
    int B64_prec = 0;       // MSHQC_CD_FP64: FP64 products; MSHQC_CD_FP16X3: int8-slice products
    // fixed-point hi/lo (BF16 carriers) of the MO vectors for the tensor-core path
    DevBuf B16;             // hi and lo interleaved (split_bf16.cuh)
    DevBuf expo;            // per-row power-of-two exponents [o][rows]
    DevBuf diag;            // exact (ia|ia) [o][rows]
    int64_t vp16 = 0, Mp16 = 0;
    double max_norm_hi = 0, max_norm_lo = 0;
    bool B16_valid = false;
    bool norms_pending = false;   // max_norm_* of the last split still on the device
    int B16_layout = 0;     // rows per orbital: 0 packed (integral tiles), 1 multiples of 256 (pair energies)
    void invalidate() {
        B64_valid = false;
        B16_valid = false;
    }
};

}  // namespace mshqc_cd

struct mshqc_cd_ctx {
    int device = 0;
    int num_sms = 148;
    cudaStream_t own = nullptr;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev[6] = {};
    void* bounce[2] = {nullptr, nullptr};
    void* hpin = nullptr;           // pinned host memory that small results arrive in
    size_t hpin_bytes = 0;
    cudaEvent_t bounce_ev[2] = {nullptr, nullptr};

    int64_t N = 0, M = 0, Mp = 0;
    bool L_set = false;
    int64_t launches = 0;           // kernels launched by this context
    // per-stage device timing of the last call (see mshqc_cd_stage_times)
    double stage_ms[8] = {};
    int64_t stage_n[8] = {};        // timed intervals per stage of the last call
    std::vector<cudaEvent_t> ev_pool;
    std::vector<std::pair<int, int>> ev_marks;   // (stage, index of the start event)
    size_t ev_used = 0;
    mshqc_cd::DevBuf L;             // [Q][N*N] FP64 (stored vectors)
    bool L_gen = false;             // vectors generated on the device, never stored
    uint64_t gen_seed = 0;
    mshqc_cd::DevBuf gen_scale;     // sigma * 10^(-6 Q / M) per Q (generated vectors)
    mshqc_cd::DevBuf Lchunk;        // one generated chunk of vectors
    mshqc_cd::SpinState spin[2];

    // workspaces
    mshqc_cd::DevBuf Y;             // half-transformed vectors
    // half-transformed vectors held in Y: per spin, the occupied orbitals
    // [lo, hi) from row `row` on (rows of M * N), made by int8 slices or not
    struct YRange {
        bool ok = false, i8 = false;
        int64_t row = 0, lo = 0, hi = 0;
    } Yr[2];
    mshqc_cd::DevBuf cpack;         // occupied orbitals of both spins, one after the other
    mshqc_cd::DevBuf occ_parts;     // dE/dC_occ of both spins in one product
    // Both spins' half-transformed vectors are held at once where they fit
    // (both_spins_fit; both_used: they were); a call that then runs out of memory is
    // done again with one spin's at a time (one_spin_retry, one_spin), and the
    // calls after it ask for twice the free memory (cautious).
    bool both_used = false, one_spin = false, cautious = false;
    bool call_open = false;         // a call that began has not finished (see begin_call)
    int L_sym = -1;                 // stored vectors symmetric to the bit (-1: not looked at yet)
    mshqc_cd::DevBuf scratch;       // uploads / unpacking
    mshqc_cd::DevBuf partial;       // per-unit energies
    mshqc_cd::DevBuf pair_sum;      // per-pair energies
    mshqc_cd::DevBuf status;        // error flags and scalar results of a call, see CallStatus
    mshqc_cd::DevBuf flag;          // error / NaN flags
    mshqc_cd::DevBuf orb_bad;       // NaN flags of set_orbitals, zero between calls
    mshqc_cd::DevBuf gemm_ws;       // split-K partials of the FP64 products
    mshqc_cd::DevBuf pace;          // wave-pacing progress counters of the persistent tile kernels
    mshqc_cd::DevBuf amp;           // backward: staged amplitudes
    mshqc_cd::DevBuf gam[2];        // backward: Gamma per spin
    mshqc_cd::DevBuf BT;            // backward: transposed MO vectors (hi/lo BF16), alpha
    mshqc_cd::DevBuf BT_b;          // backward: the same for beta
    mshqc_cd::DevBuf ampT;          // backward: transposed amplitudes
    mshqc_cd::DevBuf dsum;          // backward: per-pair row / column / total sums for dE/de
    mshqc_cd::DevBuf amp_chunks;    // backward: per-chunk column sums, energies, totals of split pairs
    mshqc_cd::DevBuf W;             // backward: integral staging / C_vir-contracted Gamma
    mshqc_cd::DevBuf grad[4];       // backward: dC / deps per spin
    mshqc_cd::DevBuf diag_os;       // sum_Q B_alpha[i][a] B_beta[i][a] (opposite-spin diagonal)
    mshqc_cd::DevBuf Hcore;         // OMP2: core Hamiltonian N*N
    bool H_set = false;
    mshqc_cd::DevBuf opdm;          // OMP2: OPDM blocks, densities, Fock matrices
    mshqc_cd::DevBuf omp2_ws;       // OMP2: split-K partials, rotation work matrices
    mshqc_cd::DevBuf Zt;            // Fock builds: P L^Q (or the factored density's L^Q X) of a chunk of vectors
    mshqc_cd::DevBuf dens_x;        // Fock builds: Cholesky factors of the densities
    mshqc_cd::DevBuf oz_a, oz_b;    // int8 slices of the transform operands (orbitals, vectors)
    mshqc_cd::DevBuf oz_ea, oz_eb;  // their row exponents and digit squares
    mshqc_cd::DevBuf oz_tiles;      // tiles of a sliced FP64 product that the FP64 product computes
    bool slices_refused = false;    // no room for FP64 slices: not tried again in this call
    mshqc_cd::DevBuf oz_p;          // per-batch FP64 partial products (transposed transforms)
    bool diag_os_valid = false;
    int fixed_point_exact = 1;      // Cauchy-Schwarz bound of the last tensor-core pass held
    // share of the backward computed by this context (mshqc_cd_set_partition):
    // the units (block pairs, or occupied blocks of the FP64 passes) of a
    // gradient call are numbered from 0 in the order the passes visit them;
    // part_owned[k] says whether unit k is this rank's (a cost-balanced plan
    // that every rank computes alike, see plan_partition in cd_mp2.cu)
    int part_rank = 0, part_size = 1;
    bool part_active = false;
    int64_t part_next = 0;
    std::vector<uint8_t> part_owned;
    // host collectives (mshqc_cd_set_collectives): with them the transforms
    // of a partitioned gradient are shared over occupied orbitals too
    mshqc_cd_collectives coll{};
    bool coll_set = false;
    std::vector<double> pair_energy[3];  // host copies, row-major [i][j]

    // what a call that stopped in between may have left half done: all but the MO
    // vectors, which are marked valid when complete (ranks that share a gradient
    // gather them together, so all or none form them again)
    void invalidate_partial() {
        for (auto& s : spin) {
            s.B16_valid = false;
            s.norms_pending = false;
        }
        diag_os_valid = false;
        Yr[0].ok = Yr[1].ok = false;
    }
    // what calls derive from the vectors and orbitals
    void invalidate_derived() {
        invalidate_partial();
        for (auto& s : spin) s.invalidate();
    }
    void invalidate_all() {
        invalidate_derived();
        L_sym = -1;
        both_used = cautious = false;
        for (auto& p : pair_energy) p.clear();
    }
    size_t held_bytes() const {
        size_t b = L.bytes + Y.bytes + scratch.bytes + partial.bytes +
                   pair_sum.bytes + flag.bytes + amp.bytes + ampT.bytes + BT.bytes + W.bytes;
        for (const auto& s : spin)
            b += s.C.bytes + s.eps.bytes + s.B64.bytes + s.B16.bytes + s.expo.bytes +
                 s.diag.bytes;
        b += gemm_ws.bytes + dens_x.bytes + Zt.bytes + diag_os.bytes + oz_a.bytes + oz_b.bytes + oz_ea.bytes + oz_eb.bytes + oz_p.bytes + oz_tiles.bytes;
        for (const auto& g : gam) b += g.bytes;
        for (const auto& g : grad) b += g.bytes;
        return b;
    }
    // what only products use, between them (int8 slices, split-K partials);
    // false: nothing held
    bool release_slices() {
        bool any = false;
        for (mshqc_cd::DevBuf* b : {&oz_a, &oz_b, &oz_p, &oz_ea, &oz_eb, &oz_tiles, &gemm_ws}) {
            any = any || b->p;
            b->release();
        }
        return any;
    }
    // what a call forms again when it needs it (scratch holds OMP2's densities)
    void release_workspaces() {
        for (mshqc_cd::DevBuf* b : {&Y, &cpack, &occ_parts, &partial, &gemm_ws, &amp, &ampT, &BT, &BT_b,
                                    &dsum, &amp_chunks, &W, &diag_os, &Zt, &oz_a, &oz_b, &oz_ea, &oz_eb, &oz_tiles,
                                    &oz_p, &gam[0], &gam[1]})
            b->release();
        for (auto& s : spin)
            for (mshqc_cd::DevBuf* b : {&s.B64, &s.B16, &s.expo, &s.diag}) b->release();
        invalidate_derived();
    }
    void release_all() {
        for (auto& e : ev_pool)
            if (e) cudaEventDestroy(e);
        ev_pool.clear();
        L.release();
        Y.release();
        scratch.release();
        partial.release();
        pair_sum.release();
        status.release();
        flag.release();
        orb_bad.release();
        gemm_ws.release();
        cpack.release();
        occ_parts.release();
        pace.release();
        amp.release();
        BT.release();
        BT_b.release();
        ampT.release();
        dsum.release();
        amp_chunks.release();
        W.release();
        for (auto& s : spin) {
            s.C.release();
            s.eps.release();
            s.B64.release();
            s.B16.release();
            s.expo.release();
            s.diag.release();
        }
        diag_os.release();
        Hcore.release();
        gen_scale.release();
        Lchunk.release();
        opdm.release();
        omp2_ws.release();
        Zt.release();
        dens_x.release();
        oz_a.release();
        oz_b.release();
        oz_ea.release();
        oz_eb.release();
        oz_tiles.release();
        oz_p.release();
        for (auto& g : gam) g.release();
        for (auto& g : grad) g.release();
    }
};

namespace mshqc_cd {
enum Stage { ST_TRANSFORM = 0, ST_SPLIT, ST_PAIR, ST_AMPLITUDE, ST_GAMMA, ST_TRANSPOSED, ST_OTHER, ST_AMP_ELEM };
// stage timing: begin_stage/end_stage record events on the context stream;
// collect_stages (after a synchronize) folds them into ctx->stage_ms
void reset_stages(mshqc_cd_ctx* ctx);
void begin_stage(mshqc_cd_ctx* ctx, int stage);
void end_stage(mshqc_cd_ctx* ctx);
void collect_stages(mshqc_cd_ctx* ctx);
int set_error(int code, const std::string& msg);
int cuda_error(cudaError_t e, const char* what);
int upload(mshqc_cd_ctx* ctx, void* dst, const void* src, size_t nbytes);
int download(mshqc_cd_ctx* ctx, void* dst, const void* src, size_t nbytes, int where);
int check_finite_device(mshqc_cd_ctx* ctx, const double* x, int64_t n, const char* what);

// status helpers for functions returning an MSHQC_CD_* code (CD_ALLOC needs
// a `ctx` in scope)
#define CD_CUDA(call)                                                     \
    do {                                                                  \
        cudaError_t _e = (call);                                          \
        if (_e != cudaSuccess) return cuda_error(_e, #call);              \
    } while (0)
#define CD_ALLOC(buf, nbytes, zero)                                                        \
    do {                                                                                   \
        cudaError_t _e = (buf).reserve((nbytes), (zero), ctx->stream);                     \
        if (_e == cudaErrorMemoryAllocation)                                               \
            return set_error(MSHQC_CD_ERR_ALLOC, "device allocation of " +                 \
                                                     std::to_string((size_t)(nbytes)) +    \
                                                     " bytes failed");                     \
        if (_e != cudaSuccess) return cuda_error(_e, "workspace");                         \
    } while (0)
// the same where no operand is waiting for its product: where the memory is
// short, what earlier products left goes first
#define CD_ALLOC_FIRST(buf, nbytes, zero)                                                     \
    do {                                                                                      \
        const cudaError_t _f = (buf).reserve((nbytes), (zero), ctx->stream);                  \
        if (_f == cudaErrorMemoryAllocation) {                                                \
            ctx->release_slices();                                                            \
            CD_ALLOC(buf, nbytes, zero);                                                      \
        } else if (_f != cudaSuccess) {                                                       \
            return cuda_error(_f, "workspace");                                               \
        }                                                                                     \
    } while (0)
#define CD_RC(x)             \
    do {                     \
        int _rc = (x);       \
        if (_rc) return _rc; \
    } while (0)

// What a call's kernels report, in ctx->status: zeroed by begin_call, copied
// back once by finish_call (one copy, one synchronization).
struct CallStatus {
    int tile_err[2];        // pair-energy / integral-tile kernel: wait given up, accumulator beyond 2^24
    int gamma_err[2];
    int slice_err[2];       // int8-slice products
    int pad[2];
    double totals[4];       // energies
    unsigned long long norms[2][2];   // largest sum hi^2, sum lo^2 of a row per spin (bit patterns)
};
// pinned host memory of at least `bytes` (grow-only; contents not kept)
int pinned(mshqc_cd_ctx* ctx, size_t bytes, void** p);
// Zeroes the status.  A call that stopped in between (an allocation that failed,
// a kernel that gave up) may have left a buffer half written, or W where Y was:
// that is then formed again.
int begin_call(mshqc_cd_ctx* ctx);
// Waits for the call's work, reports kernels that gave up, and copies `extra`
// bytes from dev to the pinned buffer behind the status (*extra_host).
int finish_call(mshqc_cd_ctx* ctx, CallStatus* st = nullptr, const void* dev = nullptr, size_t extra = 0,
                const void** extra_host = nullptr);

// Runs a call (begin_call ... finish_call), and once more with one spin's
// half-transformed vectors at a time if both were held and it ran out of memory.
template <class F>
int one_spin_retry(mshqc_cd_ctx* ctx, F call) {
    const int rc = call();
    // (ranks that share the transforms make the same collective calls: no second run)
    if (rc != MSHQC_CD_ERR_ALLOC || !ctx->both_used || (ctx->coll_set && ctx->part_size > 1)) return rc;
    cudaStreamSynchronize(ctx->stream);
    ctx->release_workspaces();
    ctx->both_used = false;
    ctx->one_spin = ctx->cautious = true;
    const int again = call();
    ctx->one_spin = false;
    return again;
}

// implemented in cd_mp2.cu
// layout: of the fixed-point operands of a mixed-precision request
// (0: integral tiles of the backward, 1: fused pair energies)
int ensure_transform(mshqc_cd_ctx* ctx, int spin, int precision, int layout = 0);
int ensure_transforms(mshqc_cd_ctx* ctx, int precision, int layout = 0);   // alpha and beta
int run_energy(mshqc_cd_ctx* ctx, int kind, int precision, mshqc_cd_energy* out);
int run_gradient(mshqc_cd_ctx* ctx, int kind, int precision, mshqc_cd_energy* e_out,
                 double* dC_a, double* dC_b, double* deps_a, double* deps_b, int where);
int invalidate_spin(mshqc_cd_ctx* ctx, int spin);   // orbitals of `spin` changed on the device

// implemented in cd_vectors.cu: the vectors Q0 .. Q0 + mc - 1 (N*N doubles
// each, contiguous): the stored array, or a chunk generated into ctx->Lchunk
// (valid until the next call); vectors_chunk_size is the chunk to ask for.
int64_t vectors_chunk_size(const mshqc_cd_ctx* ctx);
int vectors_symmetric(mshqc_cd_ctx* ctx, bool* yes);   // L[Q][mu][nu] == L[Q][nu][mu] for all
int vectors_chunk(mshqc_cd_ctx* ctx, int64_t Q0, int64_t mc, const double** out);
}  // namespace mshqc_cd

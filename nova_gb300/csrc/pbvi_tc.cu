// nova-gb300: tensor-core belief scoring for the point-based backup.
//
// The score of alpha j for (belief i, action a, observation o) is
//     score = sum_k B[i,k] * gamma * sum_l O(a,S,o) T(s_k,a,l) Gamma_j(S)
//           = sum_s A_ao[i,s] * Gamma_j[s],
//     A_ao[i,s] = gamma * O(a,s,o) * sum_{k,l : S(s_k,a,l) = s} B[i,k] T(s_k,a,l),
// a dense (r x n) . (n x |Gamma|) product per (a,o) pair. A_ao does not
// depend on Gamma: it is built once in FP16 or BF16 ([m*z][rPad][nPad],
// K-major, each row scaled by a power of two). Each update packs the unique
// alphas, shifted by a per-state midpoint c[s] (which changes every score of
// a row by the same amount), into FP16 -- or, for BF16, into a pair of BF16
// terms hi + lo whose sum carries 16 bits -- and the GEMM scores every row
// against every unique alpha on the tcgen05 tensor cores with FP32
// accumulation in TMEM. The epilogue keeps, per row, the best (score, alpha)
// pairs of each list and the best score it dropped; the scores never reach
// HBM.
//
// Exactness: for every row the kernel's score differs from the reference's
// FP32 score (pomdp_pbvi_cpu.cpp:50-83) by at most
//     E = a1 * (U * gmax + g_N * Gmax) + d1 * gmax
// (a1 = sum_s |A_ao[i,s]|, d1 = sum_s |A_ao[i,s] - half(A_ao[i,s])| the row's
// measured operand rounding, gmax = max |Gamma - c|, Gmax = max |Gamma|; U
// covers the rounding of the alphas, the FP32 build of A and the tensor-core
// accumulation; g_N = (ns + rz + 3) * 2^-24 covers the reference's own
// rounding). Every alpha within 2E of the best is re-scored in the
// reference's exact FP32 order and the argmax taken there; if the
// dropped-score bound says a candidate may be missing, the (belief, action)
// pair is rescanned exactly over all alphas. The chosen alphas are therefore
// exactly the reference's.
//
// GEMM kernel: persistent, one CTA per SM, 10 warps: warp 0 issues TMA loads
// (SWIZZLE_128B tiles 128x64 of A and 256x64 of the alphas into a 4-stage
// ring; with split alphas each A tile is loaded for the hi and then for the
// lo block), warp 1 issues tcgen05.mma (M=128, N=256, K=16, cta_group::1) into
// two 256-column TMEM accumulators, warps 2-9 drain TMEM with tcgen05.ld
// (two warps per lane quarter, alternate 32-column chunks) and list the scores
// within the row's margin of the running best, while the next tile
// accumulates. Work units are
// (a*z+o, 128-row tile, alpha group); units that run concurrently share
// their A tile and stream the same alphas, so both stay in L2. Every
// mbarrier wait is bounded; on timeout the kernel records an error word,
// stops issuing, frees its TMEM and returns.

#include "pbvi.h"

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <mutex>
#include <type_traits>
#include <vector>
#include <cmath>

namespace nova_gb300 {

__device__ unsigned int g_device_error = 0;

unsigned read_and_clear_device_error() {
    unsigned h = 0;
    if (cudaMemcpyFromSymbol(&h, g_device_error, sizeof(unsigned)) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    if (h != 0) {
        const unsigned zero = 0;
        cudaMemcpyToSymbol(g_device_error, &zero, sizeof(unsigned));
    }
    return h;
}

unsigned tc_device_error() { return read_and_clear_device_error(); }

constexpr int BM = 128;            // rows (beliefs) per tile
constexpr int BN = 256;            // alphas per tile
constexpr int BK = 64;             // K (states) per stage: 128 bytes of BF16
constexpr int STAGES = 4;
constexpr unsigned LIST_SLOTS = 32;            // a list's header and entries: 256 bytes
constexpr unsigned LIST_CAP = LIST_SLOTS - 1;  // entries per list
// Models of at most this many (padded) states choose between one and two alpha
// groups, larger ones take four; a group leaves two candidate lists per row.
constexpr size_t kTuneMaxNPad = 2048;
constexpr size_t max_lists(size_t nPad) { return nPad <= kTuneMaxNPad ? 4 : 8; }
constexpr size_t row_list_bytes(size_t nPad) { return max_lists(nPad) * LIST_SLOTS * 8; }
constexpr unsigned kNoneU = 0xffffffffu;
constexpr int A_STAGE_BYTES = BM * BK * 2;   // 16 KB
constexpr int B_STAGE_BYTES = BN * BK * 2;   // 32 KB
constexpr int EPI_WARPS = 8;          // two per TMEM lane quarter
constexpr int GEMM_THREADS = 64 + 32 * EPI_WARPS;
constexpr size_t GEMM_SMEM = (size_t)STAGES * (A_STAGE_BYTES + B_STAGE_BYTES) + 1024 + 256 + 2 * BM * 8;
constexpr long long kWaitCycles = 4000000000ll;  // ~2 s at 2 GHz

struct TcState {
    Arena arena;
    size_t nPad = 0, rPad = 0, capN = 0;
    unsigned MZ = 0, mTiles = 0;
    unsigned mode = 0;              // NOVA_SCORING_BF16 or NOVA_SCORING_FP16: element type of A and Gb
    const float *src = nullptr;     // alpha set of the last prepared launch (rows of n)
    uint16_t *A = nullptr;          // [MZ][rPad][nPad] BF16 or FP16 bits, each row scaled by a power of 2
    float *a1 = nullptr;            // [MZ][rPad] bound of sum_s |A| in the row's scaled units
    float *a1raw = nullptr;         // [MZ][rPad] the same bound unscaled
    float *d1 = nullptr;            // [MZ][rPad] sum_s |A - half(A)| (scaled units): A's actual operand rounding
    uint16_t *Gb = nullptr;         // [capN][nPad] FP16, or [capN][2 nPad] split BF16, bits of (alpha - c) * 2^gexp
    float *shift = nullptr;         // [n]
    // [0] gmax, [1] Gmax, [2] escale, [3..4] counters, [5] max half-range, [7] dscale (float bits), [8] finished
    // packing blocks; what is accumulated is 0 again after an update (scalClean).
    unsigned *scal = nullptr;
    bool scalClean = false;
    // [MZ][r][lists of the launch][LIST_SLOTS]: slot 0 of a list is {best score that found no room, entries}, then
    // {score, unique alpha}.
    uint2 *cand = nullptr;
    unsigned *rowFlag = nullptr;    // [MZ*r] rows needing the exact scan
    unsigned *rowCand = nullptr;    // [MZ*r] alphas each row re-scored exactly in the merge
    unsigned *rowList = nullptr;    // [MZ*r] their indices, compacted
    unsigned *chunkCount = nullptr; // [ceil(MZ*r / 4096)] flagged rows per chunk
    unsigned *badModel = nullptr;   // [1] set when a probability is negative or NaN
    PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    CUtensorMap tmA;
    cudaEvent_t g0 = nullptr, g1 = nullptr;
    int numSMs = 0;
    // Scoring schedule: alpha groups per row tile. Fewer groups restart the
    // running bests less often (fewer scores are listed, fewer lists merged);
    // more split the work more evenly over the SMs. The best choice depends
    // on the shape, so each solver times kSchedules on its first tensor-core
    // updates (scoring plus the exact scan it leaves, per unique alpha) and
    // keeps the fastest. Results are identical for every choice.
    int schedFixed = -1;            // chosen schedule, -1 while tuning
    unsigned tuneNext = 0;          // next trial
    bool tuneWarm = false;          // the first tensor-core update (lazy set-up) is not timed
    unsigned groupsUsed = 0;        // groups of the last launch
    float tuneCost[2] = {0, 0};  // one per tuned schedule
    // The launch prepared by tc_prepare for tc_gemm / tc_finish.
    struct Launch {
        unsigned nU = 0, nTiles = 0, groups = 0, lists = 0, kSplit = 1;
        bool fp16 = true;
        CUtensorMap tmB;
    } last;
};

// Alpha groups per row tile: the first two are timed on small models. Deep
// contractions keep the epilogue hidden behind the MMAs and take the third (the
// evenest split) without tuning. Four groups on small models were never the
// fastest by more than the timing's noise, and their lists would double the
// memory that a solver of many rows allocates.
constexpr unsigned kSchedules[3] = {2u, 1u, 4u};
constexpr int kTunedSchedules = 2, kDeepSchedule = 2;

void tc_release(TcState *tc) {
    if (!tc) return;
    if (tc->g0) cudaEventDestroy(tc->g0);
    if (tc->g1) cudaEventDestroy(tc->g1);
    delete tc;
}

bool tc_supported(const DevModel &md) {
    // While A is built, the dense row of W_a must fit in shared memory and the
    // transposed O where the candidate lists will be; the row index must stay
    // in TMA's 32-bit coordinate range.
    const size_t nPad = round_up(md.n, BK), rPad = round_up(md.r, BM);
    return md.n <= 40000 && nPad * sizeof(float) <= md.r * row_list_bytes(nPad) &&
           (size_t)md.m * md.z * rPad < (1ull << 31) && nPad < (1ull << 31) && md.r >= 1;
}

// ---------------------------------------------------------------------------
// PTX wrappers (tcgen05 / TMA / mbarrier)
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait: returns false (after recording a device error and raising
// the CTA's abort flag) if the phase does not complete in ~2 s, or if
// another role of the CTA already aborted.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abortFlag) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (true) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abortFlag) return false;
        if (clock64() - t0 > kWaitCycles) {
            *abortFlag = 1;
            atomicExch(&g_device_error, 1u);
            return false;
        }
    }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int c0, int c1, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar)
        : "memory");
}

// Shared-memory matrix descriptor for a K-major, 128-byte-swizzled tile
// whose 8-row groups are 1024 bytes apart (the layout TMA writes with
// CU_TENSOR_MAP_SWIZZLE_128B and a 128-byte inner box).
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFFu);
    d |= (uint64_t)1u << 16;              // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024u >> 4) << 32;    // stride byte offset: 8 rows x 128 B
    d |= (uint64_t)1u << 46;              // descriptor version (tcgen05)
    d |= (uint64_t)2u << 61;              // SWIZZLE_128B
    return d;
}

// Instruction descriptor, kind::f16: D FP32; A and B both BF16 (format 1) or
// both FP16 (format 0), K-major; M=128, N=256.
__host__ __device__ constexpr uint32_t make_idesc(uint32_t fmt) {
    return (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

__device__ __forceinline__ void umma_f16(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(dtmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 32; k++) v[k] = __uint_as_float(r[k]);
}

// ---------------------------------------------------------------------------
// The scoring GEMM with the listing epilogue
// ---------------------------------------------------------------------------

struct GemmBarriers {
    uint64_t full[STAGES];
    uint64_t empty[STAGES];
    uint64_t accFull[2];
    uint64_t accEmpty[2];
    uint32_t tmemBase;
    int abortFlag;
    // Running best of each row in each epilogue half, below the unit it
    // belongs to (plus 1), for the other half to read.
    unsigned long long best[2][BM];
};

__device__ __forceinline__ void decode_unit(unsigned unit, unsigned groups, unsigned mTiles, unsigned nTiles,
                                            unsigned &ao, unsigned &mt, unsigned &g, unsigned &nt0, unsigned &nt1) {
    g = unit % groups;
    const unsigned t = unit / groups;
    mt = t % mTiles;
    ao = t / mTiles;
    nt0 = (unsigned)((unsigned long long)g * nTiles / groups);
    nt1 = (unsigned)((unsigned long long)(g + 1) * nTiles / groups);
}

// The larger of three / eight scores, ignoring NaN unless all are.
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float max8(const float *v) {
    return max3(max3(max3(v[0], v[1], v[2]), v[3], v[4]), max3(v[5], v[6], v[7]), v[7]);
}
// Sorted top-K of (score, alpha) in registers; `excl` is the best score
// that fell off (or never entered) the list.
template <int K>
struct TopList {
    float v[K];
    unsigned u[K];
    float excl;
    __device__ __forceinline__ void reset() {
#pragma unroll
        for (int k = 0; k < K; k++) { v[k] = -INFINITY; u[k] = kNoneU; }
        excl = -INFINITY;
    }
    __device__ __forceinline__ void push(float x, unsigned idx) {
        if (!(x > v[K - 1])) {   // also drops NaN
            excl = fmaxf(excl, x);
            return;
        }
        excl = fmaxf(excl, v[K - 1]);
        // insertion from the bottom; equal scores keep the earlier (lower) index first
#pragma unroll
        for (int k = K - 1; k > 0; k--) {
            const bool shift = x > v[k - 1];
            const bool place = !shift && x > v[k];
            if (shift) { v[k] = v[k - 1]; u[k] = u[k - 1]; }
            else if (place) { v[k] = x; u[k] = idx; }
        }
        if (x > v[0]) { v[0] = x; u[0] = idx; }
    }
};

// Branch-free helpers over one 32-column chunk of a row's scores.
__device__ __forceinline__ unsigned chunk_mask(const float (&v)[32], float lim) {
    unsigned t[16];
#pragma unroll
    for (int k = 0; k < 16; k++)
        t[k] = (v[2 * k] >= lim ? 1u << (2 * k) : 0u) | (v[2 * k + 1] >= lim ? 1u << (2 * k + 1) : 0u);
#pragma unroll
    for (int w = 8; w > 0; w >>= 1)
#pragma unroll
        for (int k = 0; k < w; k++) t[k] = t[2 * k] | t[2 * k + 1];
    return t[0];
}
// The smallest float above a finite or -inf f (+0 and -0 step to the
// smallest subnormal): x > f is x >= next_up(f) for every non-NaN x.
__device__ __forceinline__ float next_up(float f) {
    const unsigned b = __float_as_uint(f);
    if ((b & 0x7fffffffu) == 0u) return __uint_as_float(1u);
    return __uint_as_float((b & 0x80000000u) ? b - 1u : b + 1u);
}
// v[c] for a run-time c without indexing the register array.
__device__ __forceinline__ float chunk_select(const float (&v)[32], unsigned c) {
    float t[16];
#pragma unroll
    for (int k = 0; k < 16; k++) t[k] = (c & 1u) ? v[2 * k + 1] : v[2 * k];
    unsigned bit = 2u;
#pragma unroll
    for (int w = 8; w > 0; w >>= 1, bit <<= 1)
#pragma unroll
        for (int k = 0; k < w; k++) t[k] = (c & bit) ? t[2 * k + 1] : t[2 * k];
    return t[0];
}

// Drops a list's entries below the limit; returns how many are left. Eight are
// loaded before any of them is moved (to a place not after its own): one by one,
// lists that fill (many near-tied alphas) doubled the GEMM's time (n = 500, 200
// states a belief, FP16: 118 us, 70 so; 55 with lists kept sorted in registers).
__device__ __forceinline__ unsigned list_trim(uint2 *list, unsigned count, float lim) {
    unsigned kept = 0;
#pragma unroll 1
    for (unsigned k = 1; k <= count; k += 8) {
        uint2 e[8];
#pragma unroll
        for (unsigned q = 0; q < 8; q++) e[q] = list[min(k + q, LIST_CAP)];
#pragma unroll
        for (unsigned q = 0; q < 8; q++)
            if (k + q <= count && __uint_as_float(e[q].x) >= lim) list[++kept] = e[q];
    }
    return kept;
}

// Twice the row's proven error bound (scaled units): the score gap within
// which an alpha may still be the exact argmax. The GEMM's filter and the
// merge's cut use this same expression.
__device__ __forceinline__ float row_margin(const float *__restrict__ a1, const float *__restrict__ d1, size_t idx,
                                            float escale, float dscale) {
    return 2.0f * (a1[idx] * escale + d1[idx] * dscale);
}

// What a work unit needs: its tensor maps, its place (a*z+o pair, 128-row
// tile, alpha group and the group's 256-alpha tiles) and its solver's shapes,
// bounds and candidate lists.
struct UnitParams {
    const CUtensorMap *tmA, *tmB;
    unsigned ao, mt, g, nt0, nt1;
    unsigned rPad, r, nU, kBlocks, kSplit, lists;
    const float *a1, *d1;
    const unsigned *scal;
    uint2 *cand;
};

// One solver's units (the tensor maps are kernel parameters).
struct SingleUnits {
    unsigned MZ, rPad, r, mTiles, nTiles, groups, nU, kBlocks, kSplit;
    const float *a1, *d1;
    const unsigned *scal;
    uint2 *cand;
    __device__ __forceinline__ unsigned total() const { return MZ * mTiles * groups; }
    __device__ __forceinline__ void get(unsigned unit, UnitParams &p) const {
        decode_unit(unit, groups, mTiles, nTiles, p.ao, p.mt, p.g, p.nt0, p.nt1);
        p.rPad = rPad; p.r = r; p.nU = nU; p.kBlocks = kBlocks; p.kSplit = kSplit; p.lists = 2u * groups;
        p.a1 = a1; p.d1 = d1; p.scal = scal; p.cand = cand;
    }
};

// A solver of a batched launch: its tensor maps in global memory (aligned as
// CUtensorMap requires, which the struct inherits) and its first unit in the
// launch's unit sequence.
struct BatchModel {
    CUtensorMap tmA, tmB;
    unsigned unitStart, MZ, rPad, r, mTiles, nTiles, groups, nU, kBlocks, kSplit;
    const float *a1, *d1;
    const unsigned *scal;
    uint2 *cand;
};

// The units of many solvers in one sequence (solver k owns units
// [unitStart_k, unitStart_{k+1})): a device work table the persistent CTAs
// draw from.
struct BatchUnits {
    const BatchModel *models;
    unsigned nModels, totalUnits;
    __device__ __forceinline__ unsigned total() const { return totalUnits; }
    __device__ __forceinline__ void get(unsigned unit, UnitParams &p) const {
        unsigned lo = 0, hi = nModels - 1;
        while (lo < hi) {   // last model whose first unit is <= unit
            const unsigned mid = (lo + hi + 1) >> 1;
            if (models[mid].unitStart <= unit) lo = mid;
            else hi = mid - 1;
        }
        const BatchModel &b = models[lo];
        decode_unit(unit - b.unitStart, b.groups, b.mTiles, b.nTiles, p.ao, p.mt, p.g, p.nt0, p.nt1);
        p.tmA = &b.tmA; p.tmB = &b.tmB;
        p.rPad = b.rPad; p.r = b.r; p.nU = b.nU; p.kBlocks = b.kBlocks; p.kSplit = b.kSplit;
        p.lists = 2u * b.groups;
        p.a1 = b.a1; p.d1 = b.d1; p.scal = b.scal; p.cand = b.cand;
    }
};

template <bool kSorted, class Units>
__global__ void __launch_bounds__(GEMM_THREADS, 1) tc_score_gemm_kernel(
        const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, uint32_t idesc,
        const Units units) {
    extern __shared__ uint8_t smemRaw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~(uintptr_t)1023);
    uint8_t *sA = smem;
    uint8_t *sB = smem + STAGES * A_STAGE_BYTES;
    GemmBarriers *bar = reinterpret_cast<GemmBarriers *>(smem + STAGES * (A_STAGE_BYTES + B_STAGE_BYTES));
    const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) {
            mbar_init(smem_u32(&bar->full[s]), 1);
            mbar_init(smem_u32(&bar->empty[s]), 1);
        }
        for (int k = 0; k < 2 * BM; k++) bar->best[0][k] = 0ull;  // unit 0 - 1: nobody's
        for (int a = 0; a < 2; a++) {
            mbar_init(smem_u32(&bar->accFull[a]), 1);
            mbar_init(smem_u32(&bar->accEmpty[a]), EPI_WARPS);
        }
        bar->abortFlag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;"
                     ::"r"(smem_u32(&bar->tmemBase)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bar->tmemBase;
    volatile int *abortFlag = &bar->abortFlag;
    const unsigned totalUnits = units.total();
    // Units of a single solver take the tensor maps from the kernel
    // parameters; a batch's from its work table.
    auto unit_params = [&](unsigned unit, UnitParams &p) {
        units.get(unit, p);
        if constexpr (std::is_same<Units, SingleUnits>::value) { p.tmA = &tmA; p.tmB = &tmB; }
    };

    if (warp == 0) {
        if (lane == 0) {
            // ---- TMA producer ----
            unsigned stage = 0, phase = 0;
            for (unsigned unit = blockIdx.x; unit < totalUnits && !*abortFlag; unit += gridDim.x) {
                UnitParams p;
                unit_params(unit, p);
                const int rowA = (int)(p.ao * p.rPad + p.mt * BM);
                for (unsigned nt = p.nt0; nt < p.nt1 && !*abortFlag; nt++) {
                    // kSplit B blocks per A block: the split alphas carry a hi
                    // and a lo block for each 64-state block of A.
                    for (unsigned kb = 0; kb < p.kBlocks * p.kSplit; kb++) {
                        if (!mbar_wait(smem_u32(&bar->empty[stage]), phase ^ 1u, abortFlag)) break;
                        const uint32_t fb = smem_u32(&bar->full[stage]);
                        mbar_expect_tx(fb, A_STAGE_BYTES + B_STAGE_BYTES);
                        tma_load_2d(smem_u32(sA + stage * A_STAGE_BYTES), p.tmA, (int)((kb / p.kSplit) * BK), rowA, fb);
                        tma_load_2d(smem_u32(sB + stage * B_STAGE_BYTES), p.tmB, (int)(kb * BK), (int)(nt * BN), fb);
                        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // ---- MMA issuer ----
            unsigned stage = 0, phase = 0, acc = 0, accPhase = 0;
            for (unsigned unit = blockIdx.x; unit < totalUnits && !*abortFlag; unit += gridDim.x) {
                UnitParams p;
                unit_params(unit, p);
                for (unsigned nt = p.nt0; nt < p.nt1 && !*abortFlag; nt++) {
                    if (!mbar_wait(smem_u32(&bar->accEmpty[acc]), accPhase ^ 1u, abortFlag)) break;
                    tc_fence_after();
                    const uint32_t dtmem = tmem + acc * BN;
                    for (unsigned kb = 0; kb < p.kBlocks * p.kSplit; kb++) {
                        if (!mbar_wait(smem_u32(&bar->full[stage]), phase, abortFlag)) break;
                        tc_fence_after();
                        const uint64_t adesc = smem_desc_sw128(smem_u32(sA + stage * A_STAGE_BYTES));
                        const uint64_t bdesc = smem_desc_sw128(smem_u32(sB + stage * B_STAGE_BYTES));
#pragma unroll
                        for (int kk = 0; kk < BK / 16; kk++)
                            umma_f16(dtmem, adesc + 2u * kk, bdesc + 2u * kk, idesc,
                                     (kb | (unsigned)kk) != 0u ? 1u : 0u);
                        umma_commit(smem_u32(&bar->empty[stage]));
                        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
                    }
                    umma_commit(smem_u32(&bar->accFull[acc]));
                    acc ^= 1u;
                    if (acc == 0) accPhase ^= 1u;
                }
            }
        }
    } else {
        // ---- epilogue: TMEM -> registers -> the row's candidate list ----
        // Eight warps: warps w and w+4 read the same TMEM lane quarter
        // (w & 3), one row per thread, and take alternate 32-column chunks
        // of every tile, each keeping its own list for the unit (list
        // 2g + half of the row).
        // A score below (running best - thr), thr being the row's margin as
        // the merge computes it, lies below the merge's cut for every later
        // best (the cut is fl(final best - thr) and rounding is monotonic):
        // it cannot be a candidate, so it is skipped.
        //
        // With few states the MMAs of a tile take less time than reading it,
        // and compares and selects run at half rate: what counts is the
        // instructions per chunk. Some row of the 32 has a new best in most
        // chunks (records of 79 chunks in random order), so the listing path
        // matters as much as the skipping one. Listed scores are therefore
        // appended to the row's list in global memory, unsorted, without
        // selecting them out of the registers: each 8 columns whose maximum
        // passes are compared and stored in turn. n = 150 (2,500 alphas,
        // 400,000 rows): 591 us with a sorted list in registers, 348 so; 200
        // states: 692 to 395; 512: 135 to 101 (its MMAs need 71); 700 with
        // 12 candidates a row: 354 to 225.
        // Behind a deep contraction's MMAs the epilogue costs nothing, and its
        // lists are kept sorted in registers (kSorted), so that a full one
        // loses its least entry: in BF16 at n = 4,096, whose wide margin lists
        // 24 candidates a row, 91 rows are left to the exact scan instead of
        // 17,855 (113 ms of an update of 499).
        const unsigned quarter = warp & 3u;   // TMEM lanes this warp may access
        const unsigned half = (warp - 2u) >> 2;
        const unsigned rowInTile = quarter * 32u + lane;
        const float qnan = __uint_as_float(0x7fc00000u);
        unsigned acc = 0, accPhase = 0;
        TopList<kSorted ? (int)LIST_CAP : 1> top;
        for (unsigned unit = blockIdx.x; unit < totalUnits && !*abortFlag; unit += gridDim.x) {
            UnitParams p;
            unit_params(unit, p);
            const unsigned ao = p.ao, nU = p.nU;
            const float escale = __uint_as_float(p.scal[2]);
            const float dscale = __uint_as_float(p.scal[7]);
            const unsigned iRow = p.mt * BM + rowInTile;
            const bool real = iRow < p.r;
            // Same expression as the merge's margin. An infinite margin skips
            // nothing; a NaN one skips everything, and the merge sends such
            // rows to the exact scan whatever their lists hold. Rows of the
            // tile's padding skip everything.
            const float thr = real ? row_margin(p.a1, p.d1, (size_t)ao * p.rPad + iRow, escale, dscale) : 0.0f;
            float best = real ? -INFINITY : INFINITY, lim = best;
            uint2 *list = p.cand + (((size_t)ao * p.r + (real ? iRow : 0u)) * p.lists + 2u * p.g + half) * LIST_SLOTS;
            unsigned count = 0;
            float excl = -INFINITY, limTrim = -INFINITY;
            if constexpr (kSorted) top.reset();
            volatile unsigned long long *myBest = &bar->best[half][rowInTile];
            volatile unsigned long long *otherBest = &bar->best[half ^ 1u][rowInTile];
            const unsigned long long tag = (unsigned long long)(unit + 1u) << 32;
            bool ok = true;
            for (unsigned nt = p.nt0; nt < p.nt1; nt++) {
                if (!mbar_wait(smem_u32(&bar->accFull[acc]), accPhase, abortFlag)) { ok = false; break; }
                tc_fence_after();
                // The other half's best of this row is a listed score too, so
                // it bounds the final best from below just as well.
                const unsigned long long other = *otherBest;
                if ((other & 0xffffffff00000000ull) == tag) {
                    best = fmaxf(best, __uint_as_float((unsigned)other));
                    lim = fmaxf(lim, best - thr);
                }
                const uint32_t base = tmem + ((quarter * 32u) << 16) + acc * BN;
#pragma unroll 1
                for (unsigned ch = half; ch < BN / 32; ch += 2) {
                    __syncwarp();
                    float v[32];
                    tmem_ld32(base + ch * 32u, v);
                    const unsigned u0 = nt * BN + ch * 32u;
                    if (u0 + 32u > nU) {   // columns past the unique alphas are skipped (NaN)
#pragma unroll
                        for (int c = 0; c < 32; c++)
                            if (u0 + c >= nU) v[c] = qnan;
                    }
                    float m8[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) m8[q] = max8(v + 8 * q);
                    const float mx = max3(max3(m8[0], m8[1], m8[2]), m8[3], m8[3]);
                    if (mx >= lim && real) {
                        // The chunk's maximum raises the running best first,
                        // so only its scores within thr of the new best are
                        // listed.
                        best = fmaxf(best, mx);
                        lim = best - thr;
                        if constexpr (kSorted) {
                            // Scores at or below the list's last entry f would
                            // only raise the dropped maximum (push's first
                            // branch). If any score of the chunk is above f,
                            // its insertion drops f itself, which bounds them
                            // all; otherwise the chunk's maximum is the
                            // largest of them.
                            unsigned mask = chunk_mask(v, fmaxf(lim, next_up(top.v[LIST_CAP - 1])));
                            if (mask == 0u) top.excl = fmaxf(top.excl, mx);
                            while (mask) {
                                const unsigned c = __ffs(mask) - 1;
                                mask &= mask - 1;
                                top.push(chunk_select(v, c), u0 + c);
                            }
                            continue;
                        }
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            if (!(m8[q] >= lim)) continue;
                            if (count + 8u <= LIST_CAP) {
#pragma unroll
                                for (int c = 0; c < 8; c++)
                                    if (v[8 * q + c] >= lim)
                                        list[++count] = make_uint2(__float_as_uint(v[8 * q + c]), u0 + 8 * q + c);
                            } else {
                                // Room may run out: entries that the risen
                                // limit has left behind go first; what then
                                // finds no room only raises the best dropped
                                // score, which the merge compares to its cut.
                                if (lim > limTrim) {
                                    count = list_trim(list, count, lim);
                                    limTrim = lim;
                                }
                                if (count == LIST_CAP) {
                                    excl = fmaxf(excl, m8[q]);
                                    continue;
                                }
#pragma unroll
                                for (int c = 0; c < 8; c++)
                                    if (v[8 * q + c] >= lim) {
                                        if (count < LIST_CAP)
                                            list[++count] = make_uint2(__float_as_uint(v[8 * q + c]), u0 + 8 * q + c);
                                        else
                                            excl = fmaxf(excl, v[8 * q + c]);
                                    }
                            }
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bar->accEmpty[acc]));
                *myBest = tag | __float_as_uint(best);
                acc ^= 1u;
                if (acc == 0) accPhase ^= 1u;
            }
            if (!ok) break;
            if constexpr (kSorted) {
                excl = top.excl;
#pragma unroll
                for (int k = 0; k < (int)LIST_CAP; k++)
                    if (real && top.u[k] != kNoneU) list[++count] = make_uint2(__float_as_uint(top.v[k]), top.u[k]);
            }
            if (real) list[0] = make_uint2(__float_as_uint(excl), count);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
    }
}

// ---------------------------------------------------------------------------
// Step-invariant operand: A_ao[i, s] in BF16/FP16, each row scaled by a power
// of two so its largest entry lies in [2^13, 2^14) (FP16's precision is then
// used fully and nothing overflows); a1 bounds sum_s |A| in the same units.
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint16_t to_half_bits(float v, bool fp16) {
    if (fp16) return __half_as_ushort(__float2half_rn(v));
    return __bfloat16_as_ushort(__float2bfloat16_rn(v));
}
__device__ __forceinline__ float from_half_bits(uint16_t b, bool fp16) {
    if (fp16) return __half2float(__ushort_as_half(b));
    return __bfloat162float(__ushort_as_bfloat16(b));
}

// O with the states innermost, [m][z][nPad] (0 past n): 32 x 32 tiles, the
// actions over the grid's third dimension (which ends at kMaxGridZ).
constexpr unsigned kMaxGridZ = 65535;

__global__ void tc_transpose_o_kernel(DevModel md, size_t nPad, float *__restrict__ Ot,
                                      unsigned *__restrict__ badModel) {
    __shared__ float tile[32][33];
    const unsigned s0 = blockIdx.x * 32u, o0 = blockIdx.y * 32u;
    for (unsigned a = blockIdx.z; a < md.m; a += gridDim.z) {
        for (unsigned k = threadIdx.y; k < 32u; k += 8u) {
            float v = 0.0f;
            if (s0 + k < md.n && o0 + threadIdx.x < md.z) {
                v = md.O[((size_t)a * md.n + s0 + k) * md.z + o0 + threadIdx.x];
                if (!(v >= 0.0f)) atomicOr(badModel, 1u);  // the bound assumes non-negative B, T, O
            }
            tile[k][threadIdx.x] = v;
        }
        __syncthreads();
        for (unsigned k = threadIdx.y; k < 32u; k += 8u)
            if (o0 + k < md.z) Ot[((size_t)a * md.z + o0 + k) * nPad + s0 + threadIdx.x] = tile[threadIdx.x][k];
        __syncthreads();
    }
}

// One block per action and NB beliefs: their successor distributions W in
// shared memory, then one warp per observation reads O's row once for all NB
// beliefs, twice over (the rows' maxima set their scales). Bound by its FP32
// work and by writing A: n = 1,024 (r = 1,024, m z = 128, 268 MB: 40 us at
// memory speed) 105 us; with one belief per block, all its warps on one
// observation and O as the model holds it (64-byte strides) 650 us.
template <int NB>
__global__ void __launch_bounds__(256) tc_build_a_kernel(
                                  DevModel md, const unsigned *__restrict__ succLen,
                                  const unsigned *__restrict__ suppLen, size_t rPad, size_t nPad, int fp16,
                                  const float *__restrict__ Ot, uint16_t *__restrict__ A, float *__restrict__ a1,
                                  float *__restrict__ a1raw, float *__restrict__ d1, float a1Slack, float d1Slack,
                                  unsigned *__restrict__ badModel) {
    extern __shared__ __align__(16) float W[];  // [NB][nPad]
    const unsigned i0 = blockIdx.x / md.m * NB, a = blockIdx.x % md.m;
    for (unsigned s = threadIdx.x; s < NB * nPad; s += blockDim.x) W[s] = 0.0f;
    __syncthreads();
    for (unsigned b = 0; b < NB && i0 + b < md.r; b++) {
        const unsigned i = i0 + b, Li = suppLen[i];
        for (unsigned e = threadIdx.x; e < Li * md.ns; e += blockDim.x) {
            const unsigned k = e / md.ns, l = e % md.ns;
            const int s = md.Z[(size_t)i * md.rz + k];
            if (l < succLen[(size_t)s * md.m + a]) {
                const size_t row = ((size_t)s * md.m + a) * md.ns + l;
                const float w = md.B[(size_t)i * md.rz + k] * md.T[row];
                if (!(w >= 0.0f)) atomicOr(badModel, 1u);
                atomicAdd(&W[b * nPad + md.S[row]], w);
            }
        }
    }
    __syncthreads();
    const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (unsigned o = warp; o < md.z; o += 8u) {
        const size_t ao = (size_t)a * md.z + o;
        const float4 *orow = reinterpret_cast<const float4 *>(Ot + ao * nPad);
        auto values = [&](unsigned b, unsigned s4, const float4 &ob) {
            const float4 w = reinterpret_cast<const float4 *>(W + b * nPad)[s4];
            return make_float4(md.gamma * w.x * ob.x, md.gamma * w.y * ob.y, md.gamma * w.z * ob.z,
                               md.gamma * w.w * ob.w);
        };
        float mx[NB], sum[NB], dsum[NB], scale[NB];
#pragma unroll
        for (int b = 0; b < NB; b++) mx[b] = sum[b] = dsum[b] = 0.0f;
        for (unsigned s4 = lane; s4 < nPad / 4; s4 += 32) {
            const float4 ob = __ldg(orow + s4);
#pragma unroll
            for (int b = 0; b < NB; b++) {
                const float4 v = values(b, s4, ob);
                mx[b] = fmaxf(mx[b], fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
                sum[b] += (v.x + v.y) + (v.z + v.w);
            }
        }
#pragma unroll
        for (int b = 0; b < NB; b++) {
            for (int off = 16; off > 0; off >>= 1) {
                mx[b] = fmaxf(mx[b], __shfl_xor_sync(0xffffffffu, mx[b], off));
                sum[b] += __shfl_xor_sync(0xffffffffu, sum[b], off);
            }
            int e = 0;
            if (mx[b] > 0.0f) frexpf(mx[b], &e);          // mx in [2^(e-1), 2^e)
            scale[b] = mx[b] > 0.0f ? ldexpf(1.0f, 14 - e) : 1.0f;
        }
        // d1 = sum_s |A - half(A)| in the row's scaled units: the actual
        // rounding of this row's operand (each term is exact in FP32).
        for (unsigned s4 = lane; s4 < nPad / 4; s4 += 32) {
            const float4 ob = __ldg(orow + s4);
#pragma unroll
            for (int b = 0; b < NB; b++) {
                const float4 v = values(b, s4, ob);
                const float x[4] = {v.x * scale[b], v.y * scale[b], v.z * scale[b], v.w * scale[b]};
                ushort4 h;
                h.x = to_half_bits(x[0], fp16 != 0);
                h.y = to_half_bits(x[1], fp16 != 0);
                h.z = to_half_bits(x[2], fp16 != 0);
                h.w = to_half_bits(x[3], fp16 != 0);
                dsum[b] += (fabsf(x[0] - from_half_bits(h.x, fp16 != 0)) + fabsf(x[1] - from_half_bits(h.y, fp16 != 0))) +
                           (fabsf(x[2] - from_half_bits(h.z, fp16 != 0)) + fabsf(x[3] - from_half_bits(h.w, fp16 != 0)));
                if (i0 + b < md.r) reinterpret_cast<ushort4 *>(A + (ao * rPad + i0 + b) * nPad)[s4] = h;
            }
        }
#pragma unroll
        for (int b = 0; b < NB; b++) {
            for (int off = 16; off > 0; off >>= 1) dsum[b] += __shfl_xor_sync(0xffffffffu, dsum[b], off);
            if (lane == 0 && i0 + b < md.r) {
                a1[ao * rPad + i0 + b] = sum[b] * scale[b] * a1Slack;
                a1raw[ao * rPad + i0 + b] = sum[b] * a1Slack;
                d1[ao * rPad + i0 + b] = dsum[b] * d1Slack;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Per-update packing of the unique alphas
// ---------------------------------------------------------------------------

__device__ __forceinline__ void atomic_max_nonneg(unsigned *addr, float v) {
    // Non-negative floats order like their bit patterns; NaN (all exponent
    // bits set, nonzero mantissa) compares above every finite value, which
    // disables the margin.
    atomicMax(addr, __float_as_uint(v));
}

// Per-state midpoint shift c[s] over the unique alphas, Gmax = max |alpha|
// (scal[1]) and the largest half-range max (hi - lo) / 2 (scal[5]).
__global__ void tc_shift_kernel(const float *__restrict__ Gt, size_t gtCols, unsigned n, unsigned nU,
                                float *__restrict__ shift, unsigned *__restrict__ scal) {
    const unsigned s = blockIdx.x;
    const float *row = Gt + (size_t)s * gtCols;
    float mn = INFINITY, mx = -INFINITY;
    int nanSeen = 0;
    for (unsigned u = threadIdx.x; u < nU; u += blockDim.x) {
        const float v = row[u];
        mn = fminf(mn, v);
        mx = fmaxf(mx, v);
        nanSeen |= (v != v);
    }
    __shared__ float smn[32], smx[32];
    __shared__ int snan;
    if (threadIdx.x == 0) snan = 0;
    for (int off = 16; off > 0; off >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, off));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    }
    __syncthreads();
    if (nanSeen) snan = 1;
    if ((threadIdx.x & 31) == 0) { smn[threadIdx.x >> 5] = mn; smx[threadIdx.x >> 5] = mx; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (unsigned w = 0; w < blockDim.x / 32; w++) { mn = fminf(mn, smn[w]); mx = fmaxf(mx, smx[w]); }
        shift[s] = 0.5f * mn + 0.5f * mx;
        const float nanf_ = __uint_as_float(0x7fc00000u);
        atomic_max_nonneg(&scal[1], snan ? nanf_ : fmaxf(fabsf(mn), fabsf(mx)));
        atomic_max_nonneg(&scal[5], snan ? nanf_ : 0.5f * (mx - mn));
    }
}

// Power-of-two scale for the packed alphas: the largest |alpha - c| lands
// in [2^13, 2^14) (half-range plus slack for the rounding of c).
__device__ __forceinline__ float pack_scale(const unsigned *scal) {
    const float hr = __uint_as_float(scal[5]) * 1.001f + 1e-30f;
    int e = 0;
    frexpf(hr, &e);
    return hr < 1e30f ? ldexpf(1.0f, 13 - e) : 1.0f;
}

// Gb[u] = half((alpha_u(s) - c[s]) * gscale); rows >= nU, states >= n are 0.
// Single form (FP16): one value per state, row length nPad. Split form
// (BF16): each value v is carried as hi = bf16(v) and lo = bf16(v - hi)
// (v - hi is exact in FP32), so |v - hi - lo| <= 2^-16 |v|; the row holds,
// for every 64-state block kb, the 64 hi values and then the 64 lo values
// (row length 2 nPad), and the GEMM multiplies one A block by both.
// Records gmax = max |(alpha - c) * gscale| over the FP32 values; the block
// that finishes last turns it into the margin's scales, escale = U * gmax +
// gN * Gmax * gscale and dscale = gmax (1 + 2^-22), all in the packed units
// (the per-row bound is a1 * escale + d1 * dscale). Also clears the merge's
// chunk counts.
__global__ void tc_pack_kernel(const float *__restrict__ G, unsigned n, size_t nPad, const unsigned *__restrict__ uniqJ,
                               unsigned nU, const float *__restrict__ shift, int fp16, int split,
                               uint16_t *__restrict__ Gb, unsigned *scal, float U, float gN,
                               unsigned *__restrict__ chunkCount, unsigned nChunks) {
    const unsigned u = blockIdx.x;
    const float gscale = pack_scale(scal);
    for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < nChunks; k += gridDim.x * blockDim.x) chunkCount[k] = 0u;
    const size_t rowLen = split ? 2 * nPad : nPad;
    uint16_t *out = Gb + (size_t)u * rowLen;
    float m = 0.0f;
    int nanSeen = 0;
    if (u < nU) {
        const float *row = G + (size_t)uniqJ[u] * n;
        for (unsigned s = threadIdx.x; s < nPad; s += blockDim.x) {
            float v = 0.0f;
            if (s < n) {
                v = (row[s] - shift[s]) * gscale;
                m = fmaxf(m, fabsf(v));
                nanSeen |= (v != v);
            }
            if (split) {
                const uint16_t hi = to_half_bits(v, false);
                const uint16_t lo = to_half_bits(v - from_half_bits(hi, false), false);
                const size_t at = (size_t)(s / BK) * (2 * BK) + (s % BK);
                out[at] = hi;
                out[at + BK] = lo;
            } else {
                out[s] = to_half_bits(v, fp16 != 0);
            }
        }
    } else {
        for (size_t s = threadIdx.x; s < rowLen; s += blockDim.x) out[s] = 0;
    }
    __shared__ float red[32];
    __shared__ int snan;
    if (threadIdx.x == 0) snan = 0;
    for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
    __syncthreads();
    if (nanSeen) snan = 1;
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (unsigned w = 0; w < blockDim.x / 32; w++) m = fmaxf(m, red[w]);
        atomic_max_nonneg(&scal[0], snan ? __uint_as_float(0x7fc00000u) : m);
        __threadfence();
        if (atomicAdd(&scal[8], 1u) == gridDim.x - 1) {
            __threadfence();
            const float gmax = __uint_as_float(atomicAdd(&scal[0], 0u));
            const float Gmax = __uint_as_float(scal[1]);
            scal[2] = __float_as_uint(U * gmax + gN * Gmax * gscale);
            scal[7] = __float_as_uint(gmax * (1.0f + 2.4e-7f));
        }
    }
}

// ---------------------------------------------------------------------------
// Merge the per-group lists, apply the proven margin, re-score near ties
// exactly from the projection table; rows whose candidate set may be
// incomplete go to the exact row scan.
// ---------------------------------------------------------------------------

// Without the projection table: the same exact scores straight from the
// model and the alpha rows, in the table's order: each support state's
// entry fl(gamma * sum_l C * alpha(S)) (proj_state_lanes_kernel; C3 holds the
// same products as C1, successor-contiguous), times b_k, summed in support
// order.
constexpr unsigned kDirectNs = 32;  // successors per state the direct re-score holds in registers

struct DirectScorer {
    const unsigned *succLen;
    const float *C3, *G;  // G: the update's alpha set, rows of n
    __device__ __forceinline__ float vt(const DevModel &md, unsigned a, unsigned o, unsigned s,
                                        const float *__restrict__ Gj) const {
        const unsigned Ls = __ldg(succLen + (size_t)s * md.m + a);
        const float *c = C3 + (((size_t)a * md.z + o) * md.n + s) * md.ns;
        const int *sp = md.S + ((size_t)s * md.m + a) * md.ns;
        float v = 0.0f;
        for (unsigned l = 0; l < Ls; l++) v = fadd(v, fmul(__ldg(c + l), __ldg(Gj + __ldg(sp + l))));
        return v;
    }
};

// The merge, in two launches. Most rows have one candidate, which a thread
// can see: one thread per row looks through the row's lists (their header and
// first three entries are one sector) and settles it, or queues it. The queued
// rows are re-scored by half a warp each: half warps fit rows of two to four
// candidates and 16 to 32 support states, of which each lane gathers two
// states' entries of up to kMergeBatch candidates before any is used; lane t
// then adds candidate t's products in support order from shared memory. Every
// block draws its rows from the queue, so both kinds spread over the device
// whatever their share.
// Bound by the table's random 32-byte sectors where rows have many candidates
// (n = 700: 12 candidates of 40 states, 1.3 GB of sectors, at 6 TB/s) and by
// latency and instructions elsewhere. With one warp per row from the lists to
// the argmax against this, looking and re-scoring: n = 150 (400,000 rows, 1.4
// candidates re-scored each) 285 and 145 us, n = 200 (512,000) 350 and 167,
// n = 512 (131,072) 103 and 75, n = 700 (84,000, 12 each) 239 and 210.
// The queue is in no order (the looking blocks append to it as they run). Where
// the table's slab of one (action, observation) is a good part of L2, rows are
// instead taken in their own order, a block per 16 rows as the device gets to
// them, so that the rows in flight share one slab or two: n = 4,096 with 4,096
// alphas (64 MB) 12.7 ms from the queue, 12.0 in order but dealt to resident
// blocks (which drift apart), 4.6 so (5.8 with a warp per row). n = 1,500 with
// 3,500 (21 MB): updates of 12.29 and 12.22 ms; n = 2,000 with 800 (6 MB): 245
// and 253 us of scoring; n = 512 with 1,024 (2 MB) 177 and 198.
constexpr size_t kMergeOrderedSlab = 16u << 20;
// (All this with the state-contiguous table; tc_merge_warps_kernel below has the
// other one.)
// Few rows (up to two rounds of resident blocks) are settled in one launch, 16
// of them looked at and re-scored per block: n = 64 (8,192 rows) 41 and 37 us
// of scoring with two launches and one; at four rounds n = 300 (37,800) 68 and
// 76 us, n = 100 (32,000) 93 and 99.
constexpr unsigned kMergeWholeRounds = 2;
constexpr unsigned kMergeBlocks = 4;   // resident blocks per SM (64 registers a thread)
constexpr unsigned kMergeBatch = 4;    // candidates gathered together
constexpr unsigned kMergePitch = 33;   // shared-memory row of one candidate's products

// A row's flag: kRowExact is what the compaction lists (0 and 1 once merged).
enum RowOutcome : unsigned { kRowSettled, kRowExact, kRowSeveral };

// Looks through one row's lists (per thread): the row is left to the exact
// scan, settled by its only candidate (choice: its index among the unique
// alphas, or with uniqJ among all), or has several (from *cutOut on).
__device__ __forceinline__ RowOutcome merge_look(unsigned row, const DevModel &md,
                                                 const unsigned *__restrict__ uniqJ, unsigned nLists, size_t rPad,
                                                 const float *__restrict__ a1, const float *__restrict__ d1,
                                                 const float *__restrict__ a1raw,
                                                 const unsigned *__restrict__ scal,
                                                 const uint2 *__restrict__ cand,
                                                 const unsigned *__restrict__ badModel,
                                                 unsigned *__restrict__ choice, unsigned *__restrict__ rowFlag,
                                                 unsigned *__restrict__ rowCand,
                                                 float *cutOut) {
    const unsigned ao = row / md.r, i = row % md.r;
    const uint4 *lists = reinterpret_cast<const uint4 *>(cand + (size_t)row * (nLists * LIST_SLOTS));
    const float thr = row_margin(a1, d1, (size_t)ao * rPad + i, __uint_as_float(scal[2]), __uint_as_float(scal[7]));
    const float rawBound = a1raw[(size_t)ao * rPad + i] * __uint_as_float(scal[1]);
    float best = -INFINITY, second = -INFINITY, x = -INFINITY;
    unsigned bestU = kNoneU;
    auto take = [&](unsigned score, unsigned u) {
        const float f = __uint_as_float(score);
        second = fmaxf(second, fminf(best, f));
        if (f > best) { best = f; bestU = u; }
    };
#pragma unroll 2
    for (unsigned q = 0; q < nLists; q++) {
        // The header and three entries are one sector.
        const uint4 *l = lists + (size_t)q * (LIST_SLOTS / 2);
        const uint4 w0 = __ldg(l), w1 = __ldg(l + 1);
        const unsigned len = min(w0.y, LIST_CAP);
        x = fmaxf(x, __uint_as_float(w0.x));
        if (len >= 1u) take(w0.z, w0.w);
        if (len >= 2u) take(w1.x, w1.y);
        if (len >= 3u) take(w1.z, w1.w);
        for (unsigned k = 4; k <= len; k += 4) {
            const uint4 w2 = __ldg(l + k / 2), w3 = __ldg(l + k / 2 + 1);
            take(w2.x, w2.y);
            if (k + 1u <= len) take(w2.z, w2.w);
            if (k + 2u <= len) take(w3.x, w3.y);
            if (k + 3u <= len) take(w3.z, w3.w);
        }
    }
    // Usable only with lists that the GEMM has finished, a finite margin,
    // non-negative probabilities, and scores far from the reference's -1e10
    // sentinel.
    const bool usable = (thr < 1e30f) && (best > -INFINITY) && *badModel == 0u && (rawBound < 1e9f) &&
                        g_device_error == 0u;
    const float cut = best - thr;
    const RowOutcome res = !usable || x >= cut ? kRowExact : second >= cut ? kRowSeveral : kRowSettled;
    rowFlag[row] = res;
    rowCand[row] = 0u;
    if (res == kRowSettled) {
        const size_t js = ((size_t)i * md.m + ao / md.z) * md.z + ao % md.z;
        choice[js] = uniqJ == nullptr ? bestU : uniqJ[bestU];
    }
    *cutOut = cut;
    return res;
}

// One warp re-scores a row's candidates (listed scores at or above the cut);
// returns (in every lane) how many there are. Slot e of the warp's view is
// slot e / nLists of list e % nLists, so the lists' headers (slot 0) come
// first, in lanes 0 .. nLists - 1; NE slots per lane are loaded before the
// lists' lengths are known, what lies beyond (rare: lists of more than 7
// entries, 15 of two) after that. With kTable the scores come from the
// alpha-contiguous projection table: entries of one state lie side by side
// there, so every lane takes a candidate and reads eight states' entries ahead
// of its sum. Without, from the model and the alphas.
template <int NE, bool kTable>
__device__ __forceinline__ unsigned merge_row(unsigned row, unsigned lane, const DevModel &md,
                                              const unsigned *__restrict__ suppLen, const ProjView &pv,
                                              const DirectScorer &ds, float *scratch, unsigned *list,
                                              const unsigned *__restrict__ uniqJ, unsigned nLists,
                                              const uint2 *__restrict__ cand, unsigned *__restrict__ choice,
                                              bool *flagged) {
    const unsigned ao = row / md.r, i = row % md.r;
    const unsigned a = ao / md.z, o = ao % md.z;
    const uint2 *lists = cand + (size_t)row * (nLists * LIST_SLOTS);
    const unsigned nEnt = nLists * LIST_SLOTS;
    auto slot_of = [&](unsigned e) { return lists + (size_t)(e % nLists) * LIST_SLOTS + e / nLists; };
    uint2 ent[NE];
#pragma unroll
    for (int j = 0; j < NE; j++) {
        const unsigned e = lane + 32u * j;
        ent[j] = e < nEnt ? __ldg(slot_of(e)) : make_uint2(0u, 0u);
    }
    const unsigned Li = suppLen[i];
    const int *sk = md.Z + (size_t)i * md.rz;
    const float *bk = md.B + (size_t)i * md.rz;
    // Lane l < nLists holds list l's header; list 0's has the cut.
    const float cut = __uint_as_float(__shfl_sync(0xffffffffu, ent[0].x, 0));
    const unsigned held = lane < nLists ? min(ent[0].y, LIST_CAP) : 0u;
    const unsigned steps = (__reduce_max_sync(0xffffffffu, held) + 1u) * nLists;  // e beyond these is in no list
    // The candidates, listed in shared memory.
    unsigned count = 0;
    auto keep = [&](unsigned e, uint2 en) {
        const unsigned len = __shfl_sync(0xffffffffu, held, e % nLists), k = e / nLists;
        const bool c = k != 0u && k <= len && __uint_as_float(en.x) >= cut;
        const unsigned msk = __ballot_sync(0xffffffffu, c);
        if (c) list[count + __popc(msk & ((1u << lane) - 1u))] = en.y;
        count += __popc(msk);
    };
#pragma unroll
    for (int j = 0; j < NE; j++) keep(lane + 32u * j, ent[j]);
    for (unsigned e0 = 32u * NE; e0 < steps; e0 += 32u) {
        const unsigned e = e0 + lane;
        keep(e, e < nEnt ? __ldg(slot_of(e)) : make_uint2(0u, 0u));
    }
    __syncwarp();
    const size_t js = ((size_t)i * md.m + a) * md.z + o;
    // Re-scored in the exact order, up to 32 at a time
    // (candidate t of the batch in lane t).
    float best = -INFINITY;
    unsigned bu = kNoneU;
    unsigned myU = kNoneU, nb = 0;
    auto settle = [&](float total) {
        if (lane < nb && (bu == kNoneU || total > best || (total == best && myU < bu))) { best = total; bu = myU; }
    };
    auto score_columns = [&]() {
        const float *P = pv.slab(ao) + (lane < nb ? myU : 0u) * pv.uStride;
        float total = 0.0f;
        unsigned k = 0;
        for (; k + 8u <= Li; k += 8u) {
            float p[8];
#pragma unroll
            for (unsigned q = 0; q < 8u; q++) p[q] = lane < nb ? __ldg(P + (unsigned)__ldg(sk + k + q) * pv.sStride) : 0.0f;
#pragma unroll
            for (unsigned q = 0; q < 8u; q++) total = fadd(total, fmul(p[q], __ldg(bk + k + q)));
        }
        for (; k < Li; k++)
            if (lane < nb) total = fadd(total, fmul(__ldg(P + (unsigned)__ldg(sk + k) * pv.sStride), __ldg(bk + k)));
        settle(total);
    };
    auto score_batch = [&]() {
        // The gathers of one candidate stay within one alpha row: lane k
        // computes support state k's term of every candidate of the
        // batch into the warp's scratch, then lane t adds candidate t's
        // terms in support order.
        float total = 0.0f;
        for (unsigned k0 = 0; k0 < Li; k0 += 32u) {
            const unsigned k = k0 + lane;
            const bool kv = k < Li;
            const unsigned s = kv ? (unsigned)sk[k] : 0u;
            const float b = kv ? bk[k] : 0.0f;
            if (md.ns <= kDirectNs) {
                // The state's coefficients and successors, loaded once for
                // the whole batch.
                const unsigned Ls = kv ? __ldg(ds.succLen + (size_t)s * md.m + a) : 0u;
                const float *cp = ds.C3 + (((size_t)a * md.z + o) * md.n + s) * md.ns;
                const int *spp = md.S + ((size_t)s * md.m + a) * md.ns;
                float cc[kDirectNs];
                int ss[kDirectNs];
#pragma unroll
                for (unsigned l = 0; l < kDirectNs; l++) {
                    cc[l] = l < Ls ? __ldg(cp + l) : 0.0f;
                    ss[l] = l < Ls ? __ldg(spp + l) : 0;
                }
                // Two candidates at a time: their gathers are issued
                // together, their sums are two independent chains.
                for (unsigned t = 0; t < nb; t += 2) {
                    const unsigned t1 = t + 1 < nb ? t + 1 : t;
                    const unsigned u0 = __shfl_sync(0xffffffffu, myU, t);
                    const unsigned u1 = __shfl_sync(0xffffffffu, myU, t1);
                    const float *G0 = ds.G + (size_t)__ldg(uniqJ + u0) * md.n;
                    const float *G1 = ds.G + (size_t)__ldg(uniqJ + u1) * md.n;
                    float g0[kDirectNs], g1[kDirectNs];
#pragma unroll
                    for (unsigned l = 0; l < kDirectNs; l++) {
                        if (l < Ls) {
                            g0[l] = __ldg(G0 + ss[l]);
                            g1[l] = __ldg(G1 + ss[l]);
                        }
                    }
                    float v0 = 0.0f, v1 = 0.0f;
#pragma unroll
                    for (unsigned l = 0; l < kDirectNs; l++) {
                        if (l < Ls) {
                            v0 = fadd(v0, fmul(cc[l], g0[l]));
                            v1 = fadd(v1, fmul(cc[l], g1[l]));
                        }
                    }
                    scratch[t * 32u + lane] = kv ? fmul(fmul(v0, md.gamma), b) : 0.0f;
                    if (t1 != t) scratch[t1 * 32u + lane] = kv ? fmul(fmul(v1, md.gamma), b) : 0.0f;
                }
            } else {
                for (unsigned t = 0; t < nb; t++) {
                    const unsigned uu = __shfl_sync(0xffffffffu, myU, t);
                    float p = 0.0f;
                    if (kv) p = fmul(fmul(ds.vt(md, a, o, s, ds.G + (size_t)__ldg(uniqJ + uu) * md.n), md.gamma), b);
                    scratch[t * 32u + lane] = p;
                }
            }
            __syncwarp();
            if (lane < nb) {
                const unsigned cnt = min(32u, Li - k0);
                for (unsigned q = 0; q < cnt; q++) total = fadd(total, scratch[lane * 32u + q]);
            }
            __syncwarp();
        }
        settle(total);
    };
    for (unsigned f = 0; f < count; f += 32u) {
        nb = min(32u, count - f);
        myU = lane < nb ? list[f + lane] : kNoneU;
        if constexpr (kTable) score_columns();
        else score_batch();
    }
    for (int off = 16; off > 0; off >>= 1) {
        const float b2 = __shfl_xor_sync(0xffffffffu, best, off);
        const unsigned u2 = __shfl_xor_sync(0xffffffffu, bu, off);
        if (u2 != kNoneU && (bu == kNoneU || b2 > best || (b2 == best && u2 < bu))) { best = b2; bu = u2; }
    }
    if (!(best > -1e10f)) {
        *flagged = true;  // sentinel case: the exact scan applies the reference's rule
    } else if (lane == 0) {
        choice[js] = kTable ? bu : uniqJ[bu];
    }
    return count;
}

// First half of the merge: settles the rows that one thread can and queues
// the others in rowList (their number in counters[0]), each with its cut in
// place of its first list's dropped score. Rows left to the exact scan are
// flagged and counted per compaction chunk, which the block lies in.
constexpr unsigned kCompactChunk = 4096;  // rows per block of the compaction (4 per thread)
constexpr unsigned kLookRows = 128;       // rows per block

__global__ void __launch_bounds__(kLookRows) tc_merge_look_kernel(
                                DevModel md, const unsigned *__restrict__ uniqJ, unsigned nLists, size_t rPad,
                                const float *__restrict__ a1, const float *__restrict__ d1,
                                const float *__restrict__ a1raw, const unsigned *__restrict__ scal,
                                uint2 *cand, unsigned *__restrict__ choice, unsigned *__restrict__ rowFlag, unsigned *__restrict__ rowCand,
                                unsigned *__restrict__ rowList, unsigned *__restrict__ counters,
                                unsigned *__restrict__ chunkCount, const unsigned *__restrict__ badModel) {
    const unsigned rows = md.m * md.z * md.r;  // fewer than 2^31 (tc_supported)
    const unsigned row = blockIdx.x * kLookRows + threadIdx.x, lane = threadIdx.x & 31;
    RowOutcome res = kRowSettled;
    if (row < rows) {
        float cut = 0.0f;
        res = merge_look(row, md, uniqJ, nLists, rPad, a1, d1, a1raw, scal, cand, badModel, choice, rowFlag, rowCand,
                         &cut);
        if (res == kRowSeveral) cand[(size_t)row * (nLists * LIST_SLOTS)].x = __float_as_uint(cut);
    }
    const unsigned msk = __ballot_sync(0xffffffffu, res == kRowSeveral);
    unsigned at = 0;
    if (lane == 0 && msk) at = atomicAdd(&counters[0], __popc(msk));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (res == kRowSeveral) rowList[at + __popc(msk & ((1u << lane) - 1u))] = row;
    const unsigned exact = __popc(__ballot_sync(0xffffffffu, res == kRowExact));
    if (lane == 0 && exact) atomicAdd(chunkCount + row / kCompactChunk, exact);
}

// Second half: the rows with several candidates, re-scored from the projection
// table by half a warp each: queued rows; or all rows in order, of which those
// flagged kRowSeveral are meant; or all 16 rows of a block, which has not been
// looked at before (both halves of the merge in one launch). Slot e of a half
// warp's view is slot e / nLists of list e % nLists; NE slots per lane are
// loaded before the lists' lengths are known.
enum class MergeRows { kQueued, kInOrder, kWhole };

template <int NE, MergeRows kRows>
__global__ void __launch_bounds__(256, kMergeBlocks) tc_merge_kernel(
                                DevModel md, const unsigned *__restrict__ suppLen,
                                const ProjView pv, unsigned nLists, size_t rPad, const float *__restrict__ a1,
                                const float *__restrict__ d1, const float *__restrict__ a1raw,
                                const unsigned *__restrict__ scal, const uint2 *__restrict__ cand,
                                unsigned *__restrict__ ustar, unsigned *__restrict__ rowFlag,
                                unsigned *__restrict__ rowCand, const unsigned *__restrict__ rowList,
                                unsigned *__restrict__ counters, unsigned *__restrict__ chunkCount,
                                const unsigned *__restrict__ badModel) {
    __shared__ float scratch[8][2][kMergeBatch * kMergePitch];
    extern __shared__ unsigned mergeLists[];   // [16 halves][nLists * LIST_SLOTS]
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = lane >> 4, hl = lane & 15u;
    unsigned *list = mergeLists + (size_t)(threadIdx.x >> 4) * (nLists * LIST_SLOTS);
    float *prod = scratch[warp][half];
    const unsigned nEnt = nLists * LIST_SLOTS;
    unsigned sum = 0, queued = md.m * md.z * md.r, first = (blockIdx.x * 8u + warp) * 2u;
    __shared__ unsigned severalRow[16];
    __shared__ float severalCut[16];
    if constexpr (kRows == MergeRows::kQueued) queued = counters[0];
    if constexpr (kRows == MergeRows::kWhole) {
        if (warp == 0) {
            const unsigned row = blockIdx.x * 16u + lane;
            RowOutcome res = kRowSettled;
            float cut = 0.0f;
            if (lane < 16u && row < queued)
                res = merge_look(row, md, nullptr, nLists, rPad, a1, d1, a1raw, scal, cand, badModel, ustar, rowFlag,
                                 rowCand, &cut);
            const unsigned msk = __ballot_sync(0xffffffffu, res == kRowSeveral);
            const unsigned exact = __popc(__ballot_sync(0xffffffffu, res == kRowExact));
            if (res == kRowSeveral) {
                const unsigned k = __popc(msk & ((1u << lane) - 1u));
                severalRow[k] = row;
                severalCut[k] = cut;
            }
            if (lane == 0) {
                const unsigned several = __popc(msk);
                for (unsigned k = several; k < 16u; k++) severalRow[k] = kNoneU;
                if (several) atomicAdd(&counters[0], several);
                if (exact) atomicAdd(chunkCount + row / kCompactChunk, exact);
            }
        }
        __syncthreads();
        first = warp * 2u;
        queued = 16u;
    }
    for (unsigned k0 = first; k0 < queued; k0 += gridDim.x * 16u) {
        // With an odd row at the end both halves look at it, one writes.
        bool mine = k0 + half < queued;
        unsigned row = mine ? k0 + half : k0;
        if constexpr (kRows == MergeRows::kInOrder) {
            mine = mine && rowFlag[row] == kRowSeveral;
            if (__ballot_sync(0xffffffffu, mine) == 0u) continue;
            if (!mine) row = k0 + (half ^ 1u);
        } else if constexpr (kRows == MergeRows::kWhole) {
            mine = severalRow[k0 + half] != kNoneU;
            if (severalRow[k0] == kNoneU) break;
            row = severalRow[mine ? k0 + half : k0];
        } else {
            row = __ldg(rowList + row);
        }
        const unsigned ao = row / md.r, i = row % md.r;
        const uint2 *lists = cand + (size_t)row * (nLists * LIST_SLOTS);
        auto slot_of = [&](unsigned e) { return lists + (e % nLists) * LIST_SLOTS + e / nLists; };
        uint2 ent[NE];
#pragma unroll
        for (int j = 0; j < NE; j++) {
            const unsigned e = hl + 16u * j;
            ent[j] = e < nEnt ? __ldg(slot_of(e)) : make_uint2(0u, 0u);
        }
        const unsigned Li = suppLen[i];
        const int *sk = md.Z + (size_t)i * md.rz;
        const float *bk = md.B + (size_t)i * md.rz;
        unsigned s0 = 0, s1 = 0;
        float b0 = 0.0f, b1 = 0.0f;
        if (hl < md.rz) { s0 = (unsigned)__ldg(sk + hl); b0 = __ldg(bk + hl); }
        if (hl + 16u < md.rz) { s1 = (unsigned)__ldg(sk + hl + 16u); b1 = __ldg(bk + hl + 16u); }
        // Lane l < nLists of a half holds list l's header; list 0's has the cut.
        float cut = __uint_as_float(__shfl_sync(0xffffffffu, ent[0].x, 0, 16));
        if constexpr (kRows == MergeRows::kWhole) cut = severalCut[mine ? k0 + half : k0];
        const unsigned held = hl < nLists ? min(ent[0].y, LIST_CAP) : 0u;
        const unsigned steps = (__reduce_max_sync(0xffffffffu, held) + 1u) * nLists;
        unsigned count = 0;
        auto keep = [&](unsigned e, uint2 en) {
            const unsigned len = __shfl_sync(0xffffffffu, held, e % nLists, 16), k = e / nLists;
            const bool c = k != 0u && k <= len && __uint_as_float(en.x) >= cut;
            const unsigned msk = (__ballot_sync(0xffffffffu, c) >> (16u * half)) & 0xffffu;
            if (c) list[count + __popc(msk & ((1u << hl) - 1u))] = en.y;
            count += __popc(msk);
        };
#pragma unroll
        for (int j = 0; j < NE; j++) keep(hl + 16u * j, ent[j]);
        for (unsigned e0 = 16u * NE; e0 < steps; e0 += 16u) {
            const unsigned e = e0 + hl;
            keep(e, e < nEnt ? __ldg(slot_of(e)) : make_uint2(0u, 0u));
        }
        __syncwarp();
        const float *P = pv.slab(ao);
        const unsigned most = max(count, __shfl_xor_sync(0xffffffffu, count, 16));
        const unsigned longest = max(Li, __shfl_xor_sync(0xffffffffu, Li, 16));
        float best = -INFINITY;
        unsigned bu = kNoneU;
        for (unsigned f = 0; f < most; f += kMergeBatch) {
            const unsigned nt = f < count ? min(kMergeBatch, count - f) : 0u;
            unsigned uu[kMergeBatch];
#pragma unroll
            for (unsigned t = 0; t < kMergeBatch; t++) uu[t] = t < nt ? list[f + t] : 0u;
            float total = 0.0f;
            for (unsigned q0 = 0; q0 < longest; q0 += 32u) {
                if (q0 != 0u || f != 0u) {
                    const unsigned q = q0 + hl;
                    if (q < md.rz) { s0 = (unsigned)__ldg(sk + q); b0 = __ldg(bk + q); }
                    if (q + 16u < md.rz) { s1 = (unsigned)__ldg(sk + q + 16u); b1 = __ldg(bk + q + 16u); }
                }
                const bool v0 = q0 + hl < Li, v1 = q0 + 16u + hl < Li;
                float p0[kMergeBatch], p1[kMergeBatch];
#pragma unroll
                for (unsigned t = 0; t < kMergeBatch; t++) {
                    p0[t] = t < nt && v0 ? __ldg(P + pv.at(s0, uu[t])) : 0.0f;
                    p1[t] = t < nt && v1 ? __ldg(P + pv.at(s1, uu[t])) : 0.0f;
                }
#pragma unroll
                for (unsigned t = 0; t < kMergeBatch; t++) {
                    if (t < nt) {
                        prod[t * kMergePitch + hl] = fmul(p0[t], b0);
                        prod[t * kMergePitch + hl + 16u] = fmul(p1[t], b1);
                    }
                }
                __syncwarp();
                if (hl < nt && q0 < Li) {
                    const float *row0 = prod + hl * kMergePitch;
                    const unsigned cnt = min(32u, Li - q0);
#pragma unroll 8
                    for (unsigned q = 0; q < cnt; q++) total = fadd(total, row0[q]);
                }
                __syncwarp();
            }
            if (hl < nt) {
                const unsigned u = list[f + hl];
                if (bu == kNoneU || total > best || (total == best && u < bu)) { best = total; bu = u; }
            }
        }
#pragma unroll
        for (int off = kMergeBatch / 2; off > 0; off >>= 1) {
            const float b2 = __shfl_xor_sync(0xffffffffu, best, off);
            const unsigned u2 = __shfl_xor_sync(0xffffffffu, bu, off);
            if (u2 != kNoneU && (bu == kNoneU || b2 > best || (b2 == best && u2 < bu))) { best = b2; bu = u2; }
        }
        if (hl == 0 && mine) {
            const bool exact = !(best > -1e10f);  // sentinel case: the exact scan applies the reference's rule
            rowCand[row] = count;
            rowFlag[row] = exact ? 1u : 0u;
            if (exact) {
                atomicAdd(chunkCount + row / kCompactChunk, 1u);
            } else {
                const size_t js = ((size_t)i * md.m + ao / md.z) * md.z + ao % md.z;
                ustar[js] = bu;
            }
            sum += count;
        }
        __syncwarp();
    }
    if (sum) atomicAdd(&counters[1], sum);
}

// Rows with several candidates, one warp each: with the alpha-contiguous table
// (which an update keeps after one that left more than 1 % of its rows open:
// many candidates per row, often wide beliefs) all rows in their own order, of
// which those flagged kRowSeveral are meant; without a table the queued rows.
// BF16, n = 4,096, m z = 32, 4,096 near-tied alphas (87 candidates a row): 3.5
// ms, 6.3 by half warps that gather four candidates at a time.
template <bool kTable>
__global__ void __launch_bounds__(256, kTable ? 3 : 1) tc_merge_warps_kernel(
                                DevModel md, const unsigned *__restrict__ suppLen, const ProjView pv,
                                const DirectScorer ds, const unsigned *__restrict__ uniqJ,
                                unsigned nLists, const uint2 *__restrict__ cand,
                                unsigned *__restrict__ choice, unsigned *__restrict__ rowFlag,
                                unsigned *__restrict__ rowCand, const unsigned *__restrict__ rowList,
                                unsigned *__restrict__ counters, unsigned *__restrict__ chunkCount) {
    // Each warp's candidate list; before them, without a table, [warps][32
    // candidates][32 states].
    extern __shared__ float mergeScratch[];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned queued = kTable ? md.m * md.z * md.r : counters[0];
    unsigned *list = reinterpret_cast<unsigned *>(mergeScratch + (kTable ? 0u : 8u * 1024u)) + warp * (nLists * LIST_SLOTS);
    unsigned sum = 0;
    for (unsigned k = blockIdx.x * 8u + warp; k < queued; k += gridDim.x * 8u) {
        const unsigned row = kTable ? k : __ldg(rowList + k);
        if (kTable && rowFlag[row] != kRowSeveral) continue;
        bool flagged = false;
        const unsigned rescored = merge_row<2, kTable>(row, lane, md, suppLen, pv, ds, mergeScratch + warp * 1024u, list,
                                                       uniqJ, nLists, cand, choice, &flagged);
        if (lane == 0) {
            rowCand[row] = rescored;
            rowFlag[row] = flagged ? 1u : 0u;
            if (flagged) atomicAdd(chunkCount + row / kCompactChunk, 1u);
        }
        sum += rescored;
        __syncwarp();
    }
    if (lane == 0 && sum) atomicAdd(&counters[1], sum);
}

// Indices of the flagged rows in increasing order, from the flagged rows per
// chunk of kCompactChunk: every block adds up the chunks before its own (at
// most a few thousand counts) and writes its rows behind them; the last
// block also stores the total in out[0] and, with scal (after a merge), the
// merge's counters and the error word behind it, and clears what the next
// update accumulates.
__global__ void __launch_bounds__(1024) tc_compact_write_kernel(const unsigned *__restrict__ flag, unsigned count,
                                                                const unsigned *__restrict__ chunkCount,
                                                                unsigned *__restrict__ items,
                                                                unsigned *__restrict__ out, unsigned *scal) {
    const unsigned mine = chunkCount[blockIdx.x];
    const bool lastBlock = blockIdx.x == gridDim.x - 1;
    if (mine == 0 && !lastBlock) return;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ unsigned wsum[32], before;
    unsigned c = 0;
    for (unsigned k = threadIdx.x; k < blockIdx.x; k += blockDim.x) c += chunkCount[k];
    for (int off = 16; off > 0; off >>= 1) c += __shfl_xor_sync(0xffffffffu, c, off);
    if (lane == 0) wsum[warp] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned t = 0;
        for (unsigned w = 0; w < blockDim.x / 32; w++) t += wsum[w];
        before = t;
        if (lastBlock) {
            out[0] = t + mine;
            if (scal != nullptr) {
                out[1] = scal[3];
                out[2] = scal[4];
                out[3] = atomicAdd(&g_device_error, 0u);
                scal[0] = scal[1] = scal[3] = scal[4] = scal[5] = scal[8] = 0u;
            }
        }
    }
    __syncthreads();
    if (mine == 0) return;
    const unsigned base = blockIdx.x * kCompactChunk + 4u * threadIdx.x;
    unsigned f[4], local = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        f[k] = (base + k < count && flag[base + k]) ? 1u : 0u;
        local += f[k];
    }
    unsigned incl = local;
    for (int off = 1; off < 32; off <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= (unsigned)off) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        unsigned x = lane < blockDim.x / 32 ? wsum[lane] : 0u;
        for (int off = 1; off < 32; off <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, x, off);
            if (lane >= (unsigned)off) x += y;
        }
        wsum[lane] = x;
    }
    __syncthreads();
    unsigned pos = before + (warp ? wsum[warp - 1] : 0u) + incl - local;
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (f[k]) items[pos++] = base + k;
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

static int encode_map(TcState *tc, CUtensorMap *map, const void *base, size_t rows, size_t cols, unsigned boxRows,
                      const char *fn) {
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)(cols * sizeof(uint16_t))};
    cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)boxRows};
    cuuint32_t estr[2] = {1, 1};
    const CUtensorMapDataType dt =
        tc->mode == NOVA_SCORING_FP16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    CUresult res = tc->encode(map, dt, 2, const_cast<void *>(base), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (res != CUDA_SUCCESS) {
        NOVA_ERR(fn, "Failed to encode a TMA tensor map.");
        return NOVA_ERROR_KERNEL_EXECUTION;
    }
    return NOVA_SUCCESS;
}

// Shared memory of an operand-building block (four blocks fit on an SM).
constexpr size_t kBuildSmem = 56 * 1024;

// (Re)builds A in the element type of the engine's scoring mode.
static int tc_build_operand(BackupEngine &eng, TcState *tc, const char *fn) {
    const DevModel &md = eng.md;
    // A new operand form starts its schedule choice afresh (the margins,
    // and with them the best split, differ between forms).
    if (tc->mode != eng.scoring) {
        tc->schedFixed = -1;
        tc->tuneNext = 0;
        tc->tuneWarm = false;
    }
    tc->mode = eng.scoring;
    // The build writes every column of the beliefs' rows; the padding's are 0.
    if (tc->rPad > md.r)
        cudaMemset2DAsync(tc->A + (size_t)md.r * tc->nPad, tc->rPad * tc->nPad * sizeof(uint16_t), 0,
                          (tc->rPad - md.r) * tc->nPad * sizeof(uint16_t), tc->MZ, eng.stream);
    cudaMemsetAsync(tc->a1, 0, (size_t)tc->MZ * tc->rPad * sizeof(float), eng.stream);
    cudaMemsetAsync(tc->a1raw, 0, (size_t)tc->MZ * tc->rPad * sizeof(float), eng.stream);
    cudaMemsetAsync(tc->d1, 0, (size_t)tc->MZ * tc->rPad * sizeof(float), eng.stream);
    cudaMemsetAsync(tc->badModel, 0, sizeof(unsigned), eng.stream);
    // a1 bounds sum_s |A| with A in exact arithmetic: the FP32 sums of
    // non-negative terms are inflated by their worst-case rounding.
    const float slack = 1.0f + (float)(md.n + md.rz * md.ns + 8) * 1.2e-7f;
    // d1 is an FP32 sum of nPad exact non-negative terms.
    const float dslack = 1.0f + (float)(tc->nPad + 8) * 1.2e-7f;
    float *Ot = reinterpret_cast<float *>(tc->cand);   // as the lists are written after A is built (tc_supported)
    int rc;
    const dim3 tiles((unsigned)(tc->nPad / 32), ceil_div(md.z, 32), std::min(md.m, kMaxGridZ));
    tc_transpose_o_kernel<<<tiles, dim3(32, 8), 0, eng.stream>>>(md, tc->nPad, Ot, tc->badModel);
    if ((rc = check_launch(fn, "observation transpose")) != NOVA_SUCCESS) return rc;
    const size_t wBytes = tc->nPad * sizeof(float);
    const unsigned nb = 4 * wBytes <= kBuildSmem ? 4u : 2 * wBytes <= kBuildSmem ? 2u : 1u;
    auto build = nb == 4 ? tc_build_a_kernel<4> : nb == 2 ? tc_build_a_kernel<2> : tc_build_a_kernel<1>;
    allow_dynamic_smem(build, nb * wBytes);
    build<<<ceil_div(md.r, nb) * md.m, 256, nb * wBytes, eng.stream>>>(
        md, eng.succLen, eng.suppLen, tc->rPad, tc->nPad, tc->mode == NOVA_SCORING_FP16 ? 1 : 0, Ot, tc->A, tc->a1,
        tc->a1raw, tc->d1, slack, dslack, tc->badModel);
    rc = check_launch(fn, "scoring operand build");
    if (rc != NOVA_SUCCESS) return rc;
    return encode_map(tc, &tc->tmA, tc->A, (size_t)tc->MZ * tc->rPad, tc->nPad, BM, fn);
}

// Dynamic shared memory of every scoring-kernel instantiation (once).
static bool gemm_attributes_set() {
    static std::once_flag once;
    static bool ok = false;
    std::call_once(once, [] {
        const int b = (int)GEMM_SMEM;
        const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
        ok = cudaFuncSetAttribute(tc_score_gemm_kernel<false, SingleUnits>, attr, b) == cudaSuccess &&
             cudaFuncSetAttribute(tc_score_gemm_kernel<true, SingleUnits>, attr, b) == cudaSuccess &&
             cudaFuncSetAttribute(tc_score_gemm_kernel<false, BatchUnits>, attr, b) == cudaSuccess &&
             cudaFuncSetAttribute(tc_score_gemm_kernel<true, BatchUnits>, attr, b) == cudaSuccess;
        if (!ok) cudaGetLastError();
    });
    return ok;
}

int tc_build(BackupEngine &eng, const char *fn) {
    if (eng.tc) return NOVA_SUCCESS;
    const DevModel &md = eng.md;
    std::unique_ptr<TcState> tc(new TcState());
    tc->nPad = round_up(md.n, BK);
    tc->rPad = round_up(md.r, BM);
    tc->capN = round_up(md.r, BN);
    tc->MZ = md.m * md.z;
    tc->mTiles = (unsigned)(tc->rPad / BM);
    const size_t aElems = (size_t)tc->MZ * tc->rPad * tc->nPad;
    size_t freeB = 0, totalB = 0;
    cudaMemGetInfo(&freeB, &totalB);
    const size_t slots = (size_t)tc->MZ * md.r * max_lists(tc->nPad);
    const size_t need = aElems * 2 + tc->capN * tc->nPad * 4 + slots * LIST_SLOTS * 8 + (size_t)tc->MZ * md.r * 12;
    if (need + (256ull << 20) > freeB) {
        NOVA_ERR(fn, "Not enough device memory for the tensor-core operands; using exact scoring.");
        return NOVA_ERROR_DEVICE_MALLOC;
    }
    void *fnPtr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fnPtr, 12000, cudaEnableDefault, &q) !=
            cudaSuccess || q != cudaDriverEntryPointSuccess || fnPtr == nullptr) {
        cudaGetLastError();
        NOVA_ERR(fn, "cuTensorMapEncodeTiled is not available.");
        return NOVA_ERROR_KERNEL_EXECUTION;
    }
    tc->encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fnPtr);
    int rc;
    tc->arena.add(&tc->A, aElems);
    tc->arena.add(&tc->a1, (size_t)tc->MZ * tc->rPad);
    tc->arena.add(&tc->a1raw, (size_t)tc->MZ * tc->rPad);
    tc->arena.add(&tc->d1, (size_t)tc->MZ * tc->rPad);
    tc->arena.add(&tc->Gb, tc->capN * tc->nPad * 2);
    tc->arena.add(&tc->shift, md.n);
    tc->arena.add(&tc->scal, 9);
    tc->arena.add(&tc->cand, slots * LIST_SLOTS);
    tc->arena.add(&tc->rowFlag, (size_t)tc->MZ * md.r);
    tc->arena.add(&tc->rowCand, (size_t)tc->MZ * md.r);
    tc->arena.add(&tc->rowList, (size_t)tc->MZ * md.r);
    tc->arena.add(&tc->chunkCount, ceil_div((size_t)tc->MZ * md.r, kCompactChunk));
    tc->arena.add(&tc->badModel, 1);
    if ((rc = tc->arena.commit(fn, "the tensor-core operands")) != NOVA_SUCCESS) return rc;
    if ((rc = tc_build_operand(eng, tc.get(), fn)) != NOVA_SUCCESS) return rc;
    cudaDeviceProp prop;
    cudaGetDeviceProperties(&prop, 0);
    tc->numSMs = prop.multiProcessorCount;
    cudaEventCreate(&tc->g0);
    cudaEventCreate(&tc->g1);
    if (!gemm_attributes_set()) {
        cudaGetLastError();
        NOVA_ERR(fn, "Failed to configure the scoring kernel's shared memory.");
        return NOVA_ERROR_KERNEL_EXECUTION;
    }
    eng.tc = tc.release();
    return sync_device(fn);
}

int tc_prepare(BackupEngine &eng, const float *src, unsigned nU, const char *fn) {
    int rc;
    if (!eng.tc && (rc = tc_build(eng, fn)) != NOVA_SUCCESS) return rc;
    TcState *tc = eng.tc;
    if (tc->mode != eng.scoring && (rc = tc_build_operand(eng, tc, fn)) != NOVA_SUCCESS) return rc;
    tc->src = src;
    const DevModel &md = eng.md;
    const bool fp16 = tc->mode == NOVA_SCORING_FP16;
    // BF16 carries the alphas as two BF16 terms (split); FP16 as one.
    const unsigned kSplit = fp16 ? 1u : 2u;
    const size_t nPadRows = round_up(nU, BN);
    const unsigned nTiles = (unsigned)(nPadRows / BN);
    // ---- shift, scale and pack the unique alphas ----
    if (!tc->scalClean) cudaMemsetAsync(tc->scal, 0, 9 * sizeof(unsigned), eng.stream);
    tc->scalClean = false;  // until the merge's list has cleared it again
    tc_shift_kernel<<<md.n, 256, 0, eng.stream>>>(eng.Gt, eng.gtCols, md.n, nU, tc->shift, tc->scal);
    if ((rc = check_launch(fn, "alpha shift")) != NOVA_SUCCESS) return rc;
    // The row bound is a1 * escale + d1 * dscale (packed units), with
    // escale = U * gmax + gN * Gmax * gscale and dscale = gmax (1 + 2^-22).
    // Against the reference's FP32 score, the tensor-core score of a row
    // (shifted by a row constant) differs by at most
    //  * sum_s |A - Ahalf| |alpha - c|  <= d1 gmax: A's operand rounding,
    //    measured per row when A was built;
    //  * epsA a1 gmax: the FP32 build of A itself;
    //  * (1 + uA)(uG + 2^-23) a1 gmax: the alphas' rounding to FP16 (uG =
    //    2^-11, plus the absolute error of FP16 subnormals, below 2^-25 per
    //    entry) or to the hi + lo BF16 pair (uG = 2^-16), and the FP32
    //    rounding of alpha - c;
    //  * the accumulation: each tcgen05.mma step (K=16) adds at most 2^-22 of
    //    the running sum of magnitudes, over kSplit * nPad / 16 steps;
    //  * gN a1 Gmax: the reference's own rounding over ns + rz + 3 operations.
    // uA is A's unit roundoff (2^-11 FP16, 2^-8 BF16).
    const double u24 = 1.0 / 16777216.0;
    const double epsA = (double)(md.rz * md.ns + 4) * u24;
    const double uA = fp16 ? 1.0 / 2048.0 : 1.0 / 256.0;
    const double uG = fp16 ? 1.0 / 2048.0 : 1.0 / 65536.0;
    const double steps = (double)kSplit * (double)tc->nPad / 16.0 + 2.0;
    const float U = (float)(epsA * (1.0 + 2.0 * u24) + (1.0 + uA) * (uG + 2.0 * u24) +
                            steps / 4194304.0 * (1.0 + uA) * (1.0 + uG) * (1.0 + 2.0 * u24) +
                            (fp16 ? (double)tc->nPad / 33554432.0 / 8192.0 : 0.0) + 1.0 / 1048576.0);
    const float gN = (float)((double)(md.ns + md.rz + 3) * u24 * 1.01);
    const unsigned nChunks = ceil_div((size_t)tc->MZ * md.r, kCompactChunk);
    tc_pack_kernel<<<(unsigned)nPadRows, 256, 0, eng.stream>>>(src, md.n, tc->nPad, eng.uniqMap, nU, tc->shift,
                                                              fp16 ? 1 : 0, kSplit == 2u ? 1 : 0, tc->Gb, tc->scal, U,
                                                              gN, tc->chunkCount, nChunks);
    if ((rc = check_launch(fn, "alpha packing")) != NOVA_SUCCESS) return rc;
    // ---- schedule and the alphas' tensor map ----
    TcState::Launch &L = tc->last;
    if ((rc = encode_map(tc, &L.tmB, tc->Gb, nPadRows, tc->nPad * kSplit, BN, fn)) != NOVA_SUCCESS) return rc;
    // Each alpha group leaves two lists per row (one per epilogue half).
    if (tc->schedFixed < 0 && tc->nPad > kTuneMaxNPad) tc->schedFixed = kDeepSchedule;
    const unsigned groups = kSchedules[tc->schedFixed >= 0 ? tc->schedFixed : (tc->tuneWarm ? (int)tc->tuneNext : 0)];
    L.nU = nU;
    L.nTiles = nTiles;
    L.groups = std::max(1u, std::min<unsigned>(groups, nTiles));
    L.lists = 2u * L.groups;
    L.kSplit = kSplit;
    L.fp16 = fp16;
    tc->groupsUsed = L.groups;
    return NOVA_SUCCESS;
}

// The scoring GEMM of one prepared solver on its stream.
int tc_gemm(BackupEngine &eng, bool timed, const char *fn) {
    TcState *tc = eng.tc;
    const TcState::Launch &L = tc->last;
    const unsigned totalUnits = tc->MZ * tc->mTiles * L.groups;
    const unsigned grid = std::min<unsigned>(totalUnits, (unsigned)tc->numSMs);
    if (timed) cudaEventRecord(tc->g0, eng.stream);
    const SingleUnits units{tc->MZ, (unsigned)tc->rPad, eng.md.r, tc->mTiles, L.nTiles, L.groups, L.nU,
                            (unsigned)(tc->nPad / BK), L.kSplit, tc->a1, tc->d1, tc->scal, tc->cand};
    auto gemm = tc->nPad > kTuneMaxNPad ? tc_score_gemm_kernel<true, SingleUnits> : tc_score_gemm_kernel<false, SingleUnits>;
    gemm<<<grid, GEMM_THREADS, GEMM_SMEM, eng.stream>>>(tc->tmA, L.tmB, make_idesc(L.fp16 ? 0u : 1u), units);
    int rc = check_launch(fn, "tensor-core scoring");
    if (rc != NOVA_SUCCESS) return rc;
    if (timed) cudaEventRecord(tc->g1, eng.stream);
    return NOVA_SUCCESS;
}

// After the GEMM: merge the lists, apply the margin, re-score near ties
// exactly, and list the rows left to the exact scan (count in eng.itemCount).
int tc_finish(BackupEngine &eng, const char *fn) {
    TcState *tc = eng.tc;
    const TcState::Launch &L = tc->last;
    const DevModel &md = eng.md;
    int rc;
    const size_t rows = (size_t)tc->MZ * md.r;
    // The list can hold every row: it is sized m*z*r like the flags.
    const unsigned nChunks = ceil_div(rows, kCompactChunk);
    const DirectScorer ds{eng.succLen, eng.C3, tc->src};
    const bool table = eng.useProjNow;
    const unsigned blocks = (unsigned)ceil_div(rows, 16);
    const bool whole = table && eng.projStateMajor && blocks <= kMergeWholeRounds * kMergeBlocks * (unsigned)tc->numSMs;
    if (!whole) {
        tc_merge_look_kernel<<<(unsigned)ceil_div(rows, kLookRows), kLookRows, 0, eng.stream>>>(
            md, table ? nullptr : eng.uniqMap, L.lists, tc->rPad, tc->a1, tc->d1, tc->a1raw, tc->scal, tc->cand,
            table ? eng.ustar : eng.jstar, tc->rowFlag, tc->rowCand, tc->rowList, tc->scal + 3, tc->chunkCount,
            tc->badModel);
        if ((rc = check_launch(fn, "candidate lists")) != NOVA_SUCCESS) return rc;
    }
    if (table && eng.projStateMajor) {
        const bool inOrder = eng.proj_view().slice * sizeof(float) >= kMergeOrderedSlab;
        const bool two = L.lists <= 2u;
        auto merge = whole     ? (two ? tc_merge_kernel<2, MergeRows::kWhole> : tc_merge_kernel<4, MergeRows::kWhole>)
                     : inOrder ? (two ? tc_merge_kernel<2, MergeRows::kInOrder> : tc_merge_kernel<4, MergeRows::kInOrder>)
                               : (two ? tc_merge_kernel<2, MergeRows::kQueued> : tc_merge_kernel<4, MergeRows::kQueued>);
        const unsigned grid = whole || inOrder ? blocks : std::min(blocks, kMergeBlocks * (unsigned)tc->numSMs);
        merge<<<grid, 256, 16 * L.lists * LIST_SLOTS * sizeof(unsigned), eng.stream>>>(
            md, eng.suppLen, eng.proj_view(), L.lists, tc->rPad, tc->a1, tc->d1, tc->a1raw, tc->scal, tc->cand,
            eng.ustar, tc->rowFlag, tc->rowCand, tc->rowList, tc->scal + 3, tc->chunkCount, tc->badModel);
    } else {
        const unsigned warpBlocks = (unsigned)ceil_div(rows, 8);
        const unsigned grid = table ? warpBlocks : std::min(warpBlocks, (unsigned)tc->numSMs);
        const size_t smem = 8 * ((table ? 0u : 1024u) + L.lists * LIST_SLOTS) * sizeof(float);
        (table ? tc_merge_warps_kernel<true> : tc_merge_warps_kernel<false>)<<<grid, 256, smem, eng.stream>>>(
            md, eng.suppLen, table ? eng.proj_view() : ProjView{}, ds, eng.uniqMap, L.lists, tc->cand,
            table ? eng.ustar : eng.jstar, tc->rowFlag, tc->rowCand, tc->rowList, tc->scal + 3, tc->chunkCount);
    }
    if ((rc = check_launch(fn, "candidate merge")) != NOVA_SUCCESS) return rc;
    tc_compact_write_kernel<<<nChunks, 1024, 0, eng.stream>>>(tc->rowFlag, (unsigned)rows, tc->chunkCount,
                                                              tc->rowList, eng.itemCount, tc->scal);
    if ((rc = check_launch(fn, "exact-scan list")) != NOVA_SUCCESS) return rc;
    tc->scalClean = true;
    return NOVA_SUCCESS;
}

// Flag the (belief, action) item of every listed row; each item is counted
// once, in its compaction chunk.
__global__ void tc_row_items_kernel(const unsigned *__restrict__ rowList, unsigned nRows, unsigned r, unsigned m,
                                    unsigned z, unsigned *__restrict__ itemFlag,
                                    unsigned *__restrict__ chunkCount) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nRows) return;
    const unsigned row = rowList[t];
    const unsigned ao = row / r, i = row % r;
    const size_t item = (size_t)i * m + ao / z;
    if (atomicExch(itemFlag + item, 1u) == 0u) atomicAdd(chunkCount + item / kCompactChunk, 1u);
}

// The distinct (belief, action) items of the listed rows, in increasing
// order, into eng.items (count in eng.itemCount). The row flags are free
// again once the row list is written, and hold the item flags.
int tc_rows_to_items(BackupEngine &eng, const unsigned *rowList, unsigned nRows, const char *fn) {
    TcState *tc = eng.tc;
    const DevModel &md = eng.md;
    const unsigned count = md.r * md.m;
    int rc;
    const unsigned nChunks = ceil_div(count, kCompactChunk);
    cudaMemsetAsync(tc->rowFlag, 0, (size_t)count * sizeof(unsigned), eng.stream);
    cudaMemsetAsync(tc->chunkCount, 0, nChunks * sizeof(unsigned), eng.stream);
    tc_row_items_kernel<<<ceil_div(nRows, 256), 256, 0, eng.stream>>>(rowList, nRows, md.r, md.m, md.z,
                                                                      tc->rowFlag, tc->chunkCount);
    if ((rc = check_launch(fn, "rows to items")) != NOVA_SUCCESS) return rc;
    tc_compact_write_kernel<<<nChunks, 1024, 0, eng.stream>>>(tc->rowFlag, count, tc->chunkCount, eng.items,
                                                              eng.itemCount, nullptr);
    return check_launch(fn, "item list");
}

int tc_score_launch(BackupEngine &eng, const float *src, unsigned nU, bool timed, const char *fn) {
    int rc;
    if ((rc = tc_prepare(eng, src, nU, fn)) != NOVA_SUCCESS) return rc;
    if ((rc = tc_gemm(eng, timed, fn)) != NOVA_SUCCESS) return rc;
    return tc_finish(eng, fn);
}

// ---------------------------------------------------------------------------
// Batched scoring: one persistent launch over the work units of many solvers
// ---------------------------------------------------------------------------

struct TcBatch {
    struct Group {
        unsigned totalUnits = 0, nModels = 0;
        bool fp16 = true, sorted = false;
        BatchModel *models = nullptr;   // device work table
    };
    std::vector<Group> groups;   // one per operand form and kind of list
    int numSMs = 0;
    ~TcBatch() {
        for (auto &g : groups) cudaFree(g.models);
    }
};

int tc_batch_create(BackupEngine *const *engs, unsigned count, TcBatch **out, const char *fn) {
    std::unique_ptr<TcBatch> b(new TcBatch());
    std::vector<std::vector<BatchModel>> host;
    for (unsigned k = 0; k < count; k++) {
        const BackupEngine &e = *engs[k];
        const TcState *tc = e.tc;
        if (tc == nullptr || tc->last.groups == 0) {
            NOVA_ERR(fn, "A solver of the batch has no prepared tensor-core launch.");
            return NOVA_ERROR_INVALID_DATA;
        }
        const TcState::Launch &L = tc->last;
        const bool sorted = tc->nPad > kTuneMaxNPad;
        size_t gi = 0;
        while (gi < b->groups.size() && (b->groups[gi].fp16 != L.fp16 || b->groups[gi].sorted != sorted)) gi++;
        if (gi == b->groups.size()) {
            b->groups.emplace_back();
            b->groups.back().fp16 = L.fp16;
            b->groups.back().sorted = sorted;
            host.emplace_back();
        }
        TcBatch::Group &g = b->groups[gi];
        BatchModel m;
        memset(&m, 0, sizeof(m));
        m.tmA = tc->tmA;
        m.tmB = L.tmB;
        m.unitStart = g.totalUnits;
        m.MZ = tc->MZ;
        m.rPad = (unsigned)tc->rPad;
        m.r = e.md.r;
        m.mTiles = tc->mTiles;
        m.nTiles = L.nTiles;
        m.groups = L.groups;
        m.nU = L.nU;
        m.kBlocks = (unsigned)(tc->nPad / BK);
        m.kSplit = L.kSplit;
        m.a1 = tc->a1; m.d1 = tc->d1; m.scal = tc->scal;
        m.cand = tc->cand;
        const unsigned long long units = (unsigned long long)m.MZ * m.mTiles * m.groups;
        if ((unsigned long long)g.totalUnits + units >= (1ull << 31)) {
            NOVA_ERR(fn, "Too many work units for one batched launch.");
            return NOVA_ERROR_INVALID_DATA;
        }
        g.totalUnits += (unsigned)units;
        g.nModels++;
        host[gi].push_back(m);
        b->numSMs = tc->numSMs;
    }
    for (size_t gi = 0; gi < b->groups.size(); gi++) {
        int rc;
        if ((rc = dev_alloc(&b->groups[gi].models, host[gi].size(), fn, "the batch work table")) != NOVA_SUCCESS)
            return rc;
        if ((rc = h2d(b->groups[gi].models, host[gi].data(), host[gi].size() * sizeof(BatchModel), fn,
                      "the batch work table")) != NOVA_SUCCESS)
            return rc;
    }
    *out = b.release();
    return NOVA_SUCCESS;
}

int tc_batch_gemm(TcBatch *b, cudaStream_t stream, const char *fn) {
    for (const auto &g : b->groups) {
        if (g.totalUnits == 0) continue;
        const BatchUnits units{g.models, g.nModels, g.totalUnits};
        const unsigned grid = std::min<unsigned>(g.totalUnits, (unsigned)b->numSMs);
        CUtensorMap unused;
        memset(&unused, 0, sizeof(unused));
        auto gemm = g.sorted ? tc_score_gemm_kernel<true, BatchUnits> : tc_score_gemm_kernel<false, BatchUnits>;
        gemm<<<grid, GEMM_THREADS, GEMM_SMEM, stream>>>(unused, unused, make_idesc(g.fp16 ? 0u : 1u), units);
        int rc = check_launch(fn, "batched tensor-core scoring");
        if (rc != NOVA_SUCCESS) return rc;
    }
    return NOVA_SUCCESS;
}

void tc_batch_release(TcBatch *b) { delete b; }

bool tc_schedule_fixed(const BackupEngine &eng) {
    // Fixed, and the operand is built for the solver's current mode (a
    // rebuild must not end up inside a captured update).
    return eng.tc != nullptr && eng.tc->schedFixed >= 0 && eng.tc->mode == eng.scoring;
}

const unsigned *tc_row_list(const BackupEngine &eng) { return eng.tc ? eng.tc->rowList : nullptr; }

int tc_score(BackupEngine &eng, const float *src, unsigned nU, unsigned *nRows, const unsigned **rowList,
             const char *fn) {
    int rc;
    if ((rc = tc_score_launch(eng, src, nU, true, fn)) != NOVA_SUCCESS) return rc;
    unsigned h[BackupEngine::kReport];
    if (cudaMemcpyAsync(h, eng.report, sizeof(h), cudaMemcpyDeviceToHost, eng.stream) != cudaSuccess ||
            cudaStreamSynchronize(eng.stream) != cudaSuccess) {
        cudaGetLastError();
        NOVA_ERR(fn, "Failed to read the scoring counters.");
        return NOVA_ERROR_MEMCPY_TO_HOST;
    }
    *nRows = h[1];
    *rowList = eng.tc->rowList;
    return tc_take_report(eng, h, fn);
}

int tc_take_report(BackupEngine &eng, const unsigned (&h)[BackupEngine::kReport], const char *fn) {
    const TcState *tc = eng.tc;
    if (h[4] != 0) {
        read_and_clear_device_error();
        NOVA_ERR(fn, "The tensor-core scoring kernel timed out waiting on a barrier; results are invalid.");
        return NOVA_ERROR_KERNEL_EXECUTION;
    }
    eng.stats.rowsOverflow = h[1];
    eng.stats.rowsMultiCand = h[2];
    eng.stats.candidates = h[3];
    cudaEventElapsedTime(&eng.stats.msGemm, tc->g0, tc->g1);
    eng.stats.tcGroups = tc->groupsUsed;
    return NOVA_SUCCESS;
}

int tc_row_detail(const BackupEngine &eng, unsigned *candidates, unsigned *exactRows, const char *fn) {
    const TcState *tc = eng.tc;
    const DevModel &md = eng.md;
    const size_t rows = (size_t)md.m * md.z * md.r;
    std::vector<unsigned> cand(rows), flag(rows);
    if (cudaStreamSynchronize(eng.stream) != cudaSuccess ||
            cudaMemcpy(cand.data(), tc->rowCand, rows * sizeof(unsigned), cudaMemcpyDeviceToHost) != cudaSuccess ||
            cudaMemcpy(flag.data(), tc->rowFlag, rows * sizeof(unsigned), cudaMemcpyDeviceToHost) != cudaSuccess) {
        cudaGetLastError();
        NOVA_ERR(fn, "Failed to read the per-row scoring detail.");
        return NOVA_ERROR_MEMCPY_TO_HOST;
    }
    for (unsigned i = 0; i < md.r; i++) { candidates[i] = 0; exactRows[i] = 0; }
    for (size_t row = 0; row < rows; row++) {   // row = (a*z + o) * r + i
        const unsigned i = (unsigned)(row % md.r);
        candidates[i] += cand[row];
        exactRows[i] += flag[row] ? 1u : 0u;
    }
    return NOVA_SUCCESS;
}

float tc_tuned_cost(const BackupEngine &eng) {
    const TcState *tc = eng.tc;
    if (tc == nullptr || tc->schedFixed < 0 || tc->schedFixed >= kTunedSchedules ||
            tc->tuneNext < (unsigned)kTunedSchedules)
        return -1.0f;
    return tc->tuneCost[tc->schedFixed];
}

void tc_tune_feedback(BackupEngine &eng, float msScoring, unsigned nU) {
    TcState *tc = eng.tc;
    if (tc == nullptr || tc->schedFixed >= 0 || nU == 0) return;
    if (!tc->tuneWarm) {
        tc->tuneWarm = true;
        return;
    }
    tc->tuneCost[tc->tuneNext] = msScoring / (float)nU;
    if (++tc->tuneNext < (unsigned)kTunedSchedules) return;
    unsigned best = 0;
    for (unsigned k = 1; k < (unsigned)kTunedSchedules; k++)
        if (tc->tuneCost[k] < tc->tuneCost[best]) best = k;
    tc->schedFixed = (int)best;
}

}  // namespace nova_gb300

// nova-gb300: V(b) and the policy's action for many beliefs at once.
//
// For each belief b (dense, n states) the reference evaluates
// (pomdp_alpha_vectors.cpp:52-79)
//
//   V_i = sum_s fl(Gamma_i(s) * b(s))   (added in state order, FP32)
//   V(b) = max_i V_i                     (from -1e10, strict '<': lowest i on ties)
//   a(b) = pi[argmax]
//
// Adding fl(Gamma_i(s) * 0) = +-0 changes no sum (one that starts at +0 is
// never -0) while Gamma is finite, and beliefs are mostly zeros, so beliefs
// are first compressed to their nonzeros in state order. Two kernels form the
// V_i, each with products and sums rounded separately and in state order:
//
//   * value_sparse_kernel: a block holds 4 or 8 alphas in shared memory, a
//     thread walks one belief's nonzeros;
//   * value_tiles_kernel: a register-tiled FP32 product (beliefs x states) .
//     (states x alphas) over all states, for the tiles of beliefs with too
//     many nonzeros. Two alphas per instruction: f32x2 products, summed with
//     the exact f32x2 form (fma of the product by a run-time 1.0).
//
// Either way the best alpha of a belief is kept as one 64-bit key, raised
// with atomicMax: the value's order-preserving bits above the complement of
// the alpha's index (equal values: lowest index; a V_i is never -0). Key 0
// stands for "nothing above -1e10".

#include "common.h"

#include <algorithm>

#include <nova/constants.h>
#include <nova/pomdp/policies/pomdp_alpha_vectors.h>
#include <nova/nova_gb300.h>

using nova::POMDPAlphaVectors;

namespace nova_gb300 {
namespace {

constexpr unsigned kThreads = 256;
constexpr unsigned TB = 128;          // beliefs per dense tile, and per choice of kernel
constexpr unsigned TK = 16;           // states per shared-memory stage of the dense kernel
constexpr unsigned kStagedBeliefs = 32;  // most beliefs whose lists may be staged

__device__ __forceinline__ unsigned long long value_key(float v, unsigned alpha) {
    const unsigned b = __float_as_uint(v);
    const unsigned order = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
    return ((unsigned long long)order << 32) | (unsigned)~alpha;
}
__device__ __forceinline__ float key_value(unsigned long long key) {
    const unsigned order = (unsigned)(key >> 32);
    return __uint_as_float((order & 0x80000000u) ? (order & 0x7fffffffu) : ~order);
}
// Raises the belief's key by (v, alpha); keys only grow, so a stale read
// only costs an atomic that changes nothing.
__device__ __forceinline__ void raise_key(unsigned long long *key, float v, unsigned alpha) {
    const unsigned long long k = value_key(v, alpha);
    if (k > __ldcg(key)) atomicMax(key, k);
}

// The nonzeros of every belief in state order, entry k of belief b at
// list[k * pitch + b] (so that threads on consecutive beliefs read
// consecutive entries), up to cap of them; nnz[b] counts all. One warp per
// belief; clears its key. Reads B once: 21 us of HBM time at 8,192 x 4,096.
__global__ void __launch_bounds__(kThreads) value_compress_kernel(const float *__restrict__ Bd, unsigned count,
                                                                  unsigned n, unsigned cap, unsigned pitch,
                                                                  uint2 *__restrict__ list, unsigned *__restrict__ nnz,
                                                                  unsigned long long *__restrict__ keys) {
    const unsigned lane = threadIdx.x & 31;
    const unsigned b = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    if (b >= count) return;
    const float *row = Bd + (size_t)b * n;
    unsigned filled = 0;
    for (unsigned s0 = 0; s0 < n; s0 += 128) {
        float v[4];
#pragma unroll
        for (unsigned q = 0; q < 4; q++) {
            const unsigned s = s0 + 32 * q + lane;
            v[q] = s < n ? __ldg(row + s) : 0.0f;
        }
#pragma unroll
        for (unsigned q = 0; q < 4; q++) {
            const bool some = !(v[q] == 0.0f);  // NaN is kept
            const unsigned msk = __ballot_sync(0xffffffffu, some);
            const unsigned k = filled + __popc(msk & ((1u << lane) - 1u));
            if (some && k < cap) list[(size_t)k * pitch + b] = make_uint2(s0 + 32 * q + lane, __float_as_uint(v[q]));
            filled += __popc(msk);
        }
    }
    if (lane == 0) {
        nnz[b] = filled;
        keys[b] = 0ull;
    }
}

// Whether every belief of the TB-belief tile that holds belief b is listed
// (the whole warp asks about one tile).
__device__ __forceinline__ bool tile_listed(const unsigned *__restrict__ nnz, unsigned b, unsigned count, unsigned cap,
                                            unsigned lane) {
    const unsigned t0 = b / TB * TB;
    unsigned most = 0;
#pragma unroll
    for (unsigned q = 0; q < TB / 32; q++)
        if (t0 + 32 * q + lane < count) most = max(most, nnz[t0 + 32 * q + lane]);
    return !__any_sync(0xffffffffu, most > cap);
}

// Alphas [a0, a0 + 4 H) of this block against the listed beliefs of its share:
// the alphas lie in shared memory as H planes of [state][4], so a lane's
// vector read of a nonzero's state touches one 16-byte bank group and the
// eight lanes of a phase spread over all eight. Bound by those reads (random
// states: about 2.6 passes each). A block whose alphas are not all finite adds
// every state's product instead, as the reference does. One alpha tile per
// block costs its load once per share of beliefs; 8,192 sparse beliefs (64
// nonzeros) x 8,192 alphas x 4,096 states: 1.3 ms, against 21.2 ms over all
// states with a 4 x 4 register tile.
// With few beliefs a walk is one long chain of dependent steps, so their lists
// are staged in shared memory first (kStaged; one belief of 2,699 nonzeros:
// 200 us from L2, 122 us staged).
template <int H, bool kStaged>
__global__ void __launch_bounds__(1024) value_sparse_kernel(const float *__restrict__ G, unsigned r, unsigned n,
                                                                const float *__restrict__ Bd, unsigned count,
                                                                unsigned share, unsigned cap, unsigned pitch,
                                                                const uint2 *__restrict__ list,
                                                                const unsigned *__restrict__ nnz,
                                                                unsigned long long *__restrict__ keys, float one) {
    extern __shared__ __align__(16) float4 planes[];  // [H][n]
    const unsigned a0 = blockIdx.x * 4u * H;
    int odd = 0;
    for (unsigned h = 0; h < H; h++) {
        for (unsigned s = threadIdx.x; s < n; s += blockDim.x) {
            float g[4];
#pragma unroll
            for (unsigned j = 0; j < 4; j++) {
                const unsigned ai = a0 + 4 * h + j;
                g[j] = ai < r ? __ldg(G + (size_t)ai * n + s) : 0.0f;
                odd |= !(fabsf(g[j]) <= 3.402823466e38f);
            }
            planes[h * n + s] = make_float4(g[0], g[1], g[2], g[3]);
        }
    }
    uint2 *staged = reinterpret_cast<uint2 *>(planes + (size_t)H * n);
    if constexpr (kStaged)
        for (unsigned e = threadIdx.x; e < cap * count; e += blockDim.x) staged[e] = list[e];
    odd = __syncthreads_or(odd);
    const unsigned lane = threadIdx.x & 31;
    const unsigned long long one2 = pack_f32x2(one, one);
    const unsigned bEnd = min(count, (blockIdx.y + 1) * share);
    for (unsigned b0 = blockIdx.y * share + (threadIdx.x & ~31u); b0 < bEnd; b0 += blockDim.x) {
        if (!tile_listed(nnz, b0, count, cap, lane)) continue;
        const unsigned b = b0 + lane;
        if (b >= bEnd) continue;
        unsigned long long acc[2 * H];
#pragma unroll
        for (int h = 0; h < 2 * H; h++) acc[h] = 0ull;
        auto add = [&](unsigned s, float p) {
            const unsigned long long pp = pack_f32x2(p, p);
#pragma unroll
            for (int h = 0; h < H; h++) {
                const ulonglong2 g = *reinterpret_cast<const ulonglong2 *>(planes + h * n + s);
                acc[2 * h] = fma_f32x2(mul_f32x2(g.x, pp), one2, acc[2 * h]);
                acc[2 * h + 1] = fma_f32x2(mul_f32x2(g.y, pp), one2, acc[2 * h + 1]);
            }
        };
        if (!odd) {
            // Eight entries are loaded while the eight before are added.
            constexpr unsigned kAhead = 8;
            const unsigned L = nnz[b];
            auto entry = [&](unsigned k) {
                if constexpr (kStaged) return staged[k * pitch + b];
                else return __ldg(list + (size_t)k * pitch + b);
            };
            uint2 e[kAhead], next[kAhead];
#pragma unroll
            for (unsigned q = 0; q < kAhead; q++)
                if (q < L) next[q] = entry(q);
            unsigned k = 0;
            for (; k + kAhead <= L; k += kAhead) {
#pragma unroll
                for (unsigned q = 0; q < kAhead; q++) {
                    e[q] = next[q];
                    if (k + kAhead + q < L) next[q] = entry(k + kAhead + q);
                }
#pragma unroll
                for (unsigned q = 0; q < kAhead; q++) add(e[q].x, __uint_as_float(e[q].y));
            }
#pragma unroll
            for (unsigned q = 0; q < kAhead; q++)
                if (k + q < L) add(next[q].x, __uint_as_float(next[q].y));
        } else {
            for (unsigned s = 0; s < n; s++) add(s, __ldg(Bd + (size_t)b * n + s));
        }
        float best = NOVA_FLT_MIN;
        unsigned bi = 0;
        bool any = false;
#pragma unroll
        for (int j = 0; j < 4 * H; j++) {
            const float v = f32x2_part(acc[j / 2], j & 1);
            if (a0 + j < r && best < v) { best = v; bi = a0 + j; any = true; }
        }
        if (any) raise_key(keys + b, best, bi);
    }
}

// Dense tiles: 16 NB beliefs x TA alphas, NB x TA/16 sums a thread; the next
// TK states of both operands are loaded into registers while this stage's
// products are added. Bound by FP32 issue: 2 n operations per (belief,
// alpha); with few tiles by the chain of a tile's stages, so tiles are small
// then.
template <int TA, int NB>
__global__ void __launch_bounds__(kThreads) value_tiles_kernel(const float *__restrict__ G, unsigned r, unsigned n,
                                                               const float *__restrict__ Bd, unsigned count,
                                                               unsigned cap, const unsigned *__restrict__ nnz,
                                                               unsigned long long *__restrict__ keys, float one) {
    constexpr unsigned NA = TA / 16, TBD = 16 * NB;
    constexpr unsigned LB = TBD * TK / kThreads, LA = TA * TK / kThreads;  // staged values per thread
    // State-major tiles; rows padded by 4 floats so the staging stores spread
    // over the banks and rows stay 16-byte aligned.
    __shared__ __align__(16) float sB[2][TK][TBD + 4];
    __shared__ __align__(16) float sG[2][TK][TA + 4];
    const unsigned tid = threadIdx.x;
    const unsigned b0 = blockIdx.y * TBD, a0 = blockIdx.x * TA;
    if (cap != 0u && tile_listed(nnz, b0, count, cap, tid & 31)) return;   // cap 0: no lists, no other kernel
    const unsigned tx = tid % 16, ty = tid / 16;   // alpha group, belief group
    const unsigned long long one2 = pack_f32x2(one, one);
    unsigned long long acc[NB][NA / 2];
#pragma unroll
    for (unsigned i = 0; i < (unsigned)NB; i++)
#pragma unroll
        for (unsigned j = 0; j < NA / 2; j++) acc[i][j] = 0ull;
    // Thread tid stages states (tid % TK) of rows tid / TK + (kThreads / TK) q:
    // 16 threads read 64 consecutive bytes of a row.
    const unsigned kk = tid % TK, row0 = tid / TK;
    float rb[LB], rg[LA];
    auto fetch = [&](unsigned k0) {
        const unsigned s = k0 + kk;
#pragma unroll
        for (unsigned q = 0; q < LB; q++) {
            const unsigned bi = b0 + row0 + (kThreads / TK) * q;
            rb[q] = s < n && bi < count ? __ldg(Bd + (size_t)bi * n + s) : 0.0f;
        }
#pragma unroll
        for (unsigned q = 0; q < LA; q++) {
            const unsigned ai = a0 + row0 + (kThreads / TK) * q;
            rg[q] = s < n && ai < r ? __ldg(G + (size_t)ai * n + s) : 0.0f;
        }
    };
    fetch(0);
    unsigned buf = 0;
    for (unsigned k0 = 0; k0 < n; k0 += TK, buf ^= 1) {
#pragma unroll
        for (unsigned q = 0; q < LB; q++) sB[buf][kk][row0 + (kThreads / TK) * q] = rb[q];
#pragma unroll
        for (unsigned q = 0; q < LA; q++) sG[buf][kk][row0 + (kThreads / TK) * q] = rg[q];
        __syncthreads();
        if (k0 + TK < n) fetch(k0 + TK);
        // States past n are not added: their products could be +-0 only, but
        // rows past the ends hold zeros that meet no state either.
        const unsigned kEnd = min(TK, n - k0);
        auto step = [&](unsigned k) {
            float bq[NB];
#pragma unroll
            for (unsigned i = 0; i < (unsigned)NB; i += 4) {
                const float4 v = *reinterpret_cast<const float4 *>(&sB[buf][k][NB * ty + i]);
                bq[i] = v.x; bq[i + 1] = v.y; bq[i + 2] = v.z; bq[i + 3] = v.w;
            }
            unsigned long long gq[NA / 2];
#pragma unroll
            for (unsigned j = 0; j < NA / 4; j++) {
                // Alphas 4 tx + 64 j .. + 3: the 16 threads of a row read
                // consecutive vectors.
                const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(&sG[buf][k][4 * tx + 64 * j]);
                gq[2 * j] = v.x; gq[2 * j + 1] = v.y;
            }
#pragma unroll
            for (unsigned i = 0; i < (unsigned)NB; i++) {
                const unsigned long long bb = pack_f32x2(bq[i], bq[i]);
#pragma unroll
                for (unsigned j = 0; j < NA / 2; j++) acc[i][j] = fma_f32x2(mul_f32x2(gq[j], bb), one2, acc[i][j]);
            }
        };
        if (kEnd == TK) {
#pragma unroll 4
            for (unsigned k = 0; k < TK; k++) step(k);
        } else {
            for (unsigned k = 0; k < kEnd; k++) step(k);
        }
    }
    // Best alpha of this tile per belief: the 16 threads of a belief group
    // hold NA alphas each; reduce with shuffles (max value, then lowest index).
#pragma unroll
    for (unsigned i = 0; i < (unsigned)NB; i++) {
        float best = NOVA_FLT_MIN;
        unsigned bi = 0xffffffffu;
#pragma unroll
        for (unsigned j = 0; j < NA; j++) {
            const unsigned ai = a0 + 4 * tx + 64 * (j / 4) + j % 4;
            const float v = f32x2_part(acc[i][j / 2], j & 1);
            if (ai < r && best < v) { best = v; bi = ai; }
        }
        for (int off = 8; off > 0; off >>= 1) {
            const float ov = __shfl_down_sync(0xffffffffu, best, off, 16);
            const unsigned oi = __shfl_down_sync(0xffffffffu, bi, off, 16);
            if (oi != 0xffffffffu && (bi == 0xffffffffu || ov > best || (ov == best && oi < bi))) { best = ov; bi = oi; }
        }
        const unsigned belief = b0 + NB * ty + i;
        if (tx == 0 && belief < count && bi != 0xffffffffu) raise_key(keys + belief, best, bi);
    }
}

__global__ void value_finish_kernel(unsigned count, const unsigned long long *__restrict__ keys,
                                    const unsigned *__restrict__ pi, float *__restrict__ V,
                                    unsigned *__restrict__ act) {
    const unsigned b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= count) return;
    const unsigned long long k = keys[b];
    V[b] = k == 0ull ? NOVA_FLT_MIN : key_value(k);
    act[b] = k == 0ull ? 0u : pi[~(unsigned)k];
}

}  // namespace

static int value_batched(const float *dG, const unsigned *dPi, unsigned r, unsigned n, const float *dB,
                         unsigned count, float *dV, unsigned *dA, const char *fn) {
    int dev = 0, optin = 0, sms = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        optin = 48 * 1024;
        sms = 152;
    }
    // Planes of 4 alphas that fit in shared memory: two, one, or none (then
    // every tile is dense).
    const size_t plane = (size_t)n * sizeof(float4);
    const unsigned H = 2 * plane + 1024 <= (size_t)optin ? 2u : plane + 1024 <= (size_t)optin ? 1u : 0u;
    // Nonzeros listed per belief: a nonzero costs the sparse kernel about what
    // 4.3 states cost the dense one (8,192 beliefs and alphas, 4,096 states:
    // 17.1 ms with 900 nonzeros, 18.4 ms over all states). Beliefs are listed
    // in full where the dense tiles would not fill the device.
    const bool fewTiles = (size_t)ceil_div(r, 64) * ceil_div(count, TB) < (size_t)sms;
    unsigned cap = H == 0 ? 0u : fewTiles ? n : std::max(1u, n / 4);
    // One allocation: keys, nonzero counts, lists.
    const size_t keyBytes = (size_t)count * sizeof(unsigned long long), nnzBytes = round_up((size_t)count * 4, 16);
    unsigned char *work = nullptr;
    int rc;
    if (cap != 0 && cudaMalloc(reinterpret_cast<void **>(&work), keyBytes + nnzBytes + (size_t)cap * count * 8) !=
            cudaSuccess) {
        cudaGetLastError();
        work = nullptr;
        cap = 0;  // no room for the lists
    }
    if (work == nullptr && (rc = dev_alloc(&work, keyBytes + nnzBytes, fn, "the belief keys")) != NOVA_SUCCESS)
        return rc;
    auto *keys = reinterpret_cast<unsigned long long *>(work);
    auto *nnz = reinterpret_cast<unsigned *>(work + keyBytes);
    auto *list = reinterpret_cast<uint2 *>(work + keyBytes + nnzBytes);
    value_compress_kernel<<<ceil_div(count, kThreads / 32), kThreads>>>(dB, count, n, cap, count, list, nnz, keys);
    rc = check_launch(fn, "belief nonzeros");
    if (rc == NOVA_SUCCESS && cap != 0) {
        const unsigned aTiles = ceil_div(r, 4 * H);
        const size_t listBytes = (size_t)cap * count * sizeof(uint2);
        const bool staged = count <= kStagedBeliefs && H * plane + listBytes + 1024 <= (size_t)optin;
        const size_t smem = H * plane + (staged ? listBytes : 0);
        const unsigned perSM = (unsigned)std::max<size_t>(1, std::min<size_t>(8, (size_t)optin / (smem + 1024)));
        // 32 warps an SM hide the shared-memory latency, whatever the planes
        // leave room for in blocks.
        const unsigned threads = perSM == 1 ? 1024u : perSM <= 3 ? 512u : 256u;
        // Shares of beliefs (multiples of TB) so that two rounds of blocks
        // fill the device.
        const unsigned shares = std::max(1u, std::min(ceil_div(count, 2 * TB), ceil_div(2ull * sms * perSM, aTiles)));
        const unsigned share = (unsigned)round_up(ceil_div(count, shares), 2 * TB);
        auto kernel = staged ? (H == 2 ? value_sparse_kernel<2, true> : value_sparse_kernel<1, true>)
                             : (H == 2 ? value_sparse_kernel<2, false> : value_sparse_kernel<1, false>);
        allow_dynamic_smem(kernel, smem);
        kernel<<<dim3(aTiles, ceil_div(count, share)), threads, smem>>>(dG, r, n, dB, count, share, cap, count, list,
                                                                         nnz, keys, 1.0f);
        rc = check_launch(fn, "belief values");
    }
    if (rc == NOVA_SUCCESS && cap < n) {
        // Wide tiles once they fill the device twice over, smaller ones while
        // larger would not fill it (200 alphas of 20,000 states, 50 beliefs:
        // 2.1 ms with tiles of 128 x 64, 1.3 with 64 x 64).
        const unsigned bTiles = ceil_div(count, TB), aTiles = ceil_div(r, 64);
        auto dense = [&](auto kernel, unsigned ta, unsigned tb) {
            kernel<<<dim3(ceil_div(r, ta), ceil_div(count, tb)), kThreads>>>(dG, r, n, dB, count, cap, nnz, keys, 1.0f);
        };
        if ((size_t)ceil_div(r, 128) * bTiles >= 2ull * sms) dense(value_tiles_kernel<128, 8>, 128, 128);
        else if ((size_t)aTiles * bTiles >= 2ull * sms) dense(value_tiles_kernel<64, 8>, 64, 128);
        else dense(value_tiles_kernel<64, 4>, 64, 64);
        rc = check_launch(fn, "belief values (dense)");
    }
    if (rc == NOVA_SUCCESS) {
        value_finish_kernel<<<ceil_div(count, 256), 256>>>(count, keys, dPi, dV, dA);
        rc = check_launch(fn, "belief arg-maxima");
    }
    if (rc == NOVA_SUCCESS) rc = sync_device(fn);
    cudaFree(work);
    return rc;
}

}  // namespace nova_gb300

using namespace nova_gb300;

extern "C" int pomdp_alpha_vectors_value_batched_gpu(const float *d_Gamma, const unsigned int *d_pi, unsigned int r,
                                                     unsigned int n, const float *d_B, unsigned int count,
                                                     float *d_V, unsigned int *d_a) {
    static const char *fn = "pomdp_alpha_vectors_value_batched_gpu";
    if (d_Gamma == nullptr || d_pi == nullptr || d_B == nullptr || d_V == nullptr || d_a == nullptr || r == 0 ||
            n == 0 || count == 0) {
        NOVA_ERR(fn, "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    return value_batched(d_Gamma, d_pi, r, n, d_B, count, d_V, d_a, fn);
}

extern "C" int pomdp_alpha_vectors_value_and_action_batched(const POMDPAlphaVectors *policy, const float *B,
                                                            unsigned int count, float *V, unsigned int *a) {
    static const char *fn = "pomdp_alpha_vectors_value_and_action_batched";
    if (policy == nullptr || policy->n == 0 || policy->m == 0 || policy->r == 0 || policy->Gamma == nullptr ||
            policy->pi == nullptr || B == nullptr || V == nullptr || a == nullptr || count == 0) {
        NOVA_ERR(fn, "Invalid input.");
        return NOVA_ERROR_INVALID_DATA;
    }
    const unsigned r = policy->r, n = policy->n;
    float *dG = nullptr, *dB = nullptr, *dV = nullptr;
    unsigned *dPi = nullptr, *dA = nullptr;
    Arena arena;
    int rc;
    arena.add(&dG, (size_t)r * n);
    arena.add(&dPi, r);
    arena.add(&dB, (size_t)count * n);
    arena.add(&dV, count);
    arena.add(&dA, count);
    if ((rc = arena.commit(fn, "the policy and the beliefs")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(dG, policy->Gamma, (size_t)r * n * sizeof(float), fn, "the alpha-vectors")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(dPi, policy->pi, r * sizeof(unsigned), fn, "the policy actions")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(dB, B, (size_t)count * n * sizeof(float), fn, "the beliefs")) != NOVA_SUCCESS) return rc;
    if ((rc = value_batched(dG, dPi, r, n, dB, count, dV, dA, fn)) != NOVA_SUCCESS) return rc;
    if ((rc = d2h(V, dV, count * sizeof(float), fn, "the values")) != NOVA_SUCCESS) return rc;
    return d2h(a, dA, count * sizeof(unsigned), fn, "the actions");
}

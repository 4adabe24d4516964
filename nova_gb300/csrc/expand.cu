// nova-gb300: belief-set expansion on the GB300.
//
// Replaces pomdp_expand_random_cpu, pomdp_expand_distinct_beliefs_cpu and
// pomdp_expand_pema_cpu (pomdp_expand_cpu.cpp:81-383) and
// pomdp_expand_random_gpu (pomdp_expand_gpu.cu:127-215), with the
// reference's FP32 operation order throughout, so the new beliefs are
// bit-identical:
//
//   * belief update b'(s') = O(a,s',o) * sum_{(s,i): S(s,a,i)=s'} T(s,a,i) b(s),
//     then normalised (pomdp_model_cpu.cpp:89-137). The reference scatters
//     over (s, i) in order; here each s' gathers its predecessors from a
//     per-action list sorted by (s, i), which adds the same terms in the same
//     order, so the states s' run in parallel.
//   * every sum the reference accumulates sequentially over s (observation
//     probabilities, normalisers, L1 distances, error bounds) is formed the
//     same way: the terms are computed in parallel and one thread adds them in
//     order.
//   * one block per belief (PEMA) or per trajectory (random); PEMA's L1
//     distances to all r beliefs run one belief per thread over a dense,
//     state-major copy of B.
//   * the distinct expansion needs the exact distances only where they decide
//     something: every successor's smallest distance is first bounded from the
//     beliefs' nonzeros, and the sums the reference forms are added up for the
//     successors and beliefs within that bound's error of the best.
//
// The random expansions draw from libc rand() on the host exactly as the
// reference does (srand(time(nullptr)), or a fixed seed set with
// nova_gb300_expand_seed); the draws do not depend on belief values, so the
// host lays out every trajectory first and the device runs them in parallel.

#include "common.h"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <ctime>
#include <vector>

#include <nova/constants.h>
#include <nova/pomdp/pomdp.h>
#include <nova/pomdp/policies/pomdp_alpha_vectors.h>
#include <nova/pomdp/utilities/pomdp_model_cpu.h>
#include <nova/pomdp/utilities/pomdp_expand_cpu.h>
#include <nova/pomdp/utilities/pomdp_expand_gpu.h>
#include <nova/pomdp/utilities/pomdp_sigma_cpu.h>
#include <nova/nova_gb300.h>

using nova::POMDP;
using nova::POMDPAlphaVectors;

namespace nova_gb300 {
namespace {

constexpr unsigned kThreads = 256;
constexpr unsigned kNoIndex = 0xffffffffu;

std::atomic<unsigned> g_seed_fixed{0};
std::atomic<unsigned> g_seed{0};

void seed_rand() {
    if (g_seed_fixed.load()) srand(g_seed.load());
    else srand((unsigned)time(nullptr));
}

unsigned draw(float scale) { return (unsigned)((float)rand() / (float)RAND_MAX * scale); }

struct ExpModel {
    unsigned n, ns, m, z, r, rz;
    float gamma;
    const int *S;
    const float *T, *O, *R;
    const int *Z;
    const float *B;
    const unsigned *predStart;  // [m][n+1]
    const unsigned *predState;  // predecessor s of each entry, sorted by (s, i) per (a, s')
    const float *predT;         // its T(s,a,i)
    const float *BT;            // [n][r] dense beliefs, state-major
    const float *PO;            // [m][n][z] sum_i fl(T(s,a,i) O(a,S,o)), added in i order
};

// Shared-memory layout of one block: b, bp, aux, tmp (n floats each) plus
// scalars.
struct BlockBufs {
    float *b, *bp, *aux, *tmp;
};

// Thread 0 adds v[0..n) in order; the result is returned to every thread.
__device__ float seq_sum(const float *v, unsigned n, float *slot) {
    __syncthreads();
    if (threadIdx.x == 0) {
        float acc = 0.0f;
        for (unsigned s = 0; s < n; s++) acc = fadd(acc, v[s]);
        *slot = acc;
    }
    __syncthreads();
    return *slot;
}

// The sum of term(0) .. term(n - 1) in that order, by a whole warp: the lanes
// form 128 terms (the next ones' loads under way meanwhile), lane 0 adds them.
// buf: 128 floats of the warp's.
template <typename F>
__device__ __forceinline__ float warp_ordered_sum(unsigned n, float *buf, unsigned lane, F term) {
    float acc = 0.0f, t[4];
    auto fetch = [&](unsigned s0) {
#pragma unroll
        for (unsigned q = 0; q < 4; q++) t[q] = s0 + 32 * q + lane < n ? term(s0 + 32 * q + lane) : 0.0f;
    };
    fetch(0);
    for (unsigned s0 = 0; s0 < n; s0 += 128) {
#pragma unroll
        for (unsigned q = 0; q < 4; q++) buf[32 * q + lane] = t[q];
        __syncwarp();
        if (s0 + 128 < n) fetch(s0 + 128);
        if (lane == 0) {
            if (s0 + 128 <= n) {
#pragma unroll
                for (unsigned q = 0; q < 128; q += 4) {
                    const float4 v = *reinterpret_cast<const float4 *>(buf + q);
                    acc = fadd(fadd(fadd(fadd(acc, v.x), v.y), v.z), v.w);
                }
            } else {
                for (unsigned q = 0; q < n - s0; q++) acc = fadd(acc, buf[q]);
            }
        }
        __syncwarp();
    }
    return __shfl_sync(0xffffffffu, acc, 0);
}

// PO[a][s][o]: the belief-independent part of
// pomdp_expand_probability_observation_cpu (pomdp_expand_cpu.cpp:56-78).
__global__ void prob_table_kernel(unsigned n, unsigned ns, unsigned m, unsigned z, const int *__restrict__ S,
                                  const float *__restrict__ T, const float *__restrict__ O, float *__restrict__ PO) {
    const size_t total = (size_t)m * n * z;
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const unsigned o = (unsigned)(e % z);
        const size_t as = e / z;
        const unsigned s = (unsigned)(as % n), a = (unsigned)(as / n);
        const size_t row = ((size_t)s * m + a) * ns;
        float val = 0.0f;
        for (unsigned i = 0; i < ns; i++) {
            const int sp = S[row + i];
            if (sp < 0) break;
            val = fadd(val, fmul(T[row + i], O[((size_t)a * n + sp) * z + o]));
        }
        PO[e] = val;
    }
}

// Pr(o | b, a) for one observation: sum_s fl(PO * b(s)) in state order.
__device__ __forceinline__ float prob_obs_dense(const ExpModel &md, const float *b, unsigned a, unsigned o) {
    const float *po = md.PO + (size_t)a * md.n * md.z + o;
    float acc = 0.0f;
#pragma unroll 8
    for (unsigned s = 0; s < md.n; s++) acc = fadd(acc, fmul(__ldg(po + (size_t)s * md.z), b[s]));
    return acc;
}

// pomdp_belief_update_cpu (pomdp_model_cpu.cpp:89-137). Returns true when
// the normaliser reaches FLT_ERR_TOL; otherwise bp keeps the unnormalised
// values, as the reference's does.
__device__ bool belief_update(const ExpModel &md, const float *b, float *bp, unsigned a, unsigned o, float *slot) {
    for (unsigned sp = threadIdx.x; sp < md.n; sp += blockDim.x) {
        const unsigned e0 = md.predStart[(size_t)a * (md.n + 1) + sp];
        const unsigned e1 = md.predStart[(size_t)a * (md.n + 1) + sp + 1];
        float v = 0.0f;
        for (unsigned k = e0; k < e1; k++) {
            v = fadd(v, fmul(md.predT[k], b[md.predState[k]]));
        }
        bp[sp] = fmul(v, md.O[((size_t)a * md.n + sp) * md.z + o]);
    }
    const float norm = seq_sum(bp, md.n, slot);
    if (fabs((double)fabsf(norm)) < NOVA_FLT_ERR_TOL) return false;
    for (unsigned sp = threadIdx.x; sp < md.n; sp += blockDim.x) bp[sp] = __fdiv_rn(bp[sp], norm);
    __syncthreads();
    return true;
}

__device__ void load_belief(const ExpModel &md, unsigned i, float *b) {
    for (unsigned s = threadIdx.x; s < md.n; s += blockDim.x) b[s] = md.BT[(size_t)s * md.r + i];
    __syncthreads();
}

// L1 distance sum_s |b_j(s) - bp(s)| in state order, one belief j per thread;
// returns the smallest and (in *argOut) the lowest j attaining it.
__device__ float min_distance(const ExpModel &md, const float *bp, unsigned *argOut, float *sv, unsigned *si) {
    float best = NOVA_FLT_MAX;
    unsigned bj = kNoIndex;
    for (unsigned j = threadIdx.x; j < md.r; j += blockDim.x) {
        float d = 0.0f;
#pragma unroll 8
        for (unsigned s = 0; s < md.n; s++) d = fadd(d, fabsf(__fsub_rn(__ldg(md.BT + (size_t)s * md.r + j), bp[s])));
        if (d < best) { best = d; bj = j; }
    }
    sv[threadIdx.x] = best;
    si[threadIdx.x] = bj;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (unsigned t = 1; t < blockDim.x; t++) {
            if (si[t] == kNoIndex) continue;
            if (si[0] == kNoIndex || sv[t] < sv[0] || (sv[t] == sv[0] && si[t] < si[0])) { sv[0] = sv[t]; si[0] = si[t]; }
        }
    }
    __syncthreads();
    const float v = sv[0];
    if (argOut) *argOut = si[0];
    __syncthreads();
    return v;
}

__device__ BlockBufs carve(float *smem, unsigned n) {
    return BlockBufs{smem, smem + n, smem + 2 * (size_t)n, smem + 3 * (size_t)n};
}

// ---------------------------------------------------------------------------
// pomdp_expand_distinct_beliefs_cpu (pomdp_expand_cpu.cpp:153-241): for
// belief i, the successor b'(b_i, a, o) farthest (in min L1 distance) from
// the belief set. Beliefs are expanded in chunks that share the buffers below;
// row ao = a*z + o of belief i is a successor.
// ---------------------------------------------------------------------------
struct Distinct {
    unsigned first, chunk;      // beliefs first .. first + chunk - 1
    float *W;                   // [chunk][m][n] sum over predecessors of fl(T b), before O
    float *bp;                  // [chunk][n][m*z] normalised successors, row-contiguous
    float *mass;                // [chunk][m*z] sum_s b'(s); negative: no successor
    float *bound;               // [chunk][m*z] approximate smallest distance
    uint2 *list;                // [r][cap] the beliefs' nonzeros (state, value bits) in state order
    unsigned *nnz;              // [r]
    float *total;               // [r] sum_s b_j(s)
    unsigned *odd;              // [2] a value below 0 or not finite somewhere; the largest total's bits
    unsigned cap;               // min(n, rz)
};

// Whether some observation probability sum is not finite (a zero of a belief
// then still decides something).
__global__ void distinct_check_kernel(ExpModel md, unsigned *__restrict__ odd) {
    const size_t total = (size_t)md.m * md.n * md.z;
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x)
        if (!(fabsf(md.PO[e]) <= 3.402823466e38f)) atomicOr(odd, 1u);
}

// Nonzeros of every belief in state order (one warp each), their sums, and
// whether any value is negative or not finite.
__global__ void __launch_bounds__(kThreads) distinct_list_kernel(ExpModel md, Distinct d) {
    const unsigned lane = threadIdx.x & 31, j = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    if (j >= md.r) return;
    unsigned filled = 0;
    float sum = 0.0f;
    bool odd = false;
    for (unsigned s0 = 0; s0 < md.n; s0 += 32) {
        const unsigned s = s0 + lane;
        const float v = s < md.n ? md.BT[(size_t)s * md.r + j] : 0.0f;
        const bool some = !(v == 0.0f);
        const unsigned msk = __ballot_sync(0xffffffffu, some);
        if (some) d.list[(size_t)j * d.cap + filled + __popc(msk & ((1u << lane) - 1u))] = make_uint2(s, __float_as_uint(v));
        filled += __popc(msk);
        odd |= !(v >= 0.0f && v <= NOVA_FLT_MAX);
        sum += v;
    }
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    if (__any_sync(0xffffffffu, odd) && lane == 0) atomicOr(d.odd, 1u);
    if (lane == 0) {
        d.nnz[j] = filled;
        d.total[j] = sum;
        if (sum >= 0.0f) atomicMax(d.odd + 1, __float_as_uint(sum));
    }
}

// W[i][a][s'] in the reference's order (belief_update's first sum; it does
// not depend on o). One block per belief and action.
__global__ void __launch_bounds__(kThreads) distinct_mass_kernel(ExpModel md, Distinct d) {
    extern __shared__ __align__(16) float smem[];
    const unsigned i = blockIdx.x / md.m, a = blockIdx.x % md.m;
    load_belief(md, d.first + i, smem);
    for (unsigned sp = threadIdx.x; sp < md.n; sp += blockDim.x) {
        const unsigned e0 = md.predStart[(size_t)a * (md.n + 1) + sp];
        const unsigned e1 = md.predStart[(size_t)a * (md.n + 1) + sp + 1];
        float v = 0.0f;
        for (unsigned k = e0; k < e1; k++) v = fadd(v, fmul(md.predT[k], smem[md.predState[k]]));
        d.W[((size_t)i * md.m + a) * md.n + sp] = v;
    }
}

// One thread per (belief, action, observation), observations adjacent:
// whether the successor exists (Pr(o|b,a) != 0 and the normaliser reaches
// FLT_ERR_TOL), its values and their sum. The sums the reference adds in state
// order are chains of n additions, but r*m*z of them run side by side (the
// serial form was one thread's work per block and successor).
__global__ void __launch_bounds__(kThreads) distinct_rows_kernel(ExpModel md, Distinct d) {
    const unsigned mz = md.m * md.z;
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (size_t)d.chunk * mz) return;
    const unsigned i = (unsigned)(t / mz), ao = (unsigned)(t % mz), a = ao / md.z, o = ao % md.z;
    const float *po = md.PO + (size_t)a * md.n * md.z + o;
    float pr = 0.0f;
    if (d.odd[0] == 0u) {
        // Zeros of the belief add fl(PO * 0) = 0 to the sum of finite products.
        const unsigned j = d.first + i, L = d.nnz[j];
        const uint2 *list = d.list + (size_t)j * d.cap;
        for (unsigned k = 0; k < L; k++) {
            const uint2 e = list[k];
            pr = fadd(pr, fmul(po[(size_t)e.x * md.z], __uint_as_float(e.y)));
        }
    } else {
        for (unsigned s = 0; s < md.n; s++) pr = fadd(pr, fmul(po[(size_t)s * md.z], md.BT[(size_t)s * md.r + d.first + i]));
    }
    float mass = -1.0f;
    if (!(pr == 0.0f)) {
        const float *W = d.W + ((size_t)i * md.m + a) * md.n;
        const float *Oa = md.O + (size_t)a * md.n * md.z + o;
        float norm = 0.0f;
#pragma unroll 8
        for (unsigned s = 0; s < md.n; s++) norm = fadd(norm, fmul(W[s], Oa[(size_t)s * md.z]));
        if (!(fabs((double)fabsf(norm)) < NOVA_FLT_ERR_TOL)) {
            float *out = d.bp + (size_t)i * md.n * mz + ao;
            mass = 0.0f;
            bool odd = false;
#pragma unroll 4
            for (unsigned s = 0; s < md.n; s++) {
                const float v = __fdiv_rn(fmul(W[s], Oa[(size_t)s * md.z]), norm);
                out[(size_t)s * mz] = v;
                odd |= !(v >= 0.0f && v <= NOVA_FLT_MAX);
                mass += fabsf(v);
            }
            if (odd) atomicOr(d.odd, 1u);
        }
    }
    d.mass[t] = mass;
}

// The same with a warp per row, for rows too few to fill the device with
// threads whose chains take n steps each: n = 500, 9,600 rows 175 and 53 us, n =
// 4,000, 6,400 rows 1,540 and 255, n = 2,000, 38,400 rows 752 and 701, n = 1,000,
// 64,000 rows 395 and 825.
constexpr size_t kFewRows = 32768;

__global__ void __launch_bounds__(kThreads) distinct_few_rows_kernel(ExpModel md, Distinct d) {
    __shared__ __align__(16) float terms[kThreads / 32][128];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, mz = md.m * md.z;
    const size_t t = (size_t)blockIdx.x * (kThreads / 32) + warp;
    if (t >= (size_t)d.chunk * mz) return;
    const unsigned i = (unsigned)(t / mz), ao = (unsigned)(t % mz), a = ao / md.z, o = ao % md.z;
    const float *po = md.PO + (size_t)a * md.n * md.z + o;
    float pr;
    if (d.odd[0] == 0u) {
        const unsigned j = d.first + i;
        const uint2 *list = d.list + (size_t)j * d.cap;
        pr = warp_ordered_sum(d.nnz[j], terms[warp], lane, [&](unsigned k) {
            const uint2 e = list[k];
            return fmul(po[(size_t)e.x * md.z], __uint_as_float(e.y));
        });
    } else {
        pr = warp_ordered_sum(md.n, terms[warp], lane, [&](unsigned s) {
            return fmul(po[(size_t)s * md.z], md.BT[(size_t)s * md.r + d.first + i]);
        });
    }
    float mass = -1.0f;
    if (!(pr == 0.0f)) {
        const float *W = d.W + ((size_t)i * md.m + a) * md.n;
        const float *Oa = md.O + (size_t)a * md.n * md.z + o;
        const float norm = warp_ordered_sum(md.n, terms[warp], lane,
                                            [&](unsigned s) { return fmul(__ldg(W + s), __ldg(Oa + (size_t)s * md.z)); });
        if (!(fabs((double)fabsf(norm)) < NOVA_FLT_ERR_TOL)) {
            float *out = d.bp + (size_t)i * md.n * mz + ao;
            mass = 0.0f;
            bool odd = false;
#pragma unroll 4
            for (unsigned s = lane; s < md.n; s += 32) {
                const float v = __fdiv_rn(fmul(__ldg(W + s), __ldg(Oa + (size_t)s * md.z)), norm);
                out[(size_t)s * mz] = v;
                odd |= !(v >= 0.0f && v <= NOVA_FLT_MAX);
                mass += fabsf(v);
            }
            for (int off = 16; off > 0; off >>= 1) mass += __shfl_xor_sync(0xffffffffu, mass, off);
            if (__any_sync(0xffffffffu, odd) && lane == 0) atomicOr(d.odd, 1u);
        }
    }
    if (lane == 0) d.mass[t] = mass;
}

// Half-width of the interval around an approximate distance in which the
// reference's FP32 sum lies. With both beliefs non-negative,
//     sum_s |b_j - b'| = mass - total_j + 2 sum_{s in supp j} max(b_j - b', 0).
// The reference's n-term sum rounds by at most (n + 1) u (mass + total), u =
// 2^-24; mass by n u mass, total by (n / 32 + 6) u total, the sum of the
// maxima by (nnz + 2) u total, twice, and the last three operations by 3 u
// (mass + 2 total): at most (2 n + 4) u mass + (3.1 n + 20) u total together.
__device__ __forceinline__ float distance_error(const ExpModel &md, const Distinct &d, float mass) {
    if (d.odd[0] != 0u) return INFINITY;
    return 2.0f * (float)(2 * md.n + 16) * 5.97e-8f * (mass + 2.0f * __uint_as_float(d.odd[1]));
}

// bound[i][ao] = min_j of the approximate distance. A block keeps ROWS
// successors of one belief in shared memory ([state][ROWS], kShared) and its
// warps walk the beliefs' nonzeros, lane = successor: one conflict-free read,
// a subtraction, a maximum and an addition per nonzero and successor, 16 times
// fewer terms than the sums over all states at n = 512 (32 nonzeros). Bound by
// issue: r = 1,024, m z = 128 takes 1.4 ms, the whole expansion 2.0 ms on the
// device; one block per belief forming every sum in full took 33 ms.
template <int ROWS, bool kShared>
__global__ void __launch_bounds__(1024) distinct_bound_kernel(ExpModel md, Distinct d) {
    constexpr int PER = ROWS / 32;
    extern __shared__ __align__(16) float tile[];   // [n][ROWS]; then [warps][ROWS]
    const unsigned mz = md.m * md.z, tiles = (mz + ROWS - 1) / ROWS;
    const unsigned i = blockIdx.x / tiles, r0 = (blockIdx.x % tiles) * ROWS;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const float *src = d.bp + (size_t)i * md.n * mz + r0;
    const unsigned live = min((unsigned)ROWS, mz - r0);
    float *best = tile;
    if constexpr (kShared) {
        best = tile + (size_t)md.n * ROWS;
        for (unsigned e = threadIdx.x; e < md.n * ROWS; e += blockDim.x) {
            const unsigned s = e / ROWS, q = e % ROWS;
            tile[e] = q < live ? src[(size_t)s * mz + q] : 0.0f;
        }
        __syncthreads();
    }
    float low[PER];
    unsigned at[PER];
#pragma unroll
    for (int q = 0; q < PER; q++) {
        low[q] = INFINITY;
        at[q] = min(lane + 32u * q, live - 1);
    }
    for (unsigned j = warp; j < md.r; j += warps) {
        const uint2 *list = d.list + (size_t)j * d.cap;
        const unsigned L = d.nnz[j];
        float acc[PER];
#pragma unroll
        for (int q = 0; q < PER; q++) acc[q] = 0.0f;
#pragma unroll 8
        for (unsigned k = 0; k < L; k++) {
            const uint2 e = __ldg(list + k);
            const float b = __uint_as_float(e.y);
#pragma unroll
            for (int q = 0; q < PER; q++) {
                const float p = kShared ? tile[e.x * ROWS + lane + 32u * q] : __ldg(src + (size_t)e.x * mz + at[q]);
                acc[q] += fmaxf(b - p, 0.0f);
            }
        }
        const float t = d.total[j];
#pragma unroll
        for (int q = 0; q < PER; q++) low[q] = fminf(low[q], 2.0f * acc[q] - t);
    }
#pragma unroll
    for (int q = 0; q < PER; q++) best[warp * ROWS + lane + 32 * q] = low[q];
    __syncthreads();
    for (unsigned q = threadIdx.x; q < live; q += blockDim.x) {
        float v = INFINITY;
        for (unsigned w = 0; w < warps; w++) v = fminf(v, best[w * ROWS + q]);
        const float mass = d.mass[(size_t)i * mz + r0 + q];
        d.bound[(size_t)i * mz + r0 + q] = v + mass;
    }
}

// Per belief: the successors whose bound lies within the error of the largest,
// in (a, o) order; for each, the reference's sums to the beliefs within the
// error of its smallest. The first successor with the strictly largest smallest
// distance becomes the new belief. With many states the error is wide and
// distances that are exactly equal (disjoint supports) are common: n = 12,000,
// r = 50 took 37 ms with every sum over all states, 0.23 so.
// Below kWalkStates the successor's list costs more than it saves (n = 512: 15 to
// 35 of 240 us; n = 1,000: 124 us without, 87 with).
constexpr unsigned kWalkStates = 768;

__global__ void __launch_bounds__(kThreads) distinct_select_kernel(ExpModel md, Distinct d, float *__restrict__ Bnew) {
    extern __shared__ __align__(16) float smem[];
    __shared__ float red[kThreads / 32];
    __shared__ __align__(16) float terms[kThreads / 32][128];
    __shared__ unsigned found[kThreads / 32];
    const unsigned mz = md.m * md.z, i = blockIdx.x;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float *row = smem, *star = smem + md.n;
    unsigned *states = reinterpret_cast<unsigned *>(star + md.n);   // the successor's nonzero states, in order
    const float *bound = d.bound + (size_t)i * mz, *mass = d.mass + (size_t)i * mz;
    float top = -INFINITY, heaviest = 0.0f;
    for (unsigned ao = threadIdx.x; ao < mz; ao += blockDim.x) {
        if (mass[ao] < 0.0f) continue;
        top = fmaxf(top, bound[ao]);
        heaviest = fmaxf(heaviest, mass[ao]);
    }
    auto block_max = [&](float v) {
        for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
        __syncthreads();
        if (lane == 0) red[warp] = v;
        __syncthreads();
        for (unsigned w = 0; w < kThreads / 32; w++) v = fmaxf(v, red[w]);
        return v;
    };
    top = block_max(top);
    heaviest = block_max(heaviest);
    const float err = distance_error(md, d, heaviest);
    for (unsigned s = threadIdx.x; s < md.n; s += blockDim.x) star[s] = 0.0f;
    float starValue = NOVA_FLT_MIN;
    for (unsigned ao = 0; ao < mz; ao++) {
        // A NaN mass is a successor too (err is infinite then).
        if (mass[ao] < 0.0f || bound[ao] < top - 2.0f * err) continue;
        __syncthreads();
        for (unsigned s = threadIdx.x; s < md.n; s += blockDim.x) row[s] = d.bp[((size_t)i * md.n + s) * mz + ao];
        __syncthreads();
        const bool walks = md.n >= kWalkStates;
        unsigned support = 0;
        for (unsigned s0 = 0; walks && s0 < md.n; s0 += kThreads) {
            const unsigned s = s0 + threadIdx.x;
            const bool some = s < md.n && !(row[s] == 0.0f);
            const unsigned bits = __ballot_sync(0xffffffffu, some);
            if (lane == 0) found[warp] = __popc(bits);
            __syncthreads();
            unsigned place = support;
            for (unsigned w = 0; w < kThreads / 32; w++) {
                if (w < warp) place += found[w];
                support += found[w];
            }
            if (some) states[place + __popc(bits & ((1u << lane) - 1u))] = s;
            __syncthreads();
        }
        const float cut = bound[ao] + 2.0f * err;
        float low = NOVA_FLT_MAX;
        for (unsigned j0 = warp * 32; j0 < md.r; j0 += kThreads) {
            const unsigned j = j0 + lane;
            bool near = j < md.r;
            if (near) {
                const uint2 *list = d.list + (size_t)j * d.cap;
                const unsigned L = d.nnz[j];
                float acc = 0.0f;
                for (unsigned k = 0; k < L; k++) {
                    const uint2 e = list[k];
                    acc += fmaxf(__uint_as_float(e.y) - row[e.x], 0.0f);
                }
                near = !(mass[ao] + (2.0f * acc - d.total[j]) > cut);
            }
            // Zeros of both add nothing to the sum, so a lane can walk the
            // nonzeros of its belief and of the successor side by side (about
            // 100 cycles each, 32 beliefs at once), or the warp one belief after
            // the other over all states (700 cycles per 128).
            const unsigned msk = __ballot_sync(0xffffffffu, near);
            const unsigned mine = near ? d.nnz[j] : 0u;
            const unsigned steps = support + __reduce_max_sync(0xffffffffu, mine);
            if (walks && __popc(msk) * ((md.n + 127u) / 128u) * 7u > steps) {
                if (near) {
                    const uint2 *list = d.list + (size_t)j * d.cap;
                    uint2 e = mine != 0 ? list[0] : make_uint2(kNoIndex, 0u);
                    unsigned at = support != 0 ? states[0] : kNoIndex;
                    float dist = 0.0f;
                    for (unsigned k = 0, q = 0; k < mine || q < support;) {
                        const unsigned s = min(e.x, at);
                        const float b = e.x == s ? __uint_as_float(e.y) : 0.0f;
                        dist = fadd(dist, fabsf(__fsub_rn(b, row[s])));
                        if (at == s) at = ++q < support ? states[q] : kNoIndex;
                        if (e.x == s) e = ++k < mine ? list[k] : make_uint2(kNoIndex, 0u);
                    }
                    if (dist < low) low = dist;
                }
            } else {
                for (unsigned left = msk; left != 0; left &= left - 1) {
                    const unsigned jj = j0 + __ffs(left) - 1;
                    const float dist = warp_ordered_sum(md.n, terms[warp], lane, [&](unsigned s) {
                        return fabsf(__fsub_rn(__ldg(md.BT + (size_t)s * md.r + jj), row[s]));
                    });
                    if (dist < low) low = dist;
                }
            }
        }
        for (int off = 16; off > 0; off >>= 1) low = fminf(low, __shfl_xor_sync(0xffffffffu, low, off));
        __syncthreads();
        if (lane == 0) red[warp] = low;
        __syncthreads();
        float jStar = NOVA_FLT_MAX;
        for (unsigned w = 0; w < kThreads / 32; w++)
            if (red[w] < jStar) jStar = red[w];
        if (jStar > starValue) {
            starValue = jStar;
            for (unsigned s = threadIdx.x; s < md.n; s += blockDim.x) star[s] = row[s];
        }
    }
    __syncthreads();
    for (unsigned s = threadIdx.x; s < md.n; s += blockDim.x) Bnew[(size_t)(d.first + i) * md.n + s] = star[s];
}

// One step of a random trajectory, laid out by the host.
struct Step {
    unsigned traj;      // trajectory
    unsigned a;         // action drawn
    float target;       // observation draw in [0, 1]
    unsigned out;       // row of Bnew written after the step
};

// Trajectory k starts from belief start[k] and runs steps [first[k], first[k+1]).
// checkPositive: the CPU form also requires Pr(o) > 0 for the chosen o.
__global__ void __launch_bounds__(kThreads) random_kernel(ExpModel md, const unsigned *__restrict__ start,
                                                          const unsigned *__restrict__ first,
                                                          const Step *__restrict__ steps, int checkPositive,
                                                          float *__restrict__ probs, float *__restrict__ Bnew) {
    extern __shared__ __align__(16) float smem[];
    __shared__ float slot;
    __shared__ unsigned chosen;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    BlockBufs w = carve(smem, md.n);
    float *terms = smem + (2 * md.n + 3) / 4 * 4 + warp * 128;   // where aux and tmp are not needed
    const unsigned k = blockIdx.x;
    volatile float *pr = probs + (size_t)k * md.z;
    load_belief(md, start[k], w.b);
    for (unsigned q = first[k]; q < first[k + 1]; q++) {
        const Step st = steps[q];
        // Every observation's probability is a chain of n additions, side by
        // side: a warp each, or with more observations than eight rounds of
        // the block's warps a thread each.
        if (md.z <= kThreads / 4) {
            for (unsigned o = warp; o < md.z; o += kThreads / 32) {
                const float *po = md.PO + (size_t)st.a * md.n * md.z + o;
                const float p = warp_ordered_sum(md.n, terms, lane,
                                                 [&](unsigned s) { return fmul(__ldg(po + (size_t)s * md.z), w.b[s]); });
                if (lane == 0) pr[o] = p;
            }
        } else {
            for (unsigned o = threadIdx.x; o < md.z; o += blockDim.x) pr[o] = prob_obs_dense(md, w.b, st.a, o);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            float cur = 0.0f;
            unsigned c = 0;
            for (unsigned op = 0; op < md.z; op++) {
                cur = fadd(cur, pr[op]);
                if (cur >= st.target && (!checkPositive || pr[op] > 0.0f)) { c = op; break; }
            }
            chosen = c;
        }
        __syncthreads();
        belief_update(md, w.b, w.bp, st.a, chosen, &slot);
        __syncthreads();
        for (unsigned s = threadIdx.x; s < md.n; s += blockDim.x) {
            w.b[s] = w.bp[s];
            Bnew[(size_t)st.out * md.n + s] = w.bp[s];
        }
        __syncthreads();
    }
}

// pomdp_expand_pema_cpu (pomdp_expand_cpu.cpp:244-383), per belief i: the
// best action's error bound and its (action, observation).
__global__ void __launch_bounds__(kThreads) pema_kernel(ExpModel md, unsigned pr, const float *__restrict__ Gamma,
                                                        float *__restrict__ aStarValueOut,
                                                        unsigned *__restrict__ aStarOut,
                                                        unsigned *__restrict__ oStarOut) {
    extern __shared__ __align__(16) float smem[];
    __shared__ float slot, sv[kThreads];
    __shared__ unsigned si[kThreads];
    __shared__ unsigned alphaStar, closest;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    BlockBufs w = carve(smem, md.n);
    const unsigned i = blockIdx.x;
    load_belief(md, i, w.b);
    // Rmax / (1 - gamma) and Rmin / (1 - gamma) from the reward range.
    if (threadIdx.x == 0) {
        float Rmax = NOVA_FLT_MIN, Rmin = NOVA_FLT_MAX;
        for (unsigned s = 0; s < md.n; s++)
            for (unsigned a = 0; a < md.m; a++) {
                const float v = md.R[(size_t)s * md.m + a];
                if (Rmax < v) Rmax = v;
                if (Rmin > v) Rmin = v;
            }
        sv[0] = __fdiv_rn(Rmax, __fsub_rn(1.0f, md.gamma));
        sv[1] = __fdiv_rn(Rmin, __fsub_rn(1.0f, md.gamma));
    }
    __syncthreads();
    const float hi = sv[0], lo = sv[1];
    __syncthreads();
    unsigned aStar = 0;
    float aStarValue = NOVA_FLT_MIN;
    unsigned oStarBest = 0;
    for (unsigned a = 0; a < md.m; a++) {
        float aValue = 0.0f;
        unsigned oStar = 0;
        float oStarValue = NOVA_FLT_MIN;
        for (unsigned o = 0; o < md.z; o++) {
            // Pr(o | b, a) over the belief's support, in (support, successor) order.
            if (threadIdx.x == 0) {
                float p = 0.0f;
                for (unsigned j = 0; j < md.rz; j++) {
                    const int s = md.Z[(size_t)i * md.rz + j];
                    if (s < 0) break;
                    const size_t row = ((size_t)s * md.m + a) * md.ns;
                    for (unsigned q = 0; q < md.ns; q++) {
                        const int sp = md.S[row + q];
                        if (sp < 0) break;
                        p = fadd(p, fmul(fmul(md.T[row + q], md.O[((size_t)a * md.n + sp) * md.z + o]),
                                         md.B[(size_t)i * md.rz + j]));
                    }
                }
                slot = p;
            }
            __syncthreads();
            const float p = slot;
            __syncthreads();
            if (!belief_update(md, w.b, w.bp, a, o, &slot)) continue;
            min_distance(md, w.bp, &closest, sv, si);
            float *bc = w.aux;
            for (unsigned s = threadIdx.x; s < md.n; s += blockDim.x) bc[s] = md.BT[(size_t)s * md.r + closest];
            // The reference's alpha search keeps the last j with some
            // Gamma_j(s) * bc(s) below -1e10 (its running value never moves).
            if (threadIdx.x == 0) alphaStar = 0;
            __syncthreads();
            for (unsigned j = warp; j < pr; j += kThreads / 32) {
                bool hit = false;
                for (unsigned s0 = 0; s0 < md.n && !hit; s0 += 128) {
                    bool below = false;
#pragma unroll
                    for (unsigned q = 0; q < 4; q++) {
                        const unsigned s = s0 + 32 * q + lane;
                        if (s < md.n) below |= fmul(__ldg(Gamma + (size_t)j * md.n + s), bc[s]) < NOVA_FLT_MIN;
                    }
                    hit = __any_sync(0xffffffffu, below);
                }
                if (hit && lane == 0) atomicMax(&alphaStar, j);
            }
            __syncthreads();
            const float *g = Gamma + (size_t)alphaStar * md.n;
            for (unsigned s = threadIdx.x; s < md.n; s += blockDim.x) {
                const float c = __fsub_rn(w.bp[s] >= w.b[s] ? hi : lo, g[s]);
                w.tmp[s] = fmul(c, __fsub_rn(w.bp[s], bc[s]));
            }
            const float eps = seq_sum(w.tmp, md.n, &slot);
            const float v = fmul(p, eps);
            if (v > oStarValue) { oStar = o; oStarValue = v; }
            aValue = fadd(aValue, v);
        }
        if (aValue > aStarValue) { aStar = a; aStarValue = aValue; oStarBest = oStar; }
    }
    if (threadIdx.x == 0) {
        aStarValueOut[i] = aStarValue;
        aStarOut[i] = aStar;
        oStarOut[i] = oStarBest;
    }
}

// b'(b_i, a, o), or b_i itself when the update is invalid (PEMA's final step).
__global__ void __launch_bounds__(kThreads) update_one_kernel(ExpModel md, unsigned i, unsigned a, unsigned o,
                                                              float *__restrict__ out) {
    extern __shared__ __align__(16) float smem[];
    __shared__ float slot;
    BlockBufs w = carve(smem, md.n);
    load_belief(md, i, w.b);
    const bool ok = belief_update(md, w.b, w.bp, a, o, &slot);
    for (unsigned s = threadIdx.x; s < md.n; s += blockDim.x) out[s] = ok ? w.bp[s] : w.b[s];
}

__global__ void dense_beliefs_kernel(unsigned n, unsigned r, unsigned rz, const int *__restrict__ Z,
                                     const float *__restrict__ B, float *__restrict__ BT) {
    const unsigned i = blockIdx.x;
    for (unsigned s = threadIdx.x; s < n; s += blockDim.x) BT[(size_t)s * r + i] = 0.0f;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (unsigned j = 0; j < rz; j++) {
            const int s = Z[(size_t)i * rz + j];
            if (s < 0) break;
            BT[(size_t)s * r + i] = B[(size_t)i * rz + j];
        }
    }
}

// Device copies of a host-array POMDP plus the predecessor lists and the
// dense beliefs, freed on destruction.
struct ExpWorkspace {
    Arena arena;
    ExpModel md{};
    int *S = nullptr, *Z = nullptr;
    float *T = nullptr, *O = nullptr, *R = nullptr, *B = nullptr, *BT = nullptr, *PO = nullptr, *predT = nullptr;
    unsigned *predStart = nullptr, *predState = nullptr;
    size_t smem = 0;
};

int build_workspace(const POMDP *p, ExpWorkspace &ws, const char *fn) {
    const unsigned n = p->n, ns = p->ns, m = p->m, z = p->z, r = p->r, rz = p->rz;
    const size_t nms = (size_t)n * m * ns;
    int rc;
    // Predecessors of each (a, s'), in (s, i) order: action a's lists are
    // start[a*(n+1) + s'] .. start[a*(n+1) + s' + 1] of one global array.
    std::vector<unsigned> count((size_t)m * n, 0u), start((size_t)m * (n + 1), 0u),
        state(std::max<size_t>(nms, 1));
    std::vector<float> prob(std::max<size_t>(nms, 1));
    for (unsigned s = 0; s < n; s++)
        for (unsigned a = 0; a < m; a++)
            for (unsigned i = 0; i < ns; i++) {
                const int sp = p->S[((size_t)s * m + a) * ns + i];
                if (sp < 0) break;
                if ((unsigned)sp >= n) {
                    NOVA_ERR(fn, "Invalid arguments: a successor state is out of range.");
                    return NOVA_ERROR_INVALID_DATA;
                }
                count[(size_t)a * n + sp]++;
            }
    unsigned running = 0;
    for (unsigned a = 0; a < m; a++) {
        for (unsigned sp = 0; sp < n; sp++) {
            start[(size_t)a * (n + 1) + sp] = running;
            running += count[(size_t)a * n + sp];
        }
        start[(size_t)a * (n + 1) + n] = running;
    }
    std::vector<unsigned> cursor(start);
    for (unsigned s = 0; s < n; s++)
        for (unsigned a = 0; a < m; a++)
            for (unsigned i = 0; i < ns; i++) {
                const int sp = p->S[((size_t)s * m + a) * ns + i];
                if (sp < 0) break;
                const unsigned k = cursor[(size_t)a * (n + 1) + sp]++;
                state[k] = s;
                prob[k] = p->T[((size_t)s * m + a) * ns + i];
            }
    ws.arena.add(&ws.S, nms);
    ws.arena.add(&ws.T, nms);
    ws.arena.add(&ws.O, (size_t)m * n * z);
    ws.arena.add(&ws.R, (size_t)n * m);
    ws.arena.add(&ws.Z, (size_t)r * rz);
    ws.arena.add(&ws.B, (size_t)r * rz);
    ws.arena.add(&ws.BT, (size_t)n * r);
    ws.arena.add(&ws.predStart, start.size());
    ws.arena.add(&ws.predState, std::max<size_t>(nms, 1));
    ws.arena.add(&ws.predT, std::max<size_t>(nms, 1));
    ws.arena.add(&ws.PO, (size_t)m * n * z);
    if ((rc = ws.arena.commit(fn, "the model and the beliefs")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws.S, p->S, nms * sizeof(int), fn, "the successor states")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws.T, p->T, nms * sizeof(float), fn, "the state transitions")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws.O, p->O, (size_t)m * n * z * sizeof(float), fn, "the observation transitions")) != NOVA_SUCCESS)
        return rc;
    if ((rc = h2d(ws.R, p->R, (size_t)n * m * sizeof(float), fn, "the rewards")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws.Z, p->Z, (size_t)r * rz * sizeof(int), fn, "the belief states")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws.B, p->B, (size_t)r * rz * sizeof(float), fn, "the belief values")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws.predStart, start.data(), start.size() * sizeof(unsigned), fn, "the predecessor offsets")) !=
            NOVA_SUCCESS)
        return rc;
    if ((rc = h2d(ws.predState, state.data(), nms * sizeof(unsigned), fn, "the predecessors")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws.predT, prob.data(), nms * sizeof(float), fn, "the predecessors")) != NOVA_SUCCESS) return rc;
    prob_table_kernel<<<std::min<size_t>(ceil_div((size_t)m * n * z, 256), 65535u * 8u), 256>>>(n, ns, m, z, ws.S, ws.T,
                                                                                               ws.O, ws.PO);
    if ((rc = check_launch(fn, "observation probabilities")) != NOVA_SUCCESS) return rc;
    dense_beliefs_kernel<<<r, 256>>>(n, r, rz, ws.Z, ws.B, ws.BT);
    if ((rc = check_launch(fn, "dense beliefs")) != NOVA_SUCCESS) return rc;
    ws.md = ExpModel{n, ns, m, z, r, rz, p->gamma, ws.S, ws.T, ws.O, ws.R, ws.Z, ws.B, ws.predStart, ws.predState,
                     ws.predT, ws.BT, ws.PO};
    ws.smem = 4 * (size_t)n * sizeof(float);
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
            ws.smem + 4096 > (size_t)optin) {
        cudaGetLastError();
        NOVA_ERR(fn, "Too many states for the expansion's shared-memory buffers.");
        return NOVA_ERROR_INVALID_DATA;
    }
    allow_dynamic_smem(distinct_mass_kernel, ws.smem);
    allow_dynamic_smem(distinct_select_kernel, 3 * (size_t)n * sizeof(float));
    allow_dynamic_smem(random_kernel, ws.smem);
    allow_dynamic_smem(pema_kernel, ws.smem);
    allow_dynamic_smem(update_one_kernel, ws.smem);
    return NOVA_SUCCESS;
}

bool valid_model(const POMDP *p) {
    return p != nullptr && p->n != 0 && p->ns != 0 && p->m != 0 && p->z != 0 && p->r != 0 && p->rz != 0 &&
           p->S != nullptr && p->T != nullptr && p->O != nullptr && p->R != nullptr && p->Z != nullptr &&
           p->B != nullptr;
}

// Lay out the random trajectories from the rand() stream and run them.
// fromB0: the _gpu form (every trajectory starts at belief 0, Bnew[0] is
// belief 0, no Pr(o) > 0 requirement). Returns Bnew [total][n] on the host.
int run_random(const POMDP *p, unsigned total, bool fromB0, std::vector<float> &Bnew, const char *fn) {
    ExpWorkspace ws;
    int rc = build_workspace(p, ws, fn);
    if (rc != NOVA_SUCCESS) return rc;
    seed_rand();
    std::vector<unsigned> start, first;
    std::vector<Step> steps;
    unsigned i = fromB0 ? 1u : 0u;
    while (i < total) {
        // A draw equal to RAND_MAX gives r (or m below); the reference would
        // read past its arrays there, this clamps to the last index.
        const unsigned b0 = fromB0 ? 0u : std::min(draw((float)p->r), p->r - 1);
        const unsigned h = draw((float)(p->horizon + 1));
        start.push_back(b0);
        first.push_back((unsigned)steps.size());
        for (unsigned t = 0; t < h; t++) {
            const unsigned a = draw((float)p->m);
            const float target = (float)rand() / (float)RAND_MAX;
            steps.push_back(Step{(unsigned)start.size() - 1, std::min(a, p->m - 1), target, i});
            i++;
            if (i >= total) break;
        }
    }
    first.push_back((unsigned)steps.size());
    // Trajectories without steps write nothing; drop them.
    std::vector<unsigned> s2, f2;
    for (size_t k = 0; k + 1 < first.size(); k++)
        if (first[k + 1] > first[k]) { s2.push_back(start[k]); f2.push_back(first[k]); }
    f2.push_back((unsigned)steps.size());
    float *dB = nullptr, *dProbs = nullptr;
    unsigned *dStart = nullptr, *dFirst = nullptr;
    Step *dSteps = nullptr;
    const size_t n = p->n;
    struct Free {
        float *&b, *&q; unsigned *&s, *&f; Step *&st;
        ~Free() { cudaFree(b); cudaFree(q); cudaFree(s); cudaFree(f); cudaFree(st); }
    } guard{dB, dProbs, dStart, dFirst, dSteps};
    if ((rc = dev_alloc(&dB, (size_t)total * n, fn, "the new beliefs")) != NOVA_SUCCESS) return rc;
    if (cudaMemset(dB, 0, (size_t)total * n * sizeof(float)) != cudaSuccess) {
        cudaGetLastError();
        NOVA_ERR(fn, "Failed to clear the new beliefs.");
        return NOVA_ERROR_KERNEL_EXECUTION;
    }
    if (!s2.empty()) {
        if ((rc = dev_alloc(&dStart, s2.size(), fn, "the trajectory starts")) != NOVA_SUCCESS) return rc;
        if ((rc = dev_alloc(&dFirst, f2.size(), fn, "the trajectory offsets")) != NOVA_SUCCESS) return rc;
        if ((rc = dev_alloc(&dSteps, steps.size(), fn, "the trajectory steps")) != NOVA_SUCCESS) return rc;
        if ((rc = h2d(dStart, s2.data(), s2.size() * sizeof(unsigned), fn, "the trajectory starts")) != NOVA_SUCCESS)
            return rc;
        if ((rc = h2d(dFirst, f2.data(), f2.size() * sizeof(unsigned), fn, "the trajectory offsets")) != NOVA_SUCCESS)
            return rc;
        if ((rc = h2d(dSteps, steps.data(), steps.size() * sizeof(Step), fn, "the trajectory steps")) != NOVA_SUCCESS)
            return rc;
        if ((rc = dev_alloc(&dProbs, s2.size() * p->z, fn, "the observation draws")) != NOVA_SUCCESS) return rc;
        const size_t smem = std::max(ws.smem, (round_up(2 * n, 4) + kThreads / 32 * 128) * sizeof(float));
        random_kernel<<<(unsigned)s2.size(), kThreads, smem>>>(ws.md, dStart, dFirst, dSteps, fromB0 ? 0 : 1, dProbs,
                                                                  dB);
        if ((rc = check_launch(fn, "random trajectories")) != NOVA_SUCCESS) return rc;
    }
    if (fromB0) {
        // Bnew[0] = belief 0.
        std::vector<float> b0(n, 0.0f);
        for (unsigned j = 0; j < p->rz; j++) {
            const int s = p->Z[j];
            if (s < 0) break;
            b0[s] = p->B[j];
        }
        if ((rc = h2d(dB, b0.data(), n * sizeof(float), fn, "the initial belief")) != NOVA_SUCCESS) return rc;
    }
    Bnew.assign((size_t)total * n, 0.0f);
    return d2h(Bnew.data(), dB, (size_t)total * n * sizeof(float), fn, "the new beliefs");
}

// The successor farthest from the belief set for every belief, into Bnew [r][n].
int run_distinct(const ExpWorkspace &ws, std::vector<float> &Bnew, const char *fn) {
    const ExpModel &md = ws.md;
    const size_t n = md.n, mz = (size_t)md.m * md.z, rn = md.r * n;
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
        cudaGetLastError();
        optin = 48 * 1024;
    }
    Distinct d{};
    d.cap = std::min(md.n, md.rz);
    // Beliefs whose successors are held at once: about 512 MB of them, fewer
    // where these cannot be had.
    const size_t perBelief = (n * mz + md.m * n + 2 * mz) * sizeof(float);
    d.chunk = (unsigned)std::min<size_t>(md.r, std::max<size_t>(1, (512ull << 20) / perBelief));
    float *dB = nullptr;
    Arena arena;
    int rc;
    auto allocate = [&]() {
        arena.add(&dB, rn);
        arena.add(&d.W, (size_t)d.chunk * md.m * n);
        arena.add(&d.bp, (size_t)d.chunk * n * mz);
        arena.add(&d.mass, (size_t)d.chunk * mz);
        arena.add(&d.bound, (size_t)d.chunk * mz);
        arena.add(&d.list, (size_t)md.r * d.cap);
        arena.add(&d.nnz, md.r);
        arena.add(&d.total, md.r);
        arena.add(&d.odd, 2);
        return arena.try_commit();
    };
    while (!allocate()) {
        if (d.chunk == 1) return malloc_failed(fn, "the successor beliefs");
        d.chunk = (d.chunk + 1) / 2;
    }
    if (cudaMemsetAsync(d.odd, 0, 2 * sizeof(unsigned)) != cudaSuccess) {
        cudaGetLastError();
        NOVA_ERR(fn, "Failed to clear the belief check.");
        return NOVA_ERROR_KERNEL_EXECUTION;
    }
    distinct_check_kernel<<<std::min<size_t>(ceil_div(mz * n, 256), 65535u), 256>>>(md, d.odd);
    if ((rc = check_launch(fn, "observation probabilities")) != NOVA_SUCCESS) return rc;
    distinct_list_kernel<<<ceil_div(md.r, kThreads / 32), kThreads>>>(md, d);
    if ((rc = check_launch(fn, "belief nonzeros")) != NOVA_SUCCESS) return rc;
    // Successors per block of the bound kernel: 64 where they fit in shared
    // memory (each nonzero is read once for all of them), else 32, else 32
    // read through the cache.
    const size_t tile64 = (n + 32) * 64 * sizeof(float), tile32 = (n + 32) * 32 * sizeof(float);
    const bool wide = mz > 32 && tile64 <= (size_t)optin, shared = wide || tile32 <= (size_t)optin;
    const unsigned rows = wide ? 64u : 32u;
    const size_t boundSmem = wide ? tile64 : shared ? tile32 : 32 * 32 * sizeof(float);
    auto bound = wide ? distinct_bound_kernel<64, true> : shared ? distinct_bound_kernel<32, true>
                                                                 : distinct_bound_kernel<32, false>;
    if (!allow_dynamic_smem(bound, boundSmem)) {
        NOVA_ERR(fn, "Failed to configure the distance kernel.");
        return NOVA_ERROR_KERNEL_EXECUTION;
    }
    for (d.first = 0; d.first < md.r; d.first += d.chunk) {
        const unsigned count = std::min(d.chunk, md.r - d.first);
        Distinct part = d;
        part.chunk = count;
        distinct_mass_kernel<<<count * md.m, kThreads, n * sizeof(float)>>>(md, part);
        if ((rc = check_launch(fn, "successor masses")) != NOVA_SUCCESS) return rc;
        if ((size_t)count * mz <= kFewRows)
            distinct_few_rows_kernel<<<ceil_div((size_t)count * mz, kThreads / 32), kThreads>>>(md, part);
        else
            distinct_rows_kernel<<<ceil_div((size_t)count * mz, kThreads), kThreads>>>(md, part);
        if ((rc = check_launch(fn, "successor beliefs")) != NOVA_SUCCESS) return rc;
        bound<<<count * ceil_div(mz, rows), 1024, boundSmem>>>(md, part);
        if ((rc = check_launch(fn, "distance bounds")) != NOVA_SUCCESS) return rc;
        distinct_select_kernel<<<count, kThreads, 3 * n * sizeof(float)>>>(md, part, dB);
        if ((rc = check_launch(fn, "distinct beliefs")) != NOVA_SUCCESS) return rc;
    }
    Bnew.assign(rn, 0.0f);
    return d2h(Bnew.data(), dB, rn * sizeof(float), fn, "the new beliefs");
}

}  // namespace
}  // namespace nova_gb300

using namespace nova_gb300;

extern "C" int pomdp_expand_random_cpu(POMDP *pomdp, unsigned int numBeliefsToAdd) {
    static const char *fn = "pomdp_expand_random_cpu";
    if (!valid_model(pomdp) || pomdp->horizon < 1 || numBeliefsToAdd == 0) {
        NOVA_ERR(fn, "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    std::vector<float> Bnew;
    int rc = run_random(pomdp, numBeliefsToAdd, false, Bnew, fn);
    if (rc != NOVA_SUCCESS) return rc;
    return pomdp_add_new_raw_beliefs_cpu(pomdp, numBeliefsToAdd, Bnew.data());
}

extern "C" int pomdp_expand_random_gpu(const POMDP *pomdp, unsigned int numThreads,
                                       unsigned int numDesiredBeliefPoints, unsigned int &maxNonZeroValues,
                                       float *&Bnew) {
    static const char *fn = "pomdp_expand_random_gpu";
    if (!valid_model(pomdp) || pomdp->horizon < 1 || numDesiredBeliefPoints <= 1 || Bnew != nullptr) {
        NOVA_ERR(fn, "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    (void)numThreads;  // launch shapes are fixed by the kernels
    std::vector<float> B;
    int rc = run_random(pomdp, numDesiredBeliefPoints, true, B, fn);
    if (rc != NOVA_SUCCESS) return rc;
    const size_t n = pomdp->n;
    unsigned maxNZ = 0;
    for (unsigned i = 1; i < numDesiredBeliefPoints; i++) {
        unsigned nz = 0;
        for (size_t s = 0; s < n; s++) nz += B[(size_t)i * n + s] > 0.0f ? 1u : 0u;
        maxNZ = std::max(maxNZ, nz);
    }
    maxNonZeroValues = maxNZ;
    Bnew = new float[(size_t)numDesiredBeliefPoints * n];
    memcpy(Bnew, B.data(), (size_t)numDesiredBeliefPoints * n * sizeof(float));
    return NOVA_SUCCESS;
}

extern "C" int pomdp_expand_distinct_beliefs_cpu(POMDP *pomdp) {
    static const char *fn = "pomdp_expand_distinct_beliefs_cpu";
    if (!valid_model(pomdp)) {
        NOVA_ERR(fn, "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    std::vector<float> Bnew;
    {
        ExpWorkspace ws;
        int rc = build_workspace(pomdp, ws, fn);
        if (rc != NOVA_SUCCESS) return rc;
        if ((rc = run_distinct(ws, Bnew, fn)) != NOVA_SUCCESS) return rc;
    }
    return pomdp_add_new_raw_beliefs_cpu(pomdp, pomdp->r, Bnew.data());
}

extern "C" int pomdp_expand_pema_cpu(POMDP *pomdp, const POMDPAlphaVectors *policy) {
    static const char *fn = "pomdp_expand_pema_cpu";
    if (!valid_model(pomdp) || policy == nullptr || policy->Gamma == nullptr || policy->r == 0 ||
            policy->n != pomdp->n) {
        NOVA_ERR(fn, "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    const unsigned r = pomdp->r, n = pomdp->n;
    std::vector<float> Bnew(n, 0.0f);
    {
        ExpWorkspace ws;
        int rc = build_workspace(pomdp, ws, fn);
        if (rc != NOVA_SUCCESS) return rc;
        float *dGamma = nullptr, *dVal = nullptr, *dOut = nullptr;
        unsigned *dA = nullptr, *dO = nullptr;
        struct Free {
            float *&g, *&v, *&o; unsigned *&a, *&b;
            ~Free() { cudaFree(g); cudaFree(v); cudaFree(o); cudaFree(a); cudaFree(b); }
        } guard{dGamma, dVal, dOut, dA, dO};
        if ((rc = dev_alloc(&dGamma, (size_t)policy->r * n, fn, "the policy")) != NOVA_SUCCESS) return rc;
        if ((rc = dev_alloc(&dVal, r, fn, "the error bounds")) != NOVA_SUCCESS) return rc;
        if ((rc = dev_alloc(&dA, r, fn, "the best actions")) != NOVA_SUCCESS) return rc;
        if ((rc = dev_alloc(&dO, r, fn, "the best observations")) != NOVA_SUCCESS) return rc;
        if ((rc = dev_alloc(&dOut, n, fn, "the new belief")) != NOVA_SUCCESS) return rc;
        if ((rc = h2d(dGamma, policy->Gamma, (size_t)policy->r * n * sizeof(float), fn, "the policy")) !=
                NOVA_SUCCESS)
            return rc;
        pema_kernel<<<r, kThreads, ws.smem>>>(ws.md, policy->r, dGamma, dVal, dA, dO);
        if ((rc = check_launch(fn, "error bounds")) != NOVA_SUCCESS) return rc;
        std::vector<float> val(r);
        std::vector<unsigned> A(r), O(r);
        if ((rc = d2h(val.data(), dVal, r * sizeof(float), fn, "the error bounds")) != NOVA_SUCCESS) return rc;
        if ((rc = d2h(A.data(), dA, r * sizeof(unsigned), fn, "the best actions")) != NOVA_SUCCESS) return rc;
        if ((rc = d2h(O.data(), dO, r * sizeof(unsigned), fn, "the best observations")) != NOVA_SUCCESS) return rc;
        // The reference keeps the belief of the last strict increase of the
        // running maximum, i.e. the first belief attaining the maximum.
        float bStar = NOVA_FLT_MIN;
        unsigned win = kNoIndex;
        for (unsigned i = 0; i < r; i++)
            if (val[i] > bStar) { bStar = val[i]; win = i; }
        if (win != kNoIndex) {
            update_one_kernel<<<1, kThreads, ws.smem>>>(ws.md, win, A[win], O[win], dOut);
            if ((rc = check_launch(fn, "new belief")) != NOVA_SUCCESS) return rc;
            if ((rc = d2h(Bnew.data(), dOut, n * sizeof(float), fn, "the new belief")) != NOVA_SUCCESS) return rc;
        }
    }
    return pomdp_add_new_raw_beliefs_cpu(pomdp, 1, Bnew.data());
}

extern "C" int nova_gb300_expand_seed(unsigned int fixed, unsigned int seed) {
    g_seed.store(seed);
    g_seed_fixed.store(fixed ? 1u : 0u);
    return NOVA_SUCCESS;
}

// ---------------------------------------------------------------------------
// Sigma approximation (pomdp_sigma_cpu.cpp:49-118)
// ---------------------------------------------------------------------------

namespace nova_gb300 {
namespace {

// One thread per belief: sort its rz (value, state) entries by value,
// descending (equal values keep their support order), keep the top k,
// normalise them by their sum (added largest first) and report that sum.
__global__ void sigma_kernel(unsigned r, unsigned rz, unsigned k, const int *__restrict__ Z,
                             const float *__restrict__ B, int *__restrict__ Znew, float *__restrict__ Bnew,
                             float *__restrict__ sigmaB, float *__restrict__ scratchV, int *__restrict__ scratchS) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= r) return;
    float *v = scratchV + (size_t)i * rz;
    int *st = scratchS + (size_t)i * rz;
    for (unsigned q = 0; q < rz; q++) {
        // Insertion sort keeps equal values in support order.
        const float x = B[(size_t)i * rz + q];
        const int y = Z[(size_t)i * rz + q];
        unsigned p = q;
        while (p > 0 && v[p - 1] < x) { v[p] = v[p - 1]; st[p] = st[p - 1]; p--; }
        v[p] = x;
        st[p] = y;
    }
    float sb = 0.0f;
    for (unsigned q = 0; q < k && q < rz; q++) sb = fadd(sb, v[q]);
    sigmaB[i] = sb;
    for (unsigned q = 0; q < k; q++) {
        const bool keep = q < rz && v[q] > 0.0f;
        Bnew[(size_t)i * k + q] = keep ? __fdiv_rn(v[q], sb) : 0.0f;
        Znew[(size_t)i * k + q] = keep ? st[q] : -1;
    }
}

}  // namespace
}  // namespace nova_gb300

extern "C" int pomdp_sigma_cpu(POMDP *pomdp, unsigned int numDesiredNonZeroValues, float &sigma) {
    static const char *fn = "pomdp_sigma_cpu";
    if (pomdp == nullptr || pomdp->z == 0 || pomdp->r == 0 || pomdp->rz == 0 || pomdp->Z == nullptr ||
            pomdp->B == nullptr || numDesiredNonZeroValues == 0) {
        NOVA_ERR(fn, "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    const unsigned r = pomdp->r, rz = pomdp->rz, k = numDesiredNonZeroValues;
    int *dZ = nullptr, *dZn = nullptr, *dS = nullptr;
    float *dB = nullptr, *dBn = nullptr, *dSig = nullptr, *dV = nullptr;
    struct Free {
        int *&a, *&b, *&c; float *&d, *&e, *&f, *&g;
        ~Free() { cudaFree(a); cudaFree(b); cudaFree(c); cudaFree(d); cudaFree(e); cudaFree(f); cudaFree(g); }
    } guard{dZ, dZn, dS, dB, dBn, dSig, dV};
    int rc;
    const size_t rrz = (size_t)r * rz, rk = (size_t)r * k;
    if ((rc = dev_alloc(&dZ, rrz, fn, "the belief states")) != NOVA_SUCCESS) return rc;
    if ((rc = dev_alloc(&dB, rrz, fn, "the belief values")) != NOVA_SUCCESS) return rc;
    if ((rc = dev_alloc(&dS, rrz, fn, "the sorted states")) != NOVA_SUCCESS) return rc;
    if ((rc = dev_alloc(&dV, rrz, fn, "the sorted values")) != NOVA_SUCCESS) return rc;
    if ((rc = dev_alloc(&dZn, rk, fn, "the new belief states")) != NOVA_SUCCESS) return rc;
    if ((rc = dev_alloc(&dBn, rk, fn, "the new belief values")) != NOVA_SUCCESS) return rc;
    if ((rc = dev_alloc(&dSig, r, fn, "the belief sums")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(dZ, pomdp->Z, rrz * sizeof(int), fn, "the belief states")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(dB, pomdp->B, rrz * sizeof(float), fn, "the belief values")) != NOVA_SUCCESS) return rc;
    sigma_kernel<<<ceil_div(r, 128), 128>>>(r, rz, k, dZ, dB, dZn, dBn, dSig, dV, dS);
    if ((rc = check_launch(fn, "sigma approximation")) != NOVA_SUCCESS) return rc;
    int *Znew = new int[rk];
    float *Bnew = new float[rk];
    std::vector<float> sig(r);
    if ((rc = d2h(Znew, dZn, rk * sizeof(int), fn, "the new belief states")) != NOVA_SUCCESS ||
            (rc = d2h(Bnew, dBn, rk * sizeof(float), fn, "the new belief values")) != NOVA_SUCCESS ||
            (rc = d2h(sig.data(), dSig, r * sizeof(float), fn, "the belief sums")) != NOVA_SUCCESS) {
        delete[] Znew;
        delete[] Bnew;
        return rc;
    }
    // sigma = min(1, min_i sigma_b), in belief order (pomdp_sigma_cpu.cpp:80-92).
    float s = 1.0f;
    for (unsigned i = 0; i < r; i++)
        if (sig[i] < s) s = sig[i];
    sigma = s;
    delete[] pomdp->Z;
    delete[] pomdp->B;
    pomdp->rz = k;
    pomdp->Z = Znew;
    pomdp->B = Bnew;
    return NOVA_SUCCESS;
}

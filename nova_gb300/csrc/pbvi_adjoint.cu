// nova-gb300: reverse mode of H recorded PBVI backups.
//
// With the selections of every backup held fixed (for belief i at step t:
// the action a whose alpha became Gamma_t[i], and per observation o the
// alpha index j_o chosen for (i, a, o)), a backup is the smooth map
//
//   Gamma_t[i](s) = R(s,a) + sum_o gamma * sum_l O(a,S(s,a,l),o) T(s,a,l) Gamma_{t-1}[j_o](S(s,a,l))
//
// (pomdp_pbvi_cpu.cpp:37-103 with its argmax results recorded), and
// V(b0) = b0 . Gamma_H[i*] with i* = argmax_i b0 . Gamma_H[i]
// (pomdp_alpha_vectors.cpp:52-79). This file differentiates V(b0) with
// respect to R, T and O (and Gamma_0) by the adjoint recursion, for
// lambda_t = dV/dGamma_t (r x n, FP64):
//
//   dR(s,a)          += lambda_t[i](s)
//   c_i(s')           = sum_o O(a,s',o) Gamma_{t-1}[j_o](s')
//   dT(s,a,l)        += gamma * lambda_t[i](s) * c_i(S(s,a,l))
//   w_i(s')           = sum_{(s,l): S(s,a,l)=s'} T(s,a,l) lambda_t[i](s)
//   dO(a,s',o)       += gamma * w_i(s') * Gamma_{t-1}[j_o](s')
//   lambda_{t-1}[j_o](s') += gamma * O(a,s',o) * w_i(s')
//
// Gamma_{t-1} is needed at every reverse step. The caller keeps
// checkpoints every k steps; each segment between checkpoints is
// recomputed forward in FP32 with the recorded selections, in the
// reference's operation order, so the recomputed alphas are bit-identical
// to the forward pass.

#include "common.h"

#include <algorithm>
#include <vector>

#include <nova/constants.h>
#include <nova/pomdp/pomdp.h>
#include <nova/pomdp/algorithms/pomdp_pbvi_gpu.h>
#include <nova/nova_gb300.h>

using nova::POMDP;
using nova::POMDPPBVIGPU;

namespace nova_gb300 {
namespace {

constexpr unsigned kNoRow = 0xffffffffu;

struct AdjModel {
    unsigned n, ns, m, z, r;
    float gamma;
    const int *S;
    const float *T, *O, *R;
};

__global__ void adj_len_kernel(unsigned rows, unsigned ns, const int *__restrict__ S, unsigned *__restrict__ len) {
    const unsigned row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= rows) return;
    unsigned L = ns;
    for (unsigned l = 0; l < ns; l++)
        if (S[(size_t)row * ns + l] < 0) { L = l; break; }
    len[row] = L;
}

// State-contiguous tables for the replay, so that the 32 states of a warp read
// consecutive entries: ST[a][l][s] = S(s,a,l) (0 past the row end) and
// CT[a][o][l][s] = fl(O(a,S(s,a,l),o) * T(s,a,l)), the reference's first
// product (0 past the row end).
__global__ void adj_coef_kernel(AdjModel md, const unsigned *__restrict__ len, unsigned *__restrict__ ST,
                                float *__restrict__ CT, unsigned *__restrict__ predCount) {
    const size_t total = (size_t)md.m * md.ns * md.n;
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const unsigned s = (unsigned)(e % md.n);
        size_t t = e / md.n;
        const unsigned l = (unsigned)(t % md.ns);
        const unsigned a = (unsigned)(t / md.ns);
        const bool live = l < len[(size_t)s * md.m + a];
        const size_t row = ((size_t)s * md.m + a) * md.ns + l;
        const unsigned sp = live ? (unsigned)md.S[row] : 0u;
        const float T = live ? md.T[row] : 0.0f;
        ST[e] = sp;
        if (live) atomicAdd(predCount + (size_t)a * md.n + sp, 1u);
        for (unsigned o = 0; o < md.z; o++)
            CT[(((size_t)a * md.z + o) * md.ns + l) * md.n + s] =
                live ? fmul(md.O[((size_t)a * md.n + sp) * md.z + o], T) : 0.0f;
    }
}

// Beliefs of one action in groups of kGroup, for the replays of all steps at
// once (one block per step): group g of step t backs up beliefs
// ids[(t * groups + g) * kGroup ..] (kNoRow: none) with action
// acts[t * groups + g] (kNoRow: no such group); groups = ceil(r / kGroup) + m.
constexpr unsigned kGroup = 4;

__global__ void __launch_bounds__(1024) replay_groups_kernel(unsigned r, unsigned m, unsigned groups,
                                                             const unsigned *__restrict__ act,
                                                             unsigned *__restrict__ acts, unsigned *__restrict__ ids,
                                                             unsigned *__restrict__ wideCursor) {
    extern __shared__ unsigned narrowCursor[];
    const size_t t = blockIdx.x;
    // [m] next place of each action's beliefs (in global memory for very many actions)
    unsigned *cursor = wideCursor != nullptr ? wideCursor + t * m : narrowCursor;
    act += t * r;
    acts += t * groups;
    ids += t * groups * kGroup;
    for (unsigned a = threadIdx.x; a < m; a += blockDim.x) cursor[a] = 0u;
    for (unsigned g = threadIdx.x; g < groups; g += blockDim.x) acts[g] = kNoRow;
    for (unsigned k = threadIdx.x; k < groups * kGroup; k += blockDim.x) ids[k] = kNoRow;
    __syncthreads();
    for (unsigned i = threadIdx.x; i < r; i += blockDim.x) atomicAdd(cursor + min(act[i], m - 1), 1u);
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned g = 0;
        for (unsigned a = 0; a < m; a++) {
            const unsigned n = (cursor[a] + kGroup - 1) / kGroup;
            cursor[a] = g * kGroup;
            g += n;
        }
    }
    __syncthreads();
    for (unsigned i = threadIdx.x; i < r; i += blockDim.x) {
        const unsigned a = min(act[i], m - 1);
        const unsigned k = atomicAdd(cursor + a, 1u);
        ids[k] = i;
        acts[k / kGroup] = a;
    }
}

// Gamma_t from Gamma_{t-1} with recorded selections, in the reference's
// order: alpha = R(s,a); for each o, alpha += gamma * sum_l CT * G_j(S).
// One block per (group of beliefs with one action, 1,024 states): the
// beliefs' alphas of one observation lie in shared memory (the next
// observation's are copied in meanwhile) and every coefficient is read once
// for the whole group. Bound by the shared-memory gathers (random states,
// about 3.5 passes each): 2.7e8 of them (n = r = 1,024, z = ns = 16) take
// 189 us; one belief per block reading 64-byte coefficient rows per lane
// and gathering from L1 took 1,490 us.
constexpr unsigned kReplayThreads = 256;
constexpr unsigned kReplayStates = 4;  // states per thread

__device__ __forceinline__ void copy_async(float *dst, const float *src, bool wide) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if (wide) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

template <int NB, bool kShared>
__global__ void __launch_bounds__(kReplayThreads) replay_kernel(AdjModel md, const unsigned *__restrict__ len,
                                                                const unsigned *__restrict__ ST,
                                                                const float *__restrict__ CT,
                                                                const float *__restrict__ Gin,
                                                                const unsigned *__restrict__ acts,
                                                                const unsigned *__restrict__ ids,
                                                                const unsigned *__restrict__ sel, int wide,
                                                                float *__restrict__ Gout) {
    extern __shared__ __align__(16) float rows[];  // [2][NB][pitch]
    const unsigned a = acts[blockIdx.x / (kGroup / NB)];
    if (a == kNoRow) return;
    const unsigned pitch = (md.n + 3u) & ~3u;
    unsigned id[NB];
#pragma unroll
    for (unsigned b = 0; b < NB; b++) id[b] = ids[blockIdx.x * NB + b];
    if (NB == 1 && id[0] == kNoRow) return;
    auto chosen = [&](unsigned b, unsigned o) { return Gin + (size_t)min(sel[(size_t)id[b] * md.z + o], md.r - 1) * md.n; };
    auto stage = [&](unsigned o) {
        if constexpr (kShared) {
#pragma unroll
            for (unsigned b = 0; b < NB; b++) {
                if (id[b] == kNoRow) continue;
                const float *src = chosen(b, o);
                float *dst = rows + ((o & 1u) * NB + b) * pitch;
                const unsigned w = wide ? 4u : 1u;
                for (unsigned s = threadIdx.x * w; s < md.n; s += blockDim.x * w) copy_async(dst + s, src + s, wide != 0);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    };
    const unsigned s0 = blockIdx.y * (blockDim.x * kReplayStates) + threadIdx.x;
    float alpha[kReplayStates][NB];
    unsigned L[kReplayStates];
#pragma unroll
    for (unsigned q = 0; q < kReplayStates; q++) {
        const unsigned s = s0 + q * blockDim.x;
        const bool live = s < md.n;
        L[q] = live ? len[(size_t)s * md.m + a] : 0u;
        const float R = live ? md.R[(size_t)s * md.m + a] : 0.0f;
#pragma unroll
        for (unsigned b = 0; b < NB; b++) alpha[q][b] = R;
    }
    stage(0);
    for (unsigned o = 0; o < md.z; o++) {
        const float *g[NB];
        if constexpr (kShared) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();  // observation o's rows are in, observation o - 1's free
            if (o + 1 < md.z) stage(o + 1);
#pragma unroll
            for (unsigned b = 0; b < NB; b++) g[b] = rows + ((o & 1u) * NB + b) * pitch;
        } else {
#pragma unroll
            for (unsigned b = 0; b < NB; b++) g[b] = id[b] == kNoRow ? Gin : chosen(b, o);
        }
        const float *C = CT + ((size_t)a * md.z + o) * md.ns * md.n;
        const unsigned *Sa = ST + (size_t)a * md.ns * md.n;
#pragma unroll
        for (unsigned q = 0; q < kReplayStates; q++) {
            const unsigned s = s0 + q * blockDim.x;
            float vt[NB];
#pragma unroll
            for (unsigned b = 0; b < NB; b++) vt[b] = 0.0f;
            for (unsigned l0 = 0; l0 < L[q]; l0 += 4) {
                float c[4];
                unsigned sp[4];
#pragma unroll
                for (unsigned k = 0; k < 4; k++) {
                    const bool v = l0 + k < L[q];
                    c[k] = v ? __ldg(C + (size_t)(l0 + k) * md.n + s) : 0.0f;
                    sp[k] = v ? __ldg(Sa + (size_t)(l0 + k) * md.n + s) : 0u;
                }
#pragma unroll
                for (unsigned k = 0; k < 4; k++) {
                    if (l0 + k < L[q]) {
#pragma unroll
                        for (unsigned b = 0; b < NB; b++)
                            if (kShared || id[b] != kNoRow) vt[b] = fadd(vt[b], fmul(c[k], g[b][sp[k]]));
                    }
                }
            }
#pragma unroll
            for (unsigned b = 0; b < NB; b++) alpha[q][b] = fadd(alpha[q][b], fmul(vt[b], md.gamma));
        }
    }
#pragma unroll
    for (unsigned q = 0; q < kReplayStates; q++) {
        const unsigned s = s0 + q * blockDim.x;
        if (s < md.n) {
#pragma unroll
            for (unsigned b = 0; b < NB; b++)
                if (id[b] != kNoRow) Gout[(size_t)id[b] * md.n + s] = alpha[q][b];
        }
    }
}

// vals[i] = b . Gamma[i] in FP64.
__global__ void value_rows_kernel(const float *__restrict__ G, unsigned n, const float *__restrict__ b,
                                  double *__restrict__ vals) {
    const unsigned i = blockIdx.x;
    double acc = 0.0;
    for (unsigned s = threadIdx.x; s < n; s += blockDim.x) acc += (double)G[(size_t)i * n + s] * (double)b[s];
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    __shared__ double red[32];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (unsigned w = 0; w < blockDim.x / 32; w++) t += red[w];
        vals[i] = t;
    }
}

// Maximum with the -1e10 start and lowest index on ties; seeds
// lambda_H[i*] = b.
__global__ void value_argmax_kernel(unsigned r, unsigned n, const double *__restrict__ vals,
                                    const float *__restrict__ b, double *__restrict__ Vout,
                                    unsigned *__restrict__ iout, double *__restrict__ lam,
                                    unsigned *__restrict__ live) {
    __shared__ double sv[8];
    __shared__ unsigned si[8];
    double best = (double)NOVA_FLT_MIN;
    unsigned bi = kNoRow;
    for (unsigned j = threadIdx.x; j < r; j += 256)
        if (vals[j] > best) { best = vals[j]; bi = j; }
    auto take = [&](double v, unsigned j) {
        if (j != kNoRow && (bi == kNoRow || v > best || (v == best && j < bi))) { best = v; bi = j; }
    };
    for (int off = 16; off > 0; off >>= 1) {
        const double v = __shfl_xor_sync(0xffffffffu, best, off);
        take(v, __shfl_xor_sync(0xffffffffu, bi, off));
    }
    if ((threadIdx.x & 31) == 0) { sv[threadIdx.x >> 5] = best; si[threadIdx.x >> 5] = bi; }
    __syncthreads();
    for (unsigned w = 0; w < 8; w++) take(sv[w], si[w]);
    const unsigned istar = bi;   // the same in every thread
    if (threadIdx.x == 0) {
        *Vout = best;
        *iout = bi;
    }
    if (istar == kNoRow) return;
    if (threadIdx.x == 0) live[istar] = 1u;
    for (unsigned s = threadIdx.x; s < n; s += blockDim.x) lam[(size_t)istar * n + s] = (double)b[s];
}

// Threads and shared memory of a reverse-step block.
constexpr unsigned kStepThreads = 128;
constexpr size_t kStepSmem = 56 * 1024;

// The predecessors of every (a, s'): the (s, T(s,a,l)) with S(s,a,l) = s', one
// entry per l. Counted, given places (in no particular order of the lists) and
// filled.
__global__ void adj_pred_place_kernel(size_t rows, const unsigned *__restrict__ count, unsigned long long *next,
                                      unsigned long long *__restrict__ start, unsigned *__restrict__ filled) {
    const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned lane = threadIdx.x & 31, c = k < rows ? count[k] : 0u;
    unsigned v = c;
    for (int off = 1; off < 32; off <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, v, off);
        if (lane >= (unsigned)off) v += y;
    }
    unsigned long long base = 0;
    if (lane == 31) base = atomicAdd(next, (unsigned long long)v);
    base = __shfl_sync(0xffffffffu, base, 31);
    if (k < rows) {
        start[k] = base + (v - c);
        filled[k] = 0u;
    }
}
__global__ void adj_pred_fill_kernel(AdjModel md, const unsigned *__restrict__ len,
                                     const unsigned long long *__restrict__ start, unsigned *__restrict__ filled,
                                     uint2 *__restrict__ pred, unsigned *__restrict__ predK) {
    const size_t all = (size_t)md.n * md.m * md.ns, stride = (size_t)gridDim.x * blockDim.x;
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < all; e += stride) {
        const size_t row = e / md.ns;
        if (e % md.ns >= len[row]) continue;
        const size_t k = (row % md.m) * md.n + md.S[e];
        const unsigned long long at = start[k] + atomicAdd(filled + k, 1u);
        pred[at] = make_uint2((unsigned)(row / md.m), __float_as_uint(md.T[e]));
        predK[at] = (unsigned)(e % md.ns);
    }
}

// x in FP64: the conversion instruction runs at the FP64 rate (1/64 of FP32),
// the shifts of a normal number's bits do not.
__device__ __forceinline__ double widen(float x) {
    const unsigned b = __float_as_uint(x);
    if (((b >> 23) & 255u) - 1u < 254u)
        return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + (896u << 20))), (int)(b << 29));
    return (double)x;
}

__device__ __forceinline__ bool nonzero(double x) {   // by its bits: compares run at the FP64 rate too
    return (((unsigned)__double2hiint(x) & 0x7fffffffu) | (unsigned)__double2loint(x)) != 0u;
}

// One reverse step for up to NB beliefs of one action (of a group made for the
// replay; those without an adjoint, live 0, drop out) at kStepThreads successors
// s', one per thread: c and w of the beliefs stay in registers, the s' terms of
// dT are those of its predecessors, whose lambda are gathered from L2. Shared
// memory: the beliefs' selections, and with NB > 1 a tile per warp through which
// dO's terms, computed for consecutive states, reach consecutive observations.
// Marks the rows of lamPrev that it adds to in livePrev.
// Bound by FP64 arithmetic (1/64 of the FP32 rate), so factors are widened and
// tested by integer operations, and what does not depend on the belief is
// shared by the group; blocks of a part of the states even out the groups'
// unequal numbers of beliefs. n = 1,024 (m = 8, z = ns = 16, up to 600 beliefs
// with an adjoint): 430 us a step with a block per belief and w by atomics in
// shared memory, 200 so (the FP64 pipe 70 % busy; with two beliefs per block 240,
// one 250). Copying each belief's lambda into every block's shared memory instead
// gained nothing there and cost r n ceil(n / 128) reads where few beliefs have an
// adjoint: 5.7 ms a step at n = 14,000, r = 1,000, z = 1, ns = 2, against 0.1 so.
template <int NB>
__global__ void __launch_bounds__(kStepThreads) adjoint_step_kernel(
        AdjModel md, const unsigned *__restrict__ predCount, const unsigned long long *__restrict__ predStart,
        const uint2 *__restrict__ pred, const unsigned *__restrict__ predK, const float *__restrict__ Gprev,
        const unsigned *__restrict__ acts, const unsigned *__restrict__ ids, const unsigned *__restrict__ sel,
        const double *__restrict__ lam, const unsigned *__restrict__ live, double *__restrict__ lamPrev,
        unsigned *__restrict__ livePrev, double *__restrict__ dR, double *__restrict__ dT, double *__restrict__ dO) {
    constexpr bool kStaged = NB > 1;
    extern __shared__ __align__(16) unsigned char smem[];
    double *tiles = reinterpret_cast<double *>(smem);        // [warps][32][9] with kStaged
    unsigned *jsh = reinterpret_cast<unsigned *>(tiles + (kStaged ? kStepThreads * 9 : 0));  // [NB][z]
    constexpr unsigned kParts = kGroup / NB;
    ids += (size_t)blockIdx.x * NB;
    unsigned id[NB];
#pragma unroll
    for (int q = 0; q < NB; q++) id[q] = ids[q];
    const unsigned a = acts[blockIdx.x / kParts];
    if (a == kNoRow) return;
    const unsigned lane = threadIdx.x & 31;
    const unsigned sp = blockIdx.y * kStepThreads + threadIdx.x, sp0 = sp - lane;
    const bool in = sp < md.n;
    const unsigned cnt = in ? predCount[(size_t)a * md.n + sp] : 0u;
    const size_t first = in ? predStart[(size_t)a * md.n + sp] : 0u;
    unsigned nb = 0;
    const double *lambda[NB];   // lambda of the beliefs taken
#pragma unroll
    for (int q = 0; q < NB; q++) lambda[q] = lam;
#pragma unroll
    for (int q = 0; q < NB; q++) {
        const unsigned i = id[q];
        if (i == kNoRow || live[i] == 0u) continue;   // its place is taken by the next
#pragma unroll
        for (int b = 0; b < NB; b++)
            if (b == nb) lambda[b] = lam + (size_t)i * md.n;
        for (unsigned o = threadIdx.x; o < md.z; o += kStepThreads)
            jsh[nb * md.z + o] = min(sel[(size_t)i * md.z + o], md.r - 1);
        nb++;
    }
    if (nb == 0) return;
    __syncthreads();
    const double g = (double)md.gamma;
    if (sp0 >= md.n) return;
    const size_t ob = ((size_t)a * md.n + sp) * md.z;
    double c[NB], w[NB];
#pragma unroll
    for (int b = 0; b < NB; b++) c[b] = w[b] = 0.0;
    if (in) {
        double l = 0.0;
#pragma unroll
        for (int b = 0; b < NB; b++)
            if (b < nb) l += __ldg(lambda[b] + sp);
        if (nonzero(l)) atomicAdd(dR + (size_t)sp * md.m + a, l);
#pragma unroll 2
        for (unsigned o = 0; o < md.z; o++) {
            const double po = widen(__ldg(md.O + ob + o));
#pragma unroll
            for (int b = 0; b < NB; b++)
                if (b < nb) c[b] += po * widen(__ldg(Gprev + (size_t)jsh[b * md.z + o] * md.n + sp));
        }
#pragma unroll (NB == 1 ? 4 : 2)
        for (unsigned k = 0; k < cnt; k++) {
            const uint2 e = __ldg(pred + first + k);
            const size_t row = ((size_t)e.x * md.m + a) * md.ns + __ldg(predK + first + k);
            const double t = widen(__uint_as_float(e.y));
            double u = 0.0;
            bool nz = false;
#pragma unroll
            for (int b = 0; b < NB; b++)
                if (b < nb) {
                    const double lb = __ldg(lambda[b] + e.x);
                    if (nonzero(lb)) {
                        w[b] += t * lb;
                        u += lb * c[b];
                        nz = true;
                    }
                }
            if (nz) atomicAdd(dT + row, g * u);
        }
    }
    bool nzb[NB], nz = false;
#pragma unroll
    for (int b = 0; b < NB; b++) {
        nzb[b] = nonzero(w[b]);
        nz |= nzb[b];
        w[b] *= g;
    }
    if (!__any_sync(0xffffffffu, nz)) return;
#pragma unroll
    for (int b = 0; b < NB; b++)
        if (__any_sync(0xffffffffu, nzb[b]))
            for (unsigned o = lane; o < md.z; o += 32u) livePrev[jsh[b * md.z + o]] = 1u;
    double *tile = tiles + (size_t)(threadIdx.x >> 5) * 32 * 9;
    for (unsigned o0 = 0; o0 < md.z; o0 += 8) {
        const unsigned oEnd = min(8u, md.z - o0);
        for (unsigned q = 0; q < oEnd; q++) {
            const unsigned o = o0 + q;
            const double po = nz ? widen(__ldg(md.O + ob + o)) : 0.0;
            double d = 0.0;
#pragma unroll
            for (int b = 0; b < NB; b++)
                if (nzb[b]) {
                    const size_t gj = (size_t)jsh[b * md.z + o] * md.n + sp;
                    d += w[b] * widen(__ldg(Gprev + gj));
                    atomicAdd(lamPrev + gj, po * w[b]);
                }
            if constexpr (kStaged) tile[lane * 9 + q] = d;
            else if (nz) atomicAdd(dO + ob + o, d);
        }
        if constexpr (kStaged) {
            __syncwarp();
            const size_t ob0 = ((size_t)a * md.n + sp0) * md.z + o0;
            for (unsigned t = lane; t < 32u * 8u; t += 32u) {
                const unsigned k = t >> 3, q = t & 7u;
                const double d = q < oEnd ? tile[k * 9 + q] : 0.0;
                if (nonzero(d)) atomicAdd(dO + ob0 + (size_t)k * md.z + q, d);
            }
            __syncwarp();
        }
    }
}

struct AdjBuffers {
    Arena arena;
    unsigned *len = nullptr, *ST = nullptr, *acts = nullptr, *ids = nullptr, *cursor = nullptr;
    float *CT = nullptr, *seg = nullptr;
    double *lamA = nullptr, *lamB = nullptr, *vals = nullptr, *V = nullptr;  // lambda: [r][n], then [r] marks of its rows
    unsigned *istar = nullptr;
    unsigned *predCount = nullptr, *predFilled = nullptr, *predK = nullptr;
    unsigned long long *predStart = nullptr, *predNext = nullptr;
    uint2 *pred = nullptr;
};

// Gamma_t from Gamma_{t-1} in FP64 with recorded selections:
// alpha(s) = R(s,a) + gamma * sum_l T(s,a,l) sum_o O(a,S,o) Gamma_{j_o}(S),
// every operand widened to FP64 (the same map as replay_kernel without the
// FP32 roundings; the order of the FP64 sums differs from the reference's).
__global__ void replay_f64_kernel(AdjModel md, const unsigned *__restrict__ len, const double *__restrict__ Gin,
                                  const unsigned *__restrict__ act, const unsigned *__restrict__ sel,
                                  double *__restrict__ Gout) {
    const unsigned i = blockIdx.x;
    extern __shared__ unsigned jsh[];  // [z]
    const unsigned a = min(act[i], md.m - 1);
    for (unsigned o = threadIdx.x; o < md.z; o += blockDim.x) jsh[o] = min(sel[(size_t)i * md.z + o], md.r - 1);
    __syncthreads();
    const double gamma = (double)md.gamma;
    for (unsigned s = threadIdx.x; s < md.n; s += blockDim.x) {
        const size_t row = (size_t)s * md.m + a;
        const unsigned L = len[row];
        double acc = 0.0;
        for (unsigned l = 0; l < L; l++) {
            const unsigned sp = (unsigned)md.S[row * md.ns + l];
            const float *Orow = md.O + ((size_t)a * md.n + sp) * md.z;
            double w = 0.0;
            for (unsigned o = 0; o < md.z; o++) w += (double)Orow[o] * Gin[(size_t)jsh[o] * md.n + sp];
            acc += (double)md.T[row * md.ns + l] * w;
        }
        Gout[(size_t)i * md.n + s] = (double)md.R[row] + gamma * acc;
    }
}

__global__ void widen_kernel(const float *__restrict__ in, size_t count, double *__restrict__ out) {
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < count; e += (size_t)gridDim.x * blockDim.x)
        out[e] = (double)in[e];
}

// vals[i] = b . Gamma[i] with FP64 alphas.
__global__ void value_rows_f64_kernel(const double *__restrict__ G, unsigned n, const float *__restrict__ b,
                                      double *__restrict__ vals) {
    const unsigned i = blockIdx.x;
    double acc = 0.0;
    for (unsigned s = threadIdx.x; s < n; s += blockDim.x) acc += G[(size_t)i * n + s] * (double)b[s];
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    __shared__ double red[32];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (unsigned w = 0; w < blockDim.x / 32; w++) t += red[w];
        vals[i] = t;
    }
}

}  // namespace
}  // namespace nova_gb300

using namespace nova_gb300;

extern "C" int pomdp_pbvi_adjoint_gpu(const POMDP *pomdp, unsigned int horizon, unsigned int checkpointEvery,
                                      const float *d_checkpoints, const unsigned int *d_actions,
                                      const unsigned int *d_selects, const float *d_b, double *d_dR, double *d_dT,
                                      double *d_dO, double *d_dGamma0, double *Vb, unsigned int *bestAlpha) {
    static const char *fn = "pomdp_pbvi_adjoint_gpu";
    if (pomdp == nullptr || pomdp->n == 0 || pomdp->ns == 0 || pomdp->m == 0 || pomdp->z == 0 || pomdp->r == 0 ||
            pomdp->d_S == nullptr || pomdp->d_T == nullptr || pomdp->d_O == nullptr || pomdp->d_R == nullptr ||
            horizon == 0 || checkpointEvery == 0 || d_checkpoints == nullptr || d_actions == nullptr ||
            d_selects == nullptr || d_b == nullptr || d_dR == nullptr || d_dT == nullptr || d_dO == nullptr) {
        NOVA_ERR(fn, "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    AdjModel md{pomdp->n, pomdp->ns, pomdp->m, pomdp->z, pomdp->r, pomdp->gamma,
                pomdp->d_S, pomdp->d_T, pomdp->d_O, pomdp->d_R};
    // Four beliefs per block, which share what does not depend on them; one
    // where that leaves fewer blocks than a wave (four an SM; n = 100, r = 200, m
    // = 4: 18.4 and 12.0 us a step, n = 60, r = 1,200: 10.6 and 7.8; at n = 500,
    // r = 1,500, 1,500 blocks, either way 34). With very many observations (more
    // than 2,900 or 5,900), whose selections would leave room for few blocks on
    // an SM, two or one.
    const unsigned groups = ceil_div(md.r, kGroup) + md.m;
    const bool fewSteps = (size_t)groups * ceil_div(md.n, kStepThreads) <= 4u * 152u;
    auto step_smem = [&](size_t nb) {
        return nb * md.z * sizeof(unsigned) + (nb > 1 ? kStepThreads * 9 * sizeof(double) : 0);
    };
    const unsigned nb = fewSteps ? 1u : step_smem(4) <= kStepSmem ? 4u : step_smem(2) <= kStepSmem ? 2u : 1u;
    const size_t stepSmem = step_smem(nb);
    auto step = nb == 4 ? adjoint_step_kernel<4> : nb == 2 ? adjoint_step_kernel<2> : adjoint_step_kernel<1>;
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
            2 * (size_t)md.n * sizeof(double) + md.z * sizeof(unsigned) > (size_t)optin) {
        cudaGetLastError();
        NOVA_ERR(fn, "Too many states for the reverse step's shared-memory buffers.");
        return NOVA_ERROR_INVALID_DATA;
    }
    if (!allow_dynamic_smem(step, stepSmem)) {
        cudaGetLastError();
        NOVA_ERR(fn, "Failed to configure the reverse step kernel.");
        return NOVA_ERROR_KERNEL_EXECUTION;
    }
    const unsigned n = md.n, r = md.r, z = md.z, m = md.m, ns = md.ns, k = checkpointEvery;
    const size_t rn = (size_t)r * n;
    AdjBuffers bf;
    int rc;
    bf.arena.add(&bf.len, (size_t)n * m);
    bf.arena.add(&bf.ST, (size_t)m * n * ns);
    bf.arena.add(&bf.CT, (size_t)m * z * n * ns);
    bf.arena.add(&bf.acts, (size_t)horizon * groups);
    bf.arena.add(&bf.ids, (size_t)horizon * groups * kGroup);
    bf.arena.add(&bf.seg, (size_t)(k + 1) * rn);
    const size_t lamDoubles = rn + ceil_div(r, 2);   // one piece, cleared at once
    bf.arena.add(&bf.lamA, lamDoubles);
    bf.arena.add(&bf.lamB, lamDoubles);
    bf.arena.add(&bf.vals, r);
    bf.arena.add(&bf.V, 2);          // the value, and istar beside it
    const size_t predRows = round_up((size_t)m * n, 2);
    bf.arena.add(&bf.predCount, predRows + 2);   // and predNext behind it
    bf.arena.add(&bf.predFilled, (size_t)m * n);
    bf.arena.add(&bf.predStart, (size_t)m * n);
    bf.arena.add(&bf.pred, (size_t)m * n * ns);
    bf.arena.add(&bf.predK, (size_t)m * n * ns);
    const bool manyActions = m > 8192;
    if (manyActions) bf.arena.add(&bf.cursor, (size_t)horizon * m);
    if ((rc = bf.arena.commit(fn, "the adjoint")) != NOVA_SUCCESS) return rc;
    bf.istar = reinterpret_cast<unsigned *>(bf.V + 1);
    bf.predNext = reinterpret_cast<unsigned long long *>(bf.predCount + predRows);
    if ((rc = sync_device(fn)) != NOVA_SUCCESS) return rc;

    if (cudaMemset(d_dR, 0, (size_t)n * m * sizeof(double)) != cudaSuccess ||
            cudaMemset(d_dT, 0, (size_t)n * m * ns * sizeof(double)) != cudaSuccess ||
            cudaMemset(d_dO, 0, (size_t)m * n * z * sizeof(double)) != cudaSuccess ||
            cudaMemset(bf.lamA, 0, lamDoubles * sizeof(double)) != cudaSuccess ||
            cudaMemset(bf.predCount, 0, (predRows + 2) * sizeof(unsigned)) != cudaSuccess) {
        cudaGetLastError();
        NOVA_ERR(fn, "Failed to clear the gradients.");
        return NOVA_ERROR_KERNEL_EXECUTION;
    }
    adj_len_kernel<<<ceil_div((size_t)n * m, 256), 256>>>(n * m, ns, md.S, bf.len);
    if ((rc = check_launch(fn, "successor lengths")) != NOVA_SUCCESS) return rc;
    adj_coef_kernel<<<std::min<size_t>(ceil_div((size_t)m * n * ns, 256), 65535u * 8u), 256>>>(
        md, bf.len, bf.ST, bf.CT, bf.predCount);
    if ((rc = check_launch(fn, "projection coefficients")) != NOVA_SUCCESS) return rc;
    replay_groups_kernel<<<horizon, 1024, manyActions ? 0 : m * sizeof(unsigned)>>>(r, m, groups, d_actions, bf.acts,
                                                                                  bf.ids, bf.cursor);
    if ((rc = check_launch(fn, "belief groups")) != NOVA_SUCCESS) return rc;
    // Two observations' alphas of a group in shared memory, where they fit;
    // larger models gather from the alpha rows themselves.
    const size_t rowsSmem = 2 * (size_t)kGroup * round_up(n, 4) * sizeof(float);
    const bool rowsShared = rowsSmem + 1024 <= (size_t)optin;
    // One belief per block, unstaged, where the groups would leave half the SMs
    // idle (m z = 512, ns = 32: n = 100, 41 groups, 145 and 116 us a step; n =
    // 1,000, 91 groups, 480 and 690).
    const bool fewReplays = (size_t)groups * ceil_div(n, kReplayThreads * kReplayStates) <= 76u;
    auto replay = fewReplays ? replay_kernel<1, false> : rowsShared ? replay_kernel<4, true> : replay_kernel<4, false>;
    const size_t replaySmem = !fewReplays && rowsShared ? rowsSmem : 0;
    const unsigned replayThreads = (unsigned)std::min<size_t>(kReplayThreads, round_up(n, 32));
    const dim3 replayBlocks(groups * (fewReplays ? kGroup : 1u), ceil_div(n, replayThreads * kReplayStates));
    if (!allow_dynamic_smem(replay, replaySmem)) {
        cudaGetLastError();
        NOVA_ERR(fn, "Failed to configure the replay kernel.");
        return NOVA_ERROR_KERNEL_EXECUTION;
    }
    // 16-byte copies where every alpha row starts on a 16-byte boundary (the
    // segment buffer itself does).
    const int wide = n % 4u == 0u ? 1 : 0;
    const unsigned predBlocks = (unsigned)std::min<size_t>(ceil_div((size_t)m * n * ns, 256), 65535u * 8u);
    adj_pred_place_kernel<<<ceil_div((size_t)m * n, 256), 256>>>((size_t)m * n, bf.predCount, bf.predNext,
                                                                 bf.predStart, bf.predFilled);
    if ((rc = check_launch(fn, "predecessor places")) != NOVA_SUCCESS) return rc;
    adj_pred_fill_kernel<<<predBlocks, 256>>>(md, bf.len, bf.predStart, bf.predFilled, bf.pred,
                                              bf.predK);
    if ((rc = check_launch(fn, "predecessor lists")) != NOVA_SUCCESS) return rc;

    // Recompute the segment of checkpoint c: seg[q] = Gamma_{ck + q} for
    // q = 0 .. last (last = k - 1, or horizon - ck for the final segment,
    // which also yields Gamma_H).
    auto recompute = [&](unsigned c, unsigned last) -> int {
        const size_t base = (size_t)c * k;
        if (cudaMemcpy(bf.seg, d_checkpoints + (size_t)c * rn, rn * sizeof(float), cudaMemcpyDeviceToDevice) !=
                cudaSuccess) {
            cudaGetLastError();
            NOVA_ERR(fn, "Failed to copy a checkpoint.");
            return NOVA_ERROR_KERNEL_EXECUTION;
        }
        for (unsigned q = 1; q <= last; q++) {
            const size_t step = base + q - 1;
            replay<<<replayBlocks, replayThreads, replaySmem>>>(
                md, bf.len, bf.ST, bf.CT, bf.seg + (size_t)(q - 1) * rn, bf.acts + step * groups,
                bf.ids + step * groups * kGroup, d_selects + step * r * z, wide, bf.seg + (size_t)q * rn);
            int e = check_launch(fn, "alpha recomputation");
            if (e != NOVA_SUCCESS) return e;
        }
        return NOVA_SUCCESS;
    };

    const unsigned nCk = ceil_div(horizon, k);
    unsigned segC = nCk - 1;
    unsigned segStart = segC * k;
    if ((rc = recompute(segC, horizon - segStart)) != NOVA_SUCCESS) return rc;
    const float *GH = bf.seg + (size_t)(horizon - segStart) * rn;
    value_rows_kernel<<<r, 256>>>(GH, n, d_b, bf.vals);
    if ((rc = check_launch(fn, "FP64 values")) != NOVA_SUCCESS) return rc;
    auto marks = [&](double *lam) { return reinterpret_cast<unsigned *>(lam + rn); };
    value_argmax_kernel<<<1, 256>>>(r, n, bf.vals, d_b, bf.V, bf.istar, bf.lamA, marks(bf.lamA));
    if ((rc = check_launch(fn, "FP64 argmax")) != NOVA_SUCCESS) return rc;

    for (unsigned t = horizon; t >= 1; t--) {
        const unsigned p = t - 1;  // Gamma_{t-1} and the selections of backup t
        if (p < segStart) {
            segC = p / k;
            segStart = segC * k;
            if ((rc = recompute(segC, k - 1)) != NOVA_SUCCESS) return rc;
        }
        if (cudaMemsetAsync(bf.lamB, 0, lamDoubles * sizeof(double)) != cudaSuccess) {
            cudaGetLastError();
            NOVA_ERR(fn, "Failed to clear the adjoint.");
            return NOVA_ERROR_KERNEL_EXECUTION;
        }
        step<<<dim3(groups * (kGroup / nb), ceil_div(n, kStepThreads)), kStepThreads, stepSmem>>>(
            md, bf.predCount, bf.predStart, bf.pred, bf.predK, bf.seg + (size_t)(p - segStart) * rn,
            bf.acts + (size_t)p * groups, bf.ids + (size_t)p * groups * kGroup, d_selects + (size_t)p * r * z, bf.lamA,
            marks(bf.lamA), bf.lamB, marks(bf.lamB), d_dR, d_dT, d_dO);
        if ((rc = check_launch(fn, "reverse step")) != NOVA_SUCCESS) return rc;
        std::swap(bf.lamA, bf.lamB);
    }
    if (d_dGamma0 != nullptr &&
            cudaMemcpy(d_dGamma0, bf.lamA, rn * sizeof(double), cudaMemcpyDeviceToDevice) != cudaSuccess) {
        cudaGetLastError();
        NOVA_ERR(fn, "Failed to copy the Gamma_0 gradient.");
        return NOVA_ERROR_KERNEL_EXECUTION;
    }
    if ((rc = sync_device(fn)) != NOVA_SUCCESS) return rc;
    struct { double V; unsigned istar; } h;
    if (Vb != nullptr || bestAlpha != nullptr) {
        if ((rc = d2h(&h, bf.V, sizeof(h), fn, "the value and the maximising alpha")) != NOVA_SUCCESS) return rc;
        if (Vb != nullptr) *Vb = h.V;
        if (bestAlpha != nullptr) *bestAlpha = h.istar;
    }
    return NOVA_SUCCESS;
}

extern "C" int pomdp_pbvi_execute_recorded_gpu(const POMDP *pomdp, POMDPPBVIGPU *pbvi, unsigned int horizon,
                                               unsigned int checkpointEvery, float *d_checkpoints,
                                               unsigned int *d_actions, unsigned int *d_selects) {
    static const char *fn = "pomdp_pbvi_execute_recorded_gpu";
    if (pomdp == nullptr || pbvi == nullptr || horizon == 0 || checkpointEvery == 0 || d_checkpoints == nullptr ||
            d_actions == nullptr || d_selects == nullptr || pbvi->d_Gamma == nullptr || pbvi->d_GammaPrime == nullptr) {
        NOVA_ERR(fn, "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    const size_t rn = (size_t)pomdp->r * pomdp->n;
    for (unsigned t = 0; t < horizon; t++) {
        if (t % checkpointEvery == 0) {
            const float *cur = (pbvi->currentHorizon % 2u == 0u) ? pbvi->d_Gamma : pbvi->d_GammaPrime;
            if (cudaMemcpy(d_checkpoints + (size_t)(t / checkpointEvery) * rn, cur, rn * sizeof(float),
                           cudaMemcpyDeviceToDevice) != cudaSuccess) {
                cudaGetLastError();
                NOVA_ERR(fn, "Failed to store a checkpoint.");
                return NOVA_ERROR_KERNEL_EXECUTION;
            }
        }
        int rc = pomdp_pbvi_update_record_gpu(pomdp, pbvi, d_actions + (size_t)t * pomdp->r,
                                              d_selects + (size_t)t * pomdp->r * pomdp->z);
        if (rc != NOVA_SUCCESS) return rc;
    }
    return NOVA_SUCCESS;
}

extern "C" int pomdp_pbvi_value_replay_f64_gpu(const POMDP *pomdp, unsigned int horizon, const float *d_Gamma0,
                                               const unsigned int *d_actions, const unsigned int *d_selects,
                                               const float *d_b, unsigned int alpha, double *Vb,
                                               unsigned int *bestAlpha) {
    static const char *fn = "pomdp_pbvi_value_replay_f64_gpu";
    if (pomdp == nullptr || pomdp->n == 0 || pomdp->ns == 0 || pomdp->m == 0 || pomdp->z == 0 || pomdp->r == 0 ||
            pomdp->d_S == nullptr || pomdp->d_T == nullptr || pomdp->d_O == nullptr || pomdp->d_R == nullptr ||
            d_Gamma0 == nullptr || (horizon > 0 && (d_actions == nullptr || d_selects == nullptr)) ||
            d_b == nullptr || Vb == nullptr) {
        NOVA_ERR(fn, "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    AdjModel md{pomdp->n, pomdp->ns, pomdp->m, pomdp->z, pomdp->r, pomdp->gamma,
                pomdp->d_S, pomdp->d_T, pomdp->d_O, pomdp->d_R};
    const unsigned n = md.n, r = md.r, z = md.z, m = md.m, ns = md.ns;
    const size_t rn = (size_t)r * n;
    unsigned *len = nullptr;
    double *GA = nullptr, *GB = nullptr, *vals = nullptr;
    int rc;
    auto cleanup = [&]() {
        cudaDeviceSynchronize();
        cudaFree(len); cudaFree(GA); cudaFree(GB); cudaFree(vals);
    };
    if ((rc = dev_alloc(&len, (size_t)n * m, fn, "the successor lengths")) != NOVA_SUCCESS ||
            (rc = dev_alloc(&GA, rn, fn, "the FP64 alphas")) != NOVA_SUCCESS ||
            (rc = dev_alloc(&GB, rn, fn, "the FP64 alphas")) != NOVA_SUCCESS ||
            (rc = dev_alloc(&vals, r, fn, "the values")) != NOVA_SUCCESS) {
        cleanup();
        return rc;
    }
    adj_len_kernel<<<ceil_div((size_t)n * m, 256), 256>>>(n * m, ns, md.S, len);
    if ((rc = check_launch(fn, "successor lengths")) == NOVA_SUCCESS) {
        widen_kernel<<<(unsigned)std::min<size_t>(ceil_div(rn, 256), 65535u * 8u), 256>>>(d_Gamma0, rn, GA);
        rc = check_launch(fn, "FP64 alphas");
    }
    for (unsigned t = 0; t < horizon && rc == NOVA_SUCCESS; t++) {
        replay_f64_kernel<<<r, 256, z * sizeof(unsigned)>>>(md, len, GA, d_actions + (size_t)t * r,
                                                             d_selects + (size_t)t * r * z, GB);
        rc = check_launch(fn, "FP64 replay");
        std::swap(GA, GB);
    }
    if (rc == NOVA_SUCCESS) {
        value_rows_f64_kernel<<<r, 256>>>(GA, n, d_b, vals);
        rc = check_launch(fn, "FP64 values");
    }
    if (rc == NOVA_SUCCESS) rc = sync_device(fn);
    std::vector<double> hv;
    if (rc == NOVA_SUCCESS) {
        hv.resize(r);
        rc = d2h(hv.data(), vals, r * sizeof(double), fn, "the values");
    }
    cleanup();
    if (rc != NOVA_SUCCESS) return rc;
    // The given alpha, or the maximum from the -1e10 start with the lowest
    // index on ties (pomdp_alpha_vectors.cpp:52-79).
    unsigned best = alpha;
    double V = (double)NOVA_FLT_MIN;
    if (alpha < r) {
        V = hv[alpha];
    } else {
        best = 0;
        for (unsigned i = 0; i < r; i++)
            if (hv[i] > V) { V = hv[i]; best = i; }
    }
    *Vb = V;
    if (bestAlpha != nullptr) *bestAlpha = best;
    return NOVA_SUCCESS;
}

// nova-gb300: Perseus on the GB300 (pomdp_perseus_*_gpu, new) and the
// host-buffer entry points pomdp_perseus_*_cpu.
//
// One update (pomdp_perseus_cpu.cpp:312-429):
//   * draw a belief from B~ with rand() on the host (the reference formula);
//   * back it up against V_n = Gamma[0, rGamma) (perseus_score_kernel,
//     perseus_action_kernel, perseus_assemble_kernel: the FP32 operations of
//     the point-based backup in the reference's order, for one belief);
//   * keep the new alpha if it does not lose value at the belief, else copy
//     the belief's best old alpha (pomdp_perseus_cpu.cpp:367-374), and rebuild
//     B~ = {i : V_{n+1}(b_i) < V_n(b_i)} (pomdp_perseus_cpu.cpp:387-402), in
//     perseus_commit_kernel.
// V_n(b_i) is constant within a horizon step and is computed once per step;
// V_{n+1}(b_i) is a running maximum updated with the one new alpha, which is
// exact because only the maximum value (not its index) enters the test.
//
// One belief's backup is little work (n = 512, m = 8, z = ns = 16, rz = 32,
// three alphas: 0.2 M products) and is bound by the latency of its dependent
// loads, so each of the four launches spreads it as widely as its order of
// additions allows, and the chosen alphas' projections are kept from the
// scoring for the action values. An update took 310 us with the kernels made
// for whole belief sets (one block per (belief, action) stepping through the
// support, one block for the assembly, eleven launches and three
// synchronisations); it takes 75 us.

#include "pbvi.h"

#include <algorithm>
#include <cstdlib>
#include <vector>

#include <nova/constants.h>
#include <nova/pomdp/algorithms/pomdp_perseus_cpu.h>
#include <nova/pomdp/algorithms/pomdp_perseus_gpu.h>
#include <nova/pomdp/policies/pomdp_alpha_vectors.h>

using nova::POMDP;
using nova::POMDPPerseusCPU;
using nova::POMDPPerseusGPU;
using nova::POMDPAlphaVectors;

namespace nova_gb300 {

constexpr unsigned kNoneP = 0xffffffffu;

// b_i . alpha over the belief support in the order of
// pomdp_perseus_compute_b_dot_alpha_cpu (pomdp_perseus_cpu.cpp:37-50).
__device__ __forceinline__ float belief_dot(const DevModel &md, unsigned Li, unsigned i, const float *alpha) {
    float acc = 0.0f;
    for (unsigned k = 0; k < Li; k++) {
        const int s = md.Z[(size_t)i * md.rz + k];
        acc = fadd(acc, fmul(md.B[(size_t)i * md.rz + k], alpha[s]));
    }
    return acc;
}

// V(b_i) = max over rows [0, rows) of b_i . G_j, first maximiser
// (pomdp_perseus_compute_Vb_cpu, pomdp_perseus_cpu.cpp:53-68). One block per
// belief. idxOut may be null.
__global__ void perseus_vb_kernel(DevModel md, const unsigned *__restrict__ suppLen, const float *__restrict__ G,
                                  unsigned rows, float *__restrict__ vOut, unsigned *__restrict__ idxOut) {
    const unsigned i = blockIdx.x;
    const unsigned Li = suppLen[i];
    float best = NOVA_FLT_MIN;
    unsigned bj = kNoneP;
    for (unsigned j = threadIdx.x; j < rows; j += blockDim.x) {
        const float d = belief_dot(md, Li, i, G + (size_t)j * md.n);
        if (best < d) { best = d; bj = j; }
    }
    // Larger value, lower index on ties; kNoneP: none above -1e10.
    auto take = [&](float v, unsigned j) {
        if (j != kNoneP && (bj == kNoneP || v > best || (v == best && j < bj))) { best = v; bj = j; }
    };
    __shared__ float sv[8];
    __shared__ unsigned si[8];
    for (int off = 16; off > 0; off >>= 1) {
        const float v = __shfl_xor_sync(0xffffffffu, best, off);
        take(v, __shfl_xor_sync(0xffffffffu, bj, off));
    }
    if ((threadIdx.x & 31) == 0) { sv[threadIdx.x >> 5] = best; si[threadIdx.x >> 5] = bj; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (unsigned w = 1; w < 8; w++) take(sv[w], si[w]);
        vOut[i] = best;
        // The reference's caller starts alphaPrimeIndex at 0 (pomdp_perseus_cpu.cpp:361).
        if (idxOut) idxOut[i] = bj == kNoneP ? 0u : bj;
    }
}

__device__ __forceinline__ bool better(float v1, unsigned u1, float v2, unsigned u2) {
    return v1 > v2 || (v1 == v2 && u1 < u2);
}

// fl(gamma * sum_l C3 * G_j(S)) for state s under action a, observation o
// (the reference's order). Four successors' loads are issued together.
__device__ __forceinline__ float projected_at(const DevModel &md, const float *__restrict__ C3, unsigned Ls,
                                              const float *__restrict__ Gj, unsigned a, unsigned o, unsigned s) {
    const float *c = C3 + (((size_t)a * md.z + o) * md.n + s) * md.ns;
    const int *sp = md.S + ((size_t)s * md.m + a) * md.ns;
    float vt = 0.0f;
    unsigned l = 0;
    for (; l + 8 <= Ls; l += 8) {
        float g[8], cc[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            g[q] = Gj[__ldg(sp + l + q)];
            cc[q] = __ldg(c + l + q);
        }
#pragma unroll
        for (int q = 0; q < 8; q++) vt = fadd(vt, fmul(cc[q], g[q]));
    }
    for (; l < Ls; l++) vt = fadd(vt, fmul(__ldg(c + l), Gj[__ldg(sp + l)]));
    return fmul(vt, md.gamma);
}

// Belief i against alphas [0, rows): warp (a*z+o, split) scores its share of
// them, lane k taking support state k (32 at a time), and keeps the best and
// its index (kNoneP: none above -1e10) and, in one of its two slots of
// proj [m*z][splits][2][rz], the best one's projections at the support.
__global__ void __launch_bounds__(128) perseus_score_kernel(DevModel md, const unsigned *__restrict__ succLen,
                                                            const unsigned *__restrict__ suppLen,
                                                            const float *__restrict__ C3, const float *__restrict__ G,
                                                            unsigned rows, unsigned i, unsigned splits, unsigned share,
                                                            float *__restrict__ partV, unsigned *__restrict__ partU,
                                                            float *__restrict__ proj) {
    const unsigned lane = threadIdx.x & 31, w = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (w >= md.m * md.z * splits) return;
    const unsigned ao = w / splits, split = w % splits, a = ao / md.z, o = ao % md.z;
    const unsigned Li = suppLen[i];
    float *slots = proj + (size_t)w * 2 * md.rz;
    float best = NOVA_FLT_MIN;
    unsigned bu = kNoneP, slot = 0;
    for (unsigned u = split * share; u < min(rows, (split + 1) * share); u++) {
        float *mine = slots + (slot ^ 1u) * md.rz;
        float score = 0.0f;
        for (unsigned k0 = 0; k0 < Li; k0 += 32) {
            const unsigned k = k0 + lane;
            float p = 0.0f;
            if (k < Li) {
                const unsigned s = (unsigned)md.Z[(size_t)i * md.rz + k];
                p = projected_at(md, C3, succLen[(size_t)s * md.m + a], G + (size_t)u * md.n, a, o, s);
                mine[k] = p;
                p = fmul(p, md.B[(size_t)i * md.rz + k]);
            }
            const unsigned cnt = min(32u, Li - k0);
            for (unsigned t = 0; t < cnt; t++) score = fadd(score, __shfl_sync(0xffffffffu, p, t));
        }
        if (score > best) {
            best = score;
            bu = u;
            slot ^= 1u;
        }
    }
    if (lane == 0) {
        partV[w] = best;
        partU[w] = bu == kNoneP ? kNoneP : bu << 1 | slot;
    }
}

// One warp per action: per observation the best alpha of all splits (the
// lowest index among equals; where none beat -1e10 the previous observation's,
// row 0 for the first), then the action's value at the belief: alpha_a(s_k) =
// R(s_k,a) + sum_o projection, times b_k, summed in support order.
__global__ void __launch_bounds__(32) perseus_action_kernel(DevModel md, const unsigned *__restrict__ succLen,
                                                            const unsigned *__restrict__ suppLen,
                                                            const float *__restrict__ C3, const float *__restrict__ G,
                                                            unsigned i, unsigned splits,
                                                            const float *__restrict__ partV,
                                                            const unsigned *__restrict__ partU,
                                                            const float *__restrict__ proj,
                                                            unsigned *__restrict__ jstar, float *__restrict__ actVal) {
    extern __shared__ unsigned from[];  // [z] split and slot of the choice, or kNoneP
    const unsigned a = blockIdx.x, lane = threadIdx.x;
    unsigned *js = jstar + ((size_t)i * md.m + a) * md.z;
    unsigned prev = 0;
    for (unsigned o0 = 0; o0 < md.z; o0 += 32) {
        const unsigned o = o0 + lane;
        float v = NOVA_FLT_MIN;
        unsigned u = kNoneP, at = kNoneP;
        if (o < md.z) {
            const size_t w0 = ((size_t)a * md.z + o) * splits;
            for (unsigned sp = 0; sp < splits; sp++) {
                const unsigned pu = partU[w0 + sp];
                const float pv = partV[w0 + sp];
                if (pu != kNoneP && (u == kNoneP || better(pv, pu >> 1, v, u))) {
                    v = pv;
                    u = pu >> 1;
                    at = sp << 1 | (pu & 1u);
                }
            }
            from[o] = at;
        }
        const unsigned cnt = min(32u, md.z - o0);
        for (unsigned t = 0; t < cnt; t++) {
            const unsigned ut = __shfl_sync(0xffffffffu, u, t);
            if (ut != kNoneP) prev = ut;
            if (lane == t) u = prev;
        }
        if (o < md.z) js[o] = u;
    }
    __syncwarp();
    const unsigned Li = suppLen[i];
    float value = 0.0f;
    for (unsigned k0 = 0; k0 < Li; k0 += 32) {
        const unsigned k = k0 + lane;
        float p = 0.0f;
        if (k < Li) {
            const unsigned s = (unsigned)md.Z[(size_t)i * md.rz + k];
            float alpha = md.R[(size_t)s * md.m + a];
            for (unsigned o = 0; o < md.z; o += 8) {
                float q[8];
#pragma unroll
                for (unsigned t = 0; t < 8; t++) {
                    if (o + t >= md.z) break;
                    const unsigned at = from[o + t];
                    q[t] = at != kNoneP
                        ? proj[((((size_t)a * md.z + o + t) * splits + (at >> 1)) * 2 + (at & 1u)) * md.rz + k]
                        : projected_at(md, C3, succLen[(size_t)s * md.m + a], G + (size_t)js[o + t] * md.n, a, o + t, s);
                }
#pragma unroll
                for (unsigned t = 0; t < 8; t++)
                    if (o + t < md.z) alpha = fadd(alpha, q[t]);
            }
            p = fmul(alpha, md.B[(size_t)i * md.rz + k]);
        }
        const unsigned cnt = min(32u, Li - k0);
        for (unsigned t = 0; t < cnt; t++) value = fadd(value, __shfl_sync(0xffffffffu, p, t));
    }
    if (lane == 0) actVal[a] = value;
}

// The best action's alpha (strict '>' from -1e10, lowest action on ties; none:
// *action = kNoneP and the row stays) over 32 states a block: thread (x, y)
// projects state x for observations y, y + 16, ...; sixteen at a time they are
// added in observation order.
constexpr unsigned kAssembleObs = 16;

__global__ void __launch_bounds__(32 * kAssembleObs) perseus_assemble_kernel(
        DevModel md, const unsigned *__restrict__ succLen, const float *__restrict__ C3, const float *__restrict__ G,
        unsigned i, const unsigned *__restrict__ jstar, const float *__restrict__ actVal, float *__restrict__ row,
        unsigned *__restrict__ action) {
    __shared__ float part[kAssembleObs][32];
    __shared__ unsigned bestA;
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        float best = NOVA_FLT_MIN;
        unsigned ba = kNoneP;
        for (unsigned a = 0; a < md.m; a++) {
            const float v = actVal[a];
            if (v > best) { best = v; ba = a; }
        }
        bestA = ba;
        if (blockIdx.x == 0) *action = ba;
    }
    __syncthreads();
    const unsigned a = bestA, s = blockIdx.x * 32 + threadIdx.x;
    if (a == kNoneP) return;
    const unsigned *js = jstar + ((size_t)i * md.m + a) * md.z;
    const unsigned Ls = s < md.n ? succLen[(size_t)s * md.m + a] : 0u;
    float alpha = s < md.n ? md.R[(size_t)s * md.m + a] : 0.0f;
    for (unsigned o0 = 0; o0 < md.z; o0 += kAssembleObs) {
        const unsigned o = o0 + threadIdx.y;
        if (s < md.n && o < md.z)
            part[threadIdx.y][threadIdx.x] = projected_at(md, C3, Ls, G + (size_t)js[o] * md.n, a, o, s);
        __syncthreads();
        if (threadIdx.y == 0)
            for (unsigned q = 0; q < min(kAssembleObs, md.z - o0); q++) alpha = fadd(alpha, part[q][threadIdx.x]);
        __syncthreads();
    }
    if (threadIdx.y == 0 && s < md.n) row[s] = alpha;
}

// belief_dot by a whole warp: the products side by side, added in support order.
__device__ __forceinline__ float belief_dot_warp(const DevModel &md, unsigned Li, unsigned i, const float *alpha,
                                                 unsigned lane) {
    float acc = 0.0f;
    for (unsigned k0 = 0; k0 < Li; k0 += 32) {
        const unsigned k = k0 + lane;
        const float p = k < Li ? fmul(md.B[(size_t)i * md.rz + k], alpha[md.Z[(size_t)i * md.rz + k]]) : 0.0f;
        const unsigned cnt = min(32u, Li - k0);
        for (unsigned t = 0; t < cnt; t++) acc = fadd(acc, __shfl_sync(0xffffffffu, p, t));
    }
    return acc;
}

// Keep the new alpha or take the belief's best old one, as row `slot` of V_{n+1};
// raise V_{n+1}(b_i) <- max(V_{n+1}(b_i), b_i . row) with the reference's strict
// '<'; and list B~ = {i : V_{n+1}(b_i) < V_n(b_i)} in increasing i, behind its
// size, in out [1 + r]. Every block decides about the row by itself; the one
// that finishes last makes the list. *done is 0 before and after.
__global__ void __launch_bounds__(256) perseus_commit_kernel(DevModel md, const unsigned *__restrict__ suppLen,
                                                             unsigned bIndex, const float *__restrict__ alpha,
                                                             const unsigned *__restrict__ alphaAction,
                                                             const float *__restrict__ vnb,
                                                             const unsigned *__restrict__ vnbIdx,
                                                             const float *__restrict__ G,
                                                             const unsigned *__restrict__ pi, float *__restrict__ Gp,
                                                             unsigned *__restrict__ piP, unsigned slot, float *vnp1b,
                                                             unsigned *__restrict__ out, unsigned *__restrict__ done) {
    __shared__ int keepNew;
    __shared__ bool last;
    __shared__ unsigned warpSums[8];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp == 0) {
        const float acc = belief_dot_warp(md, suppLen[bIndex], bIndex, alpha, lane);
        if (lane == 0) {
            keepNew = acc >= vnb[bIndex] ? 1 : 0;
            if (blockIdx.x == 0) {
                const unsigned act = *alphaAction == kNoneP ? 0u : *alphaAction;
                piP[slot] = keepNew ? act : pi[vnbIdx[bIndex]];
            }
        }
    }
    __syncthreads();
    const float *row = keepNew ? alpha : G + (size_t)vnbIdx[bIndex] * md.n;
    for (unsigned s = blockIdx.x * 256 + threadIdx.x; s < md.n; s += gridDim.x * 256) Gp[(size_t)slot * md.n + s] = row[s];
    for (unsigned i = blockIdx.x * 8 + warp; i < md.r; i += gridDim.x * 8) {
        const float d = belief_dot_warp(md, suppLen[i], i, row, lane);
        if (lane == 0 && vnp1b[i] < d) vnp1b[i] = d;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    // Every thread takes a range of beliefs; a block scan gives its first place.
    const unsigned per = (md.r + 255) / 256;
    const unsigned b = min(md.r, threadIdx.x * per), e = min(md.r, b + per);
    unsigned cnt = 0;
    for (unsigned i = b; i < e; i++) cnt += __ldcg(vnp1b + i) < vnb[i] ? 1u : 0u;
    unsigned v = cnt;
    for (int off = 1; off < 32; off <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, v, off);
        if (lane >= (unsigned)off) v += y;
    }
    if (lane == 31) warpSums[warp] = v;
    __syncthreads();
    unsigned pos = v - cnt;
    for (unsigned w = 0; w < warp; w++) pos += warpSums[w];
    for (unsigned i = b; i < e; i++)
        if (__ldcg(vnp1b + i) < vnb[i]) out[1 + pos++] = i;
    if (threadIdx.x == 255) {
        out[0] = pos;
        *done = 0u;
    }
}

__global__ void fill_float_kernel(float *p, unsigned count, float v) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < count) p[t] = v;
}

// Device-side Perseus state shared by the _gpu and _cpu front ends.
struct PerseusCore {
    BackupEngine eng;
    Arena arena;
    bool built = false;
    unsigned *vnbIdx = nullptr;
    // Validity of the per-horizon-step cache (V_n values).
    bool cacheValid = false;
    unsigned cacheHorizon = 0;
    unsigned *bt = nullptr;       // [1 + r] |B~| and B~
    unsigned *done = nullptr;     // [1] finished blocks of perseus_commit_kernel
    float *partV = nullptr, *proj = nullptr;   // the scoring's partial maxima and projections
    unsigned *partU = nullptr;
    Arena parts;
    unsigned maxSplits = 0;       // that these hold
    std::vector<unsigned> btHost;

    int build(const DevModel &md, const char *fn) {
        int rc = eng.build(md, fn);
        if (rc != NOVA_SUCCESS) return rc;
        arena.add(&eng.vnb, md.r);
        arena.add(&eng.vnp1b, md.r);
        arena.add(&bt, (size_t)md.r + 1);
        arena.add(&done, 1);
        arena.add(&vnbIdx, md.r);
        if ((rc = arena.commit(fn, "the Perseus values")) != NOVA_SUCCESS) return rc;
        if (cudaMemsetAsync(done, 0, sizeof(unsigned), eng.stream) != cudaSuccess) {
            cudaGetLastError();
            NOVA_ERR(fn, "Failed to clear the block counter.");
            return NOVA_ERROR_KERNEL_EXECUTION;
        }
        btHost.resize((size_t)md.r + 1);
        built = true;
        return NOVA_SUCCESS;
    }

    // Per-step cache: V_n(b_i) with maximisers, and V_{n+1}(b_i) over the rows
    // already in Gamma'.
    int refresh(const float *G, unsigned rGamma, const float *Gp, unsigned rGammaPrime, const char *fn) {
        const DevModel &md = eng.md;
        int rc;
        if (rGamma > 0) {
            perseus_vb_kernel<<<md.r, 256, 0, eng.stream>>>(md, eng.suppLen, G, rGamma, eng.vnb, vnbIdx);
        } else {
            fill_float_kernel<<<ceil_div(md.r, 256), 256, 0, eng.stream>>>(eng.vnb, md.r, NOVA_FLT_MIN);
            cudaMemsetAsync(vnbIdx, 0, md.r * sizeof(unsigned), eng.stream);
        }
        if ((rc = check_launch(fn, "V_n(b)")) != NOVA_SUCCESS) return rc;
        if (rGammaPrime > 0)
            perseus_vb_kernel<<<md.r, 256, 0, eng.stream>>>(md, eng.suppLen, Gp, rGammaPrime, eng.vnp1b, nullptr);
        else
            fill_float_kernel<<<ceil_div(md.r, 256), 256, 0, eng.stream>>>(eng.vnp1b, md.r, NOVA_FLT_MIN);
        if ((rc = check_launch(fn, "V_n+1(b)")) != NOVA_SUCCESS) return rc;
        cacheValid = true;
        return NOVA_SUCCESS;
    }

    // One Perseus update. G/pi: V_n and its actions (rGamma rows);
    // Gp/piP: V_{n+1} (rGammaPrime rows). Host bookkeeping by reference.
    // newSlot receives the row index written into Gp.
    int update(const float *G, const unsigned *pi, float *Gp, unsigned *piP, unsigned &currentHorizon,
               unsigned &rGamma, unsigned &rGammaPrime, unsigned &rTilde, unsigned *BTilde, unsigned *newSlot,
               const char *fn) {
        const DevModel &md = eng.md;
        int rc;
        if (!cacheValid || cacheHorizon != currentHorizon) {
            if ((rc = refresh(G, rGamma, Gp, rGammaPrime, fn)) != NOVA_SUCCESS) return rc;
            cacheHorizon = currentHorizon;
        }
        // Belief draw of pomdp_perseus_cpu.cpp:340-341. When rand() rounds
        // to RAND_MAX the index equals rTilde and the reference reads the
        // stale entry there; beyond the array it is clamped to the last one.
        unsigned bTildeIndex = (unsigned)((float)rand() / (float)RAND_MAX * (float)rTilde);
        if (bTildeIndex >= md.r) bTildeIndex = md.r - 1;
        const unsigned bIndex = BTilde[bTildeIndex];
        if (bIndex >= md.r) {
            NOVA_ERR(fn, "Invalid belief index in BTilde.");
            return NOVA_ERROR_INVALID_DATA;
        }
        if (rGammaPrime + 1 > md.r) {
            NOVA_ERR(fn, "Out of memory. Too many alpha-vectors added.");
            return NOVA_ERROR_OUT_OF_MEMORY;
        }
        // Backup of belief bIndex against V_n: about 8,192 scoring warps, each
        // with as many alphas as that leaves it. With V_n empty no warp has an
        // alpha, and every observation takes row 0 (the reference's best-alpha
        // index is never assigned there, pomdp_perseus_cpu.cpp:78-84).
        const unsigned mz = md.m * md.z;
        if (partV == nullptr) {
            // Room for every step's splits, allocated once; fewer splits where
            // the projections (8 rz bytes a warp) cannot be had.
            for (maxSplits = std::max(1u, std::min(md.r, 8192u / mz));; maxSplits = (maxSplits + 1) / 2) {
                const size_t most = (size_t)mz * maxSplits;
                parts.add(&partV, most);
                parts.add(&partU, most);
                parts.add(&proj, most * 2 * md.rz);
                if (parts.try_commit()) break;
                if (maxSplits == 1) return malloc_failed(fn, "the projections");
            }
        }
        const unsigned splits = std::max(1u, std::min(rGamma, maxSplits));
        const unsigned share = ceil_div(rGamma, splits);
        const size_t need = (size_t)mz * splits;
        perseus_score_kernel<<<ceil_div(need, 4), 128, 0, eng.stream>>>(md, eng.succLen, eng.suppLen, eng.C3, G, rGamma,
                                                                        bIndex, splits, share, partV, partU, proj);
        if ((rc = check_launch(fn, "belief scoring")) != NOVA_SUCCESS) return rc;
        perseus_action_kernel<<<md.m, 32, md.z * sizeof(unsigned), eng.stream>>>(
            md, eng.succLen, eng.suppLen, eng.C3, G, bIndex, splits, partV, partU, proj, eng.jstar, eng.actVal);
        if ((rc = check_launch(fn, "action values")) != NOVA_SUCCESS) return rc;
        perseus_assemble_kernel<<<ceil_div(md.n, 32), dim3(32, kAssembleObs), 0, eng.stream>>>(
            md, eng.succLen, eng.C3, G, bIndex, eng.jstar, eng.actVal, eng.rowScratch, eng.resultA);
        if ((rc = check_launch(fn, "alpha assembly")) != NOVA_SUCCESS) return rc;
        const unsigned slot = rGammaPrime;
        perseus_commit_kernel<<<std::min(608u, ceil_div(md.r, 8)), 256, 0, eng.stream>>>(
            md, eng.suppLen, bIndex, eng.rowScratch, eng.resultA, eng.vnb, vnbIdx, G, pi, Gp, piP, slot, eng.vnp1b, bt,
            done);
        if ((rc = check_launch(fn, "Perseus commit")) != NOVA_SUCCESS) return rc;
        rGammaPrime++;
        *newSlot = slot;
        // One read-back: the size and, whatever it is, the whole list.
        if (cudaMemcpyAsync(btHost.data(), bt, btHost.size() * sizeof(unsigned), cudaMemcpyDeviceToHost, eng.stream) !=
                cudaSuccess || cudaStreamSynchronize(eng.stream) != cudaSuccess) {
            cudaGetLastError();
            NOVA_ERR(fn, "Failed to copy B~ from device to host.");
            return NOVA_ERROR_MEMCPY_TO_HOST;
        }
        const unsigned count = std::min(btHost[0], md.r);
        memcpy(BTilde, btHost.data() + 1, count * sizeof(unsigned));
        rTilde = count;
        if (rTilde == 0) {
            // pomdp_perseus_cpu.cpp:405-426
            currentHorizon++;
            rGamma = 0;
            rTilde = md.r;
            for (unsigned i = 0; i < md.r; i++) BTilde[i] = i;
            cacheValid = false;
            return NOVA_CONVERGED;
        }
        return NOVA_SUCCESS;
    }
};

struct PerseusGpuWorkspace : Workspace {
    PerseusCore core;
    Arena arena;
    const void *modelKey[6] = {};
    float *d_Gamma = nullptr, *d_GammaPrime = nullptr;
    unsigned *d_pi = nullptr, *d_piPrime = nullptr;
    unsigned *hostBTilde = nullptr;
    ~PerseusGpuWorkspace() override { cudaDeviceSynchronize(); }
};

struct PerseusCpuWorkspace : Workspace {
    PerseusCore core;
    Arena arena;
    int *S = nullptr; float *T = nullptr, *O = nullptr, *R = nullptr; int *Z = nullptr; float *B = nullptr;
    float *Gamma = nullptr, *GammaPrime = nullptr;
    unsigned *pi = nullptr, *piPrime = nullptr;
    ~PerseusCpuWorkspace() override { cudaDeviceSynchronize(); }
};

static bool perseus_shape_invalid(const POMDP *p) {
    return p == nullptr || p->n == 0 || p->ns == 0 || p->m == 0 || p->z == 0 || p->r == 0 || p->rz == 0 ||
           p->gamma < 0.0f || p->gamma > 1.0f || p->horizon < 1;
}

}  // namespace nova_gb300

using namespace nova_gb300;

// ===========================================================================
// Device-buffer Perseus (new)
// ===========================================================================

static PerseusGpuWorkspace *perseus_gpu_ws(const POMDPPerseusGPU *per) {
    std::lock_guard<std::mutex> lock(registry_mutex());
    return find_workspace<PerseusGpuWorkspace>(per);
}

extern "C" int pomdp_perseus_uninitialize_gpu(const POMDP *pomdp, POMDPPerseusGPU *per) {
    (void)pomdp;
    if (per == nullptr) {
        NOVA_ERR("pomdp_perseus_uninitialize_gpu", "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    per->currentHorizon = 0;
    per->rGamma = 0; per->rGammaPrime = 0; per->rTilde = 0;
    std::lock_guard<std::mutex> lock(registry_mutex());
    auto *ws = find_workspace<PerseusGpuWorkspace>(per);
    if (ws != nullptr) {
        if (per->BTilde == ws->hostBTilde) { delete[] per->BTilde; per->BTilde = nullptr; }
        per->d_Gamma = nullptr; per->d_GammaPrime = nullptr; per->d_pi = nullptr; per->d_piPrime = nullptr;
        registry().erase(per);
    }
    return NOVA_SUCCESS;
}

extern "C" int pomdp_perseus_initialize_gpu(const POMDP *pomdp, POMDPPerseusGPU *per) {
    static const char *fn = "pomdp_perseus_initialize_gpu";
    if (pomdp == nullptr || per == nullptr || pomdp->n == 0 || pomdp->r == 0 || per->GammaInitial == nullptr) {
        NOVA_ERR(fn, "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    {
        std::lock_guard<std::mutex> lock(registry_mutex());
        auto *old = find_workspace<PerseusGpuWorkspace>(per);
        if (old != nullptr) {
            if (per->BTilde == old->hostBTilde) { delete[] per->BTilde; per->BTilde = nullptr; }
            registry().erase(per);
        }
    }
    const size_t rn = (size_t)pomdp->r * pomdp->n;
    std::unique_ptr<PerseusGpuWorkspace> ws(new PerseusGpuWorkspace());
    int rc;
    ws->arena.add(&ws->d_Gamma, rn);
    ws->arena.add(&ws->d_GammaPrime, rn);
    ws->arena.add(&ws->d_pi, pomdp->r);
    ws->arena.add(&ws->d_piPrime, pomdp->r);
    if ((rc = ws->arena.commit(fn, "the alpha sets")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws->d_Gamma, per->GammaInitial, rn * sizeof(float), fn, "Gamma")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws->d_GammaPrime, per->GammaInitial, rn * sizeof(float), fn, "Gamma (prime)")) != NOVA_SUCCESS)
        return rc;
    cudaMemset(ws->d_pi, 0, pomdp->r * sizeof(unsigned));
    cudaMemset(ws->d_piPrime, 0, pomdp->r * sizeof(unsigned));
    // pomdp_perseus_cpu.cpp:183-219: empty V_n and V_{n+1}, B~ = B.
    per->currentHorizon = 0;
    per->rGamma = 0;
    per->rGammaPrime = 0;
    per->rTilde = pomdp->r;
    per->BTilde = new unsigned int[pomdp->r];
    for (unsigned i = 0; i < pomdp->r; i++) per->BTilde[i] = i;
    ws->hostBTilde = per->BTilde;
    per->d_Gamma = ws->d_Gamma; per->d_GammaPrime = ws->d_GammaPrime;
    per->d_pi = ws->d_pi; per->d_piPrime = ws->d_piPrime;
    std::lock_guard<std::mutex> lock(registry_mutex());
    registry()[per] = std::move(ws);
    return NOVA_SUCCESS;
}

extern "C" int pomdp_perseus_update_gpu(const POMDP *pomdp, POMDPPerseusGPU *per) {
    static const char *fn = "pomdp_perseus_update_gpu";
    if (perseus_shape_invalid(pomdp) || per == nullptr || pomdp->d_S == nullptr || pomdp->d_T == nullptr ||
            pomdp->d_O == nullptr || pomdp->d_R == nullptr || pomdp->d_Z == nullptr || pomdp->d_B == nullptr ||
            per->BTilde == nullptr || per->d_Gamma == nullptr || per->d_GammaPrime == nullptr) {
        NOVA_ERR(fn, "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    PerseusGpuWorkspace *ws = perseus_gpu_ws(per);
    if (ws == nullptr) {
        NOVA_ERR(fn, "The solver is not initialized (call pomdp_perseus_initialize_gpu).");
        return NOVA_ERROR_INVALID_DATA;
    }
    const void *key[6] = {pomdp->d_S, pomdp->d_T, pomdp->d_O, pomdp->d_R, pomdp->d_Z, pomdp->d_B};
    if (!ws->core.built || memcmp(key, ws->modelKey, sizeof(key)) != 0) {
        if (ws->core.built) {
            NOVA_ERR(fn, "The device model changed during a Perseus solve.");
            return NOVA_ERROR_INVALID_DATA;
        }
        DevModel md;
        md.n = pomdp->n; md.ns = pomdp->ns; md.m = pomdp->m; md.z = pomdp->z; md.r = pomdp->r;
        md.rz = pomdp->rz; md.gamma = pomdp->gamma;
        md.S = pomdp->d_S; md.T = pomdp->d_T; md.O = pomdp->d_O; md.R = pomdp->d_R; md.Z = pomdp->d_Z;
        md.B = pomdp->d_B;
        int rc = ws->core.build(md, fn);
        if (rc != NOVA_SUCCESS) return rc;
        memcpy(ws->modelKey, key, sizeof(key));
    }
    const bool even = (per->currentHorizon % 2u) == 0u;
    unsigned slot = 0;
    if (even)
        return ws->core.update(per->d_Gamma, per->d_pi, per->d_GammaPrime, per->d_piPrime, per->currentHorizon,
                               per->rGamma, per->rGammaPrime, per->rTilde, per->BTilde, &slot, fn);
    return ws->core.update(per->d_GammaPrime, per->d_piPrime, per->d_Gamma, per->d_pi, per->currentHorizon,
                           per->rGammaPrime, per->rGamma, per->rTilde, per->BTilde, &slot, fn);
}

extern "C" int pomdp_perseus_get_policy_gpu(const POMDP *pomdp, POMDPPerseusGPU *per, POMDPAlphaVectors *policy) {
    static const char *fn = "pomdp_perseus_get_policy_gpu";
    if (pomdp == nullptr || per == nullptr || policy == nullptr) {
        NOVA_ERR(fn, "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    const bool even = (per->currentHorizon % 2u) == 0u;
    const unsigned rows = even ? per->rGamma : per->rGammaPrime;
    if (pomdp_alpha_vectors_initialize(policy, pomdp->n, pomdp->m, rows) != NOVA_SUCCESS) {
        NOVA_ERR(fn, "Could not create the policy.");
        return NOVA_ERROR_POLICY_CREATION;
    }
    int rc = d2h(policy->Gamma, even ? per->d_Gamma : per->d_GammaPrime, (size_t)rows * pomdp->n * sizeof(float),
                 fn, "Gamma");
    if (rc != NOVA_SUCCESS) return rc;
    return d2h(policy->pi, even ? per->d_pi : per->d_piPrime, rows * sizeof(unsigned), fn, "pi");
}

extern "C" int pomdp_perseus_execute_gpu(const POMDP *pomdp, POMDPPerseusGPU *per, POMDPAlphaVectors *policy) {
    static const char *fn = "pomdp_perseus_execute_gpu";
    if (perseus_shape_invalid(pomdp) || pomdp->d_S == nullptr || pomdp->d_T == nullptr || pomdp->d_O == nullptr ||
            pomdp->d_R == nullptr || pomdp->d_Z == nullptr || pomdp->d_B == nullptr || per == nullptr ||
            per->GammaInitial == nullptr || policy == nullptr) {
        NOVA_ERR(fn, "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    if (per->numThreads % 32 != 0) {
        NOVA_ERR(fn, "Invalid number of threads.");
        return NOVA_ERROR_INVALID_CUDA_PARAM;
    }
    int rc = pomdp_perseus_initialize_gpu(pomdp, per);
    if (rc != NOVA_SUCCESS) return rc;
    while (per->currentHorizon < pomdp->horizon) {
        rc = NOVA_SUCCESS;
        while (rc != NOVA_CONVERGED) {
            rc = pomdp_perseus_update_gpu(pomdp, per);
            if (rc != NOVA_CONVERGED && rc != NOVA_SUCCESS) return rc;
        }
    }
    rc = pomdp_perseus_get_policy_gpu(pomdp, per, policy);
    if (rc != NOVA_SUCCESS) return rc;
    return pomdp_perseus_uninitialize_gpu(pomdp, per);
}

// ===========================================================================
// Host-buffer Perseus (pomdp_perseus_cpu.cpp)
// ===========================================================================

static PerseusCpuWorkspace *perseus_cpu_ws(const POMDPPerseusCPU *per) {
    std::lock_guard<std::mutex> lock(registry_mutex());
    return find_workspace<PerseusCpuWorkspace>(per);
}

extern "C" int pomdp_perseus_uninitialize_cpu(const POMDP *pomdp, POMDPPerseusCPU *per) {
    (void)pomdp;
    if (per == nullptr) {
        NOVA_ERR("pomdp_perseus_uninitialize_cpu", "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    {
        std::lock_guard<std::mutex> lock(registry_mutex());
        registry().erase(per);
    }
    // pomdp_perseus_cpu.cpp:273-309
    per->currentHorizon = 0;
    delete[] per->Gamma; per->Gamma = nullptr; per->rGamma = 0;
    delete[] per->GammaPrime; per->GammaPrime = nullptr; per->rGammaPrime = 0;
    delete[] per->pi; per->pi = nullptr;
    delete[] per->piPrime; per->piPrime = nullptr;
    delete[] per->BTilde; per->BTilde = nullptr; per->rTilde = 0;
    return NOVA_SUCCESS;
}

extern "C" int pomdp_perseus_initialize_cpu(const POMDP *pomdp, POMDPPerseusCPU *per) {
    static const char *fn = "pomdp_perseus_initialize_cpu";
    if (pomdp == nullptr || per == nullptr || pomdp->n == 0 || pomdp->r == 0 || per->GammaInitial == nullptr) {
        NOVA_ERR(fn, "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    {
        std::lock_guard<std::mutex> lock(registry_mutex());
        registry().erase(per);
    }
    const size_t rn = (size_t)pomdp->r * pomdp->n;
    // Host arrays of pomdp_perseus_cpu.cpp:183-219.
    per->currentHorizon = 0;
    per->Gamma = new float[rn];
    per->GammaPrime = new float[rn];
    per->pi = new unsigned int[pomdp->r];
    per->piPrime = new unsigned int[pomdp->r];
    memcpy(per->Gamma, per->GammaInitial, rn * sizeof(float));
    memcpy(per->GammaPrime, per->GammaInitial, rn * sizeof(float));
    for (unsigned i = 0; i < pomdp->r; i++) { per->pi[i] = 0; per->piPrime[i] = 0; }
    per->rGamma = 0;
    per->rGammaPrime = 0;
    per->rTilde = pomdp->r;
    per->BTilde = new unsigned int[pomdp->r];
    for (unsigned i = 0; i < pomdp->r; i++) per->BTilde[i] = i;
    std::unique_ptr<PerseusCpuWorkspace> ws(new PerseusCpuWorkspace());
    std::lock_guard<std::mutex> lock(registry_mutex());
    registry()[per] = std::move(ws);
    return NOVA_SUCCESS;
}

// Model and solver arrays are uploaded at the first update; afterwards the
// device copies are authoritative and each update writes the one new alpha
// row and action back into the host arrays.
static int perseus_cpu_prepare(PerseusCpuWorkspace *ws, const POMDP *p, POMDPPerseusCPU *per, const char *fn) {
    if (ws->core.built) return NOVA_SUCCESS;
    if (p->S == nullptr || p->T == nullptr || p->O == nullptr || p->R == nullptr || p->Z == nullptr ||
            p->B == nullptr) {
        NOVA_ERR(fn, "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    const size_t nms = (size_t)p->n * p->m * p->ns, mnz = (size_t)p->m * p->n * p->z, nm = (size_t)p->n * p->m,
                 rrz = (size_t)p->r * p->rz, rn = (size_t)p->r * p->n;
    int rc;
    ws->arena.add(&ws->S, nms);
    ws->arena.add(&ws->T, nms);
    ws->arena.add(&ws->O, mnz);
    ws->arena.add(&ws->R, nm);
    ws->arena.add(&ws->Z, rrz);
    ws->arena.add(&ws->B, rrz);
    ws->arena.add(&ws->Gamma, rn);
    ws->arena.add(&ws->GammaPrime, rn);
    ws->arena.add(&ws->pi, p->r);
    ws->arena.add(&ws->piPrime, p->r);
    if ((rc = ws->arena.commit(fn, "the model and the alpha sets")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws->S, p->S, nms * sizeof(int), fn, "the successor states")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws->T, p->T, nms * sizeof(float), fn, "the state transitions")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws->O, p->O, mnz * sizeof(float), fn, "the observation transitions")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws->R, p->R, nm * sizeof(float), fn, "the rewards")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws->Z, p->Z, rrz * sizeof(int), fn, "the non-zero belief states")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws->B, p->B, rrz * sizeof(float), fn, "the belief points")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws->Gamma, per->Gamma, rn * sizeof(float), fn, "Gamma")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws->GammaPrime, per->GammaPrime, rn * sizeof(float), fn, "Gamma (prime)")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws->pi, per->pi, p->r * sizeof(unsigned), fn, "pi")) != NOVA_SUCCESS) return rc;
    if ((rc = h2d(ws->piPrime, per->piPrime, p->r * sizeof(unsigned), fn, "pi (prime)")) != NOVA_SUCCESS) return rc;
    DevModel md;
    md.n = p->n; md.ns = p->ns; md.m = p->m; md.z = p->z; md.r = p->r; md.rz = p->rz; md.gamma = p->gamma;
    md.S = ws->S; md.T = ws->T; md.O = ws->O; md.R = ws->R; md.Z = ws->Z; md.B = ws->B;
    return ws->core.build(md, fn);
}

extern "C" int pomdp_perseus_update_cpu(const POMDP *pomdp, POMDPPerseusCPU *per) {
    static const char *fn = "pomdp_perseus_update_cpu";
    if (perseus_shape_invalid(pomdp) || per == nullptr || per->Gamma == nullptr || per->GammaPrime == nullptr ||
            per->pi == nullptr || per->piPrime == nullptr || per->BTilde == nullptr) {
        NOVA_ERR(fn, "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    PerseusCpuWorkspace *ws = perseus_cpu_ws(per);
    if (ws == nullptr) {
        NOVA_ERR(fn, "The solver is not initialized (call pomdp_perseus_initialize_cpu).");
        return NOVA_ERROR_INVALID_DATA;
    }
    int rc = perseus_cpu_prepare(ws, pomdp, per, fn);
    if (rc != NOVA_SUCCESS) return rc;
    const bool even = (per->currentHorizon % 2u) == 0u;
    unsigned slot = 0;
    float *hostGp = even ? per->GammaPrime : per->Gamma;
    unsigned *hostPiP = even ? per->piPrime : per->pi;
    float *devGp = even ? ws->GammaPrime : ws->Gamma;
    unsigned *devPiP = even ? ws->piPrime : ws->pi;
    if (even)
        rc = ws->core.update(ws->Gamma, ws->pi, ws->GammaPrime, ws->piPrime, per->currentHorizon, per->rGamma,
                             per->rGammaPrime, per->rTilde, per->BTilde, &slot, fn);
    else
        rc = ws->core.update(ws->GammaPrime, ws->piPrime, ws->Gamma, ws->pi, per->currentHorizon, per->rGammaPrime,
                             per->rGamma, per->rTilde, per->BTilde, &slot, fn);
    if (rc != NOVA_SUCCESS && rc != NOVA_CONVERGED) return rc;
    const int rc2 = d2h(hostGp + (size_t)slot * pomdp->n, devGp + (size_t)slot * pomdp->n, pomdp->n * sizeof(float),
                        fn, "Gamma (prime)");
    if (rc2 != NOVA_SUCCESS) return rc2;
    const int rc3 = d2h(hostPiP + slot, devPiP + slot, sizeof(unsigned), fn, "pi (prime)");
    if (rc3 != NOVA_SUCCESS) return rc3;
    return rc;
}

extern "C" int pomdp_perseus_get_policy_cpu(const POMDP *pomdp, POMDPPerseusCPU *per, POMDPAlphaVectors *policy) {
    static const char *fn = "pomdp_perseus_get_policy_cpu";
    if (pomdp == nullptr || per == nullptr || policy == nullptr) {
        NOVA_ERR(fn, "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    const bool even = (per->currentHorizon % 2u) == 0u;
    const unsigned rows = even ? per->rGamma : per->rGammaPrime;
    if (pomdp_alpha_vectors_initialize(policy, pomdp->n, pomdp->m, rows) != NOVA_SUCCESS) {
        NOVA_ERR(fn, "Could not create the policy.");
        return NOVA_ERROR_POLICY_CREATION;
    }
    memcpy(policy->Gamma, even ? per->Gamma : per->GammaPrime, (size_t)rows * pomdp->n * sizeof(float));
    memcpy(policy->pi, even ? per->pi : per->piPrime, rows * sizeof(unsigned));
    return NOVA_SUCCESS;
}

extern "C" int pomdp_perseus_execute_cpu(const POMDP *pomdp, POMDPPerseusCPU *per, POMDPAlphaVectors *policy) {
    static const char *fn = "pomdp_perseus_execute_cpu";
    if (perseus_shape_invalid(pomdp) || pomdp->S == nullptr || pomdp->T == nullptr || pomdp->O == nullptr ||
            pomdp->R == nullptr || pomdp->Z == nullptr || pomdp->B == nullptr || per == nullptr ||
            per->GammaInitial == nullptr || policy == nullptr) {
        NOVA_ERR(fn, "Invalid arguments.");
        return NOVA_ERROR_INVALID_DATA;
    }
    int rc = pomdp_perseus_initialize_cpu(pomdp, per);
    if (rc != NOVA_SUCCESS) return rc;
    while (per->currentHorizon < pomdp->horizon) {
        rc = NOVA_SUCCESS;
        while (rc != NOVA_CONVERGED) {
            rc = pomdp_perseus_update_cpu(pomdp, per);
            if (rc != NOVA_CONVERGED && rc != NOVA_SUCCESS) return rc;
        }
    }
    rc = pomdp_perseus_get_policy_cpu(pomdp, per, policy);
    if (rc != NOVA_SUCCESS) return rc;
    return pomdp_perseus_uninitialize_cpu(pomdp, per);
}

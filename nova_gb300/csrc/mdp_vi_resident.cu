// nova-gb300: all sweeps of a value-iteration solve in one launch, for models
// that fit in the SMs' shared memory.
//
// A sweep of a small or middling model is mostly latency: a launch, the loads
// of S and T, the gathers of V, the residual's atomics (6.3 us for 300 rows,
// 12.7 us for 120,000 with ten successors). Here every SM keeps the successor
// entries of its states, {state, fl(gamma * T)}, in shared memory for the whole
// solve (152 SMs hold about 3.9 M entries), and a sweep is the gathers of V,
// the action scan and one barrier across the grid: 300 rows take 2.2 us, 120,000
// rows of ten 5.1 us. V is read past L1, which would keep the values of two
// sweeps before, or copied into shared memory first where that moves less. Where
// its gathers are the slower ones the ordinary sweeps run (vi_resident_sweeps).
//
// Order of operations as mdp_vi_cpu.cpp:36-63: Q = R(s,a), then Q += (gamma *
// T) * V[s'] in list order up to the row's first negative entry, gamma * T
// rounded first (here once); actions scanned in order with a strict '>'.
//
// The launch is cooperative, so all of its blocks are resident; a barrier wait
// is bounded (about 2 s), raises the state's error word when it runs out, and
// ends the block, as it does where another block's wait ran out.

#include "vi.h"

#include <algorithm>
#include <cstddef>

#include <nova/nova_gb300.h>

using nova::MDP;

namespace nova_gb300 {

namespace {

constexpr unsigned kMaxThreads = 1024;
constexpr unsigned kBatch = 8;                    // successors whose values are in flight together
constexpr unsigned kSweepsPerLaunch = 4096;
constexpr long long kWaitCycles = 4000000000ll;   // ~2 s at 2 GHz
// Models whose V does not fit beside their entries (vi_resident_sweeps).
constexpr unsigned long long kGatherSmem = 196 * 1024, kL1Entries = 2000000;
constexpr unsigned kL1States = 52000;

// One arrival per block; returns once `target` blocks have arrived in this
// launch, or false if a wait ran out here or elsewhere.
__device__ __forceinline__ bool grid_barrier(ViDeviceState *st, unsigned target, int *abortFlag) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&st->arrived, 1u);
        const long long t0 = clock64();
        while (*(volatile unsigned *)&st->arrived < target) {
            if (*(volatile unsigned *)&st->err != 0u || clock64() - t0 > kWaitCycles) {
                atomicExch(&st->err, 1u);
                *abortFlag = 1;
                break;
            }
        }
        __threadfence();
    }
    __syncthreads();
    return *abortFlag == 0;
}

template <bool kShared>
__global__ void __launch_bounds__(kMaxThreads, 1) vi_resident_kernel(
        unsigned n, unsigned m, unsigned ns, float gamma, unsigned statesPerBlock, unsigned pitch,
        const int *__restrict__ S, const float *__restrict__ T, const float *__restrict__ R, float *Va, float *Vb,
        unsigned *__restrict__ pi, ViDeviceState *st, unsigned sweeps, double tol, int early_exit) {
    extern __shared__ __align__(16) unsigned char residentShared[];
    uint2 *rec = reinterpret_cast<uint2 *>(residentShared);              // [ns][pitch]
    float *Q = reinterpret_cast<float *>(rec + (size_t)ns * pitch);      // [pitch]
    float *sV = Q + pitch;                                               // [n] (kShared)
    __shared__ int abortFlag;
    __shared__ double red[32];
    if (threadIdx.x == 0) abortFlag = 0;
    const unsigned s0 = blockIdx.x * statesPerBlock, states = min(statesPerBlock, n - s0), rows = states * m;
    const size_t first = (size_t)s0 * m * ns;
    for (unsigned e = threadIdx.x; e < rows * ns; e += blockDim.x) {
        const unsigned row = e / ns, l = e % ns;
        // (A state out of range is the model's fault; it reads the last one.)
        const int sp = min(__ldg(S + first + e), (int)(n - 1));
        rec[(size_t)l * pitch + row] = make_uint2((unsigned)sp, __float_as_uint(fmul(gamma, __ldg(T + first + e))));
    }
    __syncthreads();
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned ran = 0;
    double residual = 0.0;
    bool converged = false;
    for (unsigned k = 0; k < sweeps; k++) {
        const float *V = k % 2 == 0 ? Va : Vb;
        float *Vp = k % 2 == 0 ? Vb : Va;
        if constexpr (kShared) {
            const unsigned body = ((uintptr_t)V % 16u) == 0u ? n & ~3u : 0u;
#pragma unroll 4
            for (unsigned s = threadIdx.x * 4; s < body; s += blockDim.x * 4)
                *reinterpret_cast<float4 *>(sV + s) = __ldcg(reinterpret_cast<const float4 *>(V + s));
            for (unsigned s = body + threadIdx.x; s < n; s += blockDim.x) sV[s] = __ldcg(V + s);
            __syncthreads();
        }
        auto value = [&](unsigned s) { return kShared ? sV[s] : __ldcg(V + s); };
        for (unsigned row = threadIdx.x; row < rows; row += blockDim.x) {
            float q = __ldg(R + (size_t)s0 * m + row);
            const uint2 *p = rec + row;
            for (unsigned l0 = 0; l0 < ns; l0 += kBatch) {
                uint2 e[kBatch];
                float v[kBatch];
                bool live[kBatch];
#pragma unroll
                for (unsigned b = 0; b < kBatch; b++)
                    e[b] = l0 + b < ns ? p[(size_t)(l0 + b) * pitch] : make_uint2(0xffffffffu, 0u);
#pragma unroll
                for (unsigned b = 0; b < kBatch; b++) {
                    live[b] = (b == 0 || live[b - 1]) && (int)e[b].x >= 0;
                    v[b] = live[b] ? value(e[b].x) : 0.0f;
                }
#pragma unroll
                for (unsigned b = 0; b < kBatch; b++)
                    if (live[b]) q = fadd(q, fmul(__uint_as_float(e[b].y), v[b]));
                if (!live[kBatch - 1]) break;
            }
            Q[row] = q;
        }
        __syncthreads();
        double local = 0.0;
        for (unsigned i = threadIdx.x; i < states; i += blockDim.x) {
            const float *qs = Q + (size_t)i * m;
            float best = qs[0];
            unsigned besta = 0;
            for (unsigned a = 1; a < m; a++)
                if (qs[a] > best) { best = qs[a]; besta = a; }
            Vp[s0 + i] = best;
            pi[s0 + i] = besta;
            if (early_exit) local = fmax(local, fabs((double)best - (double)value(s0 + i)));
        }
        if (early_exit) {
            for (int off = 16; off > 0; off >>= 1) local = fmax(local, __shfl_xor_sync(0xffffffffu, local, off));
            if (lane == 0) red[warp] = local;
            __syncthreads();
            if (threadIdx.x == 0) {
                for (unsigned w = 1; w < (blockDim.x + 31) / 32; w++) local = fmax(local, red[w]);
                // Three slots in turn: this sweep's, the next one's (cleared
                // two barriers before its first use) and the last one's.
                atomicMax(&st->resid[k % 3], (unsigned long long)__double_as_longlong(local));
            }
        }
        if (!grid_barrier(st, (k + 1) * gridDim.x, &abortFlag)) return;
        ran = k + 1;
        if (early_exit) {
            residual = __longlong_as_double((long long)*(volatile unsigned long long *)&st->resid[k % 3]);
            if (blockIdx.x == 0 && threadIdx.x == 0) st->resid[(k + 2) % 3] = 0ull;
            converged = residual < tol;
            if (converged) break;
        }
    }
    if (early_exit && blockIdx.x == 0 && threadIdx.x == 0) {
        st->last_resid = residual;
        st->sweeps_done += ran;
        if (converged) st->converged = 1u;
    }
}

}  // namespace

int vi_resident_sweeps(const MDP *mdp, const int *S, const float *T, const float *R, float *V, float *Vp,
                       unsigned *pi, ViDeviceState *st, unsigned sweeps, double tol, int early_exit, unsigned *done,
                       cudaStream_t stream, const char *fn) {
    *done = 0;
    const unsigned n = mdp->n, m = mdp->m, ns = mdp->ns;
    // A single sweep gains nothing from staying; a forced tiling setting asks
    // for the sweep kernels it names.
    if (sweeps < 2 || vi_tiling_forced() || n == 0 || m == 0 || ns == 0) return NOVA_SUCCESS;
    int dev = 0, sms = 0, optin = 0, coop = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess || !coop) {
        cudaGetLastError();
        return NOVA_SUCCESS;
    }
    // A block per 1,024 rows, up to one per SM; then as many states as that
    // leaves each.
    const unsigned long long allRows = (unsigned long long)n * m;
    const unsigned want = (unsigned)std::min<unsigned long long>(sms, (allRows + kMaxThreads - 1) / kMaxThreads);
    const unsigned statesPerBlock = ceil_div(n, want);
    const unsigned grid = ceil_div(n, statesPerBlock);
    const unsigned long long rows = (unsigned long long)statesPerBlock * m;
    const unsigned long long pitch = (rows + 31) / 32 * 32;
    const unsigned long long base = pitch * ns * sizeof(uint2) + pitch * sizeof(float), reserve = 1024;
    if (base + reserve > (unsigned long long)optin) return NOVA_SUCCESS;
    // A gather moves a 32-byte sector, a copied value 4 bytes (n = 20,000, m =
    // 6, ns = 10, 7,900 gathers a block: 5.1 us a sweep copied, 10.2 gathered).
    const bool shared = base + n * sizeof(float) + reserve <= (unsigned long long)optin && n <= 4 * rows * ns;
    // Gathering pays while the SM keeps 60 KB of L1 for the loads in flight (up to
    // 196 KB of shared memory; us a sweep, resident and plain: 3.3 M entries 14 to
    // 19 and 17 to 24, 3.8 M 26 and 22), and against plain sweeps whose gathers
    // hit L1 only for fewer entries (n = 30,000 to 40,000: 1.3 M 9.5 and 13, 2.8 M
    // 20 and 15; n = 58,000, 2.8 M 16 and 16).
    if (!shared && (base + reserve > kGatherSmem || (n < kL1States && allRows * ns > kL1Entries))) return NOVA_SUCCESS;
    const size_t smem = (size_t)(base + (shared ? n * sizeof(float) : 0));
    const unsigned threads = (unsigned)std::min<unsigned long long>(kMaxThreads, std::max<unsigned long long>(128, pitch));
    const void *kernel = shared ? (const void *)vi_resident_kernel<true> : (const void *)vi_resident_kernel<false>;
    if (!allow_dynamic_smem(kernel, smem)) return NOVA_SUCCESS;
    unsigned un = n, um = m, uns = ns, usp = statesPerBlock, upitch = (unsigned)pitch;
    float gamma = mdp->gamma;
    for (unsigned k = 0; k < sweeps;) {
        // An even number of sweeps per launch keeps V the source of the next.
        unsigned count = std::min(sweeps - k, kSweepsPerLaunch);
        if (cudaMemsetAsync(&st->resid, 0, sizeof(ViDeviceState) - offsetof(ViDeviceState, resid), stream) !=
                cudaSuccess) {
            cudaGetLastError();
            NOVA_ERR(fn, "Failed to clear the sweep barrier.");
            return NOVA_ERROR_KERNEL_EXECUTION;
        }
        void *args[] = {&un, &um, &uns, &gamma, &usp, &upitch, &S, &T, &R, &V, &Vp, &pi, &st, &count, &tol, &early_exit};
        if (cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(threads), args, smem, stream) != cudaSuccess) {
            cudaGetLastError();
            if (k == 0) return NOVA_SUCCESS;  // the sweep kernels take over
            NOVA_ERR(fn, "Failed to launch the resident sweeps.");
            return NOVA_ERROR_KERNEL_EXECUTION;
        }
        const int rc = check_launch(fn, "Bellman update (resident)");
        if (rc != NOVA_SUCCESS) return rc;
        k += count;
        if (early_exit && k < sweeps) {
            ViDeviceState h;
            const int rd = d2h(&h, st, sizeof(h), fn, "the convergence state");
            if (rd != NOVA_SUCCESS) return rd;
            if (h.converged != 0 || h.err != 0) break;
        }
    }
    *done = sweeps;
    vi_note_gather();
    return NOVA_SUCCESS;
}

}  // namespace nova_gb300

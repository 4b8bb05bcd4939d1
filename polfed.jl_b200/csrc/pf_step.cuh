// pf_step.cuh -- what the step-kernel files share: the launch arguments, the
// fused-dot epilogue, the launch itself.
#pragma once
#include <utility>

#include "pf_internal.h"
#include "pf_rows.cuh"

namespace pf {

template <typename T>
struct StepArgs {
    uint32_t D;
    int s;          // columns processed per row
    int ld;         // row stride of the blocks (>= s: a column slab of a wider RI block)
    int stream;     // 1: x, p and out move with evict-first hints (slab passes)
    int G;          // column groups per row = s / V
    uint32_t items; // D * G
    const T *q;
    const T *p;     // may alias out (in-place update)
    const T *x;
    T *out;
    T cx, alpha, beta, inva, boa;
    double *partials;
    unsigned int *counter;
    double *dots;
};

constexpr int kThreads = 256;

// Deterministic "last block reduces" epilogue: every block writes its
// per-column partials, the block that finishes last sums them: each value over
// a number of strided runs fixed by the grid (of sixteen partials or more, and
// no more than the block has threads for), a run's loads sixteen in flight, then
// the runs in order.  The partials are read
// through L2 (__ldcg: other blocks wrote them before the counter told this
// block it is last).  With one run of eight loads in flight the tail took 20 us
// for 444 blocks of 128 values; as many runs as threads, whatever the grid, take
// longer to sum than to read (steps of 313 blocks, 2 values: 11.2 -> 10.1 us a
// step; of 1444 blocks, 8 values: 24.8 -> 21.8).  One block has nothing to sum:
// 6.9 -> 4.2 us a step of 32 rows.  runs: blockDim.x doubles of shared memory
// that blockvals does not overlap.
static __device__ void finish_reduction(int nvals, const double *blockvals, double *partials, unsigned int *counter,
                                        double *out, double *runs) {
    __shared__ bool last;
    if (gridDim.x == 1) {
        for (int c = threadIdx.x; c < nvals; c += blockDim.x) out[c] = blockvals[c];
        return;
    }
    for (int c = threadIdx.x; c < nvals; c += blockDim.x)
        partials[(size_t)blockIdx.x * nvals + c] = blockvals[c];
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int t = atomicAdd(counter, 1u);
        last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (last) {
        __threadfence();
        const unsigned int nb = gridDim.x;
        const int Q = max(1, min((int)blockDim.x / nvals, (int)((nb + 15) / 16)));
        for (int w = threadIdx.x; w < Q * nvals; w += blockDim.x) {
            const int c = w % nvals, q = w / nvals;
            double acc = 0.0;
            const double *col = partials + c;
            for (unsigned int b = q; b < nb; b += 16 * Q) {
                double x[16];
#pragma unroll
                for (int u = 0; u < 16; ++u) x[u] = b + u * Q < nb ? __ldcg(col + (size_t)(b + u * Q) * nvals) : 0.0;
#pragma unroll
                for (int u = 0; u < 16; ++u) acc += x[u];
            }
            if (Q == 1) out[c] = acc;
            else runs[w] = acc;
        }
        if (Q > 1) {
            __syncthreads();
            for (int c = threadIdx.x; c < nvals; c += blockDim.x) {
                double acc = 0.0;
                for (int q = 0; q < Q; ++q) acc += runs[q * nvals + c];
                out[c] = acc;
            }
        }
        if (threadIdx.x == 0) *counter = 0u;
    }
}

// Bytes of shared memory step_dots needs.
__host__ __device__ inline int step_dots_smem(int G, int V, int s) {
    const int lanes = G < 32 ? G : 32;
    return (kThreads / 32) * lanes * 2 * V * 8 + 2 * s * 8 + kThreads * 8;
}

// Per-column sums of dd1 and dd2 over the grid into dots[0 .. s) and dots[s .. 2 s).
// Every item of a thread has column group threadIdx.x % G (G divides the grid
// stride; checked on the host).  Lanes of one group are first summed with warp
// shuffles, then per warp in shared memory.
template <int V>
__device__ __forceinline__ void step_dots(double (&dd1)[V], double (&dd2)[V], int G, int s, unsigned char *smem_raw,
                                          double *partials, unsigned int *counter, double *dots) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (G < 32) {
#pragma unroll
        for (int v = 0; v < V; ++v)
            for (int o = 16; o >= G; o >>= 1) {
                dd1[v] += __shfl_xor_sync(0xffffffffu, dd1[v], o);
                dd2[v] += __shfl_xor_sync(0xffffffffu, dd2[v], o);
            }
    }
    const int lanes = G < 32 ? G : 32;
    __syncthreads();
    double *red = reinterpret_cast<double *>(smem_raw);  // [8 warps][lanes][2V]
    if (lane < lanes)
        for (int v = 0; v < V; ++v) {
            red[(warp * lanes + lane) * 2 * V + v] = dd1[v];
            red[(warp * lanes + lane) * 2 * V + V + v] = dd2[v];
        }
    __syncthreads();
    double *bv = red + (kThreads / 32) * lanes * 2 * V;  // [2 s]
    for (int c = threadIdx.x; c < s; c += blockDim.x) {
        const int g = c / V, v = c - g * V;
        double s1 = 0.0, s2 = 0.0;
        if (G < 32) {
            for (int w = 0; w < kThreads / 32; ++w) {
                s1 += red[(w * lanes + g) * 2 * V + v];
                s2 += red[(w * lanes + g) * 2 * V + V + v];
            }
        } else {
            for (int t = g; t < kThreads; t += G) {
                const int w = t >> 5, l = t & 31;
                s1 += red[(w * lanes + l) * 2 * V + v];
                s2 += red[(w * lanes + l) * 2 * V + V + v];
            }
        }
        bv[c] = s1;
        bv[s + c] = s2;
    }
    __syncthreads();
    finish_reduction(2 * s, bv, partials, counter, dots, bv + 2 * s);
}

// Launches a step kernel on st, with programmatic dependent launch when the
// handle allows it (the kernels wait for their predecessor themselves).
template <typename... KArgs, typename... Args>
static void launch_step_kernel(pf_handle *h, void (*kern)(KArgs...), int grid, int smem, cudaStream_t st,
                               Args &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = h->overlap ? 1 : 0;
    PF_CUDA(cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...));
}

// Resident CTAs per SM of a kernel instance (cached per host thread), and whether it spills registers.
int step_blocks_per_sm(const void *kern, int smem);
bool step_spills(const void *kern);

}  // namespace pf

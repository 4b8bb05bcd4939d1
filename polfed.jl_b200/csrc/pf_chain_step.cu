// pf_chain_step.cu -- spin-chain steps from a list of every row's flips.
//
// The chain step of pf_kernels.cu ranks a row's flipped states anew in every
// step and, with a narrow thread, in every one of the row's threads (61 % issue
// on the J1-J2 L = 20 chain, 64 columns FP32); with a 64-byte thread every load
// instruction touches 32 rows and the L1 data pipe is full (73 %, L = 22, s = 16
// FP32, DRAM at 12 %).  A filter, a KPM run or a Lanczos probe takes hundreds of
// steps of one operator, so here the flips are ranked once, into a list of 4
// bytes a flip; a step reads its row's chunk of the list (the lanes of a row
// broadcast it), has the next chunk on its way, and gathers 16 bytes a lane with
// eight rows in flight, so a load instruction reads whole row segments.  That
// runs at the rate at which L2 serves gathered rows (7.5 - 9.5 TB/s; 8.1
// measured for random rows).  us a step, best tuned step -> here: J1-J2 L = 24
// s = 16 FP32 736 -> 553, FP64 1248 -> 1000; L = 20 64 columns FP32 116 -> 104;
// XXZ L = 20 s = 1 FP64 17.2 -> 7.2, s = 8 30.2 -> 16.2; L = 16 s = 3 9.8 -> 3.9.
// The list costs about one step to make and is read once a step, a sixteenth of
// the gathered bytes at 64-byte rows.
//
// Gathers are added in bond order and the diagonal comes from k_chain_diag: the
// same bits as the step of pf_kernels.cu.
#include <algorithm>

#include "pf_step.cuh"

namespace pf {

template <typename T>
struct ChainCoef {
    T jhalf[PF_MAX_BONDS];
};

template <typename T>
static const ChainDesc<T> &desc_of(const pf_op *op);
template <>
const ChainDesc<double> &desc_of<double>(const pf_op *op) { return op->chain64; }
template <>
const ChainDesc<float> &desc_of<float>(const pf_op *op) { return op->chain32; }

// The flips of every row in bond order, four 32-bit entries to a chunk: chunk k
// of row i at k * D + i.  An entry is the flipped state's index (26 bits) and
// the bond; a row ends with kListEnd, which also fills its last chunk.
constexpr uint32_t kListEnd = 0xffffffffu;

__global__ void __launch_bounds__(kThreads) k_chain_list(const __grid_constant__ ChainDesc<double> d, uint32_t D,
                                                        uint4 *__restrict__ out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint32_t *tab = reinterpret_cast<uint32_t *>(smem_raw);
    if (!d.full) {
        const int n = rank_table_entries(d.nchunks);
        for (int i = threadIdx.x; i < n; i += kThreads) tab[i] = __ldg(d.rank_tab + i);
        __syncthreads();
    }
    for (uint32_t row = blockIdx.x * kThreads + threadIdx.x; row < D; row += gridDim.x * kThreads) {
        const uint32_t st = d.full ? row : __ldg(d.states + row);
        uint32_t e[4];
        int n = 0;
        size_t at = row;
        for (int b = 0; b <= d.nb; ++b) {
            uint32_t v = kListEnd;
            if (b < d.nb) {
                const uint32_t m = st & d.bmask[b];
                if (m == 0u || m == d.bmask[b]) continue;
                const uint32_t st2 = st ^ d.bmask[b];
                v = (d.full ? st2 : sector_rank(st2, tab, d.nchunks)) | ((uint32_t)b << 26);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (u == n || (b == d.nb && u > n)) e[u] = v;
            if (++n == 4 || b == d.nb) {
                out[at] = make_uint4(e[0], e[1], e[2], e[3]);
                at += D;
                n = 0;
            }
        }
    }
}

// One row segment of V columns (up to 16 bytes) per thread, neighbouring
// threads neighbouring segments.
template <typename T, int V, int FLAGS>
__global__ void __launch_bounds__(kThreads, 3)
    k_step_chain_list(const uint4 *__restrict__ ent, const T *__restrict__ diag, const __grid_constant__ ChainCoef<T> c,
                      const StepArgs<T> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    pdl_trigger();
    constexpr bool HASP = (FLAGS & StepFlags::P) != 0;
    constexpr bool HASX = (FLAGS & StepFlags::X) != 0;
    constexpr bool DOTS = (FLAGS & StepFlags::DOTS) != 0;
    T *sjh = reinterpret_cast<T *>(smem_raw);
    for (int i = threadIdx.x; i < PF_MAX_BONDS; i += kThreads) sjh[i] = c.jhalf[i];
    __syncthreads();
    pdl_wait();
    double dd1[V], dd2[V];
#pragma unroll
    for (int v = 0; v < V; ++v) dd1[v] = dd2[v] = 0.0;
    const uint32_t G = (uint32_t)a.G, stride = gridDim.x * kThreads;
    for (uint32_t it = blockIdx.x * kThreads + threadIdx.x; it < a.items; it += stride) {
        const uint32_t row = G == 1u ? it : it / G;
        const int c0 = G == 1u ? 0 : (int)(it - row * G) * V;
        const size_t off = (size_t)row * a.ld + c0;
        const T *qc = a.q + c0;
        Pack<T, V> xo, qo, po, res;
#pragma unroll
        for (int v = 0; v < V; ++v) xo.v[v] = po.v[v] = T(0);
        const uint4 *w = ent + row;
        uint4 e0 = __ldg(w), e1 = make_uint4(kListEnd, kListEnd, kListEnd, kListEnd);
        if (e0.w != kListEnd) e1 = __ldg(w + a.D);
        if constexpr (HASX) xo = ldp_hint<T, V>(a.x + off, a.stream);
        qo = ldp<T, V>(a.q + off);
        if constexpr (HASP) po = ldp_hint<T, V>(a.p + off, a.stream);
        const T dg = __ldg(diag + row);
        T acc[V];
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] = T(0);
        while (e0.x != kListEnd) {
            const uint32_t e[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
            Pack<T, V> g[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (e[u] != kListEnd) g[u] = ldp<T, V>(qc + (size_t)(e[u] & 0x3ffffffu) * a.ld);
            // the next two chunks, while the gathers are on their way
            e0.x = kListEnd;
            if (e[7] != kListEnd) {
                w += 2 * (size_t)a.D;
                e0 = __ldg(w);
                e1.x = e1.y = e1.z = e1.w = kListEnd;
                if (e0.w != kListEnd) e1 = __ldg(w + a.D);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (e[u] != kListEnd) {
                    const T cf = sjh[e[u] >> 26];
#pragma unroll
                    for (int v = 0; v < V; ++v) acc[v] = fma_t(cf, g[u].v[v], acc[v]);
                }
        }
#pragma unroll
        for (int v = 0; v < V; ++v)
            res.v[v] = step_combine<T>(HASX, true, HASP, a.cx, xo.v[v], a.alpha, acc[v], dg, qo.v[v], a.inva, a.boa, a.beta,
                                       po.v[v]);
        stp_hint<T, V>(a.out + off, res, a.stream);
        if constexpr (DOTS) {
#pragma unroll
            for (int v = 0; v < V; ++v) {
                dd1[v] += (double)res.v[v] * (double)res.v[v];
                dd2[v] += (double)res.v[v] * (double)qo.v[v];
            }
        }
    }
    if constexpr (DOTS) step_dots<V>(dd1, dd2, a.G, a.s, smem_raw, a.partials, a.counter, a.dots);
}

size_t chain_list_bytes(const pf_op *op) {
    if (op->kind != OP_CHAIN || op->chain64.diag == nullptr || op->chain32.diag == nullptr || op->chain64.nb < 1 ||
        op->dim >= (1 << 26))
        return 0;
    return (size_t)op->dim * (op->chain64.nb / 4 + 1) * sizeof(uint4);
}

void build_chain_list(pf_op *op, cudaStream_t st, void *list) {
    const ChainDesc<double> &d = op->chain64;
    const int smem = d.full ? 0 : rank_table_entries(d.nchunks) * 4;
    if (smem > 48 * 1024) PF_CUDA(cudaFuncSetAttribute(k_chain_list, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    k_chain_list<<<grid_for(op->h, op->dim, kThreads, 4), kThreads, smem, st>>>(d, (uint32_t)op->dim, static_cast<uint4 *>(list));
    PF_CUDA(cudaGetLastError());
    count_launches(1);
}

template <typename T, int V, int FLAGS>
static void launch_list_one(pf_op *op, cudaStream_t st, const void *list, StepArgs<T> a) {
    auto kern = k_step_chain_list<T, V, FLAGS>;
    const ChainDesc<T> &d = desc_of<T>(op);
    ChainCoef<T> c{};
    for (int b = 0; b < d.nb; ++b) c.jhalf[b] = d.jhalf[b];
    int smem = PF_MAX_BONDS * (int)sizeof(T);
    if constexpr ((FLAGS & StepFlags::DOTS) != 0) smem = std::max(smem, step_dots_smem(a.G, V, a.s));
    const int grid = grid_for(op->h, a.items, kThreads, step_blocks_per_sm((const void *)kern, smem));
    if constexpr ((FLAGS & StepFlags::DOTS) != 0) {
        ensure_reduction(op->h, (size_t)grid * 2 * a.s);
        a.partials = op->h->red_partials;
        a.counter = op->h->red_counter;
    }
    launch_step_kernel(op->h, kern, grid, smem, st, static_cast<const uint4 *>(list), d.diag, c, a);
    PF_CUDA(cudaGetLastError());
    count_launches(1);
}

template <typename T, int V>
static void launch_list_flags(pf_op *op, cudaStream_t st, const void *list, const StepArgs<T> &a, int flags) {
    using F = StepFlags;
    switch (flags) {
        case F::Q: launch_list_one<T, V, F::Q>(op, st, list, a); break;
        case F::Q | F::X: launch_list_one<T, V, F::Q | F::X>(op, st, list, a); break;
        case F::Q | F::P | F::X: launch_list_one<T, V, F::Q | F::P | F::X>(op, st, list, a); break;
        case F::Q | F::DOTS: launch_list_one<T, V, F::Q | F::DOTS>(op, st, list, a); break;
        case F::Q | F::P | F::DOTS: launch_list_one<T, V, F::Q | F::P | F::DOTS>(op, st, list, a); break;
        default: throw Error(PF_ERR_INVALID, "unsupported step flag combination");
    }
}

template <typename T>
void launch_chain_listed(pf_op *op, cudaStream_t st, const void *list, int s, const T *q, const T *p, const T *x, T *out,
                         double cx, double alpha, double beta, double inva, double shift, int flags, double *dots) {
    int V = 16 / (int)sizeof(T);
    while (s % V != 0) V /= 2;
    StepArgs<T> a;
    a.D = (uint32_t)op->dim;
    a.s = a.ld = s;
    a.stream = 0;
    a.G = s / V;
    PF_CHECK(op->dim * a.G < (int64_t)0xffffffffLL, PF_ERR_UNSUPPORTED, "block too large for one launch");
    PF_CHECK(!(flags & StepFlags::DOTS) || kThreads % a.G == 0, PF_ERR_UNSUPPORTED, "fused dots need s/V to divide 256");
    a.items = (uint32_t)(op->dim * a.G);
    a.q = q; a.p = p; a.x = x; a.out = out;
    a.cx = (T)cx; a.alpha = (T)alpha; a.beta = (T)beta;
    a.inva = (T)inva; a.boa = (T)(shift * inva);
    a.partials = nullptr; a.counter = nullptr; a.dots = dots;
    switch (V) {
        case 1: launch_list_flags<T, 1>(op, st, list, a, flags); break;
        case 2: launch_list_flags<T, 2>(op, st, list, a, flags); break;
        default:
            if constexpr (sizeof(T) == 4) launch_list_flags<T, 4>(op, st, list, a, flags);
    }
}
template void launch_chain_listed<double>(pf_op *, cudaStream_t, const void *, int, const double *, const double *,
                                          const double *, double *, double, double, double, double, double, int, double *);
template void launch_chain_listed<float>(pf_op *, cudaStream_t, const void *, int, const float *, const float *,
                                         const float *, float *, double, double, double, double, double, int, double *);

}  // namespace pf

// pf_cm_step.cu -- one step straight on column-major blocks.
//
// The operator-level calls (apply, recurrence, final sum) get column-major
// blocks.  Staged through row-interleaved copies, one recurrence is five
// launches that move its blocks three times (Quantum Sun 2^16, s = 8 FP64: 54 us
// with 15 us of host time).  Here a thread takes one row and up to four
// columns: the row's flips are found once, neighbouring threads read
// neighbouring rows of a column -- a spin flip maps runs of rows to runs of rows
// -- and nothing is copied.  Rows are summed in the step kernels' order with the
// same rounded operations: the same bits.
#include <algorithm>
#include <type_traits>

#include "pf_step.cuh"

namespace pf {

namespace {

template <typename T>
struct CmArgs {
    uint32_t D;
    int s;
    const T *q, *p, *x;
    T *out;
    int64_t ld, ldout;   // of q, p, x; of out
    T cx, alpha, beta, inva, boa;
};

// acc[c] += cf[u] * q[r[u]] of the thread's columns, u in order; on[u] false: left out.
template <typename T, int NC, int U>
__device__ __forceinline__ void cm_add(T (&acc)[NC], const T *__restrict__ q, int64_t ld, int nc, const uint32_t (&r)[U],
                                       const T (&cf)[U], const bool (&on)[U]) {
    T g[U][NC];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int c = 0; c < NC; ++c)
            if (on[u] && c < nc) g[u][c] = q[c * ld + r[u]];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int c = 0; c < NC; ++c)
            if (on[u] && c < nc) acc[c] = fma_t(cf[u], g[u][c], acc[c]);
}

}  // namespace

template <typename T, int NC, class Desc, bool REC>
__global__ void __launch_bounds__(kThreads) k_step_cm(const __grid_constant__ Desc d, const CmArgs<T> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int U = NC >= 4 ? 4 : 8;   // rows in flight
    const uint32_t *tab = reinterpret_cast<const uint32_t *>(smem_raw);
    if constexpr (std::is_same<Desc, ChainDesc<T>>::value) {
        if (!d.full) {
            uint32_t *t = reinterpret_cast<uint32_t *>(smem_raw);
            const int n = rank_table_entries(d.nchunks);
            for (int i = threadIdx.x; i < n; i += kThreads) t[i] = __ldg(d.rank_tab + i);
            __syncthreads();
        }
    }
    const int c0 = blockIdx.y * NC, nc = min(NC, a.s - c0);
    const T *q = a.q + c0 * a.ld;
    for (uint32_t row = blockIdx.x * kThreads + threadIdx.x; row < a.D; row += gridDim.x * kThreads) {
        T acc[NC], diag = T(0);
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[c] = T(0);
        uint32_t r[U];
        T cf[U];
        bool on[U];
        if constexpr (std::is_same<Desc, ChainDesc<T>>::value) {
            const uint32_t st = d.full ? row : __ldg(d.states + row);
            diag = __ldg(d.diag + row);
            uint64_t act = 0ull;
            for (int b = 0; b < d.nb; ++b) {
                const uint32_t m = st & d.bmask[b];
                if (m != 0u && m != d.bmask[b]) act |= 1ull << b;
            }
            while (act != 0ull) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    on[u] = act != 0ull;
                    r[u] = 0u;
                    cf[u] = T(0);
                    if (on[u]) {
                        const int b = __ffsll((long long)act) - 1;
                        act &= act - 1ull;
                        const uint32_t st2 = st ^ d.bmask[b];
                        r[u] = d.full ? st2 : sector_rank(st2, tab, d.nchunks);
                        cf[u] = d.jhalf[b];
                    }
                }
                cm_add<T, NC, U>(acc, q, a.ld, nc, r, cf, on);
            }
        } else if constexpr (std::is_same<Desc, QSunDesc<T>>::value) {
            diag = qsun_diag(d, row);
            for (int j0 = 0; j0 < d.L_loc; j0 += U) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    on[u] = j0 + u < d.L_loc;
                    r[u] = on[u] ? row ^ d.fmask[j0 + u] : 0u;
                    cf[u] = on[u] ? d.cflip[j0 + u] : T(0);
                }
                cm_add<T, NC, U>(acc, q, a.ld, nc, r, cf, on);
            }
            const uint32_t g = row & ((uint32_t)d.dg - 1u), base = row - g;
            for (int h0 = 0; h0 < d.dg; h0 += U) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    on[u] = h0 + u < d.dg;
                    r[u] = on[u] ? base + h0 + u : 0u;
                    cf[u] = on[u] ? d.grain[g * d.dg + h0 + u] : T(0);
                }
                cm_add<T, NC, U>(acc, q, a.ld, nc, r, cf, on);
            }
        } else {
            const int64_t b = __ldg(d.indptr + row), e = __ldg(d.indptr + row + 1);
            for (int64_t p0 = b; p0 < e; p0 += U) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    on[u] = p0 + u < e;
                    r[u] = on[u] ? (uint32_t)__ldg(d.indices + p0 + u) : 0u;
                    cf[u] = on[u] ? __ldg(d.values + p0 + u) : T(0);
                }
                cm_add<T, NC, U>(acc, q, a.ld, nc, r, cf, on);
            }
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            if (c >= nc) break;
            const int64_t at = (int64_t)(c0 + c) * a.ld + row;
            const T xo = REC ? a.x[at] : T(0), po = REC ? a.p[at] : T(0);
            a.out[(int64_t)(c0 + c) * a.ldout + row] =
                step_combine<T>(REC, true, REC, a.cx, xo, a.alpha, acc[c], diag, q[c * a.ld + row], a.inva, a.boa, a.beta, po);
        }
    }
}

template <typename T, int NC, class Desc>
static void launch_cm(pf_op *op, cudaStream_t st, const Desc &d, const CmArgs<T> &a, int smem) {
    auto kern = a.p ? k_step_cm<T, NC, Desc, true> : k_step_cm<T, NC, Desc, false>;
    if (smem > 48 * 1024) PF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    const int groups = (a.s + NC - 1) / NC;
    const dim3 grid((unsigned)grid_for(op->h, a.D, kThreads, std::max(1, 8 / groups)), (unsigned)groups);
    kern<<<grid, kThreads, smem, st>>>(d, a);
    PF_CUDA(cudaGetLastError());
    count_launches(1);
}

// Columns per thread.  Few rows: one, for more threads; else as many as share a row's flips at no loss.
static int cm_columns(int64_t D, int s) { return D * s <= 100000 ? 1 : s == 2 ? 2 : 4; }

template <typename T, class Desc>
static void launch_cm(pf_op *op, cudaStream_t st, const Desc &d, const CmArgs<T> &a, int smem) {
    switch (cm_columns(a.D, a.s)) {
        case 1: launch_cm<T, 1, Desc>(op, st, d, a, smem); break;
        case 2: launch_cm<T, 2, Desc>(op, st, d, a, smem); break;
        default: launch_cm<T, 4, Desc>(op, st, d, a, smem);
    }
}

template <typename T>
static void launch_cm(pf_op *op, cudaStream_t st, const ChainDesc<T> &ch, const QSunDesc<T> &qs, const CsrDesc<T> &cs,
                      const CmArgs<T> &a) {
    if (op->kind == OP_CHAIN) launch_cm<T>(op, st, ch, a, ch.full ? 0 : rank_table_entries(ch.nchunks) * 4);
    else if (op->kind == OP_QSUN) launch_cm<T>(op, st, qs, a, 0);
    else launch_cm<T>(op, st, cs, a, 0);
}

// Whether this form is at most as slow as copies and row gathers, whose gathers
// of wide blocks of many rows fill whole sectors only in the row-interleaved
// layout.  The lines lie where the two times, measured on a B200 over the widths
// 2 .. 64 and both types, cross.
//
// Chains: J1-J2 L = 22, s = 8 FP64 254 us staged, 355 here; XXZ L = 20, s = 3
// recurrence 115 and 57.
//
// Quantum Sun (2^6 .. 2^23 states), by the grain, whose dense block costs its
// rows' reads once a column: up to `narrow` columns at any size; up to `wide`
// columns, or any number, in blocks of so many elements.  Recurrences 2^16, s = 8
// FP64 55 us staged and 38 here; applies of a 4-site grain with 2^22 states, s =
// 16 FP32 996 staged, 2243 here.  An odd number of columns is staged one column
// a thread: here it is faster except for FP64 applies of a 4-site grain.
//
// CSR (200 to 1.5 million rows; chains, grids, bands, random columns): by the
// sectors gathered beyond the staged form's, those near the row at 0.3 (they
// mostly hit L1), against the copies: a number that pays for their launches, or
// one a row.  24310 rows of a chain, s = 8 recurrence 44 and 32 us; 50000 rows of
// 15 entries anywhere, s = 12 apply 46 and 72.
static bool cm_worth(const pf_op *op, int s, int elem, bool rec) {
    const double n = (double)op->dim * s;
    const int width = s * elem, fp32 = elem == 4;
    if (op->kind == OP_CHAIN) return width <= (rec ? 32 : 24) || n <= 400000;
    if (op->kind == OP_QSUN) {
        struct Lines { int narrow, wide; double wide_n, any_n; };
        static const Lines lines[2][2][3] = {   // apply, recurrence; FP64, FP32; grains of up to 2, of 3 and 4 sites
            {{{8, 8, 0, 1.6e6}, {4, 8, 4.3e6, 0.8e6}, {0, 4, 2.1e6, 0.27e6}},
             {{12, 16, 2.2e6, 1.1e6}, {6, 8, 17e6, 1.06e6}, {4, 4, 0, 0.3e6}}},
            {{{8, 8, 0, 1.6e6}, {8, 8, 0, 1.6e6}, {4, 8, 2.2e6, 0.8e6}},
             {{16, 16, 0, 1.6e6}, {12, 16, 8.4e6, 1.6e6}, {6, 8, 8.4e6, 0.8e6}}}};
        const int g = std::max(op->L_grain, 2) - 2;
        const Lines &l = lines[rec][fp32][g];
        if (s % 2 == 1 && (g < 2 || rec || fp32)) return width <= 64 || n <= 1.6e6;
        return s <= l.narrow || (s <= l.wide && n <= l.wide_n) || n <= l.any_n;
    }
    if (width > 32 && n > 600000) return false;
    static const double few[2][2] = {{1.2e6, 1.8e6}, {2.4e6, 3.0e6}}, per_row[2][2] = {{25, 30}, {42, 60}};
    const double load = op->shape.far[4] + 0.3 * (op->shape.sectors - op->shape.far[4]);
    return load * (s - 1) <= std::max(few[rec][fp32], per_row[rec][fp32] * (double)op->dim);
}

template <typename T>
bool launch_step_cm(pf_op *op, cudaStream_t st, int s, const T *q, const T *p, const T *x, T *out, int64_t ld,
                    int64_t ldout, double cx, double alpha, double beta, double inva, double shift) {
    const int64_t D = op->dim;
    if (s < 2 || (op->kind == OP_CHAIN && op->chain64.diag == nullptr)) return false;
    if ((s - 1) / cm_columns(D, s) >= 65535) return false;   // more blocks of columns than a grid's second dimension has
    if (!cm_worth(op, s, (int)sizeof(T), p != nullptr)) return false;
    // the output may be p or x itself (each element is read, then written, by
    // one thread), but not overlap q, or p or x at another place
    const size_t in = ((size_t)(s - 1) * ld + D) * sizeof(T), o = ((size_t)(s - 1) * ldout + D) * sizeof(T);
    if (overlap(out, o, q, in)) return false;
    for (const T *b : {p, x})
        if (b && overlap(out, o, b, in) && !(b == out && ld == ldout)) return false;
    CmArgs<T> a;
    a.D = (uint32_t)D;
    a.s = s;
    a.q = q; a.p = p; a.x = x; a.out = out;
    a.ld = ld; a.ldout = ldout;
    a.cx = (T)cx; a.alpha = (T)alpha; a.beta = (T)beta;
    a.inva = (T)inva; a.boa = (T)(shift * inva);
    if constexpr (sizeof(T) == 8) launch_cm<double>(op, st, op->chain64, op->qsun64, op->csr64, a);
    else launch_cm<float>(op, st, op->chain32, op->qsun32, op->csr32, a);
    return true;
}
template bool launch_step_cm<double>(pf_op *, cudaStream_t, int, const double *, const double *, const double *, double *,
                                     int64_t, int64_t, double, double, double, double, double);
template bool launch_step_cm<float>(pf_op *, cudaStream_t, int, const float *, const float *, const float *, float *,
                                    int64_t, int64_t, double, double, double, double, double);

}  // namespace pf

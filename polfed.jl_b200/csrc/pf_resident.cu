// pf_resident.cu -- whole recurrences on chip: a Chebyshev filter or a KPM
// recurrence in one launch, each column held in the shared memory of one
// thread-block cluster.
//
// A Clenshaw or KPM step reads a block at every neighbour of every row.  As one
// launch per step those reads go to L2 and a step costs a launch, a table
// set-up and a chain of dependent L2 round trips (measured on the Quantum Sun
// D = 65536, s = 8, FP64: 6.8-8.7 us a step, its gathers at the L2's own
// gather rate).  The columns of a block never mix, and one column of such an
// operator is small: here a cluster of 2^clog CTAs owns one column, each CTA a
// contiguous range of rows, and keeps b_{k+1} and b_{k+2} in its shared memory
// for all K steps.  Neighbours in the CTA's own range are shared-memory reads,
// the others distributed-shared-memory reads; a step ends in one cluster
// barrier; X and Y cross HBM once.
//
// What bounds it: shared-memory bandwidth in one CTA (the Quantum Sun D = 8192
// in one CTA: 4.9 us a step, 78 % of the 128 bytes a clock), reads of other
// CTAs' rows and the cluster barrier (about 500 clocks) on several.  Measured
// on a B200, us a step of all columns, step kernels -> here (FP64): Quantum Sun
// 2^11 s = 8 5.0 -> 1.6, 2^16 with 300 probes (KPM) 307 -> 151 for all; chain
// L = 14 s = 1 6.9 -> 1.7, L = 16 s = 8 10.3 -> 3.2; CSR 6435 rows s = 4 4.5 -> 2.4.
//
// Every row is summed in the step kernels' order with the same explicitly
// rounded operations (step_combine, fma_t), so results equal theirs bit for
// bit.
#include "pf_internal.h"
#include "pf_rows.cuh"
#include "pf_solver.h"

#include <algorithm>
#include <cmath>
#include <map>
#include <tuple>

namespace pf {

template <typename T>
struct ResArgs {
    uint32_t O;          // outer states (D / dg)
    int clog;            // log2 of the CTAs per cluster
    int K;               // filter: order; KPM: steps
    const T *X;          // filter: input; KPM: probes (null: drawn from the seed)
    int64_t xr, xc;      // element (row, column) of X at row * xr + column * xc
    T *Y;                // filter: output, laid out like X with yr, yc
    int64_t yr, yc;
    const double *coef;  // filter: K + 1 coefficients
    T inva, boa;
    int probe_kind;
    uint64_t seed;
    int ncol;            // columns of the launch
    int col0;            // KPM: number of the first of them, for drawn probes
    double *part;        // KPM: [K + 1][ncol][2^clog][2] dot partials
    // Quantum Sun, by outer spin: the XOR of a chunk's byte offset in a CTA's
    // block (spins of the CTA's own range) or of its chunk part alone (the
    // others), and the exchange inside the chunk
    uint32_t flip[PF_MAX_LOC];
    uint8_t inner[PF_MAX_LOC];
    // filters of more columns (or groups of columns) than clusters fit the device
    // at once: `slots` > 0 of them per launch, each for `steps` steps
    int slot, slots, steps;
    T *state;            // their two vectors each, between their launches
    T *xch;              // exchange blocks [2][columns][D], or null: CTAs read each other's shared memory
};

constexpr int kResListThreads = 1024;

namespace {

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// Barrier over the column's CTAs; their shared-memory writes are visible after
// it.  One warp's fence releases the whole CTA's writes (ordered before it by
// the CTA barrier): a release by every warp costs 330 clocks more with 8 warps
// and 590 more with 32.
__device__ __forceinline__ void column_sync(int clog) {
    __syncthreads();
    if (clog == 0) return;
    if (threadIdx.x < 32) asm volatile("fence.acq_rel.cluster;" ::: "memory");
    __syncwarp();   // the aligned barrier wants converged warps
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A chunk (4, 8 or 16 bytes) at a shared-memory address of any CTA of the
// cluster (CL: a mapped address) or of this one, or zeros if !on.
template <typename Ch, bool CL>
__device__ __forceinline__ Ch ld_shared_if(uint32_t addr, bool on) {
    Ch v;
    uint32_t *w = reinterpret_cast<uint32_t *>(&v);
    w[0] = 0u;
    if constexpr (sizeof(Ch) >= 8) w[1] = 0u;
    if constexpr (sizeof(Ch) == 16) w[2] = w[3] = 0u;
    if constexpr (sizeof(Ch) == 16 && CL)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\t@p ld.shared::cluster.v4.b32 {%0, %1, %2, %3}, [%4];\n\t}"
                     : "+r"(w[0]), "+r"(w[1]), "+r"(w[2]), "+r"(w[3])
                     : "r"(addr), "r"((uint32_t)on));
    else if constexpr (sizeof(Ch) == 16)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\t@p ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];\n\t}"
                     : "+r"(w[0]), "+r"(w[1]), "+r"(w[2]), "+r"(w[3])
                     : "r"(addr), "r"((uint32_t)on));
    else if constexpr (sizeof(Ch) == 8 && CL)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p ld.shared::cluster.v2.b32 {%0, %1}, [%2];\n\t}"
                     : "+r"(w[0]), "+r"(w[1])
                     : "r"(addr), "r"((uint32_t)on));
    else if constexpr (sizeof(Ch) == 8)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p ld.shared.v2.b32 {%0, %1}, [%2];\n\t}"
                     : "+r"(w[0]), "+r"(w[1])
                     : "r"(addr), "r"((uint32_t)on));
    else if constexpr (CL)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p ld.shared::cluster.b32 %0, [%1];\n\t}"
                     : "+r"(w[0])
                     : "r"(addr), "r"((uint32_t)on));
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p ld.shared.b32 %0, [%1];\n\t}"
                     : "+r"(w[0])
                     : "r"(addr), "r"((uint32_t)on));
    return v;
}
template <typename Ch, bool CL>
__device__ __forceinline__ Ch ld_shared(uint32_t addr) {
    return ld_shared_if<Ch, CL>(addr, true);
}
__device__ __forceinline__ double ld_cluster_f64(uint32_t addr) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr));
    return v;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// A chunk another CTA wrote to global memory, from L2.
template <typename Ch>
__device__ __forceinline__ Ch ld_l2(const Ch *p) {
    if constexpr (sizeof(Ch) == 16) {
        const uint4 w = __ldcg(reinterpret_cast<const uint4 *>(p));
        return *reinterpret_cast<const Ch *>(&w);
    } else {
        const uint2 w = __ldcg(reinterpret_cast<const uint2 *>(p));
        return *reinterpret_cast<const Ch *>(&w);
    }
}

// The columns (or groups of columns, `groups` in all) of a rotating launch:
// cluster i takes the i-th after the launch's first, from the step n0 its
// earlier launches reached to n1.  false: it is done (the whole cluster leaves).
template <typename T>
__device__ __forceinline__ bool res_slot(const ResArgs<T> &a, int groups, int *grp, int *n0, int *n1) {
    const int g = (*grp + a.slot) % groups;
    int before = 0;
    for (int j = 0; j < a.slot; ++j) before += (g - j + groups) % groups < a.slots;
    *grp = g;
    *n0 = min(before * a.steps, a.K);
    *n1 = min(*n0 + a.steps, a.K);
    return *n0 < *n1;
}

// The sum over the column's threads of v, the same in every one of them.
// red: one double per warp plus one.
__device__ double column_sum(double v, double *red, int clog) {
    const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) red[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < nw; ++w) t += red[w];
        red[nw] = t;
    }
    column_sync(clog);
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(red + nw);
    double t = 0.0;
    for (int r = 0; r < (1 << clog); ++r) t += clog ? ld_cluster_f64(map_rank(at, r)) : red[nw];
    column_sync(clog);   // red is free again
    return t;
}

// acc += cf * group, the elements of each chunk exchanged by `in` (0: none, 1
// or 2: with e ^ in).
template <typename T, int W, int NCH>
__device__ __forceinline__ void add_group(T *acc, const Pack<T, W> (&v)[NCH], T cf, int in) {
    if (in == 0) {
#pragma unroll
        for (int c = 0; c < NCH; ++c)
#pragma unroll
            for (int e = 0; e < W; ++e) acc[c * W + e] = fma_t(cf, v[c].v[e], acc[c * W + e]);
    } else if (W == 2 || in == 1) {
#pragma unroll
        for (int c = 0; c < NCH; ++c)
#pragma unroll
            for (int e = 0; e < W; ++e) acc[c * W + e] = fma_t(cf, v[c].v[e ^ 1], acc[c * W + e]);
    } else {
#pragma unroll
        for (int c = 0; c < NCH; ++c)
#pragma unroll
            for (int e = 0; e < W; ++e) acc[c * W + e] = fma_t(cf, v[c].v[(e ^ 2) & (W - 1)], acc[c * W + e]);
    }
}

}  // namespace

template <typename T, int LG>
struct ResQSun {
    static constexpr int DG = 1 << LG;
    static constexpr int W = DG < 16 / (int)sizeof(T) ? DG : 16 / (int)sizeof(T);   // elements per chunk
    static constexpr int NCH = DG / W;                                             // chunks per grain group
    static constexpr int threads = 512;
};

// Quantum Sun.  Row = outer state * dg + grain state.  A thread takes one grain
// group (the dg rows of one outer state) at a time, so the dense grain block is
// register arithmetic and the flip of outer spin j needs the whole group of
// outer ^ (1 << j), its elements exchanged by the grain bit.  A CTA owns an
// aligned range of outer states: flips of the low outer spins stay in its
// shared memory, the clog highest go to CTA rank ^ bit at the same place.
// Chunk c (16 bytes) of every group is stored together, so the threads of a
// warp read consecutive 16-byte words whichever spin is flipped (no bank
// conflicts) and a flip is one XOR of the byte offset.  512 threads: with 1024
// the 2^16 step took 6 % longer, and holding the far groups in registers ahead
// of the local flips (128 registers) gained nothing: L2 and shared memory are
// both near their rate.
template <typename T, int LG, bool KPM>
__global__ void __launch_bounds__(ResQSun<T, LG>::threads)
    k_res_qsun(const __grid_constant__ QSunDesc<T> d, const __grid_constant__ ResArgs<T> a) {
    using R = ResQSun<T, LG>;
    constexpr int DG = R::DG, W = R::W, NCH = R::NCH;
    using Ch = Pack<T, W>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int clog = a.clog, C = 1 << clog;
    const uint32_t rank = clog ? cluster_rank() : 0u;
    int col = blockIdx.x >> clog;
    int n0 = 0, n1 = a.K;                // steps of this launch
    if (!KPM && a.slots > 0 && !res_slot(a, a.ncol, &col, &n0, &n1)) return;
    const int Oc = (int)(a.O >> clog);   // groups of this CTA, a multiple of blockDim.x
    const int nt = blockDim.x, t = threadIdx.x;
    int lo = 0;                          // flips below lo stay in this CTA
    while ((2 << lo) <= Oc) ++lo;
    const int nloc = min(lo, d.L_loc);
    Ch *buf0 = reinterpret_cast<Ch *>(smem_raw), *buf1 = buf0 + NCH * Oc;
    Ch *xb = KPM ? buf1 : buf1 + NCH * Oc;
    T *dgs = reinterpret_cast<T *>(xb + NCH * Oc);
    double *red = reinterpret_cast<double *>(dgs + (Oc + 1) / 2 * 2);   // [2][warps][2]
    const uint32_t s0 = (uint32_t)__cvta_generic_to_shared(buf0), s1 = (uint32_t)__cvta_generic_to_shared(buf1);
    Ch *xch = reinterpret_cast<Ch *>(a.xch) + (size_t)col * C * NCH * Oc;
    const size_t xpar = (size_t)a.ncol * C * NCH * Oc;
    const bool put = a.xch != nullptr;   // the other CTAs read this one's rows from L2

    // the group of far spin nloc + i flipped: at the same place of another CTA
    auto load_far = [&](Ch (&v)[NCH], int n, uint32_t qs, int i, const uint32_t (&off)[NCH]) {
        const uint32_t m = a.flip[nloc + i], from = rank ^ (1u << i);
        if (!put) {
            const uint32_t src = map_rank(qs, from);
#pragma unroll
            for (int c = 0; c < NCH; ++c) v[c] = ld_shared<Ch, true>(src + (off[c] ^ m));
        } else {
            const unsigned char *src = reinterpret_cast<const unsigned char *>(xch + (n & 1) * xpar + (size_t)from * NCH * Oc);
#pragma unroll
            for (int c = 0; c < NCH; ++c) v[c] = ld_l2(reinterpret_cast<const Ch *>(src + (off[c] ^ m)));
        }
    };
    const T cK = KPM ? T(1) : (T)__ldg(a.coef + a.K);
    double nrm = 0.0;
    for (int ol = t; ol < Oc; ol += nt) {
        const uint32_t outer = rank * (uint32_t)Oc + ol;
        dgs[ol] = qsun_diag(d, outer << LG);
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
            Ch v, z, f;
#pragma unroll
            for (int e = 0; e < W; ++e) {
                const uint32_t row = (outer << LG) + c * W + e;
                if (!KPM || a.X) v.v[e] = __ldg(a.X + (int64_t)row * a.xr + (int64_t)col * a.xc);
                else v.v[e] = (T)probe_value(a.probe_kind, a.seed, row, a.col0 + col);
                nrm += (double)v.v[e] * (double)v.v[e];
                z.v[e] = T(0);
                f.v[e] = KPM ? v.v[e] : mul_t(cK, v.v[e]);
            }
            if (!KPM) xb[c * Oc + ol] = v;
            if (!KPM && n0 > 0) {   // b_{k+1} and b_{k+2} as the last launch left them
                const Ch *w = reinterpret_cast<const Ch *>(a.state) + (((size_t)col * 2) * C + rank) * NCH * Oc + c * Oc + ol;
                f = w[0];
                z = w[(size_t)C * NCH * Oc];
            }
            if (!KPM && a.K == 0) {
#pragma unroll
                for (int e = 0; e < W; ++e) a.Y[(int64_t)((outer << LG) + c * W + e) * a.yr + (int64_t)col * a.yc] = f.v[e];
            }
            (n0 & 1 ? buf0 : buf1)[c * Oc + ol] = z;
            (n0 & 1 ? buf1 : buf0)[c * Oc + ol] = f;
            if (put) xch[(n0 & 1) * xpar + (size_t)rank * NCH * Oc + c * Oc + ol] = f;
        }
    }
    if constexpr (KPM) {
        if (!a.X) {
            const double scl = 1.0 / sqrt(column_sum(nrm, red, clog));
            nrm = 0.0;
            for (int ol = t; ol < Oc; ol += nt)
#pragma unroll
                for (int c = 0; c < NCH; ++c) {
                    Ch v = buf0[c * Oc + ol];
#pragma unroll
                    for (int e = 0; e < W; ++e) {
                        v.v[e] = (T)((double)v.v[e] * scl);
                        nrm += (double)v.v[e] * (double)v.v[e];
                    }
                    buf0[c * Oc + ol] = v;
                    if (put) xch[(size_t)rank * NCH * Oc + c * Oc + ol] = v;
                }
        }
        nrm = column_sum(nrm, red, clog);
        if (rank == 0 && t == 0) {
            for (int r = 0; r < C; ++r) {
                double *o = a.part + ((size_t)col * C + r) * 2;
                o[0] = r == 0 ? nrm : 0.0;
                o[1] = 0.0;
            }
        }
    }

    for (int n = n0; n < n1; ++n) {
        const Ch *q = (n & 1) ? buf1 : buf0;
        Ch *out = (n & 1) ? buf0 : buf1;
        const uint32_t qs = (n & 1) ? s1 : s0;
        const bool last = n == a.K - 1;
        const T alpha = KPM ? (n == 0 ? T(1) : T(2)) : (last ? T(1) : T(2));
        const T ck = KPM ? T(0) : (T)__ldg(a.coef + a.K - 1 - n);
        double d1 = 0.0, d2 = 0.0;
        column_sync(clog);
        if constexpr (KPM) {
            if (n > 0 && t < 2) {
                double s = 0.0;
                const double *w = red + ((n - 1) & 1) * 2 * (nt >> 5);
                for (int k = 0; k < (nt >> 5); ++k) s += w[2 * k + t];
                a.part[(((size_t)n * a.ncol + col) * C + rank) * 2 + t] = s;
            }
        }
#pragma unroll 1
        for (int ol = t; ol < Oc; ol += nt) {
            T acc[DG];
#pragma unroll
            for (int e = 0; e < DG; ++e) acc[e] = T(0);
            uint32_t off[NCH];
#pragma unroll
            for (int c = 0; c < NCH; ++c) off[c] = (uint32_t)((c * Oc + ol) * (int)sizeof(Ch));
#pragma unroll 2
            for (int j = 0; j < nloc; ++j) {
                const uint32_t m = a.flip[j];
                Ch v[NCH];
#pragma unroll
                for (int c = 0; c < NCH; ++c) v[c] = *reinterpret_cast<const Ch *>(reinterpret_cast<const unsigned char *>(q) + (off[c] ^ m));
                add_group<T, W, NCH>(acc, v, d.cflip[j], a.inner[j]);
            }
#pragma unroll 1
            for (int i = 0; i < clog; ++i) {
                Ch v[NCH];
                load_far(v, n, qs, i, off);
                add_group<T, W, NCH>(acc, v, d.cflip[nloc + i], a.inner[nloc + i]);
            }
            T qo[DG];
#pragma unroll
            for (int c = 0; c < NCH; ++c) {
                const Ch v = q[c * Oc + ol];
#pragma unroll
                for (int e = 0; e < W; ++e) qo[c * W + e] = v.v[e];
            }
#pragma unroll
            for (int h = 0; h < DG; ++h)
#pragma unroll
                for (int e = 0; e < DG; ++e) acc[e] = fma_t(d.grain[e * DG + h], qo[h], acc[e]);
            const T dg = dgs[ol];
#pragma unroll
            for (int c = 0; c < NCH; ++c) {
                const Ch pv = out[c * Oc + ol];
                Ch xv = pv, v;
                if (!KPM) xv = xb[c * Oc + ol];
#pragma unroll
                for (int e = 0; e < W; ++e) {
                    // b_{k+2} starts as zero: subtracting it is exact, so the steps without it need no form of their own
                    v.v[e] = step_combine<T>(!KPM, true, true, ck, xv.v[e], alpha, acc[c * W + e], dg, qo[c * W + e],
                                             a.inva, a.boa, T(-1), pv.v[e]);
                    if constexpr (KPM) {
                        d1 += (double)v.v[e] * (double)v.v[e];
                        d2 += (double)v.v[e] * (double)qo[c * W + e];
                    }
                }
                if (!KPM && last) {
                    const uint32_t row = ((rank * (uint32_t)Oc + ol) << LG) + c * W;
#pragma unroll
                    for (int e = 0; e < W; ++e) a.Y[(int64_t)(row + e) * a.yr + (int64_t)col * a.yc] = v.v[e];
                } else {
                    out[c * Oc + ol] = v;
                    if (put) xch[((n + 1) & 1) * xpar + (size_t)rank * NCH * Oc + c * Oc + ol] = v;
                }
            }
        }
        if constexpr (KPM) {
            // lanes 0-15 go on with d1, the others with d2: one exchange, then four rounds
            const int lane = t & 31;
            const double give = lane < 16 ? d2 : d1, keep = lane < 16 ? d1 : d2;
            double s = keep + __shfl_xor_sync(0xffffffffu, give, 16);
#pragma unroll
            for (int o = 8; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if ((lane & 15) == 0) red[(n & 1) * 2 * (nt >> 5) + 2 * (t >> 5) + (lane >> 4)] = s;
        }
    }
    column_sync(clog);   // no CTA leaves while another reads its rows
    if (!KPM && n1 < a.K) {
        Ch *w = reinterpret_cast<Ch *>(a.state) + (((size_t)col * 2) * C + rank) * NCH * Oc;
        for (int i = t; i < NCH * Oc; i += nt) {
            w[i] = (n1 & 1 ? buf1 : buf0)[i];
            w[(size_t)C * NCH * Oc + i] = (n1 & 1 ? buf0 : buf1)[i];
        }
    }
    if constexpr (KPM) {
        if (a.K > 0 && t < 2) {
            double s = 0.0;
            const double *w = red + ((a.K - 1) & 1) * 2 * (nt >> 5);
            for (int k = 0; k < (nt >> 5); ++k) s += w[2 * k + t];
            a.part[(((size_t)a.K * a.ncol + col) * C + rank) * 2 + t] = s;
        }
    }
}

// ------------------------------------------------------- chains and CSR
// Neighbour lists of the rows, in groups of eight 16-bit entries: group g of row
// i at g * D + i.  An entry is a row's place in the cluster, its CTA above its
// row there (16 - clog bits), or kResNone.  Entry b of a chain's row is its
// flip by bond b (kResNone where bond b does not flip the state), so a warp's
// gathers for one bond go to runs of consecutive rows: simulated over random
// warps of the L = 16 chain, 28 shared-memory wavefronts a row slice against 45
// for lists without the gaps.  A CSR row's entries stand in storage order, with
// their values (a pack of 16 bytes h of group g at (g * NP + h) * D + i).
constexpr uint32_t kResNone = 0xffffu;

template <typename T>
struct ResList {
    uint32_t D;
    int rows;               // rows per CTA
    int groups;             // groups per row
    const uint4 *ent;
    const T *val;           // CSR values
    const T *diag;          // diagonal, or null: zero
    int x_smem, diag_smem, list_smem;
    T jhalf[PF_MAX_BONDS];
};

template <typename T>
struct ResVals {
    static constexpr int PW = 16 / (int)sizeof(T);   // values per pack
    static constexpr int NP = 8 / PW;                // packs per group
};

__device__ __forceinline__ uint16_t res_entry(uint32_t row, int rows, int clog) {
    const uint32_t c = row / (uint32_t)rows;
    return (uint16_t)((row - c * (uint32_t)rows) | (c << (16 - clog)));
}

template <typename T>
__global__ void k_res_list_chain(const __grid_constant__ ChainDesc<T> d, uint32_t D, int rows, int clog, int groups,
                                 uint16_t *__restrict__ ent) {
    for (uint32_t row = blockIdx.x * blockDim.x + threadIdx.x; row < D; row += gridDim.x * blockDim.x) {
        const uint32_t st = d.full ? row : __ldg(d.states + row);
        for (int b = 0; b < 8 * groups; ++b) {
            uint32_t e = kResNone;
            if (b < d.nb) {
                const uint32_t m = st & d.bmask[b];
                if (m != 0u && m != d.bmask[b])
                    e = res_entry(d.full ? st ^ d.bmask[b] : sector_rank(st ^ d.bmask[b], d.rank_tab, d.nchunks), rows, clog);
            }
            ent[((size_t)(b >> 3) * D + row) * 8 + (b & 7)] = (uint16_t)e;
        }
    }
}

template <typename T>
__global__ void k_res_list_csr(const CsrDesc<T> d, uint32_t D, int rows, int clog, int groups,
                               uint16_t *__restrict__ ent, T *__restrict__ val) {
    using P = ResVals<T>;
    for (uint32_t row = blockIdx.x * blockDim.x + threadIdx.x; row < D; row += gridDim.x * blockDim.x) {
        const int64_t p = d.indptr[row];
        const int cnt = (int)(d.indptr[row + 1] - p);
        for (int n = 0; n < 8 * groups; ++n) {
            const size_t g = n >> 3, u = n & 7;
            ent[(g * D + row) * 8 + u] = n < cnt ? res_entry((uint32_t)d.indices[p + n], rows, clog) : (uint16_t)kResNone;
            val[((g * P::NP + u / P::PW) * D + row) * P::PW + u % P::PW] = n < cnt ? d.values[p + n] : T(0);
        }
    }
}

// A thread owns rows and V neighbouring columns (a chunk of up to 16 bytes).
template <typename T, int V, bool CSR, bool KPM>
__global__ void __launch_bounds__(kResListThreads)
    k_res_list(const __grid_constant__ ResList<T> l, const __grid_constant__ ResArgs<T> a) {
    using Ch = Pack<T, V>;
    using P = ResVals<T>;
    using VP = Pack<T, P::PW>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int clog = a.clog, C = 1 << clog;
    const uint32_t rank = clog ? cluster_rank() : 0u;
    const int grp = blockIdx.x >> clog, col0 = grp * V;
    const int nv = min(V, a.ncol - col0);
    const int nt = blockDim.x, t = threadIdx.x, lane = t & 31, nw = nt >> 5;
    const uint32_t D = l.D, r0 = rank * (uint32_t)l.rows;
    const int R = l.rows;
    const int nr = r0 >= D ? 0 : (int)min((uint32_t)R, D - r0);
    const int lbits = 16 - clog;
    const uint32_t lmask = (1u << lbits) - 1u;
    Ch *buf0 = reinterpret_cast<Ch *>(smem_raw), *buf1 = buf0 + R;
    Ch *xb = buf1 + R;
    unsigned char *at = smem_raw + ((2 + (KPM ? 0 : l.x_smem)) * (size_t)R * sizeof(Ch) + 15) / 16 * 16;
    double *red = reinterpret_cast<double *>(at);   // [2][warps][2 V]
    at += ((size_t)nw * 4 * V + 2) * sizeof(double);
    uint4 *sval = reinterpret_cast<uint4 *>(at);
    if (CSR && l.list_smem) at += (size_t)R * l.groups * P::NP * 16;
    uint4 *sent = reinterpret_cast<uint4 *>(at);
    if (l.list_smem) at += (size_t)R * l.groups * sizeof(uint4);
    T *sdiag = reinterpret_cast<T *>(at);
    const uint32_t s0 = (uint32_t)__cvta_generic_to_shared(buf0), s1 = (uint32_t)__cvta_generic_to_shared(buf1);

    const uint4 *ent = l.ent + r0;
    const uint4 *val = CSR ? reinterpret_cast<const uint4 *>(l.val) + r0 : nullptr;
    uint32_t es = D;   // stride of a group
    if (l.list_smem) {
        for (int r = t; r < nr; r += nt)
            for (int g = 0; g < l.groups; ++g) {
                sent[g * R + r] = __ldg(ent + (size_t)g * D + r);
                if constexpr (CSR)
                    for (int h = 0; h < P::NP; ++h) sval[(g * P::NP + h) * R + r] = __ldg(val + (size_t)(g * P::NP + h) * D + r);
            }
        ent = sent;
        val = sval;
        es = (uint32_t)R;
    }
    if (l.diag_smem)
        for (int r = t; r < nr; r += nt) sdiag[r] = __ldg(l.diag + r0 + r);
    auto load_x = [&](uint32_t row) {
        Ch v;
#pragma unroll
        for (int e = 0; e < V; ++e)
            v.v[e] = e < nv ? __ldg(a.X + (int64_t)row * a.xr + (int64_t)(col0 + e) * a.xc) : T(0);
        return v;
    };
    const T cK = KPM ? T(1) : (T)__ldg(a.coef + a.K);
    double nrm[V];
#pragma unroll
    for (int e = 0; e < V; ++e) nrm[e] = 0.0;
    for (int r = t; r < nr; r += nt) {
        const uint32_t row = r0 + r;
        Ch v, z, f;
        if (!KPM || a.X) v = load_x(row);
        else {
#pragma unroll
            for (int e = 0; e < V; ++e) v.v[e] = (T)probe_value(a.probe_kind, a.seed, row, a.col0 + col0 + e);
        }
#pragma unroll
        for (int e = 0; e < V; ++e) {
            nrm[e] += (double)v.v[e] * (double)v.v[e];
            z.v[e] = T(0);
            f.v[e] = KPM ? v.v[e] : mul_t(cK, v.v[e]);
        }
        if (!KPM && l.x_smem) xb[r] = v;
        if (!KPM && a.K == 0) {
#pragma unroll
            for (int e = 0; e < V; ++e)
                if (e < nv) a.Y[(int64_t)row * a.yr + (int64_t)(col0 + e) * a.yc] = f.v[e];
        }
        buf0[r] = f;
        buf1[r] = z;
    }
    if constexpr (KPM) {
        double scl[V];
#pragma unroll
        for (int e = 0; e < V; ++e) {
            scl[e] = 1.0;
            if (!a.X) scl[e] = 1.0 / sqrt(column_sum(nrm[e], red, clog));
            nrm[e] = 0.0;
        }
        for (int r = t; r < nr; r += nt) {
            Ch v = buf0[r];
#pragma unroll
            for (int e = 0; e < V; ++e) {
                if (!a.X) v.v[e] = (T)((double)v.v[e] * scl[e]);
                nrm[e] += (double)v.v[e] * (double)v.v[e];
            }
            buf0[r] = v;
        }
#pragma unroll
        for (int e = 0; e < V; ++e) {
            const double s = column_sum(nrm[e], red, clog);
            if (rank == 0 && t == 0 && e < nv)
                for (int r = 0; r < C; ++r) {
                    double *o = a.part + ((size_t)(col0 + e) * C + r) * 2;
                    o[0] = r == 0 ? s : 0.0;
                    o[1] = 0.0;
                }
        }
    }
    // the warp sums of step m (1-based) into its partials: thread t < 2 V owns (column t / 2, dot t % 2)
    auto put_dots = [&](int m) {
        if (t < 2 * V && (t >> 1) < nv) {
            const double *w = red + (m & 1) * 2 * V * nw + t;
            double s = 0.0;
            for (int k = 0; k < nw; ++k) s += w[2 * V * k];
            a.part[(((size_t)m * a.ncol + col0 + (t >> 1)) * C + rank) * 2 + (t & 1)] = s;
        }
    };
    T ck = KPM || a.K == 0 ? T(0) : (T)__ldg(a.coef + a.K - 1);
    for (int n = 0; n < a.K; ++n) {
        const Ch *q = (n & 1) ? buf1 : buf0;
        Ch *out = (n & 1) ? buf0 : buf1;
        const uint32_t qs = (n & 1) ? s1 : s0;
        const bool last = n == a.K - 1;
        const T alpha = KPM ? (n == 0 ? T(1) : T(2)) : (last ? T(1) : T(2));
        const T cnext = KPM || last ? T(0) : (T)__ldg(a.coef + a.K - 2 - n);
        double d1[V], d2[V];
#pragma unroll
        for (int e = 0; e < V; ++e) d1[e] = d2[e] = 0.0;
        column_sync(clog);
        if constexpr (KPM) {
            if (n > 0) put_dots(n);
        }
        for (int r = t; r < nr; r += nt) {
            const T dg = l.diag_smem ? sdiag[r] : l.diag ? __ldg(l.diag + r0 + r) : T(0);
            T acc[V];
#pragma unroll
            for (int e = 0; e < V; ++e) acc[e] = T(0);
            const uint4 *w = ent + r;
            const uint4 *wv = val + r;
            uint4 en = w[0];
            for (int g = 0; g < l.groups; ++g) {
                const uint32_t e8[8] = {en.x & 0xffffu, en.x >> 16, en.y & 0xffffu, en.y >> 16,
                                        en.z & 0xffffu, en.z >> 16, en.w & 0xffffu, en.w >> 16};
                if (CSR && e8[0] == kResNone) break;   // rows are full up to their length
                if (g + 1 < l.groups) en = w[(size_t)(g + 1) * es];
                Ch x[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const uint32_t off = (e8[u] & lmask) * (uint32_t)sizeof(Ch);
                    if (clog == 0) x[u] = ld_shared_if<Ch, false>(qs + off, e8[u] != kResNone);
                    else x[u] = ld_shared_if<Ch, true>(map_rank(qs, e8[u] >> lbits) + off, e8[u] != kResNone);
                }
                T cf[8];
                if constexpr (CSR) {
#pragma unroll
                    for (int h = 0; h < P::NP; ++h) {
                        const uint4 u = wv[(size_t)(g * P::NP + h) * es];
                        const VP v = *reinterpret_cast<const VP *>(&u);
#pragma unroll
                        for (int i = 0; i < P::PW; ++i) cf[h * P::PW + i] = v.v[i];
                    }
                } else {
#pragma unroll
                    for (int u = 0; u < 8; ++u) cf[u] = l.jhalf[8 * g + u];
                }
                // a missing entry reads as zero: adding coefficient * 0 is exact
#pragma unroll
                for (int u = 0; u < 8; ++u)
#pragma unroll
                    for (int e = 0; e < V; ++e) acc[e] = fma_t(cf[u], x[u].v[e], acc[e]);
            }
            const Ch qo = q[r], po = out[r];
            Ch xo = po, v;
            if (!KPM) xo = l.x_smem ? xb[r] : load_x(r0 + r);
#pragma unroll
            for (int e = 0; e < V; ++e) {
                v.v[e] = step_combine<T>(!KPM, true, true, ck, xo.v[e], alpha, acc[e], dg, qo.v[e], a.inva, a.boa, T(-1),
                                         po.v[e]);
                if constexpr (KPM) {
                    d1[e] += (double)v.v[e] * (double)v.v[e];
                    d2[e] += (double)v.v[e] * (double)qo.v[e];
                }
            }
            if (!KPM && last) {
#pragma unroll
                for (int e = 0; e < V; ++e)
                    if (e < nv) a.Y[(int64_t)(r0 + r) * a.yr + (int64_t)(col0 + e) * a.yc] = v.v[e];
            } else {
                out[r] = v;
            }
        }
        ck = cnext;
        if constexpr (KPM) {
            __syncwarp();
#pragma unroll
            for (int e = 0; e < V; ++e) {
                const double give = lane < 16 ? d2[e] : d1[e], keep = lane < 16 ? d1[e] : d2[e];
                double s = keep + __shfl_xor_sync(0xffffffffu, give, 16);
#pragma unroll
                for (int o = 8; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if ((lane & 15) == 0) red[((n + 1) & 1) * 2 * V * nw + 2 * V * (t >> 5) + 2 * e + (lane >> 4)] = s;
            }
        }
    }
    column_sync(clog);
    if constexpr (KPM) {
        if (a.K > 0) put_dots(a.K);
    }
}

// The filter of a chain whose CTAs hold at most a row per thread: a thread's
// list stays in registers as ready addresses, with its X, its diagonal and its
// own values, so a step is one barrier, its gathers (eight in flight) and their
// sum.  us a step, k_res_list -> here: XXZ L = 14 s = 1 1.76 -> 1.69, L = 16 s = 1
// 3.07 -> 2.47, s = 8 3.99 -> 3.16.  More than 24 entries or 1024 rows a CTA do
// not fit its 64 registers a thread: those stay with k_res_list.
template <typename T, int V, int G>
__global__ void __launch_bounds__(1024)
    k_res_pinned(const __grid_constant__ ResList<T> l, const __grid_constant__ ResArgs<T> a) {
    using Ch = Pack<T, V>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int clog = a.clog;
    const uint32_t rank = clog ? cluster_rank() : 0u;
    int grp = blockIdx.x >> clog, n0 = 0, n1 = a.K;
    if (a.slots > 0 && !res_slot(a, (a.ncol + V - 1) / V, &grp, &n0, &n1)) return;
    const int col0 = grp * V, nv = min(V, a.ncol - col0);
    const int t = threadIdx.x, R = l.rows;
    const uint32_t row = rank * (uint32_t)R + t;
    const bool mine = t < R && row < l.D;
    const int lbits = 16 - clog;
    Ch *buf0 = reinterpret_cast<Ch *>(smem_raw), *buf1 = buf0 + R;
    const uint32_t s0 = (uint32_t)__cvta_generic_to_shared(buf0), s1 = (uint32_t)__cvta_generic_to_shared(buf1);
    uint32_t at[8 * G], on = 0u;
    Ch x, qo, po;
    T dg = T(0);
    const T cK = (T)__ldg(a.coef + a.K);
#pragma unroll
    for (int e = 0; e < V; ++e) x.v[e] = qo.v[e] = po.v[e] = T(0);
#pragma unroll
    for (int g = 0; g < G; ++g) {
        uint4 w = make_uint4(~0u, ~0u, ~0u, ~0u);
        if (mine) w = __ldg(l.ent + (size_t)g * l.D + row);
        const uint32_t w4[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const uint32_t e = (w4[u >> 1] >> (16 * (u & 1))) & 0xffffu;
            if (e != kResNone) on |= 1u << (8 * g + u);
            at[8 * g + u] = (clog ? map_rank(s0, e >> lbits) : s0) + (e & ((1u << lbits) - 1u)) * (uint32_t)sizeof(Ch);
        }
    }
    if (mine) {
        dg = __ldg(l.diag + row);
#pragma unroll
        for (int e = 0; e < V; ++e) {
            if (e < nv) x.v[e] = __ldg(a.X + (int64_t)row * a.xr + (int64_t)(col0 + e) * a.xc);
            qo.v[e] = mul_t(cK, x.v[e]);
            if (a.K == 0 && e < nv) a.Y[(int64_t)row * a.yr + (int64_t)(col0 + e) * a.yc] = qo.v[e];
        }
    }
    Ch *state = reinterpret_cast<Ch *>(a.state) + ((size_t)(2 * grp) << clog) * R + rank * (uint32_t)R + t;   // then po
    const size_t spo = (size_t)R << clog;
    if (mine && n0 > 0) {
        qo = state[0];
        po = state[spo];
    }
    if (mine) (n0 & 1 ? buf1 : buf0)[t] = qo;
    T ck = a.K == 0 ? T(0) : (T)__ldg(a.coef + a.K - 1 - n0);
    for (int n = n0; n < n1; ++n) {
        const uint32_t dq = (n & 1) ? s1 - s0 : 0u;
        Ch *out = (n & 1) ? buf0 : buf1;
        const bool last = n == a.K - 1;
        const T alpha = last ? T(1) : T(2);
        const T cnext = last ? T(0) : (T)__ldg(a.coef + a.K - 2 - n);
        column_sync(clog);
        Ch v;
        T acc[V];
#pragma unroll
        for (int e = 0; e < V; ++e) acc[e] = T(0);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            Ch f[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) f[u] = ld_shared_if<Ch, true>(at[8 * g + u] + dq, (on >> (8 * g + u)) & 1u);
#pragma unroll
            for (int u = 0; u < 8; ++u)
#pragma unroll
                for (int e = 0; e < V; ++e) acc[e] = fma_t(l.jhalf[8 * g + u], f[u].v[e], acc[e]);
        }
#pragma unroll
        for (int e = 0; e < V; ++e) {
            v.v[e] = step_combine<T>(true, true, true, ck, x.v[e], alpha, acc[e], dg, qo.v[e], a.inva, a.boa, T(-1), po.v[e]);
            po.v[e] = qo.v[e];
            qo.v[e] = v.v[e];
        }
        if (mine && last) {
#pragma unroll
            for (int e = 0; e < V; ++e)
                if (e < nv) a.Y[(int64_t)row * a.yr + (int64_t)(col0 + e) * a.yc] = v.v[e];
        } else if (mine) {
            out[t] = v;
        }
        ck = cnext;
    }
    column_sync(clog);   // no CTA leaves while another reads its rows
    if (mine && n1 < a.K) {
        state[0] = qo;
        state[spo] = po;
    }
}

// out[(m * 2 + v) * ncol + c] = the sum over a column's CTAs of its partial dots, in rank order
__global__ void k_res_dots(const double *__restrict__ part, int64_t n, int C, int ncol, double *__restrict__ out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int v = (int)(i & 1);
        const int64_t mc = i >> 1, m = mc / ncol, c = mc - m * ncol;
        double s = 0.0;
        for (int r = 0; r < C; ++r) s += part[(mc * C + r) * 2 + v];
        out[(m * 2 + v) * ncol + c] = s;
    }
}

// ------------------------------------------------------------------- launch
constexpr size_t kResSmem = 227 * 1024;

// Where CTAs read each other's rows: from shared memory up to this many bytes
// per CTA and step, above it from global memory (L2), where each step also
// writes them.  Remote shared-memory reads pass 16-35 bytes a clock and SM and
// L2 reads about as many, but behind a barrier that has 1000 instead of 500
// clocks to wait for the global writes (a step of 2^13 rows on 8 CTAs: 2.64
// against 2.70 us; 2^14 rows: 3.56 against 3.11; 2^16 rows: 10.0 against 7.4).
constexpr size_t kResFarShared = 32 * 1024;

// The plan of a Quantum Sun column on 2^clog CTAs, if it fits.  us: estimated
// time of a step of one cluster that has its SMs to itself (measured: shared
// memory at 105 of its 128 bytes a clock, 0.5 us for the barrier and the
// latencies, 0.9 us and 100 KB/us for rows from L2).
template <typename T, int LG>
static bool qsun_plan(uint32_t O, int L_loc, int ncol, int clog, bool kpm, ResPlan *p) {
    using R = ResQSun<T, LG>;
    const uint32_t Oc = O >> clog;
    if (Oc < 32) return false;
    p->clog = clog;
    p->cols = 1;
    p->threads = (int)std::min<uint32_t>(Oc, R::threads);
    const size_t block = (size_t)Oc * R::DG * sizeof(T);
    p->smem = (kpm ? 2 : 3) * block + Oc * sizeof(T) + ((p->threads / 32) * 4 + 2) * sizeof(double);
    p->kern = kpm ? (const void *)k_res_qsun<T, LG, true> : (const void *)k_res_qsun<T, LG, false>;
    const size_t far = clog * block;
    p->far = far > kResFarShared;
    const size_t exchange = p->far ? 2 * (size_t)O * R::DG * sizeof(T) : 0;   // of a column
    p->work = kpm ? 0 : (size_t)ncol * exchange;
    p->work_col = exchange;
    p->busy_us = (double)block * (L_loc - clog + (kpm ? 3 : 4)) / 200e3 + far / 100e3;
    p->us = p->busy_us + 0.5 + (p->far ? 0.9 : clog ? 0.5 : 0.0);
    return p->smem <= kResSmem;
}

template <typename T>
static bool qsun_plan(const pf_op *op, int ncol, int clog, bool kpm, ResPlan *p) {
    const uint32_t O = (uint32_t)(op->dim >> op->L_grain);
    switch (op->L_grain) {
        case 1: return qsun_plan<T, 1>(O, op->L_loc, ncol, clog, kpm, p);
        case 2: return qsun_plan<T, 2>(O, op->L_loc, ncol, clog, kpm, p);
        case 3: return qsun_plan<T, 3>(O, op->L_loc, ncol, clog, kpm, p);
        case 4: return qsun_plan<T, 4>(O, op->L_loc, ncol, clog, kpm, p);
        default: return false;
    }
}

template <typename T, int V>
static const void *list_kernel(bool csr, bool kpm) {
    if (csr) return kpm ? (const void *)k_res_list<T, V, true, true> : (const void *)k_res_list<T, V, true, false>;
    return kpm ? (const void *)k_res_list<T, V, false, true> : (const void *)k_res_list<T, V, false, false>;
}

template <typename T, int V>
static const void *pinned_kernel(int groups) {
    return groups == 1 ? (const void *)k_res_pinned<T, V, 1> : groups == 2 ? (const void *)k_res_pinned<T, V, 2>
                                                             : (const void *)k_res_pinned<T, V, 3>;
}

// Entries of a row of a chain or CSR operator, on average.
static double list_terms(const pf_op *op) {
    if (op->kind == OP_CSR) return (double)op->nnz / (double)op->dim;
    const double L = op->L, up = op->Lup, nb = op->chain64.nb;
    return op->Lup < 0 || op->L < 2 ? nb / 2 : nb * 2 * up * (L - up) / (L * (L - 1));
}

// The plan of V columns of a chain or CSR operator on 2^clog CTAs, if it fits.
// us as for qsun_plan.  Chains (measured): 0.18 ns a row and entry in one CTA,
// 0.27 ns on several, where a quarter of the entries are remote; wider chunks
// cost a quarter more; 0.4 and 1.2 us for the barrier and latencies.
// CSR rows may have their entries anywhere.  Measured over 40 matrices of 200 to
// 50000 rows (chains, grids, bands, random columns; 3 to 60 entries a row), on
// several CTAs: 1.3 ns a sector of remote columns, 0.8 ns a row, 0.38 us for each
// eight entries of a row that wait for remote ones, as much for each eight read
// from a list in L2, 1.05 us for the barrier, within a standard deviation of 10 to
// 15 %; in one CTA the row places alone.
template <typename T>
static bool list_plan(const pf_op *op, int V, int clog, bool kpm, ResPlan *p) {
    const bool csr = op->kind == OP_CSR;
    if (!csr && op->chain64.diag == nullptr) return false;
    const int width = csr ? op->shape.max_row : op->chain64.nb;
    const int64_t D = op->dim;
    const int64_t rows = (D + (1 << clog) - 1) >> clog;
    // the last CTA's last row would be kResNone
    if (width < 1 || width > PF_MAX_BONDS || rows >= (1 << (16 - clog))) return false;
    p->clog = clog;
    p->cols = V;
    p->rows = (int)rows;
    p->groups = (width + 7) / 8;
    p->threads = (int)std::min<int64_t>(kResListThreads, (rows + 31) / 32 * 32);
    const size_t vec = (size_t)rows * V * sizeof(T);
    size_t smem = 2 * vec + 16 + ((p->threads / 32) * 4 * V + 2) * sizeof(double);
    if (smem > kResSmem) return false;
    // what room is left holds the lists, then X, then the diagonal
    const size_t list = (size_t)rows * p->groups * (16 + (csr ? 8 * sizeof(T) : 0));
    p->list_smem = smem + list <= kResSmem;
    if (p->list_smem) smem += list;
    p->x_smem = !kpm && smem + vec <= kResSmem;
    if (p->x_smem) smem += vec;
    p->diag_smem = !csr && smem + (size_t)rows * sizeof(T) <= kResSmem;
    if (p->diag_smem) smem += (size_t)rows * sizeof(T);
    p->smem = smem;
    p->work = (size_t)D * p->groups * (16 + (csr ? 8 * sizeof(T) : 0));
    const int bytes = V * (int)sizeof(T);
    const double wide = bytes == 16 ? 1.25 : bytes == 4 ? 0.85 : 1.0;
    if (csr) {
        const CsrShape &sh = op->shape;
        const double C = 1 << clog, slots = sh.slots / C;
        if (clog == 0) {
            p->busy_us = (slots * (bytes == 16 ? 0.18 : bytes == 8 ? 0.115 : 0.08) + (p->list_smem ? 0.0 : 0.4 * rows)) * 1e-3;
            p->us = p->busy_us + (kpm ? 0.8 : 0.4);
        } else {
            p->busy_us = (sh.far[clog] / C * 1.3 + 0.8 * rows + slots * (bytes == 16 ? 0.09 : bytes == 8 ? 0.015 : 0.01)) * 1e-3;
            const double turns = std::ceil((double)rows / p->threads), entries = std::max(1.0, (double)op->nnz);
            p->us = p->busy_us + (kpm ? 1.3 : 1.05) + 0.38 * turns * p->groups * sh.far_entries[clog] / entries;
            if (!p->list_smem) p->us += turns * sh.slots / 8 / (double)D * (sizeof(T) == 4 ? 0.25 : V == 1 ? 0.45 : 0.75);
        }
    } else {
        p->busy_us = (double)rows * list_terms(op) * (clog ? 0.27e-3 : 0.18e-3) * wide;
        p->us = p->busy_us + (clog ? 1.2 : 0.4);
    }
    if (!csr && !kpm && p->groups <= 3 && rows <= 1024) {
        // measured: 1.35 us for the barrier and the latency of remote rows, 0.042
        // ns a row and entry for every doubling of the CTAs (the remote share
        // grows so); in one CTA 0.35 us and 0.1 ns
        const double size = V * (int)sizeof(T) == 16 ? 1.9 : V * (int)sizeof(T) == 4 ? 0.7 : 1.0;
        p->busy_us = (double)rows * list_terms(op) * (clog ? 0.042e-3 * clog * size : 0.1e-3 * wide);
        p->us = p->busy_us + (clog ? 1.35 : 0.35);
        p->threads = (int)(rows + 31) / 32 * 32;
        p->smem = 2 * vec;
        p->pinned = 1;
        if constexpr (sizeof(T) == 8) p->kern = V == 1 ? pinned_kernel<T, 1>(p->groups) : pinned_kernel<T, 2>(p->groups);
        else p->kern = V == 1 ? pinned_kernel<T, 1>(p->groups) : V == 2 ? pinned_kernel<T, 2>(p->groups) : pinned_kernel<T, 4>(p->groups);
        return true;
    }
    if constexpr (sizeof(T) == 8) p->kern = V == 1 ? list_kernel<T, 1>(csr, kpm) : list_kernel<T, 2>(csr, kpm);
    else p->kern = V == 1 ? list_kernel<T, 1>(csr, kpm) : V == 2 ? list_kernel<T, 2>(csr, kpm) : list_kernel<T, 4>(csr, kpm);
    return true;
}

static int res_groups(const ResPlan &p, int ncol) { return (ncol + p.cols - 1) / p.cols; }

static cudaLaunchConfig_t res_config(const ResPlan &p, int ncol, cudaStream_t st, cudaLaunchAttribute *attr) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)res_groups(p, ncol) << p.clog);
    cfg.blockDim = dim3((unsigned)p.threads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1u << p.clog;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// Clusters of a plan that are resident on the device at once (cached per host thread).
static int res_resident(const ResPlan &p) {
    thread_local std::map<std::tuple<const void *, int, int, size_t>, int> cache;
    const auto key = std::make_tuple(p.kern, p.clog, p.threads, p.smem);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    PF_CUDA(cudaFuncSetAttribute(p.kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResSmem));
    PF_CUDA(cudaFuncSetAttribute(p.kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = res_config(p, 64 * p.cols, nullptr, attr);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, p.kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    return cache[key] = n;
}

// A CSR step of s columns, V a thread, in us (measured over the matrices of
// list_plan): a launch, a dependent gather for every batch of a row, the gathered
// sectors, the blocks' bytes.
static double csr_step_us(const pf_op *op, int s, int elem, int V, bool dots) {
    const int bytes = V * elem, batch = bytes >= 64 ? 2 : bytes >= 16 ? 4 : 8;
    const double waits = std::ceil((double)op->shape.max_row / batch) * (bytes < 16 ? 0.8 : 0.55);
    const double sectors = (double)op->nnz * (s / V) * std::max(1.0, bytes / 32.0), moved = (double)op->dim * s * elem;
    if (dots) return (bytes < 32 ? 3.0 : 4.9) + waits + sectors * (bytes < 32 ? 9e-6 : 2e-6) + moved * 0.7e-6;
    return (bytes < 64 ? 1.4 : 2.2) + waits + sectors * 3.5e-6 + moved * 0.12e-6;
}

// A step of ncol columns by the step kernels, in us: what the kernels, autotuned
// or a chain's listed ones, measured over D = 2^11 .. 2^17 (a launch floor, then
// the gathered values).  KPM: a step of every block of columns, with fused dots,
// of chains and the Quantum Sun about twice a filter's.  CSR filters depend on
// the columns a thread takes: the default, or the best if they are (to be) tuned
// (whose gather batch saves a fifth more);
// a CSR KPM run pays 55 us a block beyond its K steps (its probes and their norms).
static double step_us(const pf_op *op, int ncol, int elem, bool kpm, int K, bool tuned) {
    const double D = (double)op->dim, w = elem == 8 ? 1.0 : 0.7;
    if (op->kind == OP_CSR) {
        double us = 0.0;
        if (kpm) {
            const double block = 55.0 / std::max(K, 1);
            if (ncol >= 64) us = (ncol / 64) * (block + csr_step_us(op, 64, elem, dots_width(64, elem), true));
            for (int nb = 32; nb >= 1; nb /= 2)
                if (ncol % 64 & nb) us += block + csr_step_us(op, nb, elem, dots_width(nb, elem), true);
            return us;
        }
        us = csr_step_us(op, ncol, elem, default_width(ncol, elem), false);
        if (tuned)
            for (int V = 1; V * elem <= 64 && ncol % V == 0; V *= 2) us = std::min(us, 0.8 * csr_step_us(op, ncol, elem, V, false));
        return us;
    }
    const int n = kpm ? std::min(ncol, 64) : ncol;
    const double us = op->kind == OP_QSUN ? 2.8 + D * n * (op->L_loc + (1 << op->L_grain)) * 0.42e-6 * w
                                          : 3.0 + D * n * list_terms(op) * 0.9e-6 * (elem == 8 ? 1.0 : 0.5);
    return kpm ? 2 * us * std::ceil(ncol / 64.0) : us;
}

// A filter of g columns (or groups of columns) with n < g clusters resident runs
// as g launches of n of them and K / n steps each, every one resting in g - n
// launches, so no launch leaves clusters idle: eight columns on 7 clusters of 16
// CTAs take 8/7 rounds instead of two.  A launch costs about 10 us beyond its
// steps (its start, the vectors to memory and back).  A chain's filter beside
// others in a pool does not rotate: two columns a cluster then take half the
// clusters for 12 % more time each, and the others run on the rest (eight XXZ L =
// 16 solves in flight 511 ms rotating, 390 not; the Quantum Sun's CTAs hold one
// column only).
constexpr double kResSlotUs = 10.0;

// A KPM run takes its columns in launches of whole rounds of clusters, so many
// that the columns' exchange blocks and dot partials stay below kResKpmBytes or
// the two blocks of 64 columns the step kernels would hold, whichever is more
// (a round's exchange blocks are at most the SMs' shared memory twice).  A
// launch's last round waits for its slowest cluster: the Quantum Sun 2^16 with
// 300 probes takes 18.32 ms in one launch, 18.49 in two, 18.69 in the six of 67
// MB.  false: not even a round fits.
static bool kpm_launch(ResPlan *p, int64_t D, int elem, int ncol, int M, int resident) {
    const double each = (double)p->work_col + 16.0 * (M + 1) * (1 << p->clog);
    const double room = std::max((double)kResKpmBytes, 2.0 * (double)D * 64 * elem);
    const int64_t fit = (int64_t)std::min(room / each, 1e9), round = (int64_t)resident * p->cols;
    if (fit < std::min<int64_t>(round, ncol)) return false;
    p->launch = (int)std::min<int64_t>(ncol, std::max<int64_t>(fit / round, 1) * round);
    p->work += p->work_col * p->launch;
    return true;
}

// Of the cluster sizes and widths that fit, the one with the least estimated
// time for all columns: as many rounds of clusters as are not resident at once,
// or the SMs' total work where that is more.  K: a filter's order, a KPM run's steps.
// A CSR matrix has to be ahead by 6 %: of 880 filters and KPM runs whose forms were
// all measured, the choice then is more than 5 % slower than the step kernels in
// 5, by 24 % at most (by a model without its columns' places in 183, by up to a
// factor of 9.6).
template <typename T>
bool resident_plan(const pf_op *op, int ncol, bool kpm, int K, bool tuned, ResPlan *best) {
    const double sms = op->h->num_sms;
    double bt = step_us(op, ncol, (int)sizeof(T), kpm, K, tuned) / (op->kind == OP_CSR ? 1.06 : 1.0);
    bool have = false;
    for (int clog = 0; clog <= 4; ++clog)
        for (int V = 1; V * (int)sizeof(T) <= (op->kind == OP_QSUN ? (int)sizeof(T) : 16); V *= 2) {
            ResPlan p;
            const bool ok = op->kind == OP_QSUN ? qsun_plan<T>(op, ncol, clog, kpm, &p) : list_plan<T>(op, V, clog, kpm, &p);
            if (!ok) continue;
            const int n = res_resident(p);
            if (n < 1) continue;
            const int groups = res_groups(p, ncol);
            if (kpm && !kpm_launch(&p, op->dim, (int)sizeof(T), ncol, K, n)) continue;
            double t = std::max((groups + n - 1) / n * p.us, groups * (1 << clog) * p.busy_us / sms);
            if (op->kind == OP_CSR) {
                // beyond the clusters that have their SMs to themselves, the next share them
                ResPlan alone = p;
                alone.smem = kResSmem;
                const int n1 = std::max(1, res_resident(alone));
                t = (groups + n - 1) / n * (p.us - p.busy_us) + (groups + n1 - 1) / n1 * p.busy_us;
            }
            const bool rotates = op->kind == OP_QSUN || (p.pinned && !op->h->shared);
            if (rotates && !kpm && K > 0 && groups > n) {
                const int steps = (K + n - 1) / n;
                const double ts = groups * (steps * p.us + kResSlotUs) / std::max(K, 1);
                if (ts < t) {
                    t = ts;
                    p.slots = n;
                    p.work += 2 * (size_t)groups * p.cols * sizeof(T) *
                              (p.pinned ? (size_t)p.rows << p.clog : (size_t)op->dim);
                }
            }
            if (t < bt) {
                bt = t;
                *best = p;
                have = true;
            }
        }
    return have;
}

template <typename T>
static const QSunDesc<T> &res_qsun(const pf_op *op);
template <>
const QSunDesc<double> &res_qsun<double>(const pf_op *op) { return op->qsun64; }
template <>
const QSunDesc<float> &res_qsun<float>(const pf_op *op) { return op->qsun32; }
template <typename T>
static const ChainDesc<T> &res_chain(const pf_op *op);
template <>
const ChainDesc<double> &res_chain<double>(const pf_op *op) { return op->chain64; }
template <>
const ChainDesc<float> &res_chain<float>(const pf_op *op) { return op->chain32; }
template <typename T>
static const CsrDesc<T> &res_csr(const pf_op *op);
template <>
const CsrDesc<double> &res_csr<double>(const pf_op *op) { return op->csr64; }
template <>
const CsrDesc<float> &res_csr<float>(const pf_op *op) { return op->csr32; }

// The workspace of a list operator: entries, CSR values.
template <typename T>
static void list_parts(const pf_op *op, const ResPlan &p, void *work, uint16_t **ent, T **val) {
    unsigned char *w = static_cast<unsigned char *>(work);
    *ent = reinterpret_cast<uint16_t *>(w);
    *val = reinterpret_cast<T *>(w + (size_t)op->dim * p.groups * 16);
}

template <typename T>
void resident_prepare(pf_op *op, cudaStream_t st, const ResPlan &p, void *work) {
    if (op->kind == OP_QSUN) return;
    uint16_t *ent;
    T *val;
    list_parts<T>(op, p, work, &ent, &val);
    const int grid = grid_for(op->h, op->dim, 128, 16);
    const uint32_t D = (uint32_t)op->dim;
    if (op->kind == OP_CHAIN)
        k_res_list_chain<T><<<grid, 128, 0, st>>>(res_chain<T>(op), D, p.rows, p.clog, p.groups, ent);
    else k_res_list_csr<T><<<grid, 128, 0, st>>>(res_csr<T>(op), D, p.rows, p.clog, p.groups, ent, val);
    PF_CUDA(cudaGetLastError());
    count_launches(1);
}

// The launch, or the plan's rotating launches.  args: the kernel's, with &a.
template <typename T>
static void res_launch_slots(cudaLaunchConfig_t &cfg, const ResPlan &p, void **args, ResArgs<T> &a, int ncol) {
    const int launches = p.slots > 0 ? res_groups(p, ncol) : 1;
    if (p.slots > 0) {
        cfg.gridDim = dim3((unsigned)p.slots << p.clog);
        a.slots = p.slots;
        a.steps = (a.K + p.slots - 1) / p.slots;
    }
    for (a.slot = 0; a.slot < launches; ++a.slot) {
        PF_CUDA(cudaLaunchKernelExC(&cfg, p.kern, args));
        count_launches(1);
    }
}

template <typename T>
static void res_launch(pf_op *op, const ResPlan &p, void *work, int ncol, cudaStream_t st, ResArgs<T> &a) {
    a.clog = p.clog;
    a.ncol = ncol;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = res_config(p, ncol, st, attr);
    PF_CUDA(cudaFuncSetAttribute(p.kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResSmem));
    PF_CUDA(cudaFuncSetAttribute(p.kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    if (op->kind == OP_QSUN) {
        a.O = (uint32_t)(op->dim >> op->L_grain);
        a.xch = p.far ? static_cast<T *>(work) : nullptr;
        a.state = static_cast<T *>(work) + (p.far ? 2 * (size_t)ncol * op->dim : 0);
        QSunDesc<T> d = res_qsun<T>(op);
        {
            const int dg = 1 << op->L_grain, W = std::min(dg, 16 / (int)sizeof(T)), ch = W * (int)sizeof(T);
            const uint32_t Oc = a.O >> p.clog;
            for (int j = 0; j < op->L_loc; ++j) {
                const uint32_t g = d.fmask[j] & (uint32_t)(dg - 1);
                a.flip[j] = g / W * Oc * ch + ((1u << j) < Oc ? ch << j : 0u);
                a.inner[j] = (uint8_t)(g % W);
            }
        }
        void *args[2] = {&d, &a};
        res_launch_slots(cfg, p, args, a, ncol);
    } else {
        ResList<T> l{};
        uint16_t *ent;
        T *val;
        list_parts<T>(op, p, work, &ent, &val);
        l.D = (uint32_t)op->dim;
        l.rows = p.rows;
        l.groups = p.groups;
        l.ent = reinterpret_cast<const uint4 *>(ent);
        l.val = val;
        l.x_smem = p.x_smem;
        l.diag_smem = p.diag_smem;
        l.list_smem = p.list_smem;
        if (op->kind == OP_CHAIN) {
            const ChainDesc<T> &d = res_chain<T>(op);
            l.diag = d.diag;
            for (int b = 0; b < d.nb; ++b) l.jhalf[b] = d.jhalf[b];
        }
        a.state = val;   // a rotating chain filter's vectors, in the place of CSR values
        void *args[2] = {&l, &a};
        res_launch_slots(cfg, p, args, a, ncol);
    }
}

template <typename T>
void resident_filter(pf_op *op, cudaStream_t st, const ResPlan &p, void *work, int s, int K, const double *coef,
                     double a, double b, const T *X, int64_t xr, int64_t xc, T *Y, int64_t yr, int64_t yc) {
    ResArgs<T> r{};
    r.K = K;
    r.X = X; r.xr = xr; r.xc = xc;
    r.Y = Y; r.yr = yr; r.yc = yc;
    r.coef = coef;
    r.inva = (T)(1.0 / a);
    r.boa = (T)(b * (1.0 / a));
    res_launch<T>(op, p, work, s, st, r);
}

template <typename T>
void resident_kpm(pf_op *op, cudaStream_t st, const ResPlan &p, void *work, int M, int R, int col0, double a, double b,
                  const T *probes, int64_t ldp, int kind, uint64_t seed, double *part, double *dots) {
    ResArgs<T> r{};
    r.K = M;
    r.X = probes; r.xr = 1; r.xc = ldp;
    r.col0 = col0;
    r.inva = (T)(1.0 / a);
    r.boa = (T)(b * (1.0 / a));
    r.probe_kind = kind;
    r.seed = seed;
    r.part = part;
    res_launch<T>(op, p, work, R, st, r);
    const int64_t n = (int64_t)(M + 1) * R * 2;
    k_res_dots<<<(int)std::min<int64_t>((n + 255) / 256, 148 * 8), 256, 0, st>>>(part, n, 1 << p.clog, R, dots);
    PF_CUDA(cudaGetLastError());
    count_launches(1);
}

#define PF_RES_INST(T)                                                                                              \
    template bool resident_plan<T>(const pf_op *, int, bool, int, bool, ResPlan *);                                   \
    template void resident_prepare<T>(pf_op *, cudaStream_t, const ResPlan &, void *);                             \
    template void resident_filter<T>(pf_op *, cudaStream_t, const ResPlan &, void *, int, int, const double *,     \
                                     double, double, const T *, int64_t, int64_t, T *, int64_t, int64_t);         \
    template void resident_kpm<T>(pf_op *, cudaStream_t, const ResPlan &, void *, int, int, int, double, double,   \
                                  const T *, int64_t, int, uint64_t, double *, double *);
PF_RES_INST(double)
PF_RES_INST(float)

}  // namespace pf

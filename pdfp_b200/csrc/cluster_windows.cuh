// cluster_windows.cuh -- whole evaluation windows of a small member in one launch.
//
// For members of up to a few thousand rows and columns every launch and every host poll
// costs more than the work of a window.  Here one thread-block cluster (of one block for
// the smallest) runs whole windows of a member's solve (src/pdfp.jl:258-285,
// src/pdlp.jl:332-370): step 1, the evaluation after a restart, steps 2 .. freq-1, step
// freq, the full evaluation, the controller (termination, should_restart, PID) and the
// restart copy, window after window, until the member stops, asks for the FP64 polish, or
// max_windows windows have run.
//
// A step is bound by latency alone: two passes of a sum, an epilogue and a barrier, and in
// each an instruction issues only every few cycles, because each scheduler has one or two
// warps.  So every warp has one slice of 32 lanes (ResSlice, layout.hpp) of one side, its
// rows' vectors in registers and nothing else to decide; every block holds all of x_bar
// and z, which the warps of the cluster's other blocks write directly; and the cluster has
// as many blocks as that takes.
//
// What bounds it: the chain sum -> x_bar -> barrier -> sum -> z -> barrier, about 790
// cycles a pass at 133 x 201 with 1,854 nonzeros (one block); with several blocks the
// barrier of the cluster (380 cycles against 30) and the stores to the other blocks.
// Measured on one B200, FP64, whole solves, against one block that read the CSR arrays
// from shared memory: that model, 600 iterations, 1.65 -> 0.58 ms; two 6 x 56 knapsacks
// 1.11 -> 0.47; 601 x 1,503 with 15k nonzeros, 400 iterations, seven blocks, 8.6 -> 0.94;
// the root LP of 133 x 201, whole call, 2.4 -> 1.27.  Rows are whole whatever their length
// (more than 512 entries: 32 lanes of more than 16): a 6 x 606 knapsack, 600 iterations,
// 1.91 -> 1.00 ms, 2.43 with its rows in pieces on the resident window.
//
// A row's order of summation depends on its length alone and an evaluation's on the rows'
// numbers alone, so the results do not depend on the cluster's size: a batch member takes
// the steps of its own handle bit for bit.
#pragma once
#include "resident_steps.cuh"

namespace pdfp {

constexpr int kCluWarps = 16;  // at most; one slice of 32 lanes per warp, and no idle warps
constexpr int kCluThreads = 32 * kCluWarps;
constexpr int kCluMaxBlocks = 8;  // the portable cluster size
constexpr int kCluWindowsPerLaunch = 64;

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// The address, in block `rank` of the cluster, of this block's shared address `a`.
__device__ __forceinline__ uint32_t cluster_map(uint32_t a, uint32_t rank) {
    uint32_t d;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(rank));
    return d;
}
__device__ __forceinline__ void cluster_put(uint32_t a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_put(uint32_t a, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void cluster_put(uint32_t a, int32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
// All threads of the cluster meet; what each wrote before (shared memory of any of its
// blocks, global memory) is visible to all after.  A block of one member alone meets at its
// barrier 0 by number: the warps of the columns, of the rows and idle ones arrive from
// different places in the code, which __syncthreads() does not allow.  In a cluster the
// compiler's barrier functions, after a warp-wide join: every lane of a warp arrives at the
// same instruction.
template <bool CL>
__device__ __forceinline__ void cluster_meet() {
    if (CL) {
        __syncwarp();
        __cluster_barrier_arrive();
        __cluster_barrier_wait();
    } else {
        asm volatile("barrier.sync 0;" ::: "memory");
    }
}

// What a block's threads share about the solve.
template <typename T>
struct alignas(16) CluCtl {
    T tau, sigma, omega, omw;
    int64_t inner;
    int32_t go;       // run another window
    int32_t restart;  // 1: the evaluation after step 1 is due; 2: the restart copy is due
};

// A lane's entries: the products with the gathered vector, added in order.  The indices
// are the entries' shared addresses in that vector (empty lanes: its zero) and depth is a
// multiple of kCluDepthUnit, so that nothing is tested: a warp that runs alone issues an
// instruction only every few cycles.  The first kCluKept entries stay in registers.
// 4: 1,902 cycles a step at 133 x 201, 8: 1,762, 12: 1,572, 16: 1,457, but at 601 x 1,503
// (seven blocks) 4,340, 4,170, 3,970 and 4,070
constexpr int kCluKept = 12;
template <typename T>
__device__ __forceinline__ T clu_load(uint32_t a);
template <>
__device__ __forceinline__ double clu_load<double>(uint32_t a) {
    double x;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(x) : "r"(a) : "memory");
    return x;
}
template <>
__device__ __forceinline__ float clu_load<float>(uint32_t a) {
    float x;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(a) : "memory");
    return x;
}
template <typename T>
struct CluEntries {
    uint32_t c[kCluKept];
    T a[kCluKept];
    const uint32_t* ip;  // the entries after them
    const T* vp;
    int32_t depth;  // how many, a multiple of kCluDepthUnit
    // A lane of more than kCluLaneNnz entries: one of 32 lanes of a row of more than 512.
    __device__ __forceinline__ bool wide() const { return depth + kCluKept > kCluLaneNnz; }
    // zero: a shared address that holds 0
    __device__ __forceinline__ void take(const uint32_t* i, const T* v, int32_t d, uint32_t zero) {
#pragma unroll
        for (int e = 0; e < kCluKept; ++e) {
            c[e] = e < d ? i[32 * e] : zero;
            a[e] = e < d ? v[32 * e] : T(0);
        }
        ip = i + 32 * kCluKept;
        vp = v + 32 * kCluKept;
        depth = d - kCluKept;
    }
    __device__ __forceinline__ T sum() const {
        T x[kCluKept], acc = T(0);
#pragma unroll
        for (int e = 0; e < kCluKept; ++e) x[e] = clu_load<T>(c[e]);
#pragma unroll
        for (int e = 0; e < kCluKept; ++e) acc = add_rn(acc, mul_rn(a[e], x[e]));  // + 0 leaves the sum as it is
        const uint32_t* i = ip;
        const T* v = vp;
#pragma unroll 1
        for (int d = depth; d > 0; d -= kCluDepthUnit, i += 32 * kCluDepthUnit, v += 32 * kCluDepthUnit) {
            T y[kCluDepthUnit];
#pragma unroll
            for (int e = 0; e < kCluDepthUnit; ++e) y[e] = clu_load<T>(i[32 * e]);
#pragma unroll
            for (int e = 0; e < kCluDepthUnit; ++e) acc = add_rn(acc, mul_rn(v[32 * e], y[e]));
        }
        return acc;
    }
    // The same products, added in FP64: the lanes' sums of a wide row in the FP32 form.
    __device__ __forceinline__ double sum64() const {
        double acc = 0.0;
#pragma unroll
        for (int e = 0; e < kCluKept; ++e) acc += static_cast<double>(mul_rn(a[e], clu_load<T>(c[e])));
        for (int e = 0; e < depth; ++e) acc += static_cast<double>(mul_rn(vp[32 * e], clu_load<T>(ip[32 * e])));
        return acc;
    }
};

// A warp's part in the solve: one slice of one side, its rows' vectors in registers.
template <class P>
struct CluWarp {
    CluEntries<typename P::T> entries;  // its lane's
    int32_t lanes;         // per row
    int32_t i;             // the lane's row (packed), -1: none to update
    uint32_t out;          // shared address of the row's entry in x_bar / z
    typename P::T v[P::NCV];  // rows: the first NRV
};

template <bool ROW, class P>
__device__ __forceinline__ CluWarp<P> clu_warp(const P& prob, unsigned char* sm, const ResDev& d, const ResBlock& b,
                                                   int slice, uint32_t idx, uint32_t val, uint32_t vec, int32_t base,
                                                   const typename P::T* zero) {
    using T = typename P::T;
    const int lane = threadIdx.x & 31;
    const ResSlice m = d.slices[b.slice0 + slice];
    CluWarp<P> w;
    w.entries.take(reinterpret_cast<const uint32_t*>(sm + idx) + m.off + lane,
                   reinterpret_cast<const T*>(sm + val) + m.off + lane, m.shape >> 3, smem_addr(zero));
    w.lanes = 1 << (m.shape & 7);
    const int32_t r = d.lane_row[32 * static_cast<int64_t>(b.slice0 + slice) + lane];
    w.i = r >= 0 && (lane & (w.lanes - 1)) == 0 ? b.row0 + r : -1;
    w.out = smem_addr(sm + vec) + static_cast<uint32_t>(sizeof(T)) * (w.i < 0 ? 0 : w.i - base);
#pragma unroll
    for (int q = 0; q < P::NCV; ++q)
        w.v[q] = w.i >= 0 && (!ROW || q < P::NRV) ? (ROW ? prob.row_vec(q) : prob.col_vec(q))[w.i] : T(0);
    return w;
}

template <bool CL, typename T>
__device__ __forceinline__ void clu_put_all(uint32_t at, T y, uint32_t n_ranks) {
    if (CL) {
#pragma unroll 1
        for (uint32_t c = 0; c < n_ranks; ++c) cluster_put(cluster_map(at, c), y);
    } else {
        cluster_put(at, y);
    }
}

// Steps from .. to - 1 as a warp of the columns (ROW false) or of the rows sees them: a
// pass of its own and a barrier, a pass of the other side and a barrier.  A column's own
// iterates are formed while the rows work: the rows wait only for x_bar.  The steps'
// weights k / (k + 1) are computed by the lanes, 32 steps at a time.
template <bool ROW, bool MAJOR, bool CL, class P>
__device__ __forceinline__ void clu_steps(const P& prob, CluWarp<P>& w, const CluCtl<typename P::T>& ctl, bool eq,
                                          int32_t from, int32_t to, uint32_t n_ranks) {
    using T = typename P::T;
    const int lane = threadIdx.x & 31;
    StepParams<T> p{ctl.tau, ctl.sigma, T(0), T(0), ctl.omega, ctl.omw};
    double weights = 0.0;
    auto weight = [&](int32_t k) {
        if (((k - from) & 31) == 0) {
            const double kk = static_cast<double>(ctl.inner + k + lane);
            weights = kk / (kk + 1.0);
        }
        const double x = __shfl_sync(0xffffffffu, weights, (k - from) & 31);
        p.weight = static_cast<T>(x);
        p.omwt = static_cast<T>(1.0 - x);
    };
    weight(from);
#pragma unroll 1
    for (int32_t k = from; k < to; ++k) {
        if (ROW) cluster_meet<CL>();
        T acc;
        if (sizeof(T) == 4 && w.entries.wide()) {  // the same for the whole warp
            double sum = w.entries.sum64();
#pragma unroll 1
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            acc = static_cast<T>(sum);
        } else {
            acc = w.entries.sum();
            if (w.lanes > 1)
#pragma unroll 1
                for (int o = w.lanes >> 1; o > 0; o >>= 1) acc = add_rn(acc, __shfl_xor_sync(0xffffffffu, acc, o));
        }
        if constexpr (ROW) {
            T in[P::NRV];
#pragma unroll
            for (int q = 0; q < P::NRV; ++q) in[q] = w.v[q];
            if (w.i >= 0) clu_put_all<CL>(w.out, prob.template row<MAJOR>(p, eq, w.i, in, w.v, 1, acc), n_ranks);
            cluster_meet<CL>();
        } else {
            const typename P::X x = prob.col_x(p, w.v, acc);
            if (w.i >= 0) clu_put_all<CL>(w.out, x.rx, n_ranks);
            cluster_meet<CL>();
            if (w.i >= 0) prob.template col_rest<MAJOR>(p, w.i, w.v, x, w.v, 1);
        }
        weight(k + 1);
        if (!ROW) cluster_meet<CL>();
    }
}

// The partial sums of an evaluation Op over 32 consecutive rows (chunk c of the member's
// rows [r0, r1)), one row per lane (a row of more than kCluEvalLong entries: the whole
// warp), its NP terms' sums to the shared address dst.
constexpr int kCluEvalLong = 64;
template <class Op, int NP>
__device__ __forceinline__ void clu_eval(const Op& op, const int32_t* rp, const int32_t* ci, int32_t r0, int32_t r1,
                                         int32_t c, int inst, uint32_t dst) {
    constexpr int NV = Op::NV, U = 8;
    const double* vals = op.values();
    const int lane = threadIdx.x & 31;
    const double* none[1] = {nullptr};
    const int32_t r = r0 + c * kCluEvalRows + lane;
    const int32_t k0 = r < r1 ? rp[r] : 0, k1 = r < r1 ? rp[r + 1] : 0;
    double s[NV], acc[NP];
#pragma unroll
    for (int v = 0; v < NV; ++v) s[v] = 0.0;
#pragma unroll
    for (int k = 0; k < NP; ++k) acc[k] = 0.0;
    if (k1 - k0 <= kCluEvalLong)
#pragma unroll 1
        for (int32_t k = k0; k < k1; k += U) {
            int32_t j[U];
            double a[U], g[U][NV];
#pragma unroll
            for (int e = 0; e < U; ++e) {
                const int32_t at = k + e < k1 ? k + e : k1 - 1;
                j[e] = ci[at];
                a[e] = vals[at];
            }
#pragma unroll
            for (int e = 0; e < U; ++e) op.gather(j[e], g[e]);
#pragma unroll
            for (int e = 0; e < U; ++e)
#pragma unroll
                for (int v = 0; v < NV; ++v) s[v] = add_rn(s[v], k + e < k1 ? mul_rn(a[e], g[e][v]) : 0.0);
        }
    __syncwarp();
    for (unsigned left = __ballot_sync(0xffffffffu, k1 - k0 > kCluEvalLong); left; left &= left - 1) {
        const int who = __ffs(left) - 1;
        const int32_t b = __shfl_sync(0xffffffffu, k0, who), e = __shfl_sync(0xffffffffu, k1, who);
        double t[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) t[v] = 0.0;
        for (int32_t k = b + lane; k < e; k += 32) {
            double g[NV];
            op.gather(ci[k], g);
#pragma unroll
            for (int v = 0; v < NV; ++v) t[v] = add_rn(t[v], mul_rn(vals[k], g[v]));
        }
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            for (int o = 16; o > 0; o >>= 1) t[v] = add_rn(t[v], __shfl_xor_sync(0xffffffffu, t[v], o));
            if (lane == who) s[v] = t[v];
        }
    }
    if (r < r1) op.row(r, r - r0, inst, op.tile_params(inst), none, s, acc);
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < NP; ++k) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NP; ++k) cluster_put(dst + 8u * k, acc[k]);
}

// Windows of members[blockIdx.x / n_ranks].  P: the steps (as the resident window's), the
// evaluation Ops and the controller.  any_stop: a member that stops sets it, and the others
// leave after their window; each runs one at least, also where more members than the GPU
// holds clusters at a time wait for the first ones to leave (of eight blocks, 16 or so).
template <class P, bool CL>
__global__ void __launch_bounds__(kCluThreads, 1)
    cluster_windows_kernel(const P prob, const ResDev dt, const ResDev da, const int32_t* rp_t,
                           const int32_t* ci_t, const int32_t* rp_a, const int32_t* ci_a,
                           const int32_t* col_off, const int32_t* row_off, const ClusterMember* members,
                           uint32_t n_ranks, int32_t max_windows, int32_t* any_stop) {
    using T = typename P::T;
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ CluCtl<T> ctl;
    __shared__ double terms[12];
    __shared__ double ray_terms[3];
    const uint32_t rank = CL ? cluster_rank() : 0u;
    const ClusterMember who = members[blockIdx.x / n_ranks];
    const int p = who.inst, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
    const int32_t c0 = col_off[p], n = col_off[p + 1] - c0, r0 = row_off[p], m = row_off[p + 1] - r0;
    const ResBlock bt = dt.blocks[who.block0 + rank], ba = da.blocks[who.block0 + rank];
    const CluSmem o = clu_smem(bt, ba, sizeof(T), n, m);
    T* const xs = reinterpret_cast<T*>(sm + o.xs);
    T* const zs = reinterpret_cast<T*>(sm + o.zs);
    if (threadIdx.x == 0) {
        const InstState& st = prob.st[p];
        const StepParams<T> q = step_params<T>(st, 0);
        ctl = CluCtl<T>{q.tau, q.sigma, q.omega, q.omw, st.inner, prob.active(p) ? 1 : 0, st.do_restart ? 1 : 0};
        xs[n] = T(0);
        zs[m] = T(0);
    }
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        const ResDev& d = h ? da : dt;
        const ResBlock& b = h ? ba : bt;
        uint32_t* sidx = reinterpret_cast<uint32_t*>(sm + (h ? o.idx_a : o.idx_t));
        T* sval = reinterpret_cast<T*>(sm + (h ? o.val_a : o.val_t));
        const T* gval = static_cast<const T*>(d.val) + b.elem0;
        const uint32_t vec = smem_addr(h ? xs : zs);
        const int32_t base = h ? c0 : r0, zero = h ? n : m;
        for (int32_t k = threadIdx.x; k < b.n_elem; k += blockDim.x) {
            const int32_t c = d.idx[b.elem0 + k];
            sidx[k] = vec + static_cast<uint32_t>(sizeof(T)) * (c >= 0 ? c - base : zero);
            sval[k] = gval[k];
        }
    }
    for (int32_t k = threadIdx.x; k < m; k += blockDim.x) zs[k] = prob.row_vec(0)[r0 + k];
    __syncthreads();
    // the warps of the columns, then those of the rows, then idle ones
    const bool is_col = warp < bt.n_slices, is_row = !is_col && warp < bt.n_slices + ba.n_slices;
    CluWarp<P> w{};
    w.i = -1;
    if (is_col) w = clu_warp<false, P>(prob, sm, dt, bt, warp, o.idx_t, o.val_t, o.xs, c0, zs + m);
    if (is_row) w = clu_warp<true, P>(prob, sm, da, ba, warp - bt.n_slices, o.idx_a, o.val_a, o.zs, r0, xs + n);
    const bool eq = is_row && w.i >= 0 && w.i < prob.eq_end(p);
    cluster_meet<CL>();
    auto minor = [&](int32_t from, int32_t to) {
        if (is_col) {
            clu_steps<false, false, CL>(prob, w, ctl, false, from, to, n_ranks);
        } else if (is_row) {
            clu_steps<true, false, CL>(prob, w, ctl, eq, from, to, n_ranks);
        } else {
#pragma unroll 1
            for (int32_t k = 2 * from; k < 2 * to; ++k) cluster_meet<CL>();
        }
    };
    auto major = [&](int32_t k) {
        if (is_col) {
            clu_steps<false, true, CL>(prob, w, ctl, false, k, k + 1, n_ranks);
        } else if (is_row) {
            clu_steps<true, true, CL>(prob, w, ctl, eq, k, k + 1, n_ranks);
        } else {
            cluster_meet<CL>();
            cluster_meet<CL>();
        }
    };
    // one evaluation and the controller (the first block's first thread), whose outcome
    // goes to every block
    auto evaluate = [&](int32_t which) {
        // the chunks of the columns, then those of the rows, over the cluster's warps
        const int32_t nc = (n + kCluEvalRows - 1) / kCluEvalRows, nr = (m + kCluEvalRows - 1) / kCluEvalRows;
        uint32_t to_c = smem_addr(sm + o.part_c), to_r = smem_addr(sm + o.part_r);
        if (CL) {
            to_c = cluster_map(to_c, 0);
            to_r = cluster_map(to_r, 0);
        }
        for (int32_t c = rank * n_warps + warp; c < nc + nr; c += n_ranks * n_warps)
            if (c < nc)
                clu_eval<typename P::EvalCol, 8>(prob.eval_col(which), rp_t, ci_t, c0, c0 + n, c, p, to_c + 64u * c);
            else
                clu_eval<typename P::EvalRow, 4>(prob.eval_row(which), rp_a, ci_a, r0, r0 + m, c - nc, p, to_r + 32u * (c - nc));
        cluster_meet<CL>();
        if (rank == 0) {
            const int t = threadIdx.x;
            if (t < 12) {
                const int np = t < 8 ? 8 : 4, len = ((t < 8 ? n : m) + kCluEvalRows - 1) / kCluEvalRows;
                const double* q = reinterpret_cast<const double*>(sm + (t < 8 ? o.part_c : o.part_r)) + (t < 8 ? t : t - 8);
                double sum = 0.0;
                for (int c = 0; c < len; ++c) sum += q[np * c];
                terms[t] = sum;
            }
        }
        if constexpr (P::kRays) {
            if (which == EVAL_FULL) {
                // the ray passes: the rays themselves, then their products, both over the
                // chunks above; the partial sums take the places of the terms'
                if (rank == 0) prob.rays_begin();
                cluster_meet<CL>();
                for (int32_t c = rank * n_warps + warp; c < nc + nr; c += n_ranks * n_warps) {
                    const int32_t i = kCluEvalRows * (c < nc ? c : c - nc) + (threadIdx.x & 31);
                    if (c < nc) {
                        if (i < n) prob.ray_col(c0 + i);
                        continue;
                    }
                    double s = i < m ? prob.ray_row(r0 + i) : 0.0;
                    __syncwarp();
#pragma unroll
                    for (int q = 16; q > 0; q >>= 1) s += __shfl_xor_sync(0xffffffffu, s, q);
                    if ((threadIdx.x & 31) == 0) cluster_put(to_r + 32u * (c - nc), s);
                }
                cluster_meet<CL>();
                for (int32_t c = rank * n_warps + warp; c < nc + nr; c += n_ranks * n_warps)
                    if (c < nc)
                        clu_eval<typename P::RayCol, 2>(prob.ray_col_op(), rp_t, ci_t, c0, c0 + n, c, p, to_c + 64u * c);
                    else  // no sums: one place that nothing reads
                        clu_eval<typename P::RayRow, 1>(prob.ray_row_op(), rp_a, ci_a, r0, r0 + m, c - nc, p, to_r + 32u * (c - nc) + 8u);
                cluster_meet<CL>();
                if (rank == 0 && threadIdx.x < 3) {
                    const int t = threadIdx.x, np = t < 2 ? 8 : 4, len = t < 2 ? nc : nr;
                    const double* q = reinterpret_cast<const double*>(sm + (t < 2 ? o.part_c : o.part_r)) + (t < 2 ? t : 0);
                    double sum = 0.0;
                    for (int c = 0; c < len; ++c) sum += q[np * c];
                    ray_terms[t] = sum;
                }
            }
        }
        if (rank == 0) {
            const int t = threadIdx.x;
            __syncthreads();
            if (t == 0) {
                if constexpr (P::kRays)
                    if (which == EVAL_FULL) prob.rays_finalize(p, ray_terms);
                prob.finalize(p, terms, which);
                const InstState& st = prob.st[p];
                const StepParams<T> q = step_params<T>(st, 0);
                int32_t go = st.status == ST_RUNNING && !prob.polish(p);
                if (which == EVAL_FULL && any_stop) {
                    if (st.status != ST_RUNNING) atomicExch(any_stop, 1);
                    go = go && !*reinterpret_cast<volatile int32_t*>(any_stop);
                }
                for (uint32_t b = 0; b < n_ranks; ++b) {
                    auto to = [&](const void* f) { return CL ? cluster_map(smem_addr(f), b) : smem_addr(f); };
                    if (which == EVAL_FULL) {
                        cluster_put(to(&ctl.tau), q.tau);
                        cluster_put(to(&ctl.sigma), q.sigma);
                        cluster_put(to(&ctl.inner), static_cast<int32_t>(st.inner));
                        cluster_put(to(&ctl.inner) + 4, static_cast<int32_t>(st.inner >> 32));
                        cluster_put(to(&ctl.go), go);
                        cluster_put(to(&ctl.restart), st.restart_now ? 2 : 0);
                    } else {
                        cluster_put(to(&ctl.restart), 0);
                    }
                }
            }
        }
        cluster_meet<CL>();
    };
    const int32_t freq = prob.st[p].freq;
#pragma unroll 1
    for (int32_t win = 0; win < max_windows && ctl.go; ++win) {
        major(1);
        if (ctl.restart == 1) evaluate(EVAL_AFTER_RESTART);
        if (freq > 1) {
            minor(2, freq);
            major(freq);
        }
        evaluate(EVAL_FULL);
        if (ctl.restart == 2) {  // initial = current = pdhg
            if (w.i >= 0 && is_col) prob.col_restart(w.i, w.v);
            if (w.i >= 0 && is_row) prob.row_restart(w.i, w.v);
            for (int32_t k = threadIdx.x; k < m; k += blockDim.x) zs[k] = prob.row_pdhg()[r0 + k];
            __syncthreads();
            if (threadIdx.x == 0) ctl.restart = 1;
        }
        cluster_meet<CL>();
    }
#pragma unroll
    for (int q = 0; q < P::NCV; ++q)  // the iterates back to global memory
        if (P::col_changes(q) && is_col && w.i >= 0) prob.col_vec(q)[w.i] = w.v[q];
#pragma unroll
    for (int q = 0; q < P::NRV; ++q)
        if (P::row_changes(q) && is_row && w.i >= 0) prob.row_vec(q)[w.i] = w.v[q];
}

// The cluster form of one handle and precision on the host.  Members that need the same
// number of blocks run in one launch; the launches of different numbers run side by side, on
// streams of their own that fork from the handle's and join it again.  (One number for all,
// the largest: 999 members of 133 x 201 and one of 601 x 1,503, 400 iterations, 34.7 ms on
// the device, 2.4 now; 16.0 when each ran in one block.)
struct ClusterForm {
    bool tried = false;
    DeviceMatrix::Resident r;  // blocks of every member in turn; n_blocks == 0: does not fit
    std::vector<DeviceMatrix::ClusterGroup> groups;
    bool ready() const { return r.n_blocks > 0; }
    ClusterForm() = default;
    ClusterForm(const ClusterForm&) = delete;
    ClusterForm& operator=(const ClusterForm&) = delete;
    ~ClusterForm() {
        for (const Side& s : sides_) {
            if (s.done) cudaEventDestroy(s.done);
            if (s.stream) cudaStreamDestroy(s.stream);
        }
        if (fork_) cudaEventDestroy(fork_);
    }

    // Lays every member out, if each fits a cluster; the values follow with fill().
    template <class P>
    void prepare(const DeviceMatrix& M, DeviceArena& ar, int max_smem_block) {
        using T = typename P::T;
        if (tried) return;
        tried = true;
        const uint32_t cap = static_cast<uint32_t>(max_smem_block) - 2048;  // its static memory
        DeviceMatrix::Resident f;
        if (!M.make_cluster(ar, kCluMaxBlocks, sizeof(T), kCluWarps, cap, f, groups)) return;
        for (const auto& g : groups)
            if (g.n_ranks == 1) set_attr(cluster_windows_kernel<P, false>, cap); else set_attr(cluster_windows_kernel<P, true>, cap);
        if (groups.size() > 1) {
            PDFP_CK(cudaEventCreateWithFlags(&fork_, cudaEventDisableTiming));
            sides_.resize(groups.size() - 1);
            for (Side& s : sides_) {
                PDFP_CK(cudaStreamCreateWithFlags(&s.stream, cudaStreamNonBlocking));
                PDFP_CK(cudaEventCreateWithFlags(&s.done, cudaEventDisableTiming));
            }
        }
        r = f;
    }
    // The matrix's values into the layout, once; stream-ordered.
    template <class P>
    void fill(const DeviceMatrix& M, DeviceArena& ar, cudaStream_t stream) {
        if (ready() && !r.t.val) M.fill_resident(ar, r, std::is_same<typename P::T, float>::value, stream);
    }

    template <class P>
    void launch(const P& prob, const DeviceMatrix& M, int32_t* any_stop, cudaStream_t stream) const {
        if (!sides_.empty()) PDFP_CK(cudaEventRecord(fork_, stream));
        for (size_t k = 0; k < groups.size(); ++k) {
            const Side side = k > 0 ? sides_[k - 1] : Side{stream, nullptr};
            if (k > 0) PDFP_CK(cudaStreamWaitEvent(side.stream, fork_, 0));
            launch_group(groups[k], prob, M, any_stop, side.stream);
            if (k > 0) {
                PDFP_CK(cudaEventRecord(side.done, side.stream));
                PDFP_CK(cudaStreamWaitEvent(stream, side.done, 0));
            }
        }
    }

  private:
    struct Side {
        cudaStream_t stream = nullptr;
        cudaEvent_t done = nullptr;
    };
    std::vector<Side> sides_;  // of the groups after the first
    cudaEvent_t fork_ = nullptr;

    template <class P>
    void launch_group(const DeviceMatrix::ClusterGroup& g, const P& prob, const DeviceMatrix& M, int32_t* any_stop,
                      cudaStream_t stream) const {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>(g.n_ranks) * static_cast<unsigned>(g.count));
        cfg.blockDim = dim3(static_cast<unsigned>(32 * g.n_warps));
        cfg.dynamicSmemBytes = g.smem;
        cfg.stream = stream;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = static_cast<unsigned>(g.n_ranks);
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = g.n_ranks > 1 ? 1 : 0;
        auto run = [&](auto kern) {
            PDFP_CK(cudaLaunchKernelEx(&cfg, kern, prob, r.t, r.a, static_cast<const int32_t*>(M.rp_t),
                                       static_cast<const int32_t*>(M.ci_t), static_cast<const int32_t*>(M.rp_a),
                                       static_cast<const int32_t*>(M.ci_a), static_cast<const int32_t*>(M.col_off),
                                       static_cast<const int32_t*>(M.row_off), g.members,
                                       static_cast<uint32_t>(g.n_ranks), static_cast<int32_t>(kCluWindowsPerLaunch),
                                       any_stop));
        };
        if (g.n_ranks > 1) run(cluster_windows_kernel<P, true>); else run(cluster_windows_kernel<P, false>);
    }
    template <class K>
    static void set_attr(K kern, uint32_t cap) {  // the same for every handle: never lowered under another one
        PDFP_CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(cap)));
    }
};

}  // namespace pdfp

// resident_steps.cuh -- a window's steps in one cooperative launch that keeps the
// whole problem on the chip.
//
// A handle of some thousands to about a million nonzeros is bound by latency: its step
// launches take 5-7 us each for 1-3 us of work (two launches per step, each waiting for
// the previous one's drain, then for item, row pointer, index and gather in turn).
// Here one block per SM owns a fixed range of the rows of A' (columns) and of A and
// keeps everything of theirs in shared memory for the whole launch: indices and values
// as 32-lane slices (ResSlice, layout.hpp), the iterates, the anchors and the data.
// Only x_bar and z cross between blocks, and they cross without a barrier: an entry is
// written to global memory together with the step it belongs to, in one 16-byte (FP32:
// 8-byte) access, and a gather repeats until it reads the step it needs.  One buffer per
// vector is enough: x_bar_j of the next step is written only after column j has read the
// new z of every row it meets, and each of these rows has read the old x_bar_j by then
// (and the same with rows and columns exchanged).  The launch is cooperative, so every
// block is resident and every wait ends; all the same each wait is bounded (kResWaitNs).
//
// What bounds it: an entry takes about 950 cycles from one SM to another (a ping-pong of
// tagged entries), a pass that only exchanges 700 gathers per SM 2,300 cycles and one
// with 3,400 gathers 5,000 (an SM gets about one scattered gather per cycle through).
// Measured per PDHG iteration (one B200, FP64, whole solves): 4,001 x 10,007 with 100k
// nonzeros 13.7 -> 4.3 us, 20,000 x 50,000 with 500k 15.4 -> 7.8 us (mixed form 12.8 ->
// 7.8).  What does not depend on the pass is read before the wait (4.7 and 8.2 us when it
// was read after).  The same passes with a grid barrier after each instead of tagged entries
// (release, atomic, acquire, then the gathers) took 6.3 and 11 us.
//
// The order in which a row's terms are added depends on its length alone (its lanes
// take every 2^lg-th term, then an xor tree; pieces of a long row, which are summed in FP64,
// in order), so a batch member with its own handle's step size takes its steps bit for bit.
#pragma once
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "device.hpp"
#include "layout.hpp"
#include "pdfp_ops.cuh"

namespace pdfp {

// 16 warps with 128 registers (timed before the reads moved ahead of the wait): 1.87 / 3.26 / 3.39 ms for 400 iterations of the models above
// (100k FP64, 500k mixed, 500k FP64) against 2.31 / 3.43 / 3.96 with 32 warps, whose passes
// spill, and 2.08 / 3.63 / 3.74 with 24.
constexpr int kResThreads = 512;
constexpr uint64_t kResWaitNs = 2000000000ull;  // a wait for an entry longer than 2 s is declared hung

// One entry of a vector that crosses between blocks, with the step it belongs to.
template <typename T>
struct ResWord;
template <>
struct alignas(16) ResWord<double> {
    double v;
    unsigned long long tag;
};
template <>
struct alignas(8) ResWord<float> {
    float v;
    unsigned tag;
};
__device__ __forceinline__ void res_put(ResWord<double>* p, double v, int32_t tag) {
    asm volatile("{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"(static_cast<long long>(tag)) : "memory");
}
__device__ __forceinline__ void res_put(ResWord<float>* p, float v, int32_t tag) {
    const unsigned long long w = static_cast<unsigned long long>(static_cast<unsigned>(tag)) << 32 | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ void res_get(const ResWord<double>* p, double& v, int32_t& tag) {
    long long a, t;
    asm volatile("{\n\t.reg .b128 w;\n\tld.relaxed.gpu.global.b128 w, [%2];\n\tmov.b128 {%0, %1}, w;\n\t}"
                 : "=l"(a), "=l"(t) : "l"(p) : "memory");
    v = __longlong_as_double(a);
    tag = static_cast<int32_t>(t);
}
__device__ __forceinline__ void res_get(const ResWord<float>* p, float& v, int32_t& tag) {
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    v = __uint_as_float(static_cast<unsigned>(w));
    tag = static_cast<int32_t>(w >> 32);
}

// The projector's steps (src/pdfp.jl:119-156) as the resident window runs them.
template <typename TT>
struct PdfpResident {
    using T = TT;
    static constexpr int NCV = 8, NRV = 3;
    IterVecs<T> v;
    const InstState* st;
    const int32_t *row_off, *n_eq;
    int32_t mode;
    int32_t* errp;
    __device__ bool active(int p) const { return st[p].status == ST_RUNNING && st[p].mode == mode; }
    __device__ int32_t eq_end(int p) const { return row_off[p] + n_eq[p]; }
    __device__ T* col_vec(int q) const {
        T* const s[NCV] = {v.cx, v.ix, v.cy, v.iy, v.lb, v.ub, v.xt, v.w};
        return s[q];
    }
    __device__ T* row_vec(int q) const {
        T* const s[NRV] = {v.cz, v.iz, v.b};
        return s[q];
    }
    // column j with its vectors, read as `in`, at pv[q * n]: first x_bar_j (.rx), for which
    // others wait, then its own iterates
    using X = PrimalX<T>;
    __device__ __forceinline__ X col_x(const StepParams<T>& p, const T (&in)[NCV], T sum) const {
        return primal_x(p, in, sum);
    }
    template <bool MAJOR>
    __device__ __forceinline__ void col_rest(const StepParams<T>& p, int32_t j, const T (&in)[NCV], const X& x,
                                             T* pv, int n) const {
        const PrimalRest<T> o = primal_rest(p, in, x.rx);
        pv[0] = o.cx;
        pv[2 * n] = o.cy;
        if (MAJOR) {
            v.rx[j] = x.rx;
            v.px[j] = x.px;
            v.ds[j] = sub_rn(x.px, x.t) / p.tau;
            v.py[j] = o.py;
            v.ry[j] = o.ry;
        }
    }
    // row i likewise; returns z_i
    template <bool MAJOR>
    __device__ __forceinline__ T row(const StepParams<T>& p, bool eq, int32_t i, const T (&in)[NRV], T* pv,
                                     int, T sum) const {
        const DualCell<T> o = dual_cell(p, eq, in, sum);
        pv[0] = o.cz;
        if (MAJOR) {
            v.pz[i] = o.pz;
            v.rz[i] = o.rz;
        }
        return o.cz;
    }
    // the vectors that the steps change (row vector 0 is the one that columns gather)
    __device__ static bool col_changes(int q) { return q == 0 || q == 2; }
    __device__ static bool row_changes(int q) { return q == 0; }
};

// An instance in a block's shared memory: its parameters for the launch, and the step's
// weights for even and odd steps.
template <typename T>
struct alignas(16) ResPar {
    T tau, sigma, omega, omw;
    T weight[2], omwt[2];
    int64_t inner;
    int32_t eq_end, act;
};

// One block's share of one side: shared-memory offsets, and the vectors that cross.
template <typename T>
struct ResSide {
    const ResWord<T>* in;  // the entries this side gathers
    ResWord<T>* out;       // and the ones it writes
    uint32_t idx, val, prod, slices, lane, longs, vec, slots, arr, par;
    int32_t n_slices, n_elem, row0, rows;
    int32_t first_warp;    // the warp that sums slice 0
    uint32_t par_all;      // the parameter entries of both sides (they adjoin)
    int32_t n_par;
};

// After 64 fruitless looks: whether the wait is over for good.
static __device__ __noinline__ bool res_gave_up(unsigned* dead, int32_t* err, uint64_t& t0,
                                                uint64_t limit_ns = kResWaitNs) {
    const uint64_t now = globaltimer_ns();
    if (t0 == 0) t0 = now;
    if (*reinterpret_cast<volatile unsigned*>(dead)) return true;
    if (now - t0 <= limit_ns) return false;
    atomicExch(dead, 1u);
    if (err) atomicExch(err, DEV_ERR_TIMEOUT);
    return true;
}

// Waits for an entry of step `want`; `off` once this or another wait gave up.
template <typename T>
__device__ __forceinline__ void res_wait(const ResWord<T>* entry, int32_t want, unsigned* dead, int32_t* err, bool& off,
                                         uint64_t limit_ns = kResWaitNs) {
    uint64_t t0 = 0;
    unsigned spins = 0;
    while (!off) {
        T x;
        int32_t t;
        res_get(entry, x, t);
        if (t == want) break;
        if ((++spins & 63u) == 0) off = res_gave_up(dead, err, t0, limit_ns);
    }
}

// A piece of a long row: the lanes' products pp[0], pp[32], .. (depth of them) and then the
// lanes are summed in FP64, as in every engine's long rows; the piece that arrives last adds
// the row's pieces in order.  Returns the row (lane 0 of that warp; its sum in acc), else -1.
template <typename T>
__device__ __noinline__ int32_t res_long(unsigned char* sm, const ResSide<T>& s, const ResSlice& m,
                                         int32_t q, const T* pp, T& acc) {
    double part = 0.0;
    for (int u = 0; u < (m.shape >> 3); ++u) part += static_cast<double>(pp[32 * u]);
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if ((threadIdx.x & 31) != 0) return -1;
    const int32_t ln = reinterpret_cast<const int32_t*>(sm + s.lane)[q * 32];
    const ResLong l = reinterpret_cast<const ResLong*>(sm + s.longs)[ln];
    volatile double* slots = reinterpret_cast<volatile double*>(sm + s.slots);
    int32_t* arr = reinterpret_cast<int32_t*>(sm + s.arr);
    slots[m.slot] = part;
    __threadfence_block();
    if (atomicAdd(arr + ln, 1) != l.np - 1) return -1;
    __threadfence_block();
    arr[ln] = 0;
    double tot = 0.0;
    for (int32_t e = 0; e < l.np; ++e) tot += slots[l.slot0 + e];
    acc = static_cast<T>(tot);
    return l.row;
}

// The weights k / (k + 1) of step k of every instance of the block.
template <typename T>
__device__ __forceinline__ void res_weights(unsigned char* sm, const ResSide<T>& s, int32_t k, int t, int n) {
    ResPar<T>* par = reinterpret_cast<ResPar<T>*>(sm + s.par_all);
    for (int32_t p = t; p < s.n_par; p += n) {
        const double kk = static_cast<double>(par[p].inner + k);
        const double weight = kk / (kk + 1.0);
        par[p].weight[k & 1] = static_cast<T>(weight);
        par[p].omwt[k & 1] = static_cast<T>(1.0 - weight);
    }
}

// The sum of a lane's products, in order.
template <typename T>
__device__ __forceinline__ T res_sum(const T* pp, int depth) {
    T acc = T(0);
#pragma unroll 1
    for (; depth >= 8; depth -= 8, pp += 256) {
        T x[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = pp[32 * e];
#pragma unroll
        for (int e = 0; e < 8; ++e) acc = add_rn(acc, x[e]);
    }
    T x[7];
#pragma unroll
    for (int e = 0; e < 7; ++e) x[e] = e < depth ? pp[32 * e] : T(0);
#pragma unroll
    for (int e = 0; e < 7; ++e) acc = add_rn(acc, x[e]);  // + 0 leaves the sum as it is
    return acc;
}

// One pass of one side in step k: gathers entries of step `want`, writes its own entries
// with tag `tag`.
//  1. Every thread of the block gathers and multiplies the entries threadIdx.x + e *
//     kResThreads, wherever their rows are: one warp gets a 16-byte gather of 32 lanes
//     through in about 230 cycles (eight of them: 2,030; eight warps with one each:
//     417), so the gathers are spread over all warps, few per lane.  One lane per warp
//     watches for an entry first: all lanes polling would saturate L2.
//  2. One barrier of the block.
//  3. One thread per row (2^lg for a row of more than kResLaneNnz entries) sums the
//     products in order and runs the epilogue: as many rows per FP64 instruction as
//     lanes.  The other warps are already waiting for the next pass's entries.
// The products of the two sides have their own memory, so the next pass may form its
// products while this one's are summed.
// Both sides run through the same code, and what is rare (major steps, long rows, the
// wait's limit) stays out of it: a step is one pass through a few hundred instructions
// by warps that have just been idle, so instructions that miss the small instruction
// cache cost more than the arithmetic.
template <class P, bool MAJOR>
__device__ __forceinline__ void res_pass(const P& prob, unsigned char* sm, const ResSide<typename P::T>& s,
                                         bool is_row, int32_t k, unsigned* dead, bool& off) {
    using T = typename P::T;
    constexpr int U = 4;  // gathers in flight per thread: 2 and 8 measured slower (1.92 and 2.29 ms for 1.87)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int32_t want = k;
    const int32_t* idx = reinterpret_cast<const int32_t*>(sm + s.idx);
    const T* val = reinterpret_cast<const T*>(sm + s.val);
    T* prod = reinterpret_cast<T*>(sm + s.prod);
    // the warp's first slice, its lanes' rows with their vectors and the step's parameters,
    // read before the wait
    int32_t q = (warp + kResThreads / 32 - s.first_warp) % (kResThreads / 32), r = -1;
    ResSlice m{};
    StepParams<T> p{};
    int32_t eq_end = 0;
    bool act = false;
    T in[P::NCV];
    auto read_vecs = [&](int32_t row) {
        const T* pv = reinterpret_cast<const T*>(sm + s.vec) + row;
#pragma unroll
        for (int e = 0; e < P::NCV; ++e)
            if (e < P::NRV || !is_row) in[e] = pv[e * s.rows];
    };
    auto next_slice = [&]() {
        if (q >= s.n_slices) return;
        m = reinterpret_cast<const ResSlice*>(sm + s.slices)[q];
        r = reinterpret_cast<const int32_t*>(sm + s.lane)[q * 32 + lane];
        if (m.slot >= 0) r = 0;
        const ResPar<T>& pr = reinterpret_cast<const ResPar<T>*>(sm + s.par)[m.inst];
        p = StepParams<T>{pr.tau, pr.sigma, T(0), T(0), pr.omega, pr.omw};
        eq_end = pr.eq_end;
        act = pr.act != 0;
        read_vecs(r < 0 ? 0 : r);
    };
    next_slice();
    if (lane == 0 && static_cast<int32_t>(threadIdx.x) < s.n_elem) {
        const int32_t c = idx[threadIdx.x];
        if (c >= 0) res_wait(s.in + c, want, dead, prob.errp, off);
    }
    __syncwarp();
#pragma unroll 1
    for (int32_t e0 = threadIdx.x; e0 < s.n_elem; e0 += U * kResThreads) {
        int32_t c[U], t[U];
        T x[U];
#pragma unroll
        for (int e = 0; e < U; ++e) c[e] = e0 + e * kResThreads < s.n_elem ? idx[e0 + e * kResThreads] : -1;
#pragma unroll
        for (int e = 0; e < U; ++e) {
            t[e] = want;
            if (c[e] >= 0) res_get(s.in + c[e], x[e], t[e]);
        }
        uint64_t t0 = 0;
        unsigned spins = 0;
        while (!off) {
            bool ready = true;
#pragma unroll
            for (int e = 0; e < U; ++e) ready = ready && t[e] == want;
            if (ready) break;
#pragma unroll
            for (int e = 0; e < U; ++e)
                if (t[e] != want) res_get(s.in + c[e], x[e], t[e]);
            if ((++spins & 63u) == 0) off = res_gave_up(dead, prob.errp, t0);
        }
#pragma unroll
        for (int e = 0; e < U; ++e)
            if (c[e] >= 0) prod[e0 + e * kResThreads] = mul_rn(val[e0 + e * kResThreads], x[e]);
    }
    __syncthreads();
#pragma unroll 1
    while (q < s.n_slices) {
        if (act) {
            const bool piece = m.slot >= 0;
            const ResPar<T>& pr = reinterpret_cast<const ResPar<T>*>(sm + s.par)[m.inst];
            p.weight = pr.weight[k & 1];  // written in the pass before
            p.omwt = pr.omwt[k & 1];
            const T* const pp = prod + m.off + lane;
            T acc = T(0);
            if (piece) {
                r = res_long<T>(sm, s, m, q, pp, acc);
                if (r >= 0) read_vecs(r);
            } else {
                acc = res_sum(pp, m.shape >> 3);
            }
            if (!piece && (m.shape & 7)) {
                const int G = 1 << (m.shape & 7);
#pragma unroll 1
                for (int o = G >> 1; o > 0; o >>= 1) acc = add_rn(acc, __shfl_xor_sync(0xffffffffu, acc, o));
                if (lane & (G - 1)) r = -1;
            }
            if (r >= 0) {
                const int32_t i = s.row0 + r;
                T* pv = reinterpret_cast<T*>(sm + s.vec) + r;
                if (is_row) {
                    T in3[P::NRV];
#pragma unroll
                    for (int e = 0; e < P::NRV; ++e) in3[e] = in[e];
                    res_put(s.out + i, prob.template row<MAJOR>(p, i < eq_end, i, in3, pv, s.rows, acc), k + 1);
                } else {
                    const typename P::X x = prob.col_x(p, in, acc);
                    res_put(s.out + i, x.rx, k);
                    prob.template col_rest<MAJOR>(p, i, in, x, pv, s.rows);
                }
            }
            __syncwarp();
        }
        q += kResThreads / 32;
        next_slice();
    }
    if (is_row && warp == kResThreads / 32 - 1) res_weights<T>(sm, s, k + 1, lane, 32);  // before the next barrier
}

// Steps i0 .. i1 of every active instance (K of them), i0 >= 1; step i1 is major.
// wx / wz: the tagged copies of x_bar and z, all tags zero at launch.  One block per SM,
// cooperative, blocks as dealt by deal_resident.
template <class P>
__global__ void __launch_bounds__(kResThreads, 1)
    resident_steps_kernel(const P prob, const ResDev dt, const ResDev da, ResWord<typename P::T>* wx,
                          ResWord<typename P::T>* wz, unsigned* dead, int K, int32_t i0, int32_t i1) {
    using T = typename P::T;
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ ResSide<T> sides[2];  // 0: columns, 1: rows
    int any = 0;
    for (int p = threadIdx.x; p < K; p += kResThreads) any |= prob.active(p) ? 1 : 0;
    if (!__syncthreads_or(any)) return;  // the same answer in every block
    {
        const ResBlock bt = dt.blocks[blockIdx.x], ba = da.blocks[blockIdx.x];
        const ResSmem o = res_smem(bt, ba, sizeof(T), P::NCV, P::NRV, sizeof(ResPar<T>));
        if (threadIdx.x == 0) {
            sides[0] = ResSide<T>{wz, wx, o.idx_t, o.val_t, o.prod_t, o.slice_t, o.lane_t, o.long_t, o.col,
                                  o.slots_t, o.arr_t, o.par_t, bt.n_slices, bt.n_elem, bt.row0,
                                  bt.row1 - bt.row0, 0, o.par_t, bt.n_inst + ba.n_inst};
            // the row slices go to the warps after those of the column slices
            sides[1] = ResSide<T>{wx, wz, o.idx_a, o.val_a, o.prod_a, o.slice_a, o.lane_a, o.long_a, o.row,
                                  o.slots_a, o.arr_a, o.par_a, ba.n_slices, ba.n_elem, ba.row0,
                                  ba.row1 - ba.row0, bt.n_slices % (kResThreads / 32), o.par_t, bt.n_inst + ba.n_inst};
        }
        __syncthreads();
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
            const ResSide<T>& s = sides[h];
            const ResDev& d = h ? da : dt;
            const ResBlock& b = h ? ba : bt;
            int32_t* sidx = reinterpret_cast<int32_t*>(sm + s.idx);
            T* sval = reinterpret_cast<T*>(sm + s.val);
            T* sprod = reinterpret_cast<T*>(sm + s.prod);
            const T* gval = static_cast<const T*>(d.val) + b.elem0;
#pragma unroll 2
            for (int32_t k = threadIdx.x; k < b.n_elem; k += kResThreads) {
                sidx[k] = __ldcs(d.idx + b.elem0 + k);
                sval[k] = __ldcs(gval + k);
                sprod[k] = T(0);  // entries without a gather stay 0
            }
#pragma unroll 1
            for (int32_t k = threadIdx.x; k < 32 * b.n_slices; k += kResThreads)
                reinterpret_cast<int32_t*>(sm + s.lane)[k] = d.lane_row[static_cast<int64_t>(32) * b.slice0 + k];
#pragma unroll 1
            for (int32_t k = threadIdx.x; k < b.n_slices; k += kResThreads)
                reinterpret_cast<ResSlice*>(sm + s.slices)[k] = d.slices[b.slice0 + k];
#pragma unroll 1
            for (int32_t k = threadIdx.x; k < b.n_long; k += kResThreads) {
                reinterpret_cast<ResLong*>(sm + s.longs)[k] = d.longs[b.long0 + k];
                reinterpret_cast<int32_t*>(sm + s.arr)[k] = 0;
            }
#pragma unroll 1
            for (int32_t k = threadIdx.x; k < b.n_inst; k += kResThreads) {
                const int p = b.inst0 + k;
                const StepParams<T> q = step_params<T>(prob.st[p], 0);
                reinterpret_cast<ResPar<T>*>(sm + s.par)[k] =
                    ResPar<T>{q.tau, q.sigma, q.omega, q.omw, {T(0), T(0)}, {T(0), T(0)}, prob.st[p].inner,
                              prob.eq_end(p), prob.active(p) ? 1 : 0};
            }
            T* vec = reinterpret_cast<T*>(sm + s.vec);
#pragma unroll 1
            for (int q = 0; q < (h ? P::NRV : P::NCV); ++q) {
                const T* src = (h ? prob.row_vec(q) : prob.col_vec(q)) + b.row0;
                for (int32_t k = threadIdx.x; k < s.rows; k += kResThreads) {
                    const T v = src[k];
                    vec[q * s.rows + k] = v;
                    if (h && q == 0) res_put(wz + b.row0 + k, v, i0);  // z as the first step gathers it
                }
            }
        }
        __syncthreads();
        // the entries of instances that do not run: nobody writes what they would wait for
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
            const ResSide<T>& s = sides[h];
            for (int32_t q = threadIdx.x >> 5; q < s.n_slices; q += kResThreads / 32) {
                const ResSlice m = reinterpret_cast<const ResSlice*>(sm + s.slices)[q];
                if (!reinterpret_cast<const ResPar<T>*>(sm + s.par)[m.inst].act)
                    for (int u = 0; u < (m.shape >> 3); ++u)
                        reinterpret_cast<int32_t*>(sm + s.idx)[m.off + 32 * u + (threadIdx.x & 31)] = -1;
            }
        }
    }
    res_weights<T>(sm, sides[0], i0, threadIdx.x, kResThreads);
    __syncthreads();
    bool off = false;
#pragma unroll 1
    for (int32_t h = 2 * i0; h < 2 * i1; ++h)
        res_pass<P, false>(prob, sm, sides[h & 1], h & 1, h >> 1, dead, off);
#pragma unroll 1
    for (int h = 0; h < 2; ++h)
        res_pass<P, true>(prob, sm, sides[h], h != 0, i1, dead, off);
    __syncthreads();
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        const ResSide<T>& s = sides[h];
        const T* vec = reinterpret_cast<const T*>(sm + s.vec);
#pragma unroll 1
        for (int q = 0; q < (h ? P::NRV : P::NCV); ++q)
            if (h ? P::row_changes(q) : P::col_changes(q)) {
                T* dst = (h ? prob.row_vec(q) : prob.col_vec(q)) + s.row0;
                for (int32_t k = threadIdx.x; k < s.rows; k += kResThreads) dst[k] = vec[q * s.rows + k];
            }
    }
}

// The resident form of one handle and precision on the host.
struct ResidentForm {
    DeviceMatrix::Resident r;  // n_blocks == 0: not laid out
    bool ready() const { return r.n_blocks > 0; }

    // Whether the handle fits, decided the first time on the host: nothing goes to the device.
    template <class P>
    bool plan(const DeviceMatrix& M, int num_sms, int max_smem_block) {
        using T = typename P::T;
        if (planned_) return fits_;
        planned_ = true;
        if (M.L.NNZ == 0) return false;
        const uint32_t cap = static_cast<uint32_t>(max_smem_block) - 1024;  // its static memory
        // Where it stops to pay: 400 iterations of general-integer models, resident against
        // per-step launches, FP64 500k nonzeros (187 KB a block) 3.2 / 5.7 ms, 610k (about
        // 226 KB) 5.1 / 7.5; mixed 900k (194 KB) 4.5 / 6.3, 970k (200 KB) 4.6 / 6.4, 1M
        // (205 KB) 7.0 / 6.5: what shared memory takes, the gathers' misses lack in L1.
        const uint32_t most = sizeof(T) == 4 ? std::min(cap, 200u * 1024u) : cap;
        if (!M.plan_resident(num_sms, sizeof(T), P::NCV, P::NRV, sizeof(ResPar<T>), most, t_, a_, smem_)) {
            t_ = a_ = HostResident();
            return false;
        }
        auto kern = resident_steps_kernel<P>;
        int coop = 0, dev = 0, per_sm = 0;
        PDFP_CK(cudaGetDevice(&dev));
        PDFP_CK(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
        PDFP_CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(cap)));
        PDFP_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kResThreads, smem_));
        fits_ = coop && per_sm >= 1;
        return fits_;
    }

    // Lays the handle out for P's steps the first time, if it fits; stream-ordered.
    template <class P>
    void prepare(const DeviceMatrix& M, DeviceArena& ar, int num_sms, int max_smem_block, cudaStream_t stream) {
        using T = typename P::T;
        if (ready() || !plan<P>(M, num_sms, max_smem_block)) return;
        DeviceMatrix::Resident f;
        M.upload_resident(ar, t_, a_, 32 * kResLaneNnz, f);
        t_ = a_ = HostResident();
        f.smem = smem_;
        M.fill_resident(ar, f, std::is_same<T, float>::value, stream);
        words_bytes = sizeof(ResWord<T>) * (M.L.N + M.L.M) + 16;
        words = ar.alloc<unsigned char>(words_bytes);
        n_cols = M.L.N;
        n_rows = M.L.M;
        r = f;
    }

    // Steps i0 .. i1 of every active instance of K, the last one major.
    template <class P>
    void launch(const P& prob, int K, int i0, int i1, cudaStream_t stream) const {
        using T = typename P::T;
        ResWord<T>* const wx = static_cast<ResWord<T>*>(words);
        ResWord<T>* const wz = wx + n_cols;
        unsigned* const dead = reinterpret_cast<unsigned*>(wz + n_rows);
        PDFP_CK(cudaMemsetAsync(words, 0, words_bytes, stream));  // no entry of any step, nobody gave up
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>(r.n_blocks));
        cfg.blockDim = dim3(kResThreads);
        cfg.dynamicSmemBytes = r.smem;
        cfg.stream = stream;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        PDFP_CK(cudaLaunchKernelEx(&cfg, resident_steps_kernel<P>, prob, r.t, r.a, wx, wz, dead, K,
                                   static_cast<int32_t>(i0), static_cast<int32_t>(i1)));
    }

  private:
    bool planned_ = false, fits_ = false;
    HostResident t_, a_;  // from plan() to prepare()
    uint32_t smem_ = 0;   // of the largest block
    void* words = nullptr;     // the tagged x_bar (N) and z (M), and the give-up word
    size_t words_bytes = 0;
    int64_t n_cols = 0, n_rows = 0;
};

}  // namespace pdfp

// precond.cu -- the diagonal preconditioner on the device.
//
// scale_problem, src/preconditioner.jl:26-99: ten Ruiz rounds (1/sqrt of the
// largest |a| per row and column), one Pock-Chambolle pass (1/sqrt of the sum
// of |a|^alpha per row, |a|^(2-alpha) per column), then the scaled bounds and
// the optional bound/objective rescaling.  Row sums are taken by one thread per row of
// A (and of A') in ascending index order, row maxima, which no order changes, by eight
// lanes, so the scaling factors and scaled values are bit-identical to the reference's CPU
// arithmetic (Julia walks its CSC matrix column by column, which gives each row
// sum its terms in ascending column order and each column sum in ascending row
// order).  The scaled bounds, costs and the optional bound/objective rescaling
// (two sequential norms, as the reference's loops) run on the device too.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "device.hpp"
#include "kernels.cuh"
#include "power.cuh"
#include "solvers.hpp"

namespace pdfp {

static constexpr double SCALING_EPSILON = 1e-12;  // src/preconditioner.jl:11

// One Ruiz round over both sides of the matrix in one launch: entries times the scales of
// the round before (none in the first), D times the row's own, and from the new entries
// the row's next scale, 1/sqrt(max |v|) (1 if below SCALING_EPSILON; none in the last).
// kRoundLanes lanes per row, since no result depends on the order of a maximum.  The
// rounds used to be six launches each (maxima, products and D of each side, one thread
// per row): on 20,000 x 50,000 with 500k nonzeros 80 us a round, now 13.
constexpr int kRoundLanes = 8;
struct ScaleSide {
    const int32_t *rp, *ci;
    double* v;
    int32_t rows;
    const double *own, *other;  // this round's scales: of the rows, of the columns
    double *next, *D;
};
__device__ __forceinline__ void scale_round(const ScaleSide& s, int32_t row, bool rows_first, bool first, bool last) {
    const int gl = threadIdx.x & (kRoundLanes - 1);
    const bool valid = row < s.rows;
    double mx = 0.0;
    if (valid) {
        const double mine = first ? 1.0 : s.own[row];
        const int32_t e = s.rp[row + 1];
        for (int32_t p = s.rp[row] + gl; p < e; p += kRoundLanes) {
            double x = s.v[p];
            if (!first) {
                const double c = s.other[s.ci[p]];
                // row scale times column scale, whichever side this is
                x = __dmul_rn(x, rows_first ? __dmul_rn(mine, c) : __dmul_rn(c, mine));
                s.v[p] = x;
            }
            const double a = fabs(x);
            if (a > mx) mx = a;
        }
    }
    for (int o = kRoundLanes >> 1; o > 0; o >>= 1) {
        const double a = __shfl_xor_sync(0xffffffffu, mx, o);
        if (a > mx) mx = a;
    }
    if (valid && gl == 0) {
        if (!first) s.D[row] = __dmul_rn(s.D[row], s.own[row]);
        if (!last) s.next[row] = mx < SCALING_EPSILON ? 1.0 : 1.0 / sqrt(mx);
    }
}
__global__ void __launch_bounds__(256) scale_round_kernel(const ScaleSide a, const ScaleSide t, int blocks_a, int first,
                                                          int last) {
    const bool is_a = static_cast<int>(blockIdx.x) < blocks_a;
    const int32_t row = static_cast<int32_t>((is_a ? blockIdx.x : blockIdx.x - blocks_a) * (256 / kRoundLanes) +
                                             threadIdx.x / kRoundLanes);
    scale_round(is_a ? a : t, row, is_a, first != 0, last != 0);
}

// Pock-Chambolle: scale[i] = 1/sqrt(sum_p |v_p|^e), terms in ascending order
__global__ void pc_scale_kernel(const int32_t* __restrict__ rp, const double* __restrict__ v,
                                int32_t rows, double e, double* __restrict__ scale) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += gridDim.x * blockDim.x) {
        double s = 0.0;
        for (int32_t p = rp[i]; p < rp[i + 1]; ++p) {
            const double a = fabs(v[p]);
            s = __dadd_rn(s, e == 1.0 ? a : pow(a, e));
        }
        scale[i] = s < SCALING_EPSILON ? 1.0 : 1.0 / sqrt(s);
    }
}

// scaled bounds and costs, src/preconditioner.jl:66-70:
// c_s = c .* D_c; var bounds / D_c and row bounds .* D_r where finite
__global__ void scale_vectors_kernel(const double* __restrict__ c, const double* __restrict__ lb,
                                     const double* __restrict__ ub, const double* __restrict__ D_c,
                                     int32_t n, const double* __restrict__ clb,
                                     const double* __restrict__ cub, const double* __restrict__ D_r,
                                     int32_t m, double* __restrict__ c_s, double* __restrict__ lb_s,
                                     double* __restrict__ ub_s, double* __restrict__ clb_s,
                                     double* __restrict__ cub_s) {
    for (int32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        c_s[j] = __dmul_rn(c[j], D_c[j]);
        lb_s[j] = isfinite(lb[j]) ? lb[j] / D_c[j] : lb[j];
        ub_s[j] = isfinite(ub[j]) ? ub[j] / D_c[j] : ub[j];
    }
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        clb_s[i] = isfinite(clb[i]) ? __dmul_rn(clb[i], D_r[i]) : clb[i];
        cub_s[i] = isfinite(cub[i]) ? __dmul_rn(cub[i], D_r[i]) : cub[i];
    }
}

// bound/objective rescaling, src/preconditioner.jl:72-96: the two squared norms
// (sequential sums, as the reference's loops), then the scaling.  Block 0 sums the bounds,
// block 1 the costs: the block's threads form a chunk of terms in shared memory (a term
// that the reference skips is +0, which changes no sum of squares) while thread 0 adds the
// chunk before it, one dependent addition (8 cycles) after another; reading the terms in
// the adding thread took 2.4 ms at 20,000 x 50,000, this takes 0.25.
constexpr int kNormChunk = 2048;
__global__ void __launch_bounds__(256) rescale_norms_kernel(const double* __restrict__ clb, const double* __restrict__ cub,
                                                            const double* __restrict__ clb_s,
                                                            const double* __restrict__ cub_s, int32_t m,
                                                            const double* __restrict__ c_s, int32_t n,
                                                            double* __restrict__ out /* bound_sq, c_sq */) {
    __shared__ double term[2][kNormChunk];
    const bool bounds = blockIdx.x == 0;
    const int64_t len = bounds ? 2 * int64_t(m) : n;  // bounds: lower, upper of each row in turn
    double sum = 0.0;
    for (int64_t base = 0, buf = 0; base - kNormChunk < len; base += kNormChunk, buf ^= 1) {
        if (threadIdx.x == 0) {
            if (base > 0) {  // the chunk formed in the round before
                const double* q = term[buf ^ 1];
#pragma unroll 16
                for (int k = 0; k < kNormChunk; ++k) sum = __dadd_rn(sum, q[k]);
            }
        } else if (threadIdx.x >= 32) {
            for (int k = threadIdx.x - 32; k < kNormChunk; k += 224) {
                const int64_t at = base + k;
                double x = 0.0;
                if (at < len) {
                    if (bounds) {
                        const int64_t i = at >> 1;
                        const bool flo = isfinite(clb[i]), fhi = isfinite(cub[i]);
                        const double lo = clb_s[i], hi = cub_s[i];
                        if (at & 1)
                            x = fhi ? __dmul_rn(hi, hi) : 0.0;
                        else if (flo && (!fhi || fabs(lo - hi) > SCALING_EPSILON))
                            x = __dmul_rn(lo, lo);
                    } else {
                        x = __dmul_rn(c_s[at], c_s[at]);
                    }
                }
                term[buf][k] = x;
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) out[bounds ? 0 : 1] = sum;
}

__global__ void rescale_apply_kernel(const double* __restrict__ lb, const double* __restrict__ ub,
                                     int32_t n, const double* __restrict__ clb,
                                     const double* __restrict__ cub, int32_t m,
                                     const double* __restrict__ sq, double* __restrict__ c_s,
                                     double* __restrict__ lb_s, double* __restrict__ ub_s,
                                     double* __restrict__ clb_s, double* __restrict__ cub_s,
                                     double* __restrict__ scales /* bound, objective */) {
    const double bs = 1.0 / (sqrt(sq[0]) + 1.0);
    const double os = 1.0 / (sqrt(sq[1]) + 1.0);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        scales[0] = bs;
        scales[1] = os;
    }
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        if (isfinite(clb[i])) clb_s[i] = __dmul_rn(clb_s[i], bs);
        if (isfinite(cub[i])) cub_s[i] = __dmul_rn(cub_s[i], bs);
    }
    for (int32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        if (isfinite(lb[j])) lb_s[j] = __dmul_rn(lb_s[j], bs);
        if (isfinite(ub[j])) ub_s[j] = __dmul_rn(ub_s[j], bs);
        c_s[j] = __dmul_rn(c_s[j], os);
    }
}

// Small matrices (at most kScaleTinyMaxDim rows + columns and kScaleTinyMaxNnz
// nonzeros): every Ruiz round and the Pock-Chambolle pass in one launch of one
// block -- the same per-row and per-entry operations as the kernels above, in the
// same order (no value depends on how rows are shared among threads), with block
// barriers where those kernels end.
constexpr int64_t kScaleTinyMaxDim = 4096;
constexpr int64_t kScaleTinyMaxNnz = 65536;
constexpr int kScaleTinyThreads = 1024;

__global__ void __launch_bounds__(kScaleTinyThreads)
    scale_tiny_kernel(const int32_t* __restrict__ rp_a, const int32_t* __restrict__ ci_a,
                      double* __restrict__ v_a, const int32_t* __restrict__ rp_t,
                      const int32_t* __restrict__ ci_t, double* __restrict__ v_t, int32_t m,
                      int32_t n, int32_t ruiz_iterations, double alpha, double* __restrict__ rs,
                      double* __restrict__ cs, double* __restrict__ D_r, double* __restrict__ D_c) {
    const int t = threadIdx.x;
    for (int32_t it = 0; it <= ruiz_iterations; ++it) {
        const bool pc = it == ruiz_iterations;  // the last pass: Pock-Chambolle
        for (int32_t i = t; i < m; i += kScaleTinyThreads) {
            if (pc) {
                double sum = 0.0;
                for (int32_t p = rp_a[i]; p < rp_a[i + 1]; ++p) {
                    const double a = fabs(v_a[p]);
                    sum = __dadd_rn(sum, alpha == 1.0 ? a : pow(a, alpha));
                }
                rs[i] = sum < SCALING_EPSILON ? 1.0 : 1.0 / sqrt(sum);
            } else {
                double mx = 0.0;
                for (int32_t p = rp_a[i]; p < rp_a[i + 1]; ++p) {
                    const double a = fabs(v_a[p]);
                    if (a > mx) mx = a;
                }
                rs[i] = mx < SCALING_EPSILON ? 1.0 : 1.0 / sqrt(mx);
            }
        }
        for (int32_t j = t; j < n; j += kScaleTinyThreads) {
            if (pc) {
                const double e = 2.0 - alpha;
                double sum = 0.0;
                for (int32_t p = rp_t[j]; p < rp_t[j + 1]; ++p) {
                    const double a = fabs(v_t[p]);
                    sum = __dadd_rn(sum, e == 1.0 ? a : pow(a, e));
                }
                cs[j] = sum < SCALING_EPSILON ? 1.0 : 1.0 / sqrt(sum);
            } else {
                double mx = 0.0;
                for (int32_t p = rp_t[j]; p < rp_t[j + 1]; ++p) {
                    const double a = fabs(v_t[p]);
                    if (a > mx) mx = a;
                }
                cs[j] = mx < SCALING_EPSILON ? 1.0 : 1.0 / sqrt(mx);
            }
        }
        __syncthreads();
        for (int32_t i = t; i < m; i += kScaleTinyThreads)
            for (int32_t p = rp_a[i]; p < rp_a[i + 1]; ++p)
                v_a[p] = __dmul_rn(v_a[p], __dmul_rn(rs[i], cs[ci_a[p]]));
        for (int32_t j = t; j < n; j += kScaleTinyThreads)
            for (int32_t p = rp_t[j]; p < rp_t[j + 1]; ++p)
                v_t[p] = __dmul_rn(v_t[p], __dmul_rn(rs[ci_t[p]], cs[j]));
        for (int32_t i = t; i < m; i += kScaleTinyThreads) D_r[i] = __dmul_rn(D_r[i], rs[i]);
        for (int32_t j = t; j < n; j += kScaleTinyThreads) D_c[j] = __dmul_rn(D_c[j], cs[j]);
        __syncthreads();
    }
}

static int blocks_for(int64_t n) { return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 8192))); }

__global__ void fill_kernel(double* __restrict__ d, int64_t n, double v) {
    for (int64_t i = blockIdx.x * 256 + threadIdx.x; i < n; i += int64_t(gridDim.x) * 256) d[i] = v;
}

void scale_uploaded(const DeviceMatrix& M, DeviceArena& ar, int32_t ruiz_iterations, double alpha,
                    bool rescale, const double* const vin[5], double* const vout[5], double* D_r,
                    double* D_c, double* scales, cudaStream_t st) {
    const int32_t m = static_cast<int32_t>(M.L.M), n = static_cast<int32_t>(M.L.N);
    double* rs = ar.alloc<double>(2 * static_cast<size_t>(m));  // two rounds' scales in turn
    double* cs = ar.alloc<double>(2 * static_cast<size_t>(n));
    const int bm = blocks_for(m), bn = blocks_for(n);
    if (m) fill_kernel<<<bm, 256, 0, st>>>(D_r, m, 1.0);
    if (n) fill_kernel<<<bn, 256, 0, st>>>(D_c, n, 1.0);
    fill_kernel<<<1, 256, 0, st>>>(scales, 2, 1.0);
    // products with the scales in buffer `b`, and the next round's scales into the other
    auto round = [&](int b, bool first, bool last) {
        const int64_t per = 256 / kRoundLanes;
        const int64_t ga = (m + per - 1) / per, gt = (n + per - 1) / per;
        if (ga + gt == 0) return;
        const ScaleSide a{M.rp_a, M.ci_a, M.v64_a, m, rs + b * int64_t(m), cs + b * int64_t(n), rs + (b ^ 1) * int64_t(m), D_r};
        const ScaleSide t{M.rp_t, M.ci_t, M.v64_t, n, cs + b * int64_t(n), rs + b * int64_t(m), cs + (b ^ 1) * int64_t(n), D_c};
        scale_round_kernel<<<static_cast<unsigned>(ga + gt), 256, 0, st>>>(a, t, static_cast<int>(ga), first, last);
    };
    const char* te = std::getenv("PDFP_TINY");
    const bool tiny = !(te && te[0] == '0') && static_cast<int64_t>(m) + n <= kScaleTinyMaxDim &&
                      M.L.NNZ <= kScaleTinyMaxNnz && m > 0 && n > 0;
    if (tiny) {  // every round in one launch
        scale_tiny_kernel<<<1, kScaleTinyThreads, 0, st>>>(M.rp_a, M.ci_a, M.v64_a, M.rp_t, M.ci_t,
                                                           M.v64_t, m, n, std::max(ruiz_iterations, 0),
                                                           alpha, rs, cs, D_r, D_c);
    } else {
        int b = 0;
        if (ruiz_iterations > 0) {  // src/preconditioner.jl:36-49
            round(b ^ 1, true, false);  // the first scales, into buffer b
            for (int32_t it = 0; it < ruiz_iterations; ++it, b ^= 1) round(b, false, it + 1 == ruiz_iterations);
        }
        // Pock-Chambolle, src/preconditioner.jl:51-64
        if (m) pc_scale_kernel<<<bm, 256, 0, st>>>(M.rp_a, M.v64_a, m, alpha, rs + b * int64_t(m));
        if (n) pc_scale_kernel<<<bn, 256, 0, st>>>(M.rp_t, M.v64_t, n, 2.0 - alpha, cs + b * int64_t(n));
        round(b, false, true);
    }
    // the scaled vectors and the optional bound/objective rescaling
    double* sq = ar.alloc<double>(2);
    const int bb = blocks_for(std::max(m, n));
    scale_vectors_kernel<<<bb, 256, 0, st>>>(vin[0], vin[1], vin[2], D_c, n, vin[3], vin[4], D_r, m,
                                             vout[0], vout[1], vout[2], vout[3], vout[4]);
    if (rescale) {
        rescale_norms_kernel<<<2, 256, 0, st>>>(vin[3], vin[4], vout[3], vout[4], m, vout[0], n, sq);
        rescale_apply_kernel<<<bb, 256, 0, st>>>(vin[1], vin[2], n, vin[3], vin[4], m, sq, vout[0],
                                                 vout[1], vout[2], vout[3], vout[4], scales);
    }
    PDFP_CK(cudaGetLastError());
}

// ---- A' on the device, for scale_problem of a matrix that is not small --------------
//
// scale_problem needs A' only to read each column's entries in ascending row order.  The
// host's transposition (a pass of scattered writes over every nonzero) and its second
// upload took most of the call at 500k nonzeros; here the device counts the columns'
// entries, scans the counts, drops every entry into its column and orders each column by
// row.  Below kDeviceTransposeNnz the host's way costs less than these launches.
constexpr int64_t kDeviceTransposeNnz = 1 << 16;
constexpr int kScanThreads = 1024;
constexpr int32_t kShortColumn = 64;   // ordered by one thread; a longer one by a block
constexpr int32_t kRankColumn = 1024;  // and one longer than this by marks

__global__ void count_columns_kernel(const int32_t* __restrict__ ci, int64_t nnz, int32_t* __restrict__ count) {
    for (int64_t e = blockIdx.x * int64_t(256) + threadIdx.x; e < nnz; e += int64_t(gridDim.x) * 256)
        atomicAdd(count + ci[e], 1);
}
// rp[0 .. n] = exclusive sums of count[0 .. n); cursor = rp; one block
__global__ void __launch_bounds__(kScanThreads) scan_columns_kernel(const int32_t* __restrict__ count, int32_t n,
                                                                    int32_t* __restrict__ rp, int32_t* __restrict__ cursor) {
    __shared__ int32_t warp_sum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t carry = 0;
    for (int64_t base = 0; base < n; base += kScanThreads) {
        const int64_t j = base + threadIdx.x;
        const int32_t x = j < n ? count[j] : 0;
        int32_t v = x;
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += y;
        }
        if (lane == 31) warp_sum[warp] = v;
        __syncthreads();
        if (warp == 0) {
            int32_t w = warp_sum[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int32_t y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += y;
            }
            warp_sum[lane] = w;
        }
        __syncthreads();
        const int32_t before = carry + (warp > 0 ? warp_sum[warp - 1] : 0) + v - x;
        if (j < n) {
            rp[j] = before;
            cursor[j] = before;
        }
        carry += warp_sum[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) rp[n] = carry;
}
// every entry into its column, in any order: its row and its place in A
__global__ void fill_columns_kernel(const int32_t* __restrict__ rp_a, const int32_t* __restrict__ ci_a, int32_t m,
                                    int32_t* __restrict__ cursor, int2* __restrict__ entry) {
    const int lane = threadIdx.x & 31;
    for (int32_t i = (blockIdx.x * 256 + threadIdx.x) >> 5; i < m; i += (gridDim.x * 256) >> 5)
        for (int32_t e = rp_a[i] + lane; e < rp_a[i + 1]; e += 32) entry[atomicAdd(cursor + ci_a[e], 1)] = make_int2(i, e);
}
// columns in ascending row order: ci_t the rows, v_t the values.  A column holds a row at
// most once, so an entry's place is the number of smaller rows.
__global__ void order_short_columns_kernel(const int32_t* __restrict__ rp_t, int32_t n, const int2* __restrict__ entry,
                                           const double* __restrict__ v_a, int32_t* __restrict__ ci_t,
                                           double* __restrict__ v_t) {
    for (int32_t j = blockIdx.x * 256 + threadIdx.x; j < n; j += gridDim.x * 256) {
        const int32_t b = rp_t[j], len = rp_t[j + 1] - b;
        if (len > kShortColumn) continue;
        for (int32_t k = 0; k < len; ++k) {
            const int2 x = entry[b + k];
            int32_t at = b;
            for (int32_t q = 0; q < len; ++q) at += entry[b + q].x < x.x ? 1 : 0;
            ci_t[at] = x.x;
            v_t[at] = v_a[x.y];
        }
    }
}
__global__ void __launch_bounds__(256) order_long_columns_kernel(const int32_t* __restrict__ rp_t, int32_t n,
                                                                 const int2* __restrict__ entry,
                                                                 const double* __restrict__ v_a,
                                                                 int32_t* __restrict__ ci_t, double* __restrict__ v_t) {
    __shared__ int32_t rows[kRankColumn];
    for (int32_t j = blockIdx.x; j < n; j += gridDim.x) {
        const int32_t b = rp_t[j], len = rp_t[j + 1] - b;
        if (len <= kShortColumn || len > kRankColumn) continue;  // the same for the whole block
        __syncthreads();
        for (int32_t q = threadIdx.x; q < len; q += 256) rows[q] = entry[b + q].x;
        __syncthreads();
        for (int32_t k = threadIdx.x; k < len; k += 256) {
            const int2 x = entry[b + k];
            int32_t at = b;
            for (int32_t q = 0; q < len; ++q) at += rows[q] < x.x ? 1 : 0;
            ci_t[at] = x.x;
            v_t[at] = v_a[x.y];
        }
    }
}
// A column of more than kRankColumn entries, of which counting would take the square: a
// block marks the rows that occur in a bitmap, kRowWindow rows at a time, and an entry's
// place is the number of marks before its own -- two passes over the column per window,
// whatever its length.  The blocks of the grid's second dimension take the windows in turn
// and each counts the entries before its window.  scale_problem with one column in every
// row: 100,000 rows 55 ms (by counting 380, transposed by the host 182), 500,000 rows 286
// (host 943).
constexpr int kMarkThreads = 1024;
constexpr int kMarkWords = 5 * kMarkThreads;
constexpr int32_t kRowWindow = 32 * kMarkWords;
// The sum of v over the block, to all its threads.
__device__ __forceinline__ int32_t mark_total(int32_t v, int32_t* warp_sum) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = v;
    __syncthreads();
    int32_t all = 0;
    for (int q = 0; q < kMarkThreads / 32; ++q) all += warp_sum[q];
    __syncthreads();
    return all;
}
__global__ void __launch_bounds__(kMarkThreads) order_marked_columns_kernel(const int32_t* __restrict__ rp_t, int32_t n,
                                                                            int32_t m, const int2* __restrict__ entry,
                                                                            const double* __restrict__ v_a,
                                                                            int32_t* __restrict__ ci_t,
                                                                            double* __restrict__ v_t) {
    __shared__ uint32_t bits[kMarkWords];   // a window's marks
    __shared__ int32_t before[kMarkWords];  // the column's entries before each word's rows
    __shared__ int32_t found[kMarkThreads], n_found, warp_sum[kMarkThreads / 32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    // a share of the columns per block, so that long ones side by side go to different blocks
    const int64_t j0 = int64_t(n) * blockIdx.x / gridDim.x, j1 = int64_t(n) * (blockIdx.x + 1) / gridDim.x;
    for (int64_t base_j = j0; base_j < j1; base_j += kMarkThreads) {
        __syncthreads();
        if (t == 0) n_found = 0;
        __syncthreads();
        const int64_t j = base_j + t;
        if (j < j1 && rp_t[j + 1] - rp_t[j] > kRankColumn) found[atomicAdd(&n_found, 1)] = static_cast<int32_t>(j);
        __syncthreads();
        for (int c = 0; c < n_found; ++c) {  // the same for the whole block
            const int32_t b = rp_t[found[c]], len = rp_t[found[c] + 1] - b;
            for (int64_t lo = int64_t(blockIdx.y) * kRowWindow; lo < m; lo += int64_t(gridDim.y) * kRowWindow) {
                __syncthreads();
                for (int w = t; w < kMarkWords; w += kMarkThreads) bits[w] = 0u;
                __syncthreads();
                int32_t earlier = 0;
#pragma unroll 4
                for (int32_t k = t; k < len; k += kMarkThreads) {
                    const int64_t d = entry[b + k].x - lo;
                    if (d < 0)
                        ++earlier;
                    else if (d < kRowWindow)
                        atomicOr(bits + (d >> 5), 1u << (d & 31));
                }
                const int32_t base = b + mark_total(earlier, warp_sum);
                // exclusive sums of the words' marks, a few adjacent words per thread
                constexpr int per = kMarkWords / kMarkThreads;
                int32_t own = 0;
#pragma unroll
                for (int w = 0; w < per; ++w) own += __popc(bits[per * t + w]);
                int32_t v = own;
                for (int o = 1; o < 32; o <<= 1) {
                    const int32_t y = __shfl_up_sync(0xffffffffu, v, o);
                    if (lane >= o) v += y;
                }
                if (lane == 31) warp_sum[warp] = v;
                __syncthreads();
                int32_t at = base + v - own;
                for (int q = 0; q < warp; ++q) at += warp_sum[q];
#pragma unroll
                for (int w = 0; w < per; ++w) {
                    before[per * t + w] = at;
                    at += __popc(bits[per * t + w]);
                }
                __syncthreads();
#pragma unroll 4
                for (int32_t k = t; k < len; k += kMarkThreads) {
                    const int2 x = entry[b + k];
                    const int64_t d = x.x - lo;
                    if (d < 0 || d >= kRowWindow) continue;
                    const int32_t place = before[d >> 5] + __popc(bits[d >> 5] & ((1u << (d & 31)) - 1u));
                    ci_t[place] = x.x;
                    v_t[place] = v_a[x.y];
                }
            }
        }
    }
}

// build_layout's checks of one problem, without its layout.
static std::string check_csr(const pdfp_csr& A, const int32_t* rp) {
    if (A.m < 0 || A.n < 0) return "negative dimension";
    if (A.m > 0 && !A.row_ptr) return "null row_ptr";
    if (A.m > 0 && rp[0] != 0) return "row_ptr[0] must be 0";
    for (int32_t i = 0; i < A.m; ++i) {
        if (rp[i + 1] < rp[i]) return "row_ptr is not monotone";
        for (int32_t q = rp[i]; q < rp[i + 1]; ++q) {
            if (A.col_idx[q] < 0 || A.col_idx[q] >= A.n) return "column index out of range";
            if (q > rp[i] && A.col_idx[q] <= A.col_idx[q - 1])
                return "column indices must be strictly ascending within a row";
            if (!std::isfinite(A.val[q])) return "non-finite matrix value";
        }
    }
    if (A.m > 0 && rp[A.m] > 0x7fffff00LL) return "problem too large for int32 indexing";
    return "";
}

// The caller's matrix and its transpose on the device, on the default stream.
static void upload_transposed(const pdfp_csr& A, DeviceArena& ar, DeviceMatrix& M) {
    const int32_t m = A.m, n = A.n;
    const int64_t nnz = A.row_ptr[m];
    M.L.K = 1;
    M.L.M = m;
    M.L.N = n;
    M.L.NNZ = nnz;
    M.rp_a = ar.alloc<int32_t>(static_cast<size_t>(m) + 1);
    M.ci_a = ar.alloc<int32_t>(nnz);
    M.v64_a = ar.alloc<double>(nnz);
    M.rp_t = ar.alloc<int32_t>(static_cast<size_t>(n) + 1);
    M.ci_t = ar.alloc<int32_t>(nnz);
    M.v64_t = ar.alloc<double>(nnz);
    int32_t* const count = ar.alloc<int32_t>(n);  // zero-filled
    int32_t* const cursor = ar.alloc<int32_t>(n);
    int2* const entry = ar.alloc<int2>(nnz);
    PDFP_CK(cudaMemcpyAsync(M.rp_a, A.row_ptr, sizeof(int32_t) * (size_t(m) + 1), cudaMemcpyHostToDevice, 0));
    PDFP_CK(cudaMemcpyAsync(M.ci_a, A.col_idx, sizeof(int32_t) * nnz, cudaMemcpyHostToDevice, 0));
    const int be = static_cast<int>(std::min<int64_t>((nnz + 255) / 256, 8192)), bn = blocks_for(n);
    count_columns_kernel<<<be, 256>>>(M.ci_a, nnz, count);
    scan_columns_kernel<<<1, kScanThreads>>>(count, n, M.rp_t, cursor);
    fill_columns_kernel<<<be, 256>>>(M.rp_a, M.ci_a, m, cursor, entry);
    PDFP_CK(cudaMemcpyAsync(M.v64_a, A.val, sizeof(double) * nnz, cudaMemcpyHostToDevice, 0));
    order_short_columns_kernel<<<bn, 256>>>(M.rp_t, n, entry, M.v64_a, M.ci_t, M.v64_t);
    order_long_columns_kernel<<<std::min(n, 4 * 148), 256>>>(M.rp_t, n, entry, M.v64_a, M.ci_t, M.v64_t);
    const dim3 mark_grid(static_cast<unsigned>(std::min(n, 2 * 148)),
                         static_cast<unsigned>(std::min<int64_t>((int64_t(m) + kRowWindow - 1) / kRowWindow, 16)));
    order_marked_columns_kernel<<<mark_grid, kMarkThreads>>>(M.rp_t, n, m, entry, M.v64_a, M.ci_t, M.v64_t);
    PDFP_CK(cudaGetLastError());
}

void scale_problem_device(const pdfp_csr& A, const double* c, const double* var_lb,
                          const double* var_ub, const double* con_lb, const double* con_ub,
                          int32_t ruiz_iterations, double alpha, bool rescale, double* val_out,
                          double* c_out, double* var_lb_out, double* var_ub_out, double* con_lb_out,
                          double* con_ub_out, double* D_r_out, double* D_c_out, double* bound_scale,
                          double* objective_scale) {
    static const int32_t zero_rp = 0;
    const int32_t m = A.m, n = A.n;
    ProblemIn in{m, n, m > 0 ? A.row_ptr : &zero_rp, A.col_idx, A.val, nullptr};
    DeviceMatrix M;
    DeviceArena ar;
    if (m > 0 && n > 0 && A.row_ptr && A.row_ptr[m] >= kDeviceTransposeNnz) {
        const std::string msg = check_csr(A, A.row_ptr);
        if (!msg.empty()) throw Error(E_INVALID, msg);
        upload_transposed(A, ar, M);
    } else {
        std::string msg = build_layout({in}, false, M.L);
        if (!msg.empty()) throw Error(E_INVALID, msg);
        M.upload(ar, false);
    }
    // inputs in one block: c, lb, ub (n each), con_lb, con_ub (m each), then the outputs,
    // D_c, D_r and the two scales
    const int64_t tot = 3 * int64_t(n) + 2 * int64_t(m);
    std::vector<double> hin(std::max<int64_t>(tot, 1));
    const double* src[5] = {c, var_lb, var_ub, con_lb, con_ub};
    const int64_t len[5] = {n, n, n, m, m};
    double* const din = ar.alloc<double>(hin.size());
    double* const dout = ar.alloc<double>(tot + n + m + 2);
    const double* vin[5];
    double* vout[5];
    int64_t off = 0;
    for (int k = 0; k < 5; ++k) {
        if (len[k]) std::copy(src[k], src[k] + len[k], hin.begin() + off);
        vin[k] = din + off;
        vout[k] = dout + off;
        off += len[k];
    }
    double* D_c = dout + tot;
    double* D_r = D_c + n;
    double* scales = D_r + m;
    if (tot) PDFP_CK(cudaMemcpy(din, hin.data(), sizeof(double) * tot, cudaMemcpyHostToDevice));
    scale_uploaded(M, ar, ruiz_iterations, alpha, rescale, vin, vout, D_r, D_c, scales, 0);
    PDFP_CK(cudaDeviceSynchronize());
    std::vector<double> hout(tot + n + m + 2);
    PDFP_CK(cudaMemcpy(hout.data(), dout, sizeof(double) * hout.size(), cudaMemcpyDeviceToHost));
    if (M.L.NNZ) PDFP_CK(cudaMemcpy(val_out, M.v64_a, sizeof(double) * M.L.NNZ, cudaMemcpyDeviceToHost));
    double* dst[5] = {c_out, var_lb_out, var_ub_out, con_lb_out, con_ub_out};
    off = 0;
    for (int k = 0; k < 5; ++k) {
        if (len[k]) std::copy(hout.begin() + off, hout.begin() + off + len[k], dst[k]);
        off += len[k];
    }
    if (n) std::copy(hout.begin() + tot, hout.begin() + tot + n, D_c_out);
    if (m) std::copy(hout.begin() + tot + n, hout.begin() + tot + n + m, D_r_out);
    *bound_scale = hout[tot + n + m];
    *objective_scale = hout[tot + n + m + 1];
}

double estimate_sv_device(const pdfp_csr& A, int32_t max_iterations, double tolerance,
                          int32_t* iterations) {
    static const int32_t zero_rp = 0;
    ProblemIn in{A.m, A.n, A.m > 0 ? A.row_ptr : &zero_rp, A.col_idx, A.val, nullptr};
    DeviceMatrix M;
    std::string msg = build_layout({in}, false, M.L);
    if (!msg.empty()) throw Error(E_INVALID, msg);
    DeviceArena ar;
    M.upload(ar, false);
    StageGeom gev{8, 8, 8, 0, 2, 32 * 1024, 2048};
    DeviceMatrix::Tiling ta = M.make_tiling(ar, false, gev);
    DeviceMatrix::Tiling tt = M.make_tiling(ar, true, gev);
    int dev = 0, sms = 148;
    PDFP_CK(cudaGetDevice(&dev));
    PDFP_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    cudaStream_t s;
    PDFP_CK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    int32_t* err = ar.alloc<int32_t>(4);
    std::vector<int32_t> its;
    std::vector<double> r;
    try {
        r = power_iteration(M, ar, ta, tt, {1}, max_iterations, tolerance, s, sms, err, &its);
    } catch (...) {
        cudaStreamDestroy(s);
        throw;
    }
    cudaStreamDestroy(s);
    if (iterations) *iterations = its.empty() ? 0 : its[0];
    return r[0];
}

}  // namespace pdfp

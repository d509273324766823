// device.cu -- uploads of the packed matrix and its tilings.
#include "device.hpp"

#include <cstdlib>
#include <mutex>
#include <string>

namespace pdfp {

static thread_local std::string g_last_error;
void set_last_error(const std::string& msg) { g_last_error = msg; }

namespace {
constexpr int kMaxPoolDevices = 64;
constexpr uint64_t kPoolKeepBytes = 256ull << 20;
std::mutex g_pool_mu;
cudaMemPool_t g_pools[kMaxPoolDevices] = {};
bool g_pool_failed[kMaxPoolDevices] = {};
int g_pool_enabled = -1;  // -1: not read yet

cudaMemPool_t current_pool() {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    if (g_pool_enabled < 0) {
        const char* e = std::getenv("PDFP_POOL");
        g_pool_enabled = (e && e[0] == '0') ? 0 : 1;
    }
    if (!g_pool_enabled) return nullptr;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxPoolDevices) return nullptr;
    if (g_pools[dev] || g_pool_failed[dev]) return g_pools[dev];
    int supported = 0;
    cudaDeviceGetAttribute(&supported, cudaDevAttrMemoryPoolsSupported, dev);
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    if (!supported || cudaMemPoolCreate(&g_pools[dev], &props) != cudaSuccess) {
        g_pools[dev] = nullptr;
        g_pool_failed[dev] = true;
        cudaGetLastError();
        return nullptr;
    }
    uint64_t keep = kPoolKeepBytes;
    cudaMemPoolSetAttribute(g_pools[dev], cudaMemPoolAttrReleaseThreshold, &keep);
    return g_pools[dev];
}
}  // namespace

namespace {
constexpr int kPinnedClasses = 32;
constexpr size_t kPinnedKeep = 8;  // blocks kept per size class
std::mutex g_pinned_mu;
std::vector<void*> g_pinned_free[kPinnedClasses];
int pinned_class(size_t bytes) {
    int c = 0;
    while ((size_t(256) << c) < bytes && c < kPinnedClasses - 1) ++c;
    return c;
}
}  // namespace

void* pinned_take(size_t bytes) {
    const int c = pinned_class(bytes);
    if ((size_t(256) << c) < bytes) throw Error(E_INVALID, "pinned block too large");
    {
        std::lock_guard<std::mutex> lk(g_pinned_mu);
        if (!g_pinned_free[c].empty()) {
            void* p = g_pinned_free[c].back();
            g_pinned_free[c].pop_back();
            return p;
        }
    }
    void* p = nullptr;
    PDFP_CK(cudaMallocHost(&p, size_t(256) << c));
    return p;
}

void pinned_give(void* p, size_t bytes) {
    if (!p) return;
    const int c = pinned_class(bytes);
    {
        std::lock_guard<std::mutex> lk(g_pinned_mu);
        if (g_pinned_free[c].size() < kPinnedKeep) {
            g_pinned_free[c].push_back(p);
            return;
        }
    }
    cudaFreeHost(p);
}

void* arena_malloc(size_t bytes, bool* pooled) {
    void* p = nullptr;
    *pooled = false;
    if (cudaMemPool_t pool = current_pool()) {
        // on the legacy default stream, then waited for: the memory is zero and
        // usable from every stream when this returns
        PDFP_CK(cudaMallocFromPoolAsync(&p, bytes, pool, 0));
        *pooled = true;
        cudaError_t e = cudaMemsetAsync(p, 0, bytes, 0);
        if (e == cudaSuccess) e = cudaStreamSynchronize(0);
        if (e != cudaSuccess) {
            cudaFreeAsync(p, 0);
            throw Error(E_CUDA, std::string("arena zero-fill: ") + cudaGetErrorString(e));
        }
        return p;
    }
    PDFP_CK(cudaMalloc(&p, bytes));
    cudaError_t e = cudaMemset(p, 0, bytes);
    if (e != cudaSuccess) {
        cudaFree(p);
        throw Error(E_CUDA, std::string("arena zero-fill: ") + cudaGetErrorString(e));
    }
    return p;
}

void arena_free(const std::vector<void*>& ptrs, const std::vector<bool>& pooled) {
    // no kernel of any stream may still use the memory (cudaFree's own guarantee)
    cudaDeviceSynchronize();
    for (size_t i = 0; i < ptrs.size(); ++i) {
        if (pooled[i]) cudaFreeAsync(ptrs[i], 0); else cudaFree(ptrs[i]);
    }
    cudaStreamSynchronize(0);
}
const char* last_error_cstr() { return g_last_error.c_str(); }

__global__ void f64_to_f32_kernel(const double* __restrict__ a, float* __restrict__ b, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        b[i] = static_cast<float>(a[i]);
}

template <class T>
static std::pair<const void*, size_t> part(const std::vector<T>& v) {
    return {v.data(), v.size() * sizeof(T)};
}

void DeviceMatrix::upload(DeviceArena& ar, bool want_f32) {
    const std::vector<void*> d = ar.upload_group(
        {part(L.A.rp), part(L.A.ci), part(L.A.v), part(L.At.rp), part(L.At.ci), part(L.At.v),
         part(L.row_off), part(L.col_off), part(L.n_eq), part(L.row_orig), part(L.col_orig)});
    rp_a = static_cast<int32_t*>(d[0]);
    ci_a = static_cast<int32_t*>(d[1]);
    v64_a = static_cast<double*>(d[2]);
    rp_t = static_cast<int32_t*>(d[3]);
    ci_t = static_cast<int32_t*>(d[4]);
    v64_t = static_cast<double*>(d[5]);
    row_off = static_cast<int32_t*>(d[6]);
    col_off = static_cast<int32_t*>(d[7]);
    n_eq = static_cast<int32_t*>(d[8]);
    row_orig = static_cast<int32_t*>(d[9]);
    col_orig = static_cast<int32_t*>(d[10]);
    max_m = max_n = 0;
    for (int p = 0; p < L.K; ++p) {
        max_m = std::max(max_m, L.row_off[p + 1] - L.row_off[p]);
        max_n = std::max(max_n, L.col_off[p + 1] - L.col_off[p]);
    }
    if (want_f32) {
        v32_a = ar.alloc<float>(L.NNZ);
        v32_t = ar.alloc<float>(L.NNZ);
        refresh_f32(0);
        PDFP_CK(cudaDeviceSynchronize());
    }
}

__global__ void recip_kernel(const double* __restrict__ s, double* __restrict__ d, int64_t n) {
    for (int64_t i = blockIdx.x * 256 + threadIdx.x; i < n; i += int64_t(gridDim.x) * 256)
        d[i] = __ddiv_rn(1.0, s[i]);
}

void cast_f64_to_f32(const double* src, float* dst, int64_t n, cudaStream_t s) {
    if (n <= 0) return;
    const int blocks = static_cast<int>(std::min<int64_t>((n + 255) / 256, 4096));
    f64_to_f32_kernel<<<blocks, 256, 0, s>>>(src, dst, n);
    PDFP_CK(cudaGetLastError());
}

void reciprocal(const double* src, double* dst, int64_t n, cudaStream_t s) {
    if (n <= 0) return;
    const int blocks = static_cast<int>(std::min<int64_t>((n + 255) / 256, 4096));
    recip_kernel<<<blocks, 256, 0, s>>>(src, dst, n);
    PDFP_CK(cudaGetLastError());
}

void DeviceMatrix::refresh_f32(cudaStream_t s) {
    if (!v32_a || L.NNZ == 0) return;
    int blocks = static_cast<int>(std::min<int64_t>((L.NNZ + 255) / 256, 4096));
    f64_to_f32_kernel<<<blocks, 256, 0, s>>>(v64_a, v32_a, L.NNZ);
    f64_to_f32_kernel<<<blocks, 256, 0, s>>>(v64_t, v32_t, L.NNZ);
    PDFP_CK(cudaGetLastError());
}

// Upload a built tiling of the CSR whose device arrays are rp / ci.
static DeviceMatrix::Tiling upload_tiling(DeviceArena& ar, DeviceMatrix::Tiling&& t, int32_t rows,
                                          const int32_t* rp, const int32_t* ci, const StageGeom& g) {
    SideDev& s = t.dev;
    s.rows = rows;
    s.n_tiles = static_cast<int32_t>(t.host.tile_inst.size());
    s.n_chunks = static_cast<int32_t>(t.host.chunk_k0.size());
    s.max_tile_rows = t.host.max_tile_rows;
    s.stage_bytes = g.stage_bytes;
    s.rp = rp;
    s.ci = ci;
    std::vector<ChunkDesc> desc(t.host.chunk_k0.size());
    for (size_t c = 0; c < desc.size(); ++c) {
        const int32_t tile = t.host.chunk_tile[c];
        desc[c] = ChunkDesc{t.host.chunk_k0[c], t.host.chunk_k1[c], t.host.tile_row[tile],
                            t.host.tile_row_end[tile], tile, t.host.tile_inst[tile],
                            t.host.chunk_flags[c], t.host.tile_chunk[tile] == (int32_t)c ? 1 : 0};
    }
    const std::vector<void*> d = ar.upload_group({part(t.host.tile_row), part(t.host.tile_chunk),
                                                  part(t.host.tile_inst), part(desc),
                                                  part(t.host.inst_tile0)});
    s.tile_row = static_cast<const int32_t*>(d[0]);
    s.tile_chunk = static_cast<const int32_t*>(d[1]);
    s.tile_inst = static_cast<const int32_t*>(d[2]);
    s.chunks = static_cast<const ChunkDesc*>(d[3]);
    t.inst_tile0 = static_cast<int32_t*>(d[4]);
    return std::move(t);
}

DeviceMatrix::Tiling DeviceMatrix::make_tiling(DeviceArena& ar, bool transpose,
                                               const StageGeom& g,
                                               const std::vector<uint8_t>* skip) const {
    Tiling t;
    const HostCsr& csr = transpose ? L.At : L.A;
    build_tiling(csr, transpose ? L.col_off : L.row_off, g, t.host, skip);
    return upload_tiling(ar, std::move(t), csr.rows, transpose ? rp_t : rp_a, transpose ? ci_t : ci_a, g);
}

bool DeviceMatrix::make_seg(DeviceArena& ar, int nseg, int long_min, const StageGeom& g,
                            SegDev& d, Tiling& pairs, std::vector<uint8_t>& is_long) const {
    HostSeg h;
    if (!build_seg(L.A, L.row_off, nseg, long_min, h)) return false;
    const int64_t nl = static_cast<int64_t>(h.long_row.size());
    d = SegDev();
    d.nseg = h.nseg;
    d.seg_len = h.seg_len;
    d.n_cols = h.n_cols;
    d.n_long = static_cast<int32_t>(nl);
    d.long_row = ar.upload(h.long_row);
    d.long_inst = ar.upload(h.long_inst);
    std::vector<float> v32(h.pairs.v.size());
    for (size_t k = 0; k < v32.size(); ++k) v32[k] = static_cast<float>(h.pairs.v[k]);  // as refresh_f32 rounds
    d.val = ar.upload(v32);
    d.partial = ar.alloc<float>(static_cast<size_t>(nl) * nseg);
    // tiles of the pairs, the segments as instances, interleaved one block per segment
    std::vector<int32_t> off(nseg + 1);
    for (int s = 0; s <= nseg; ++s) off[s] = static_cast<int32_t>(s * nl);
    HostTiling by_seg;
    build_tiling(h.pairs, off, g, by_seg);
    Tiling t;
    interleave_tiles(by_seg, nseg, t.host);
    const int32_t* rp = ar.upload(h.pairs.rp);
    const int32_t* ci = ar.upload(h.pairs.ci);
    pairs = upload_tiling(ar, std::move(t), h.pairs.rows, rp, ci, g);
    is_long.swap(h.is_long);
    return true;
}

constexpr int32_t kResHotRow = 512;
constexpr int64_t kResHotNnz = int64_t(1) << 18;

bool DeviceMatrix::plan_resident(int n_blocks, int esize, int ncv, int nrv, int par_bytes, uint32_t max_smem,
                                 HostResident& ht, HostResident& ha, uint32_t& smem) const {
    // entries and vectors alone, spread evenly: no need to lay out what cannot fit
    const double least = 2.0 * L.NNZ * (4 + 2 * esize) +
                         static_cast<double>(esize * ncv + 4) * L.N + static_cast<double>(esize * nrv + 4) * L.M;
    if (n_blocks <= 0 || least > static_cast<double>(n_blocks) * max_smem) return false;
    // Every block gathers the entries of long rows again and again, and from L2, where they
    // share a few lines; the step launches have them in L1.  400 iterations of Zipf-skewed
    // models with nearly all nonzeros in rows of 1,000 to 2,000, resident against launches:
    // 129k nonzeros 3.9 / 5.5 ms, 240k (FP64) 4.8 / 5.8, 359k (FP64) 5.6 / 5.2, 656k 8.0 / 5.5.
    if (L.NNZ > kResHotNnz) {
        int64_t hot = 0;
        for (const HostCsr* s : {&L.A, &L.At})
            for (int32_t i = 0; i < s->rows; ++i)
                if (s->rp[i + 1] - s->rp[i] >= kResHotRow) hot += s->rp[i + 1] - s->rp[i];
        if (2 * hot > L.NNZ) return false;
    }
    deal_resident(L.At, L.col_off, n_blocks, kResLaneNnz, 1, false, ht);
    deal_resident(L.A, L.row_off, n_blocks, kResLaneNnz, 1, false, ha);
    smem = 0;
    for (int b = 0; b < n_blocks; ++b)
        smem = std::max(smem, res_smem(ht.blocks[b], ha.blocks[b], esize, ncv, nrv, par_bytes).total);
    return smem <= max_smem;
}

bool DeviceMatrix::make_cluster(DeviceArena& ar, int max_blocks, int esize, int max_warps, uint32_t max_smem,
                                Resident& r, std::vector<ClusterGroup>& groups) const {
    r = Resident();
    groups.clear();
    HostResident ht, ha;
    std::vector<ClusterGroup> by(max_blocks + 1);
    std::vector<std::vector<ClusterMember>> in(max_blocks + 1);
    for (int p = 0; p < L.K; ++p) {
        const int32_t n = L.col_off[p + 1] - L.col_off[p], m = L.row_off[p + 1] - L.row_off[p];
        const int32_t b0 = static_cast<int32_t>(ht.blocks.size());
        int warps = 0;
        uint32_t smem = 0;
        // the fewest blocks that hold the member, every row whole: a lane sums a long
        // row's every 32nd entry
        auto fits = [&](int c) {
            for (HostResident* o : {&ht, &ha}) {  // without the blocks of the number tried before
                if (static_cast<int32_t>(o->blocks.size()) == b0) continue;
                o->slices.resize(o->blocks[b0].slice0);
                o->lane_row.resize(size_t(32) * o->slices.size());
                o->blocks.resize(b0);
            }
            deal_member(L.At, L.col_off, p, c, kCluLaneNnz, INT32_MAX, kCluDepthUnit, ht);
            deal_member(L.A, L.row_off, p, c, kCluLaneNnz, INT32_MAX, kCluDepthUnit, ha);
            warps = 1;
            smem = 0;
            for (int b = b0; b < b0 + c; ++b) {
                warps = std::max(warps, ht.blocks[b].n_slices + ha.blocks[b].n_slices);
                smem = std::max(smem, clu_smem(ht.blocks[b], ha.blocks[b], esize, n, m).total);
            }
            return warps <= max_warps && smem <= max_smem;
        };
        int c = 1;
        if (!fits(1)) {  // more blocks never make fewer slices
            c = std::max(2, (warps + max_warps - 1) / max_warps);
            while (c <= max_blocks && !fits(c)) ++c;
            if (c > max_blocks) return false;
        }
        by[c].n_warps = std::max(by[c].n_warps, warps);
        by[c].smem = std::max(by[c].smem, smem);
        in[c].push_back(ClusterMember{p, b0});
    }
    std::vector<ClusterMember> all;
    for (int c = max_blocks; c >= 1; --c) {  // the largest members first
        if (in[c].empty()) continue;
        by[c].n_ranks = c;
        by[c].first = static_cast<int32_t>(all.size());
        by[c].count = static_cast<int32_t>(in[c].size());
        groups.push_back(by[c]);
        all.insert(all.end(), in[c].begin(), in[c].end());
    }
    upload_resident(ar, ht, ha, INT32_MAX, r);
    const ClusterMember* d = ar.upload(all);
    for (ClusterGroup& g : groups) g.members = d + g.first;
    return true;
}

void DeviceMatrix::upload_resident(DeviceArena& ar, const HostResident& ht, const HostResident& ha, int32_t piece,
                                   Resident& r) const {
    const std::vector<void*> d = ar.upload_group({part(ht.blocks), part(ht.slices), part(ht.longs), part(ht.lane_row),
                                                  part(ha.blocks), part(ha.slices), part(ha.longs), part(ha.lane_row)});
    auto side = [&](int k) {
        ResDev s;
        s.blocks = static_cast<const ResBlock*>(d[k]);
        s.slices = static_cast<const ResSlice*>(d[k + 1]);
        s.longs = static_cast<const ResLong*>(d[k + 2]);
        s.lane_row = static_cast<const int32_t*>(d[k + 3]);
        return s;
    };
    auto entries = [](const HostResident& h) {
        return h.blocks.empty() ? int64_t(0) : int64_t(h.blocks.back().elem0) + h.blocks.back().n_elem;
    };
    r.t = side(0);
    r.a = side(4);
    r.n_t = entries(ht);
    r.n_a = entries(ha);
    r.piece = piece;
    r.n_blocks = static_cast<int>(ht.blocks.size());
    // the copies from pageable memory may still be under way on the default stream, which
    // the handle's own stream does not wait for
    PDFP_CK(cudaStreamSynchronize(0));
}

// The entries of a layout in slices, one warp per slice: fill_resident() of layout.cpp, which
// states what goes where, on the arrays of the CSR matrix.  A new handle's first solve of one
// window, in per-step launches / resident with this / with the entries made by a host thread
// and uploaded: FP64 600k nonzeros 9.4 / 8.5 / 12.2 ms, mixed 900k 16.0 / 15.0 / 20.4.
template <typename T>
__global__ void __launch_bounds__(256) fill_slices_kernel(const ResDev d, int n_blocks, int32_t piece,
                                                          const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                                                          const T* __restrict__ v, int32_t* __restrict__ idx,
                                                          T* __restrict__ val) {
    const int lane = threadIdx.x & 31;
    for (int b = blockIdx.x; b < n_blocks; b += gridDim.x) {
        const ResBlock B = d.blocks[b];
        for (int32_t q = blockIdx.y * 8 + (threadIdx.x >> 5); q < B.n_slices; q += gridDim.y * 8) {
            const ResSlice m = d.slices[B.slice0 + q];
            const int lg = m.shape & 7;
            const int32_t ln = d.lane_row[int64_t(32) * (B.slice0 + q) + lane];
            int32_t k = 0, end = 0;  // the lane's entries: every 2^lg-th of its row or piece
            if (ln >= 0) {
                const ResLong l = m.slot >= 0 ? d.longs[B.long0 + ln] : ResLong{};
                const int32_t row = B.row0 + (m.slot >= 0 ? l.row : ln);
                const int32_t k0 = rp[row] + (m.slot >= 0 ? (m.slot - l.slot0) * piece : 0);
                end = m.slot >= 0 && rp[row + 1] - k0 > piece ? k0 + piece : rp[row + 1];
                k = k0 + (lane & ((1 << lg) - 1));
            }
            int64_t x = int64_t(B.elem0) + m.off + lane;
            for (int u = 0; u < (m.shape >> 3); ++u, x += 32, k += 1 << lg) {
                idx[x] = k < end ? ci[k] : -1;
                val[x] = k < end ? v[k] : T(0);
            }
        }
    }
}

template <typename T>
static void fill_slices(DeviceArena& ar, ResDev& d, int64_t n, int n_blocks, int32_t piece, const int32_t* rp,
                        const int32_t* ci, const T* v, cudaStream_t s) {
    int32_t* const idx = ar.alloc<int32_t>(n);
    T* const val = ar.alloc<T>(n);
    fill_slices_kernel<T><<<dim3(std::min(n_blocks, 4096), 8), 256, 0, s>>>(d, n_blocks, piece, rp, ci, v, idx, val);
    PDFP_CK(cudaGetLastError());
    d.idx = idx;
    d.val = val;
}

void DeviceMatrix::fill_resident(DeviceArena& ar, Resident& r, bool f32, cudaStream_t s) const {
    if (f32) {
        fill_slices(ar, r.t, r.n_t, r.n_blocks, r.piece, rp_t, ci_t, v32_t, s);
        fill_slices(ar, r.a, r.n_a, r.n_blocks, r.piece, rp_a, ci_a, v32_a, s);
    } else {
        fill_slices(ar, r.t, r.n_t, r.n_blocks, r.piece, rp_t, ci_t, v64_t, s);
        fill_slices(ar, r.a, r.n_a, r.n_blocks, r.piece, rp_a, ci_a, v64_a, s);
    }
}

VecDev DeviceMatrix::make_vec(DeviceArena& ar, bool transpose, int lane_nnz, int64_t min_items) const {
    const HostCsr& csr = transpose ? L.At : L.A;
    const std::vector<int32_t>& off = transpose ? L.col_off : L.row_off;
    std::vector<VecItem> items;
    int32_t slots = 0;
    if (min_items > 0) {
        // four times the default rows per item (fewer items to fetch per warp) while
        // that still leaves at least min_items items for the warps of the grid
        slots = build_vec_items(csr, off, lane_nnz, items, std::max(1, 32 / std::max(1, lane_nnz)));
        if (static_cast<int64_t>(items.size()) < min_items) items.clear();
    }
    if (items.empty()) slots = build_vec_items(csr, off, lane_nnz, items);
    VecDev v;
    v.n_items = static_cast<int32_t>(items.size());
    v.n_slots = slots;
    v.rp = transpose ? rp_t : rp_a;
    v.ci = transpose ? ci_t : ci_a;
    v.items = ar.upload(items);
    v.piece_sum = ar.alloc<double>(slots > 0 ? slots : 1);  // zero-filled
    v.piece_cnt = ar.alloc<int32_t>(slots > 0 ? slots : 1);
    return v;
}

}  // namespace pdfp

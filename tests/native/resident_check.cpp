// resident_check.cpp -- CPU checks of the resident window's layout (deal_resident and
// fill_resident in pdfp_b200/csrc/layout.cpp): walks every block's slices with the kernel's own index
// arithmetic and checks every bound, that each row is summed exactly once from its own
// nonzeros, and that a row's order of summation depends on its length alone.
#include <algorithm>
#include <cstdint>
#include <vector>

#include "../../pdfp_b200/csrc/layout.hpp"

using namespace pdfp;

// The order in which a row's nonzeros are added, as one number per nonzero: its place
// in the slice (depth and lane relative to the row's first lane, piece).
static int check_side(const HostCsr& csr, const std::vector<int32_t>& off, int n_blocks, int lane_nnz,
                      int unit, bool per_member, HostResident& h) {
    const int kResLaneNnz = lane_nnz, kResPiece = 32 * lane_nnz;
    deal_resident(csr, off, n_blocks, lane_nnz, unit, per_member, h);
    fill_resident(csr, lane_nnz, h);
    const int K = static_cast<int>(off.size()) - 1;
    if (static_cast<int>(h.blocks.size()) != (per_member ? K : 1) * n_blocks) return 1;
    for (size_t b = 0; per_member && b < h.blocks.size(); ++b)  // a member's blocks hold its rows
        if (h.blocks[b].row0 < off[b / n_blocks] || h.blocks[b].row1 > off[b / n_blocks + 1]) return 24;
    if (h.lane_row.size() != 32 * h.slices.size() || h.idx.size() != h.src.size()) return 2;
    std::vector<int> rows_done(csr.rows, 0), nz_done(csr.ci.size(), 0);
    int32_t next_row = 0, next_slice = 0, next_elem = 0, next_long = 0;
    for (const ResBlock& b : h.blocks) {
        if (b.row0 != next_row || b.row1 < b.row0 || b.row1 > csr.rows) return 3;
        if (b.slice0 != next_slice || b.elem0 != next_elem || b.long0 != next_long) return 4;
        next_row = b.row1;
        next_slice += b.n_slices;
        next_elem += b.n_elem;
        next_long += b.n_long;
        std::vector<int> slot_row(b.n_slots, -1), slot_piece(b.n_slots, -1);
        for (int32_t q = 0; q < b.n_long; ++q) {
            const ResLong& m = h.longs[b.long0 + q];
            if (m.row < 0 || m.row >= b.row1 - b.row0 || m.slot0 < 0 || m.slot0 + m.np > b.n_slots) return 5;
            if (m.inst < 0 || m.inst >= b.n_inst) return 6;
            const int32_t r = b.row0 + m.row, len = csr.rp[r + 1] - csr.rp[r];
            if (len <= kResPiece || m.np != (len + kResPiece - 1) / kResPiece) return 7;
            if (r < off[b.inst0 + m.inst] || r >= off[b.inst0 + m.inst + 1]) return 8;
            for (int s = 0; s < m.np; ++s) {
                if (slot_row[m.slot0 + s] >= 0) return 9;
                slot_row[m.slot0 + s] = r;
                slot_piece[m.slot0 + s] = s;
            }
            ++rows_done[r];
        }
        for (int32_t q = 0; q < b.n_slices; ++q) {
            const ResSlice& m = h.slices[b.slice0 + q];
            const int lg = m.shape & 7, depth = m.shape >> 3, G = 1 << lg;
            if (lg > 5 || depth < 0 || depth % unit || m.off < 0 || m.off + 32 * depth > b.n_elem) return 10;
            if (m.inst < 0 || m.inst >= b.n_inst) return 11;
            if (q > 0 && depth > (h.slices[b.slice0 + q - 1].shape >> 3)) return 12;
            for (int lane = 0; lane < 32; ++lane) {
                const int32_t lr = h.lane_row[32 * (b.slice0 + q) + lane];
                int32_t r = -1, k0 = 0;
                if (m.slot >= 0) {
                    if (m.slot >= b.n_slots || slot_row[m.slot] < 0 || lg != 5) return 13;
                    if (lr < 0 || lr >= b.n_long || b.row0 + h.longs[b.long0 + lr].row != slot_row[m.slot]) return 23;
                    r = slot_row[m.slot];
                    k0 = csr.rp[r] + slot_piece[m.slot] * kResPiece;
                } else if (lr >= 0) {
                    if (lr >= b.row1 - b.row0) return 14;
                    r = b.row0 + lr;
                    k0 = csr.rp[r];
                    const int32_t len = csr.rp[r + 1] - csr.rp[r];
                    // the lanes by the row's length alone
                    if ((lg < 5 && G * kResLaneNnz < len) || (lg > 0 && G / 2 * kResLaneNnz >= len)) return 15;
                    if (len > kResPiece || r < off[b.inst0 + m.inst] || r >= off[b.inst0 + m.inst + 1]) return 16;
                    // the G lanes of a row are consecutive and aligned
                    if (h.lane_row[32 * (b.slice0 + q) + (lane & ~(G - 1))] != lr) return 17;
                    if ((lane & (G - 1)) == 0) ++rows_done[r];
                }
                const int32_t kend = r < 0 ? 0 : m.slot >= 0 ? std::min(k0 + kResPiece, csr.rp[r + 1]) : csr.rp[r + 1];
                for (int u = 0; u < depth; ++u) {
                    const size_t e = static_cast<size_t>(b.elem0) + m.off + 32 * u + lane;
                    const int32_t want = r < 0 ? -1 : k0 + u * G + (lane & (G - 1));
                    if (want < 0 || want >= kend) {
                        if (h.idx[e] != -1 || h.src[e] != -1) return 18;
                    } else {
                        if (h.src[e] != want || h.idx[e] != csr.ci[want]) return 19;
                        ++nz_done[want];
                    }
                }
            }
        }
    }
    if (next_row != csr.rows || next_slice != (int)h.slices.size() || next_elem != (int)h.idx.size() ||
        next_long != (int)h.longs.size())
        return 20;
    for (int v : rows_done) if (v != 1) return 21;
    for (int v : nz_done) if (v != 1) return 22;
    return 0;
}

extern "C" int resident_check(int K, const int32_t* ms, const int32_t* ns, const int32_t* const* rps,
                              const int32_t* const* cis, const double* const* vs,
                              const uint8_t* const* is_eqs, int n_blocks, int64_t* stats) {
    std::vector<ProblemIn> probs;
    for (int p = 0; p < K; ++p) probs.push_back(ProblemIn{ms[p], ns[p], rps[p], cis[p], vs[p], is_eqs[p]});
    for (int permute = 0; permute < 2; ++permute) {  // the projector's order and the root LP's
        HostLayout L;
        if (!build_layout(probs, permute != 0, L).empty()) return 100;
        HostResident t, a;
        for (int c = 1; c <= 8; ++c) {  // small members' clusters
            if (int rc = check_side(L.At, L.col_off, c, kCluLaneNnz, kCluDepthUnit, true, t)) return 500 + rc;
            if (int rc = check_side(L.A, L.row_off, c, kCluLaneNnz, kCluDepthUnit, true, a)) return 600 + rc;
            for (size_t b = 0; b < t.blocks.size(); ++b) {
                const CluSmem s = clu_smem(t.blocks[b], a.blocks[b], 8, ns[b / c], ms[b / c]);
                if (s.total % 16 || s.idx_a > s.total) return 700;
                // what other blocks write lies at the same place in all of a member's blocks
                const size_t f = b / c * c;
                const CluSmem s0 = clu_smem(t.blocks[f], a.blocks[f], 8, ns[b / c], ms[b / c]);
                if (s.xs != s0.xs || s.zs != s0.zs || s.part_c != s0.part_c || s.part_r != s0.part_r) return 701;
            }
        }
        if (int rc = check_side(L.At, L.col_off, n_blocks, kResLaneNnz, 1, false, t)) return 200 + rc;
        if (int rc = check_side(L.A, L.row_off, n_blocks, kResLaneNnz, 1, false, a)) return 300 + rc;
        stats[0] = stats[1] = 0;
        for (int b = 0; b < n_blocks; ++b) {
            const ResSmem s = res_smem(t.blocks[b], a.blocks[b], 8, 8, 3, 48);
            if (s.total % 16 || s.long_a > s.total) return 400;
            stats[0] = std::max<int64_t>(stats[0], s.total);
        }
        stats[1] = static_cast<int64_t>(t.longs.size() + a.longs.size());
    }
    return 0;
}

// rows_plan.h -- host tables of the assembled stiffness (MeshView::bsr_*) and
// of the solve on resident rows (cg_rows.cu).
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

namespace femgb {

// The assembled stiffness's pattern and contributions (MeshView::bsr_*): row n
// holds n's neighbours through its elements and n itself, ascending, padded
// with n to a multiple of four; slot (n, j), j other than n, sums the corner
// pairs (li of n, lj of j) of the elements holding both, in element order.
struct BsrPattern {
    std::vector<uint32_t> row, used, col, cptr, contrib;
};
// False: too large. ptr/idx: the node CSR of element corners.
inline bool bsr_pattern(uint32_t N, uint32_t T, const uint32_t* tets, const std::vector<uint32_t>& ptr,
                 const std::vector<uint32_t>& idx, BsrPattern& p)
{
    if ((uint64_t)T >= (1ull << 28)) return false;  // contributions pack the element in 28 bits
    std::vector<uint32_t> seen(N, 0xffffffffu), place(N), at(12 * (size_t)T), nb;
    p.row.assign(N + 1, 0);
    p.used.resize(N);
    p.col.reserve(18 * (size_t)N);
    std::vector<uint32_t> count;
    count.reserve(18 * (size_t)N);
    size_t k = 0;
    for (uint32_t n = 0; n < N; n++) {
        nb.assign(1, n);
        seen[n] = n;
        for (uint32_t j = ptr[n]; j < ptr[n + 1]; j++)
            for (int i = 0; i < 4; i++) {
                const uint32_t c = tets[4 * (size_t)(idx[j] >> 2) + i];
                if (seen[c] != n) {
                    seen[c] = n;
                    nb.push_back(c);
                }
            }
        std::sort(nb.begin(), nb.end());
        p.used[n] = (uint32_t)nb.size();
        const uint32_t base = (uint32_t)p.col.size();
        for (uint32_t i = 0; i < nb.size(); i++) place[nb[i]] = base + i;
        while (nb.size() % 4) nb.push_back(n);
        p.col.insert(p.col.end(), nb.begin(), nb.end());
        if (p.col.size() >= (1ull << 28)) return false;
        p.row[n + 1] = (uint32_t)(p.col.size() / 4);
        count.resize(p.col.size(), 0);
        for (uint32_t j = ptr[n]; j < ptr[n + 1]; j++)
            for (uint32_t lj = 0; lj < 4; lj++) {
                if (lj == (idx[j] & 3u)) continue;
                at[k] = place[tets[4 * (size_t)(idx[j] >> 2) + lj]];
                count[at[k++]]++;
            }
    }
    const size_t slots = p.col.size();
    p.cptr.assign(slots + 1, 0);
    for (size_t i = 0; i < slots; i++) p.cptr[i + 1] = p.cptr[i] + count[i];
    std::copy(p.cptr.begin(), p.cptr.end() - 1, count.begin());  // where the next one goes
    p.contrib.resize(12 * (size_t)T);
    k = 0;
    for (uint32_t n = 0; n < N; n++)
        for (uint32_t j = ptr[n]; j < ptr[n + 1]; j++) {
            const uint32_t e = idx[j] >> 2, li = idx[j] & 3u;
            for (uint32_t lj = 0; lj < 4; lj++)
                if (lj != li) p.contrib[count[at[k++]]++] = (e << 4) | (li << 2) | lj;
        }
    return true;
}

// The CG or MINRES solve of a C_WRP solid in one launch, its rows in shared
// memory (cg_rows.cu). Block g owns node[node0 .. node0 + nn), rows of `lanes`
// lanes, 32 / lanes rows per group; a group's units [group[group0 + w],
// group[group0 + w + 1]) hold one 3x3 block per lane: its bsr slot (kCgRowsPad:
// none) and its column, as the index of the node in the block or nn + its
// index in the block's rim, halo[halo0 .. halo0 + nhalo). owner: where a rim
// node's r is: the CTA of the cluster << 16 | the node's index in its block,
// or kCgRowsFar (another cluster's). The marks in node: some rim of the
// cluster, or of another one, holds it.
constexpr uint32_t kCgRowsPad = 0xffffffffu, kCgRowsFar = 0xffffffffu;
constexpr uint32_t kCgRowsFarShared = 0x80000000u, kCgRowsNearShared = 0x40000000u, kCgRowsNode = 0x3fffffffu;
constexpr uint32_t kCgRowsMaxThreads = 768, kCgRowsMaxBlocks = 160, kCgRowsMaxWords = 160;  // words: five per lane of a warp
constexpr size_t kCgRowsMaxSmem = 226 * 1024;
constexpr uint32_t kCgRowsPolls = 1u << 20;  // default poll limit of a wait, each an L2 round trip
struct CgRowsBlock {
    uint32_t node0, nn, group0, ngroups, unit0, units, halo0, nhalo;
};
// warps: of a block, one component per thread; npb: nodes per block; units,
// records: the most of any block (shared memory before the words that the
// cluster's CTAs address in one another).
struct CgRowsPlan {
    uint32_t blocks = 0, cluster = 0, threads = 0, lanes = 0, warps = 0, npb = 0, units = 0, records = 0;
    size_t smem = 0;
};
inline size_t cg_rows_smem_bytes(const CgRowsPlan& p, const CgRowsBlock& b)
{
    return 288 * 2 * sizeof(int32_t) * (size_t)p.units + 32 * (size_t)p.records + 16 * (2 * (size_t)p.cluster * p.warps + 3 * (size_t)p.npb) +
           (24 + 4) * (size_t)b.nn + (48 + 8) * (size_t)b.nhalo + 4 * (size_t)(b.ngroups + 1) + 32 * sizeof(uint16_t) * (size_t)b.units;
}

// The layout of the solve on resident rows (CgRowsBlock).
struct CgRowsLayout {
    CgRowsPlan plan;
    std::vector<CgRowsBlock> blk;
    std::vector<uint32_t> node, group, slot, halo, owner;
    std::vector<uint16_t> col;
};

// Nodes [g npb, (g + 1) npb) to block g, longest rows first (a group's units
// are those of its longest row). False when the rows do not fit the GPU's
// shared memory. max_blocks(plan): the blocks of that shape that are resident
// together (cg_rows_max_blocks).
// One cluster of up to 16 blocks, kRowsPerBlock rows in each before there are
// 16 (160 tets, a step: 399 us; 12 rows 417, 24 rows 424, 48 rows 485), as long
// as its blocks' sums fit the words a warp polls; a mesh of 3,000 tets takes
// 512 us on it, 575 us on all clusters, whose sums go through L2 (1.3 us more
// each). Above that clusters of 8, all that are resident together with one
// block per SM (20,480 tets: 637 us on 15 clusters; 727 us on 36 of 4, 746 us
// on 76 of 2, 648 us on 7 of 16), of 2 for the last of the SMs' memory. 16
// lanes per row while a block has up to 16 rows, else 8 (20,480 tets: 660 us
// with 16, 658 us with 4), else 4.
constexpr uint32_t kRowsPerBlock = 8;
template <typename F>
bool cg_rows_layout(uint32_t N, const BsrPattern& p, F&& max_blocks, CgRowsLayout& o)
{
    if (N > kCgRowsNode) return false;
    std::vector<uint32_t> order(N), seen(N, 0), place(N);
    uint32_t sorted = 0;  // rows per block that order is sorted for
    auto build = [&](uint32_t blocks, uint32_t cluster, uint32_t lanes) {
        const uint32_t npb = (N + blocks - 1) / blocks, rows = 32 / lanes, warps = (3 * npb + 31) / 32;
        if (3 * npb + (blocks > 1 ? 32u : 0u) > kCgRowsMaxThreads || (lanes > 4 && lanes * npb > kCgRowsMaxThreads) ||
            cluster * warps > kCgRowsMaxWords || blocks / cluster > 96)
            return false;
        if (sorted != npb) {
            for (uint32_t n = 0; n < N; n++) order[n] = n;
            for (uint32_t a = 0; a < N; a += npb)
                std::sort(order.begin() + a, order.begin() + std::min(N, a + npb),
                          [&](uint32_t i, uint32_t j) { return p.used[i] != p.used[j] ? p.used[i] > p.used[j] : i < j; });
            sorted = npb;
        }
        o = CgRowsLayout{};
        CgRowsPlan& plan = o.plan;
        plan.blocks = blocks;
        plan.cluster = cluster;
        plan.lanes = lanes;
        plan.warps = warps;
        plan.npb = npb;
        plan.threads = 64;
        // the shared memory without the rims first
        for (uint32_t a = 0; a < N; a += npb) {
            uint32_t units = 0;
            for (uint32_t n = a; n < std::min(N, a + npb); n += rows) units += (p.used[order[n]] + lanes - 1) / lanes;
            plan.units = std::max(plan.units, units);
        }
        if (cg_rows_smem_bytes(plan, CgRowsBlock{}) > kCgRowsMaxSmem) return false;
        o.node = order;
        std::fill(seen.begin(), seen.end(), 0u);
        for (uint32_t g = 0; g < blocks; g++) {
            const uint32_t a = std::min(N, g * npb), e = std::min(N, a + npb), mark = g + 1;
            CgRowsBlock b{a, e - a, (uint32_t)o.group.size(), 0, (uint32_t)(o.slot.size() / 32), 0, (uint32_t)o.halo.size(), 0};
            for (uint32_t i = a; i < e; i++) {
                seen[order[i]] = mark;
                place[order[i]] = i - a;
            }
            for (uint32_t g0 = a; g0 < e; g0 += rows) {
                o.group.push_back(b.units);
                const uint32_t units = (p.used[order[g0]] + lanes - 1) / lanes;
                for (uint32_t u = 0; u < units; u++)
                    for (uint32_t l = 0; l < 32; l++) {
                        const uint32_t i = g0 + l / lanes, k = lanes * u + l % lanes;
                        if (i >= e || k >= p.used[order[i]]) {
                            o.slot.push_back(kCgRowsPad);
                            o.col.push_back((uint16_t)(std::min(i, e - 1) - a));
                            continue;
                        }
                        const uint32_t s = 4 * p.row[order[i]] + k, c = p.col[s];
                        if (seen[c] != mark) {
                            seen[c] = mark;
                            place[c] = b.nn + b.nhalo++;
                            o.halo.push_back(c);
                        }
                        o.slot.push_back(s);
                        o.col.push_back((uint16_t)place[c]);
                    }
                b.units += units;
                b.ngroups++;
            }
            o.group.push_back(b.units);
            plan.records = std::max(plan.records, b.nn + b.nhalo);
            const uint32_t rim = std::min((3 * b.nhalo + 31) / 32 * 32, 256u);
            plan.threads = std::max({plan.threads, 32 * b.ngroups, 32 * warps + rim});
            o.blk.push_back(b);
        }
        plan.threads = std::min(plan.threads, kCgRowsMaxThreads);
        for (const CgRowsBlock& b : o.blk) plan.smem = std::max(plan.smem, cg_rows_smem_bytes(plan, b));
        if (plan.smem > kCgRowsMaxSmem) return false;
        if (blocks > 1) plan.smem = std::max(plan.smem, kCgRowsMaxSmem / 2 + 4096);  // one block per SM
        for (uint32_t i = 0; i < N; i++) place[order[i]] = i;
        std::vector<uint32_t> shared(N, 0);
        o.owner.resize(o.halo.size());
        for (uint32_t g = 0; g < blocks; g++)
            for (uint32_t i = o.blk[g].halo0; i < o.blk[g].halo0 + o.blk[g].nhalo; i++) {
                const uint32_t at = place[o.halo[i]], from = at / npb;
                const bool near = from / cluster == g / cluster;
                shared[at] |= near ? kCgRowsNearShared : kCgRowsFarShared;
                o.owner[i] = near ? (from % cluster) << 16 | (at - from * npb) : kCgRowsFar;
            }
        for (uint32_t i = 0; i < N; i++) o.node[i] |= shared[i];
        return blocks <= max_blocks(plan);
    };
    auto lay = [&](uint32_t blocks, uint32_t cluster) {
        return ((N + blocks - 1) / blocks <= 16 && build(blocks, cluster, 16)) || build(blocks, cluster, 8) || build(blocks, cluster, 4);
    };
    const uint32_t near = std::max(1u, std::min(16u, (N + kRowsPerBlock - 1) / kRowsPerBlock));
    if (lay(near, near)) return true;
    for (uint32_t cluster : {8u, 2u}) {
        CgRowsPlan shape;
        shape.lanes = 4;
        shape.threads = kCgRowsMaxThreads;
        shape.smem = kCgRowsMaxSmem;
        shape.cluster = cluster;
        const uint32_t blocks = max_blocks(shape) / cluster * cluster;
        if (blocks && lay(blocks, cluster)) return true;
    }
    return false;
}

}  // namespace femgb

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
// False: too large. ptr/idx: the node CSR of element corners. One pass over
// the corners finds a row's columns and counts its contributions, which start
// at three per corner.
inline bool bsr_pattern(uint32_t N, uint32_t T, const uint32_t* tets, const std::vector<uint32_t>& ptr,
                 const std::vector<uint32_t>& idx, BsrPattern& p)
{
    if ((uint64_t)T >= (1ull << 28)) return false;  // contributions pack the element in 28 bits
    std::vector<uint32_t> seen(N, 0xffffffffu), place(N), count, which;
    std::vector<uint64_t> nb;  // column << 32 | the order it was met in
    p.row.assign(N + 1, 0);
    p.used.resize(N);
    p.col.reserve(18 * (size_t)N);
    p.cptr.reserve(18 * (size_t)N + 1);
    p.contrib.resize(12 * (size_t)T);
    for (uint32_t n = 0; n < N; n++) {
        const uint32_t beg = ptr[n], end = ptr[n + 1];
        const size_t most = 3 * (size_t)(end - beg) + 1;
        if (nb.size() < most) {
            nb.resize(2 * most);
            count.resize(2 * most);
            which.resize(2 * most);
        }
        uint64_t* const col = nb.data();
        uint32_t *const at = count.data(), *w = which.data();
        uint32_t used = 1;
        col[0] = (uint64_t)n << 32;
        at[0] = place[n] = 0;
        seen[n] = n;
        for (uint32_t j = beg; j < end; j++)
            for (uint32_t k = 1; k < 4; k++) {
                const uint32_t c = tets[(size_t)(idx[j] & ~3u) + ((idx[j] + k) & 3u)];
                if (seen[c] != n) {
                    seen[c] = n;
                    place[c] = used;
                    at[used] = 0;
                    col[used] = (uint64_t)c << 32 | used;
                    used++;
                }
                at[*w++ = place[c]]++;
            }
        std::sort(col, col + used);
        p.used[n] = used;
        uint32_t next = 3 * beg;
        for (uint32_t i = 0; i < used; i++) {
            uint32_t& k = at[(uint32_t)col[i]];
            p.col.push_back((uint32_t)(col[i] >> 32));
            p.cptr.push_back(next);
            next += k;
            k = next - k;  // where its next contribution goes
        }
        while (p.col.size() % 4) {
            p.col.push_back(n);
            p.cptr.push_back(next);
        }
        if (p.col.size() >= (1ull << 28)) return false;
        p.row[n + 1] = (uint32_t)(p.col.size() / 4);
        w = which.data();
        for (uint32_t j = beg; j < end; j++)
            for (uint32_t k = 1; k < 4; k++) p.contrib[at[*w++]++] = idx[j] << 2 | ((idx[j] + k) & 3u);
    }
    p.cptr.push_back(12 * T);
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

// The plan of a shape and its blocks from each block's units and rim; false when
// they do not fit the shared memory.
struct CgRowsCount {
    uint32_t units, halo;
};
inline bool cg_rows_plan(uint32_t N, uint32_t blocks, uint32_t cluster, uint32_t lanes, const CgRowsCount* count,
                         CgRowsPlan& plan, std::vector<CgRowsBlock>& blk)
{
    plan = CgRowsPlan{};
    plan.blocks = blocks;
    plan.cluster = cluster;
    plan.lanes = lanes;
    plan.npb = (N + blocks - 1) / blocks;
    plan.warps = (3 * plan.npb + 31) / 32;
    plan.threads = 64;
    blk.clear();
    CgRowsBlock b{};
    for (uint32_t g = 0; g < blocks; g++) {
        b.node0 = std::min(N, g * plan.npb);
        b.nn = std::min(N, b.node0 + plan.npb) - b.node0;
        b.ngroups = (b.nn + 32 / lanes - 1) / (32 / lanes);
        b.units = count[g].units;
        b.nhalo = count[g].halo;
        blk.push_back(b);
        plan.units = std::max(plan.units, b.units);
        plan.records = std::max(plan.records, b.nn + b.nhalo);
        const uint32_t rim = std::min((3 * b.nhalo + 31) / 32 * 32, 256u);
        plan.threads = std::max({plan.threads, 32 * b.ngroups, 32 * plan.warps + rim});
        b.group0 += b.ngroups + 1;
        b.unit0 += b.units;
        b.halo0 += b.nhalo;
    }
    plan.threads = std::min(plan.threads, kCgRowsMaxThreads);
    for (const CgRowsBlock& c : blk) plan.smem = std::max(plan.smem, cg_rows_smem_bytes(plan, c));
    if (plan.smem > kCgRowsMaxSmem) return false;
    if (blocks > 1) plan.smem = std::max(plan.smem, kCgRowsMaxSmem / 2 + 4096);  // one block per SM
    return true;
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
// 16, as long as its blocks' sums fit the words a warp polls. Above that
// clusters of 8, all that are resident together with one block per SM, of 2 for
// the last of the SMs' memory. 16 lanes per row while a block has up to 16
// rows, else 8, else 4. Measured side by side, whole steps in early forms of
// the kernel (now 300, 421 and 515 us): 160 tets, rows in each 8 / 12 / 24 / 48:
// 399 / 417 / 424 / 485 us; 3,000 tets on one cluster 512, on all clusters, whose
// sums go through L2 (1.3 us more each), 575; 20,480 tets on clusters of 8 / 4 /
// 2 / 16: 637 / 727 / 746 / 648, with 8 / 16 / 4 lanes 637 / 660 / 658.
constexpr uint32_t kRowsPerBlock = 8;
// lay(blocks, cluster) for each shape, the best one first, until one is true.
template <typename F, typename L>
bool cg_rows_shapes(uint32_t N, F&& max_blocks, L&& lay)
{
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
// build(lanes) for each number of lanes per row, the best one first, until one is true.
template <typename B>
bool cg_rows_lanes(uint32_t N, uint32_t blocks, B&& build)
{
    return ((N + blocks - 1) / blocks <= 16 && build(16)) || build(8) || build(4);
}
inline bool cg_rows_shape_ok(uint32_t npb, uint32_t blocks, uint32_t cluster, uint32_t lanes)
{
    return 3 * npb + (blocks > 1 ? 32u : 0u) <= kCgRowsMaxThreads && (lanes <= 4 || lanes * npb <= kCgRowsMaxThreads) &&
           cluster * ((3 * npb + 31) / 32) <= kCgRowsMaxWords && blocks / cluster <= 96;
}

// Whether cg_rows_layout can succeed, from three blocks of each shape: the
// least their rows, vectors and rims take. Ahead of the pattern, which takes
// far longer (109,760 tets, which do not fit: 0.1 ms against 4.3 and 3.5 for
// pattern and layout).
template <typename F>
bool cg_rows_may_fit(uint32_t N, const uint32_t* tets, const std::vector<uint32_t>& ptr,
                     const std::vector<uint32_t>& idx, F&& max_blocks)
{
    std::vector<uint32_t> in_row(N, 0), in_rim(N, 0), used;
    uint32_t row = 0, mark = 0;
    return cg_rows_shapes(N, max_blocks, [&](uint32_t blocks, uint32_t cluster) {
        CgRowsPlan plan;
        plan.cluster = cluster;
        plan.npb = (N + blocks - 1) / blocks;
        plan.warps = (3 * plan.npb + 31) / 32;
        if (!cg_rows_shape_ok(plan.npb, blocks, cluster, 4)) return false;
        for (uint32_t g : {blocks / 2, blocks / 4, blocks - 1 - blocks / 4}) {
            const uint32_t a = std::min(N, g * plan.npb), e = std::min(N, a + plan.npb);
            CgRowsBlock b{a, e - a, 0, 0, 0, 0, 0, 0};
            used.assign(e - a, 1);
            mark++;
            for (uint32_t n = a; n < e; n++) {
                in_row[n] = ++row;
                for (uint32_t j = ptr[n]; j < ptr[n + 1]; j++)
                    for (uint32_t k = 1; k < 4; k++) {
                        const uint32_t c = tets[(size_t)(idx[j] & ~3u) + ((idx[j] + k) & 3u)];
                        if (in_row[c] == row) continue;
                        in_row[c] = row;
                        used[n - a]++;
                        if ((c < a || c >= e) && in_rim[c] != mark) {
                            in_rim[c] = mark;
                            b.nhalo++;
                        }
                    }
            }
            plan.records = b.nn + b.nhalo;
            std::sort(used.begin(), used.end(), [](uint32_t i, uint32_t j) { return i > j; });
            size_t least = ~(size_t)0;
            for (uint32_t lanes : {4u, 8u, 16u}) {
                b.units = b.ngroups = 0;
                for (uint32_t i = 0; i < e - a; i += 32 / lanes, b.ngroups++) b.units += (used[i] + lanes - 1) / lanes;
                plan.units = b.units;
                least = std::min(least, cg_rows_smem_bytes(plan, b));
            }
            if (least > kCgRowsMaxSmem) return false;
        }
        return true;
    });
}

// The layout on the host: what the device's (rows_build.h) is checked against.
template <typename F>
bool cg_rows_layout(uint32_t N, const BsrPattern& p, F&& max_blocks, CgRowsLayout& o)
{
    if (N > kCgRowsNode) return false;
    std::vector<uint32_t> order(N), seen(N, 0), place(N);
    uint32_t sorted = 0;  // rows per block that order is sorted for
    auto build = [&](uint32_t blocks, uint32_t cluster, uint32_t lanes) {
        const uint32_t npb = (N + blocks - 1) / blocks, rows = 32 / lanes;
        if (!cg_rows_shape_ok(npb, blocks, cluster, lanes)) return false;
        if (sorted != npb) {
            for (uint32_t n = 0; n < N; n++) order[n] = n;
            for (uint32_t a = 0; a < N; a += npb)
                std::sort(order.begin() + a, order.begin() + std::min(N, a + npb),
                          [&](uint32_t i, uint32_t j) { return p.used[i] != p.used[j] ? p.used[i] > p.used[j] : i < j; });
            sorted = npb;
        }
        o = CgRowsLayout{};
        std::vector<CgRowsCount> count(blocks);
        std::vector<uint32_t> rim;
        std::fill(seen.begin(), seen.end(), 0u);
        for (uint32_t g = 0; g < blocks; g++) {
            const uint32_t a = std::min(N, g * npb), e = std::min(N, a + npb), mark = g + 1;
            for (uint32_t i = a; i < e; i++) {
                seen[order[i]] = mark;
                place[order[i]] = i - a;
            }
            rim.clear();
            for (uint32_t i = a; i < e; i++)
                for (uint32_t k = 0; k < p.used[i]; k++) {
                    const uint32_t c = p.col[4 * p.row[i] + k];
                    if (seen[c] != mark) {
                        seen[c] = mark;
                        rim.push_back(c);
                    }
                }
            std::sort(rim.begin(), rim.end());
            for (uint32_t i = 0; i < rim.size(); i++) place[rim[i]] = e - a + i;
            o.halo.insert(o.halo.end(), rim.begin(), rim.end());
            uint32_t units = 0;
            for (uint32_t g0 = a; g0 < e; g0 += rows) {
                o.group.push_back(units);
                const uint32_t most = (p.used[order[g0]] + lanes - 1) / lanes;
                for (uint32_t u = 0; u < most; u++)
                    for (uint32_t l = 0; l < 32; l++) {
                        const uint32_t i = g0 + l / lanes, k = lanes * u + l % lanes;
                        const bool pad = i >= e || k >= p.used[order[i]];
                        const uint32_t s = pad ? kCgRowsPad : 4 * p.row[order[i]] + k;
                        o.slot.push_back(s);
                        o.col.push_back((uint16_t)(pad ? std::min(i, e - 1) - a : place[p.col[s]]));
                    }
                units += most;
            }
            o.group.push_back(units);
            count[g] = CgRowsCount{units, (uint32_t)rim.size()};
        }
        if (!cg_rows_plan(N, blocks, cluster, lanes, count.data(), o.plan, o.blk)) return false;
        o.node = order;
        for (uint32_t i = 0; i < N; i++) place[order[i]] = i;
        o.owner.resize(o.halo.size());
        for (uint32_t g = 0; g < blocks; g++)
            for (uint32_t i = o.blk[g].halo0; i < o.blk[g].halo0 + o.blk[g].nhalo; i++) {
                const uint32_t at = place[o.halo[i]], from = at / npb;
                const bool near = from / cluster == g / cluster;
                o.node[at] |= near ? kCgRowsNearShared : kCgRowsFarShared;
                o.owner[i] = near ? (from % cluster) << 16 | (at - from * npb) : kCgRowsFar;
            }
        return blocks <= max_blocks(o.plan);
    };
    return cg_rows_shapes(N, max_blocks, [&](uint32_t blocks, uint32_t cluster) {
        return cg_rows_lanes(N, blocks, [&](uint32_t lanes) { return build(blocks, cluster, lanes); });
    });
}

}  // namespace femgb

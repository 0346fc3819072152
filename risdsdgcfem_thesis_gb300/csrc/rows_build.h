// rows_build.h -- the tables of rows_plan.h made where the mesh is, on the
// device (rows_build.cu). Each step is a function of a thread and the number of
// threads, with a barrier between steps, so that the CPU can run the same code
// over all threads in turn against bsr_pattern and cg_rows_layout.
//
// On the host they were a pass over every corner and one over every block after
// reading the mesh's tables back. First step of a new solid less a later one, 3
// iterations: 160 tets 0.21 -> 0.15 ms, 2,560 0.52 -> 0.31, 20,480 1.80 -> 0.37,
// 87,880 6.5 -> 0.45, of which capturing the step's graph is about 0.1; most of
// the rest is allocation.
#pragma once
#include "fx.cuh"
#include "rows_plan.h"

namespace femgb {

// The most entries of a row (itself and three per corner) that a warp takes;
// meshes with a longer one (a hub of more than 341 corners) take bsr_pattern.
constexpr uint32_t kRowEntries = 1024;

// e[0] = n, then the other nodes of n's corners, in the corners' order.
FX_HD void row_entries(uint32_t n, uint32_t beg, uint32_t entries, const uint32_t* tets, const uint32_t* idx, uint32_t* e,
                       uint32_t t, uint32_t threads)
{
    for (uint32_t i = t; i < entries; i += threads) {
        const uint32_t v = i ? idx[beg + (i - 1) / 3] : 0u;
        e[i] = i ? tets[(size_t)(v & ~3u) + ((v + 1 + (i - 1) % 3) & 3u)] : n;
    }
}
// before[i]: the entries ahead of i with its node; returns this thread's
// entries with none, which are the row's columns.
FX_HD uint32_t row_columns(const uint32_t* e, uint32_t entries, uint32_t* before, uint32_t t, uint32_t threads)
{
    uint32_t columns = 0;
    for (uint32_t i = t; i < entries; i += threads) {
        uint32_t k = 0;
        for (uint32_t m = 0; m < i; m++) k += e[m] == e[i] ? 1u : 0u;
        before[i] = k;
        columns += k == 0 ? 1u : 0u;
    }
    return columns;
}
// The row's part of BsrPattern from its first slot on: columns ascending, each
// with its contributions in the corners' order, which start at three per corner.
FX_HD void row_write(const uint32_t* e, const uint32_t* before, uint32_t entries, uint32_t beg, uint32_t used,
                     uint32_t slot, const uint32_t* idx, uint32_t* col, uint32_t* cptr, uint32_t* contrib, uint32_t t,
                     uint32_t threads)
{
    for (uint32_t i = t; i < entries; i += threads) {
        uint32_t rank = 0, start = 3 * beg;
        for (uint32_t m = 0; m < entries; m++)
            if (e[m] < e[i]) {
                rank += before[m] == 0 ? 1u : 0u;
                start += m ? 1u : 0u;
            }
        if (before[i] == 0) {
            col[slot + rank] = e[i];
            cptr[slot + rank] = start;
        }
        if (i) {
            const uint32_t v = idx[beg + (i - 1) / 3];
            contrib[start + before[i] - (e[i] == e[0] ? 1u : 0u)] = v << 2 | ((v + 1 + (i - 1) % 3) & 3u);
        }
    }
    for (uint32_t k = used + t; k < (used + 3) / 4 * 4; k += threads) {
        col[slot + k] = e[0];
        cptr[slot + k] = 3 * beg + entries - 1;
    }
}

// A block of the layout: its rows by length, its groups' units, its rim as a
// bit per node.
constexpr uint32_t kLayoutRows = 256, kLayoutThreads = 256;
constexpr uint32_t kLayoutWords = (kCgRowsMaxBlocks * (kCgRowsMaxThreads / 3) + 31) / 32;
struct LayoutWork {
    uint32_t used[kLayoutRows], order[kLayoutRows], rank[kLayoutRows], start[kLayoutRows + 1];
    uint32_t bits[kLayoutWords], ahead[kLayoutWords], part[kLayoutThreads];
    uint32_t units, halo;
};
struct LayoutShape {
    uint32_t N, npb, lanes, cluster;
};
// (a block's columns are in col from 4 row[n] on)
struct LayoutRows {
    const uint32_t *used, *row, *col;
};
struct LayoutOut {
    CgRowsBlock* blk;  // node0, nn, group0, unit0, halo0 given
    uint32_t *node, *place, *group, *slot, *halo, *owner;
    uint16_t* col;
};
struct LayoutSpan {
    uint32_t a, e, groups, words;
};
FX_HD LayoutSpan layout_span(const LayoutShape& s, uint32_t g)
{
    const uint32_t a = g * s.npb < s.N ? g * s.npb : s.N, e = a + s.npb < s.N ? a + s.npb : s.N, rows = 32 / s.lanes;
    return LayoutSpan{a, e, (e - a + rows - 1) / rows, (s.N + 31) / 32};
}
FX_HD uint32_t layout_popc(uint32_t v)
{
#ifdef __CUDA_ARCH__
    return (uint32_t)__popc(v);
#else
    return (uint32_t)__builtin_popcount(v);
#endif
}
FX_HD void layout_or(uint32_t* p, uint32_t v)
{
#ifdef __CUDA_ARCH__
    atomicOr(p, v);
#else
    *p |= v;
#endif
}
FX_HD void layout_begin(const LayoutSpan& b, const LayoutRows& m, LayoutWork& w, uint32_t t, uint32_t threads)
{
    for (uint32_t i = t; i < b.e - b.a; i += threads) w.used[i] = m.used[b.a + i];
    for (uint32_t i = t; i < b.words; i += threads) w.bits[i] = 0;
}
FX_HD void layout_rim(const LayoutSpan& b, const LayoutRows& m, LayoutWork& w, uint32_t t, uint32_t threads)
{
    const uint32_t nn = b.e - b.a;
    for (uint32_t i = t; i < nn; i += threads) {
        uint32_t r = 0;
        for (uint32_t k = 0; k < nn; k++) r += w.used[k] > w.used[i] || (w.used[k] == w.used[i] && k < i) ? 1u : 0u;
        w.order[r] = i;
        w.rank[i] = r;
        const uint32_t* c = m.col + 4 * (size_t)m.row[b.a + i];
        for (uint32_t k = 0; k < w.used[i]; k++)
            if (c[k] < b.a || c[k] >= b.e) layout_or(w.bits + (c[k] >> 5), 1u << (c[k] & 31u));
    }
}
FX_HD void layout_parts(const LayoutShape& s, const LayoutSpan& b, LayoutWork& w, uint32_t t, uint32_t threads)
{
    const uint32_t per = (b.words + threads - 1) / threads, rows = 32 / s.lanes;
    uint32_t n = 0;
    for (uint32_t i = t * per; i < (t + 1) * per && i < b.words; i++) n += layout_popc(w.bits[i]);
    w.part[t] = n;
    if (t != 0) return;
    uint32_t units = 0;
    for (uint32_t g = 0; g < b.groups; g++) {
        w.start[g] = units;
        units += (w.used[w.order[g * rows]] + s.lanes - 1) / s.lanes;
    }
    w.start[b.groups] = w.units = units;
}
FX_HD void layout_sum(LayoutWork& w, uint32_t t, uint32_t threads)
{
    if (t != 0) return;
    uint32_t n = 0;
    for (uint32_t i = 0; i < threads; i++) {
        const uint32_t k = w.part[i];
        w.part[i] = n;
        n += k;
    }
    w.halo = n;
}
FX_HD void layout_ahead(const LayoutSpan& b, LayoutWork& w, uint32_t t, uint32_t threads)
{
    const uint32_t per = (b.words + threads - 1) / threads;
    uint32_t n = w.part[t];
    for (uint32_t i = t * per; i < (t + 1) * per && i < b.words; i++) {
        w.ahead[i] = n;
        n += layout_popc(w.bits[i]);
    }
}
FX_HD void layout_write(const LayoutShape& s, const LayoutSpan& b, uint32_t g, const LayoutRows& m, const LayoutWork& w,
                        const LayoutOut& o, uint32_t t, uint32_t threads)
{
    const uint32_t nn = b.e - b.a, rows = 32 / s.lanes, lane = t & 31u;
    const CgRowsBlock B = o.blk[g];
    for (uint32_t r = t; r < nn; r += threads) {
        o.node[b.a + r] = b.a + w.order[r];
        o.place[b.a + w.order[r]] = b.a + r;
    }
    for (uint32_t i = t; i <= b.groups; i += threads) o.group[B.group0 + i] = b.groups ? w.start[i] : 0u;
    for (uint32_t i = t; i < b.words; i += threads) {
        uint32_t at = B.halo0 + w.ahead[i];
        for (uint32_t k = 0; k < 32; k++)
            if (w.bits[i] >> k & 1u) o.halo[at++] = 32 * i + k;
    }
    for (uint32_t q = t >> 5; q < b.groups; q += threads >> 5)
        for (uint32_t u = w.start[q]; u < w.start[q + 1]; u++) {
            const uint32_t r = q * rows + lane / s.lanes, k = s.lanes * (u - w.start[q]) + lane % s.lanes;
            const size_t at = 32 * ((size_t)B.unit0 + u) + lane;
            if (r >= nn || k >= w.used[w.order[r]]) {
                o.slot[at] = kCgRowsPad;
                o.col[at] = (uint16_t)(r < nn ? r : nn - 1);
                continue;
            }
            const uint32_t slot = 4 * m.row[b.a + w.order[r]] + k, c = m.col[slot];
            o.slot[at] = slot;
            o.col[at] = (uint16_t)(c >= b.a && c < b.e
                                       ? w.rank[c - b.a]
                                       : nn + w.ahead[c >> 5] + layout_popc(w.bits[c >> 5] & ((1u << (c & 31u)) - 1u)));
        }
}
// Where the rim's values come from, and the marks of the nodes they are; after
// every block's layout_write.
FX_HD void layout_owners(const LayoutShape& s, uint32_t g, const LayoutOut& o, uint32_t t, uint32_t threads)
{
    const CgRowsBlock B = o.blk[g];
    for (uint32_t i = B.halo0 + t; i < B.halo0 + B.nhalo; i += threads) {
        const uint32_t at = o.place[o.halo[i]], from = at / s.npb;
        const bool near = from / s.cluster == g / s.cluster;
        o.owner[i] = near ? (from % s.cluster) << 16 | (at - from * s.npb) : kCgRowsFar;
        layout_or(o.node + at, near ? kCgRowsNearShared : kCgRowsFarShared);
    }
}

}  // namespace femgb

"""Host tables of the CG solve on resident rows (rows_plan.h) on the CPU: a
product through them against the mesh's own adjacency, every index in range."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from risdsdgcfem_thesis_gb300 import scenes

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "risdsdgcfem_thesis_gb300", "csrc")
SHIM = r"""
#include "rows_plan.h"
using namespace femgb;
// y = A d with A(n, c) = a[n] b[c] for neighbours c, n itself included;
// returns 0, -1 without a layout, else the line of a failed check.
#define CHECK(x) do { if (!(x)) return __LINE__; } while (0)
extern "C" int rows(uint32_t N, uint32_t T, const uint32_t* tets, uint32_t sms, const double* a, const double* d,
                    double* y, uint32_t* contribs, uint32_t* blocks)
{
    std::vector<uint32_t> ptr(N + 1, 0), idx(4 * (size_t)T);
    for (size_t i = 0; i < 4 * (size_t)T; i++) ptr[tets[i] + 1]++;
    for (uint32_t n = 0; n < N; n++) ptr[n + 1] += ptr[n];
    std::vector<uint32_t> fill(ptr.begin(), ptr.end() - 1);
    for (size_t i = 0; i < 4 * (size_t)T; i++) idx[fill[tets[i]]++] = (uint32_t)i;
    BsrPattern p;
    CHECK(bsr_pattern(N, T, tets, ptr, idx, p));
    const size_t slots = p.col.size();
    CHECK(p.row[N] * (size_t)4 == slots && p.cptr[slots] == 12 * (size_t)T && p.contrib.size() == 12 * (size_t)T);
    for (uint32_t n = 0; n < N; n++)
        for (uint32_t s = 4 * p.row[n]; s < 4 * p.row[n + 1]; s++) {
            CHECK(p.col[s] < N);
            for (uint32_t k = p.cptr[s]; k < p.cptr[s + 1]; k++) {
                const uint32_t e = p.contrib[k] >> 4, li = (p.contrib[k] >> 2) & 3, lj = p.contrib[k] & 3;
                CHECK(e < T && li != lj && tets[4 * e + li] == n && tets[4 * e + lj] == p.col[s]);
                contribs[0]++;
            }
        }
    CgRowsLayout l;
    if (!cg_rows_layout(N, p, [&](const CgRowsPlan& q) {
            return q.threads > kCgRowsMaxThreads || q.smem > kCgRowsMaxSmem || q.cluster > sms ? 0u : sms;
        }, l)) return -1;
    const uint32_t L = l.plan.lanes, rows = 32 / L;
    CHECK(l.plan.blocks == l.blk.size() && l.plan.blocks <= sms && l.node.size() == N);
    CHECK(l.plan.threads % 32 == 0 && l.plan.threads <= kCgRowsMaxThreads);
    const uint32_t G = l.plan.blocks, K = l.plan.cluster;
    CHECK(G % K == 0 && K * l.plan.warps <= 160 && G / K <= 96 && l.owner.size() == l.halo.size());
    std::vector<int> used(slots, 0), seen(N, 0);
    std::vector<uint32_t> in_rim(N, 0);
    for (size_t g = 0; g < l.blk.size(); g++) {
        const CgRowsBlock b = l.blk[g];
        CHECK(3 * b.nn <= 32 * l.plan.warps && 32 * l.plan.warps + (b.nhalo ? 32 : 0) <= l.plan.threads);
        CHECK(cg_rows_smem_bytes(l.plan, b) <= l.plan.smem && b.nn <= l.plan.npb && b.units <= l.plan.units);
        CHECK(b.nn + b.nhalo <= l.plan.records);
        CHECK(l.group.size() >= b.group0 + b.ngroups + 1 && l.group[b.group0] == 0 && l.group[b.group0 + b.ngroups] == b.units);
        CHECK(rows * b.ngroups >= b.nn && 32 * (size_t)(b.unit0 + b.units) <= l.slot.size() && l.slot.size() == l.col.size());
        for (uint32_t w = 0; w < b.ngroups; w++)
            for (uint32_t lane = 0; lane < 32; lane++) {
                const uint32_t row = rows * w + lane / L;
                for (uint32_t u = l.group[b.group0 + w]; u < l.group[b.group0 + w + 1]; u++) {
                    const size_t at = 32 * (size_t)(b.unit0 + u) + lane;
                    const uint32_t s = l.slot[at], c = l.col[at];
                    CHECK(c < b.nn + b.nhalo);
                    if (s == kCgRowsPad) continue;
                    CHECK(row < b.nn && s < slots);
                    const uint32_t n = l.node[b.node0 + row] & kCgRowsNode;
                    const uint32_t gc = c < b.nn ? l.node[b.node0 + c] & kCgRowsNode : l.halo[b.halo0 + c - b.nn];
                    CHECK(n < N && gc < N && p.col[s] == gc && s >= 4 * p.row[n] && s < 4 * p.row[n + 1]);
                    used[s]++;
                    if (c >= b.nn) {
                        const uint32_t o = l.owner[b.halo0 + c - b.nn], near = g / K * K + (o >> 16);
                        in_rim[gc] |= o == kCgRowsFar ? kCgRowsFarShared : kCgRowsNearShared;
                        CHECK(o == kCgRowsFar || (near < G && (o & 0xffff) < l.blk[near].nn &&
                                                  (l.node[l.blk[near].node0 + (o & 0xffff)] & kCgRowsNode) == gc));
                    }
                    y[n] += a[n] * a[gc] * d[gc];
                }
            }
        for (uint32_t i = 0; i < b.nn; i++) seen[l.node[b.node0 + i] & kCgRowsNode]++;
    }
    for (uint32_t n = 0; n < N; n++) CHECK(seen[n] == 1);
    for (uint32_t w : l.node) CHECK((w & ~kCgRowsNode) == in_rim[w & kCgRowsNode]);
    for (uint32_t n = 0; n < N; n++)
        for (uint32_t k = 0; k < 4 * (p.row[n + 1] - p.row[n]); k++) CHECK(used[4 * p.row[n] + k] == (k < p.used[n]));
    *blocks = l.plan.blocks;
    return 0;
}
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("rows")
    src, lib = d / "rows.cpp", d / "rows.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(lib)], check=True)
    return C.CDLL(str(lib))


def _star(k):
    """k tets around one node, which every other node neighbours."""
    t = np.arange(3 * k, dtype=np.uint32).reshape(k, 3) + 1
    return 3 * k + 1, np.concatenate([np.zeros((k, 1), np.uint32), t], 1)


def _grid(*dims):
    rest, tets, _ = scenes.grid_mesh(*dims, 0.1, 0.01, 5)
    return len(rest), tets


@pytest.mark.parametrize("sms", [2, 16, 152])
@pytest.mark.parametrize("mesh,shuffle", [(_grid(1, 1, 1), False), (_grid(5, 5, 5), False), (_grid(6, 6, 5), True),
                                          (_grid(17, 16, 15), False), (_grid(17, 16, 15), True), (_star(150), False),
                                          ((9, _grid(1, 1, 1)[1]), False), (_grid(45, 40, 40), False)],
                         ids=["cell", "216", "294shuffled", "20400", "20400shuffled", "star", "lone", "360000"])
def test_layout_covers_the_rows(shim, mesh, shuffle, sms):
    n, tets = mesh
    rng = np.random.default_rng(2)
    if shuffle:
        tets = rng.permutation(n).astype(np.uint32)[tets]
    tets = np.ascontiguousarray(tets, np.uint32)
    a, d, y = rng.integers(-9, 10, n).astype(float), rng.integers(-9, 10, n).astype(float), np.zeros(n)
    contribs, blocks = C.c_uint32(0), C.c_uint32(0)
    dp = lambda v: v.ctypes.data_as(C.POINTER(C.c_double))
    rc = shim.rows(n, len(tets), tets.ctypes.data_as(C.POINTER(C.c_uint32)), sms, dp(a), dp(d), dp(y),
                   C.byref(contribs), C.byref(blocks))
    assert contribs.value == 12 * len(tets)
    if rc == -1:
        assert n > 200 * sms  # about 1,000 bytes a row
        return
    assert rc == 0
    pairs = np.unique(np.concatenate([np.stack([tets[:, i], tets[:, j]], 1) for i in range(4) for j in range(4)] +
                                     [np.stack([np.arange(n)] * 2, 1)]), axis=0)
    ref = np.zeros(n)
    np.add.at(ref, pairs[:, 0], a[pairs[:, 0]] * a[pairs[:, 1]] * d[pairs[:, 1]])
    assert np.array_equal(y, ref)


FITS = r"""
#include "rows_plan.h"
using namespace femgb;
// Bit 0: the layout succeeds; bit 1: cg_rows_may_fit; bit 2: some block does not hold its own range of nodes.
extern "C" int fits(uint32_t N, uint32_t T, const uint32_t* tets)
{
    std::vector<uint32_t> ptr(N + 1, 0), idx(4 * (size_t)T);
    for (size_t i = 0; i < 4 * (size_t)T; i++) ptr[tets[i] + 1]++;
    for (uint32_t n = 0; n < N; n++) ptr[n + 1] += ptr[n];
    std::vector<uint32_t> fill(ptr.begin(), ptr.end() - 1);
    for (size_t i = 0; i < 4 * (size_t)T; i++) idx[fill[tets[i]]++] = (uint32_t)i;
    auto blocks = [](const CgRowsPlan& q) {
        return q.threads > kCgRowsMaxThreads || q.smem > kCgRowsMaxSmem ? 0u : q.cluster == 2 ? 152u : 120u;
    };
    BsrPattern p;
    CgRowsLayout l;
    int r = bsr_pattern(N, T, tets, ptr, idx, p) && cg_rows_layout(N, p, blocks, l) ? 1 : 0;
    if (cg_rows_may_fit(N, tets, ptr, idx, blocks)) r |= 2;
    if (r & 1)
        for (const CgRowsBlock& b : l.blk)
            for (uint32_t i = b.node0; i < b.node0 + b.nn; i++) {
                const uint32_t n = l.node[i] & kCgRowsNode;
                if (n < b.node0 || n >= b.node0 + b.nn) r |= 4;
            }
    return r;
}
"""


@pytest.fixture(scope="module")
def fits(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("fits")
    src, so = d / "fits.cpp", d / "fits.so"
    src.write_text(FITS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    return C.CDLL(str(so)).fits


@pytest.mark.parametrize("mesh,fit", [(_grid(1, 1, 1), True), (_grid(12, 12, 12), True), (_grid(16, 16, 16), True),
                                      (_grid(26, 26, 26), True), (_grid(28, 28, 27), True), (_grid(80, 80, 2), True),
                                      (_grid(28, 28, 28), False), (_grid(60, 20, 18), False), (_grid(100, 30, 6), False),
                                      (_grid(200, 11, 11), False), (_grid(1000, 5, 5), False), (_star(150), True),
                                      (_star(3000), False)],
                         ids=["5", "8640", "20480", "87880", "105840", "flat64000", "109760", "108000", "flat90000",
                              "long121000", "long125000", "star", "star3000"])
def test_whether_the_rows_fit_is_known_ahead(fits, mesh, fit):
    """cg_rows_may_fit agrees with the layout (it may only err towards a try),
    and the layout's blocks hold ranges of nodes whatever shape was tried first."""
    n, tets = mesh
    tets = np.ascontiguousarray(tets, np.uint32)
    r = fits(n, len(tets), tets.ctypes.data_as(C.POINTER(C.c_uint32)))
    assert bool(r & 1) == fit and not r & 4
    assert bool(r & 2) == fit if len(tets) > 3000 else r & 2 or not fit


WORDS = r"""
#include "rows_words.h"
using namespace femgb;
struct W { unsigned long long x, y; };
// The words a solve starts with after number seq: 0 unless one of them reads
// as one of the solve's first numbers.
extern "C" int taken(uint32_t seq)
{
    W w[8];
    rows_words_start(w, 3, 5, seq, 0, 1);
    for (uint32_t ahead = 1; ahead < 5; ahead++)
        for (int i = 0; i < 8; i++) {
            Part p;
            double v;
            if (i < 3 ? rows_word_is(w[i], p, seq + ahead) : rows_word_is(w[i], v, seq + ahead)) return i + 1;
        }
    return 0;
}
extern "C" double through(double v) { return part_value(part_of(v)); }
extern "C" double infinities(int plus, int minus) { return part_value(Part{(int64_t)(plus - minus) * (1ll << 42) - 5120, kPartInf}); }
extern "C" int kept(double v, int64_t m, int32_t e, uint32_t seq)
{
    Part p;
    double u;
    return rows_word_is(rows_word<W>(v, seq), u, seq) && fx_bits(u) == fx_bits(v) &&
           rows_word_is(rows_word<W>(Part{m, e}, seq), p, seq) && p.m == m && p.e == e;
}
"""


def test_words_between_blocks(tmp_path):
    """Data survives the words, and what they hold at the start of a solve is
    no answer to its first exchanges, whatever the number (both formats wrap)."""
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    src, so = tmp_path / "words.cpp", tmp_path / "words.so"
    src.write_text(WORDS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wno-unknown-pragmas", "-shared", "-fPIC", "-I", CSRC, str(src),
                    "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    lib.taken.argtypes = [C.c_uint32]
    lib.kept.argtypes = [C.c_double, C.c_int64, C.c_int32, C.c_uint32]
    edges = [k + d for k in (0, 0xffff, 0x10000, 0xfffeffff, 0xffff0000, 0xffffffff, 0x7fffffff) for d in (-1, 0, 1)]
    for seq in [e & 0xffffffff for e in edges] + [0x10001 * k for k in range(0, 0x10000, 257)]:
        assert lib.taken(seq) == 0, hex(seq)
        for v, m, e in ((0.0, 0, 0), (-1.5, -(1 << 62), 2046), (np.inf, (1 << 62), 0x7fff), (5e-324, -1, 1)):
            assert lib.kept(v, m, e, seq), hex(seq)

    lib.through.argtypes, lib.through.restype, lib.infinities.restype = [C.c_double], C.c_double, C.c_double
    for v in (0.0, 1.0, -1.5, 2.2250738585072014e-308, 1.7976931348623157e308, np.inf, -np.inf):
        assert lib.through(v) == v
    assert np.isnan(lib.through(np.nan))
    assert lib.infinities(3, 1) == np.inf and lib.infinities(1, 2) == -np.inf and np.isnan(lib.infinities(2, 2))


QUOTIENT = r"""
#include <math.h>
#include "rows_words.h"
using namespace femgb;
#include <float.h>
#if LDBL_MANT_DIG >= 113
typedef long double Q;
#else
typedef __float128 Q;
#endif
// The error of t / d in units of its last place; -1 where it is to be divided.
extern "C" double ulps(double t, double d)
{
    double q;
    if (!rows_quotient(t, d, 1.0 / d, q)) return -1.0;
    int e;
    frexp(q, &e);
    const Q err = ((Q)q - (Q)t / (Q)d) / (Q)ldexp(1.0, e - 53);
    return (double)(err < 0 ? -err : err);
}
"""


def test_quotient_by_the_reciprocal(tmp_path):
    """Half a unit in the last place, and 2^-50 for the corrected product's
    own error, wherever it is taken."""
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    src, so = tmp_path / "quotient.cpp", tmp_path / "quotient.so"
    src.write_text(QUOTIENT)
    subprocess.run(["g++", "-std=gnu++17", "-O2", "-ffp-contract=off", "-Wno-unknown-pragmas", "-shared", "-fPIC", "-I", CSRC,
                    str(src), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    lib.ulps.argtypes, lib.ulps.restype = [C.c_double, C.c_double], C.c_double
    rng = np.random.default_rng(9)
    taken = 0
    for span in (0.001, 1, 30, 280, 307):
        t, d = (rng.uniform(1, 2, 20000) * 10.0 ** rng.uniform(-span, span, 20000) for _ in range(2))
        for a, b in zip(t, d):
            u = lib.ulps(a, b)
            assert u <= 0.5 + 2.0 ** -50, (a, b, u)
            taken += u >= 0
    assert taken > 60000
    edges = [0.0, 5e-324, 2.2250738585072014e-308, 1e-300, 1.0, np.nextafter(1, 2), 1.7976931348623157e308, np.inf, np.nan]
    for a in edges:
        for b in edges:
            u = lib.ulps(a, b)
            assert u <= 0.5 + 2.0 ** -50 and (u == -1.0 or np.isfinite([a, b]).all()), (a, b, u)


BUILD = r"""
#include <memory>
#include "rows_build.h"
using namespace femgb;
// The device's pattern and layout, every thread of a step in turn, against the
// host's; returns 0, or the line of the first difference (-1: no layout, both).
#define CHECK(x) do { if (!(x)) return __LINE__; } while (0)
extern "C" int build(uint32_t N, uint32_t T, const uint32_t* tets, uint32_t sms)
{
    std::vector<uint32_t> ptr(N + 1, 0), idx(4 * (size_t)T);
    for (size_t i = 0; i < 4 * (size_t)T; i++) ptr[tets[i] + 1]++;
    for (uint32_t n = 0; n < N; n++) ptr[n + 1] += ptr[n];
    std::vector<uint32_t> fill(ptr.begin(), ptr.end() - 1);
    for (size_t i = 0; i < 4 * (size_t)T; i++) idx[fill[tets[i]]++] = (uint32_t)i;
    BsrPattern p;
    CHECK(bsr_pattern(N, T, tets, ptr, idx, p));
    const size_t slots = p.col.size();
    std::vector<uint32_t> e(kRowEntries), before(kRowEntries), col(slots, ~0u), cptr(slots + 1, ~0u), contrib(12 * (size_t)T, ~0u);
    cptr[slots] = 12 * T;
    for (uint32_t n = 0; n < N; n++) {
        const uint32_t entries = 3 * (ptr[n + 1] - ptr[n]) + 1;
        CHECK(entries <= kRowEntries);
        uint32_t used = 0;
        for (uint32_t t = 0; t < 32; t++) row_entries(n, ptr[n], entries, tets, idx.data(), e.data(), t, 32);
        for (uint32_t t = 0; t < 32; t++) used += row_columns(e.data(), entries, before.data(), t, 32);
        CHECK(used == p.used[n]);
        for (uint32_t t = 0; t < 32; t++)
            row_write(e.data(), before.data(), entries, ptr[n], used, 4 * p.row[n], idx.data(), col.data(), cptr.data(),
                      contrib.data(), t, 32);
    }
    CHECK(col == p.col && cptr == p.cptr && contrib == p.contrib);
    auto most = [&](const CgRowsPlan& q) {
        return q.threads > kCgRowsMaxThreads || q.smem > kCgRowsMaxSmem || q.cluster > sms ? 0u : sms;
    };
    CgRowsLayout l;
    const bool laid = cg_rows_layout(N, p, most, l);
    CgRowsPlan plan;
    std::vector<CgRowsBlock> blk;
    const LayoutRows rows{p.used.data(), p.row.data(), p.col.data()};
    std::unique_ptr<LayoutWork> w(new LayoutWork);
    const uint32_t K = kLayoutThreads;
    LayoutShape shape{};
    auto count = [&](const LayoutShape& s, uint32_t g) {
        const LayoutSpan b = layout_span(s, g);
        for (uint32_t t = 0; t < K; t++) layout_begin(b, rows, *w, t, K);
        for (uint32_t t = 0; t < K; t++) layout_rim(b, rows, *w, t, K);
        for (uint32_t t = 0; t < K; t++) layout_parts(s, b, *w, t, K);
        for (uint32_t t = 0; t < K; t++) layout_sum(*w, t, K);
    };
    const bool built = cg_rows_shapes(N, most, [&](uint32_t blocks, uint32_t cluster) {
        return cg_rows_lanes(N, blocks, [&](uint32_t lanes) {
            shape = LayoutShape{N, (N + blocks - 1) / blocks, lanes, cluster};
            if (!cg_rows_shape_ok(shape.npb, blocks, cluster, lanes)) return false;
            if (shape.npb > kLayoutRows || (N + 31) / 32 > kLayoutWords) __builtin_trap();
            std::vector<CgRowsCount> c(blocks);
            for (uint32_t g = 0; g < blocks; g++) {
                count(shape, g);
                c[g] = CgRowsCount{w->units, w->halo};
            }
            return cg_rows_plan(N, blocks, cluster, lanes, c.data(), plan, blk) && blocks <= most(plan);
        });
    });
    CHECK(built == laid);
    if (!laid) return -1;
    CHECK(plan.blocks == l.plan.blocks && plan.threads == l.plan.threads && plan.smem == l.plan.smem);
    const CgRowsBlock& z = blk.back();
    std::vector<uint32_t> node(N, ~0u), place(N, ~0u), group(z.group0 + z.ngroups + 1, ~0u), slot(32 * (size_t)(z.unit0 + z.units), ~1u),
        halo(z.halo0 + z.nhalo, ~0u), owner(halo.size(), ~1u);
    std::vector<uint16_t> lcol(slot.size(), 0xffff);
    const LayoutOut o{blk.data(), node.data(), place.data(), group.data(), slot.data(), halo.data(), owner.data(), lcol.data()};
    for (uint32_t g = 0; g < plan.blocks; g++) {
        count(shape, g);
        const LayoutSpan b = layout_span(shape, g);
        for (uint32_t t = 0; t < K; t++) layout_ahead(b, *w, t, K);
        for (uint32_t t = 0; t < K; t++) layout_write(shape, b, g, rows, *w, o, t, K);
    }
    for (uint32_t g = 0; g < plan.blocks; g++)
        for (uint32_t t = 0; t < K; t++) layout_owners(shape, g, o, t, K);
    CHECK(node == l.node && group == l.group && slot == l.slot && halo == l.halo && owner == l.owner && lcol == l.col);
    for (uint32_t g = 0; g < plan.blocks; g++) CHECK(memcmp(&blk[g], &l.blk[g], sizeof(CgRowsBlock)) == 0);
    return 0;
}
"""


@pytest.fixture(scope="module")
def build(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("build")
    src, so = d / "build.cpp", d / "build.so"
    src.write_text(BUILD)
    subprocess.run(["g++", "-std=c++17", "-O1", "-D_GLIBCXX_ASSERTIONS", "-fsanitize=undefined", "-fno-sanitize-recover",
                    "-Wno-unknown-pragmas", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    return C.CDLL(str(so)).build


@pytest.mark.parametrize("sms", [2, 16, 152])
@pytest.mark.parametrize("mesh,shuffle", [(_grid(1, 1, 1), False), (_grid(2, 2, 1), False), (_grid(5, 5, 5), False),
                                          (_grid(6, 6, 5), True), (_grid(12, 12, 11), False), (_grid(17, 16, 15), True),
                                          (_grid(24, 24, 24), False), (_grid(26, 26, 26), False), (_star(100), False),
                                          ((9, _grid(1, 1, 1)[1]), False), ((45, _grid(1, 1, 1)[1] + 20), False)],
                         ids=["cell", "20", "625", "900shuffled", "7920", "20400shuffled", "69120", "87880", "star", "lone",
                              "apart"])
def test_tables_made_on_the_device(build, mesh, shuffle, sms):
    """The device's steps (rows_build.h) give the host's tables, whatever the
    mesh, entry for entry."""
    n, tets = mesh
    if shuffle:
        tets = np.random.default_rng(2).permutation(n).astype(np.uint32)[tets]
    tets = np.ascontiguousarray(tets, np.uint32)
    assert build(n, len(tets), tets.ctypes.data_as(C.POINTER(C.c_uint32)), sms) in ((0,) if sms == 152 else (0, -1))


def test_tables_of_a_degenerate_mesh(build):
    """Elements that name a node twice, and twice the same element."""
    tets = np.array([[0, 1, 2, 3], [1, 1, 2, 4], [3, 2, 1, 0], [4, 5, 5, 5], [0, 1, 2, 3]], np.uint32)
    assert build(7, len(tets), tets.ctypes.data_as(C.POINTER(C.c_uint32)), 152) == 0

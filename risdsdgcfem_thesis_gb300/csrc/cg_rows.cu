// cg_rows.cu -- the whole of ILSS_CG::Solve (ILSS_CG.h:38-151) or
// ILSS_MINRES::Solve (ILSS_MINRES.h:51-168) for a C_WRP solid in one launch,
// the assembled stiffness's rows resident in shared memory (rows_plan.h).
//
// Block g owns a range of nodes: their rows as fixed-point 3x3 blocks (fx.cuh),
// and their y, r, d, q and b, one component per thread, in registers. An
// iteration is bound by latency, so nothing of it goes through a kernel
// boundary or a grid barrier: what another block needs is stored in 64-bit
// words that carry the exchange's number beside the data, in the shared memory
// of a CTA of the cluster (about 700 clocks) or in L2 (1,000 to 2,300, a
// polled word), and the reader polls the word itself. Two exchanges make an
// iteration, the sums of d.q and of |r|^2; r of the nodes on a block's rim goes
// out beside the second, and every block keeps the d of its rim by the same
// recurrence as the owner (MINRES: v1.v, |v1|^2 and v1, which the norm makes
// v). Sums stay integers from the lanes to the total, and
// every block adds them all, so all take the same scalar steps and leave
// together. A word is overwritten only after an exchange that its reader has
// taken part in since it read it: the two sums by each other, r by the d.q
// before it; every solve writes both sums' words, so that no number comes round
// to a word that is still there. Every wait is bounded; a block that gives up
// says so in a word of its own (StepScalars::gave_up), and the others give up
// at their next exchange.
//
// Per iteration of CG: 3.2 us at 160 tets and 4.6 us at 3,000 on one cluster,
// 6.3 us at 20,480 on 15, 10.3 at 87,880 on 76 of two (MINRES 4.2, 7.0 at
// 7,215, 7.5 at 20,480); the product over the rows is a fifth of it, the rest are
// the sums (half on 15 clusters), the division, and the vector arithmetic (one
// FP64 instruction of a warp holds its sub-partition 64 clocks). The four launches
// per iteration it replaces took 22 us at 20,480 tets, and its predecessor on
// one cluster with element products 7 us at 160 and 14 us at 3,000.
#include "bounds.cuh"
#include "fem_device.cuh"
#include "fx_device.cuh"
#include "rows_words.h"

#include <algorithm>

namespace femgb {

namespace {

// A 128-bit word, each half with the exchange's number in its top bits.
__device__ __forceinline__ void word_put(ulonglong2* p, unsigned long long a, unsigned long long b)
{
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ ulonglong2 word_get(const ulonglong2* p)
{
    ulonglong2 w;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(w.x), "=l"(w.y) : "l"(p) : "memory");
    return w;
}
// The same in the shared memory of a CTA of the cluster.
__device__ __forceinline__ uint32_t near_address(const void* p, uint32_t rank)
{
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void near_put(uint32_t p, unsigned long long a, unsigned long long b)
{
    asm volatile("st.relaxed.cluster.shared::cluster.v2.b64 [%0], {%1, %2};" ::"r"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ ulonglong2 near_get(uint32_t p)
{
    ulonglong2 w;
    asm volatile("ld.relaxed.cluster.shared::cluster.v2.b64 {%0, %1}, [%2];" : "=l"(w.x), "=l"(w.y) : "r"(p) : "memory");
    return w;
}
// The warp's sum of m 2^e (|m| <= 2^62), in every lane: added in three limbs.
template <int K>
__device__ __forceinline__ Part part_sum(const Part (&v)[K])
{
    int32_t E = v[0].e;
#pragma unroll
    for (int k = 1; k < K; k++) E = max(E, v[k].e);
    E = __reduce_max_sync(0xffffffffu, E);
    uint32_t l0 = 0, l1 = 0;
    int32_t l2 = 0;
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int64_t m = v[k].m >> fx_min63(E - v[k].e);
        l0 += (uint32_t)m & 0xffffffu;
        l1 += (uint32_t)(m >> 24) & 0xffffffu;
        l2 += (int32_t)(m >> 48);
    }
    l0 = __reduce_add_sync(0xffffffffu, l0);
    l1 = __reduce_add_sync(0xffffffffu, l1) + (l0 >> 24);
    l2 = __reduce_add_sync(0xffffffffu, l2);
    const int64_t t = (int64_t)l1 + (int64_t)((uint64_t)(int64_t)l2 << 24);  // units of 2^24, the rest in l0
    const int32_t sh = max(0, 64 - fx_clz(fx_mag(t) | 1u) - 38);             // at most 9
    return Part{(int64_t)((uint64_t)t << (24 - sh)) | (int64_t)((l0 & 0xffffffu) >> sh), E >= kPartInf ? E : E + sh};
}
// Out of line: the compiler would otherwise divide on every path.
__device__ __noinline__ double divide(double a, double b) { return a / b; }

// Polls n words (get(i), one per lane and turn) and adds them, in every lane
// of the warp; bad when the wait gave up.
template <int K, typename F>
__device__ __forceinline__ Part words_sum(F&& get, uint32_t n, uint32_t seq, uint32_t limit, bool& bad)
{
    const uint32_t lane = threadIdx.x & 31u;
    Part part[K];
    bool ok;
    uint32_t polls = 0;
    do {
        ok = true;
#pragma unroll
        for (int i = 0; i < K; i++) {  // all in flight together
            const bool on = lane + 32 * i < n;
            const bool there = rows_word_is(get(on ? lane + 32 * i : 0u), part[i], seq);
            ok = ok && (there || !on);
            if (!on) part[i] = Part{0, 0};
        }
        ok = __all_sync(0xffffffffu, ok);
    } while (!ok && ++polls <= limit);
    bad = bad || !ok;
    return part_sum(part);
}

__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.aligned;\n barrier.cluster.wait.aligned;" ::: "memory");
}

// v = h 2^30 + l, |l| <= 2^29: an entry (below 2^60) times a component (below
// 2^59) drops l l, 2^-61 of full scale.
__device__ __forceinline__ FxL split30(int64_t v)
{
    FxL s;
    s.h = (int32_t)((v + (1ll << 29)) >> 30);
    s.l = (int32_t)((uint32_t)v - ((uint32_t)s.h << 30));
    asm("" : "+r"(s.l), "+r"(s.h));  // as in fx_split
    return s;
}

// A node's components as the product reads them: each in units of 2^(e - 1081).
struct __align__(16) RowRecord {
    long long v[3];
    uint16_t e[4];
};

}  // namespace

// ILSS_MINRES's Givens rotation from |v1|^2 (ILSS_MINRES.h:131-144) by a warp:
// its two roots and its four quotients each on four lanes.
__device__ __forceinline__ void givens_by_warp(MinresScalars& s, double total)
{
    const uint32_t q = threadIdx.x & 3u;
    const MinresScalars mr = s;
    const double be = mr.beta_new;
    const double r2 = mr.s * mr.alpha + mr.c * mr.c_old * be;
    const double r3 = mr.s_old * be;
    const double r1_hat = mr.c * mr.alpha - mr.c_old * mr.s * be;
    const double root = ::sqrt(q == 0 ? total : r1_hat * r1_hat + total);
    const double beta_new = __shfl_sync(0xffffffffu, root, 0), r1 = __shfl_sync(0xffffffffu, root, 1);
    const double part = (q == 1 ? r1_hat : (q == 2 ? beta_new : 1.0)) / (q == 0 ? beta_new : r1);
    const double inv_beta = __shfl_sync(0xffffffffu, part, 0), c = __shfl_sync(0xffffffffu, part, 1);
    const double sn = __shfl_sync(0xffffffffu, part, 2), ir1 = __shfl_sync(0xffffffffu, part, 3);
    if (threadIdx.x == 0) {
        s.beta = be;
        s.beta_new = beta_new;
        s.inv_beta = inv_beta;
        s.c_old = mr.c;
        s.s_old = mr.s;
        s.c = c;
        s.s = sn;
        s.neg_r2 = -r2;
        s.neg_r3 = -r3;
        s.inv_r1 = ir1;
        s.x_coef = mr.beta_one * c * mr.eta;
        s.norm_r_sq = mr.norm_r_sq * (sn * sn);
        s.eta = -sn * mr.eta;
    }
    __syncwarp();
}

template <int L, bool kMinres>  // L: lanes per row
__global__ void __launch_bounds__(kCgRowsMaxThreads, 1)
    k_cg_rows_fp64(MeshView<double> m, StepConsts c, CgRowsView p, const double* __restrict__ b, double* y,
                   StepScalars* st)
{
    extern __shared__ __align__(16) unsigned char rows_smem[];
    __shared__ double s_scalar;
    __shared__ MinresScalars s_mr;
    __shared__ int s_go, s_ok;  // the loop test; the first sum is there (0: breakdown)
    const uint32_t tid = threadIdx.x, nt = blockDim.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t G = gridDim.x, g = blockIdx.x, C = p.cluster, row0 = g / C * C, rank = g - row0, nrow = G / C;
    const CgRowsBlock B = p.blk[g];
    const uint32_t nn = B.nn, nh = B.nhalo, n3 = 3 * nn, h3 = 3 * nh;
    int2* A = reinterpret_cast<int2*>(rows_smem);                              // [units][9][32]
    RowRecord* rec = reinterpret_cast<RowRecord*>(A + 288 * (size_t)p.units);  // [nn + nh]
    ulonglong2* sums = reinterpret_cast<ulonglong2*>(rec + p.records);        // [2][C vwarps]: the same place in every CTA
    ulonglong2* myr = sums + 2 * (size_t)C * p.warps;                          // [3 npb]: r for the cluster
    double* ku = reinterpret_cast<double*>(myr + 3 * (size_t)p.npb);           // [3 nn]
    double* rimd = ku + n3;                                                    // [3 nh]: d on the rim
    double* rimr = rimd + h3;                                                  // [3 nh]: r on the rim
    int32_t* rowx = reinterpret_cast<int32_t*>(rimr + h3);                     // [nn]
    uint32_t* rim = reinterpret_cast<uint32_t*>(rowx + nn);                    // [nh]
    uint32_t* rimw = rim + nh;                                                 // [nh]: where r is
    uint32_t* group = rimw + nh;                                               // [ngroups + 1]
    uint16_t* col = reinterpret_cast<uint16_t*>(group + B.ngroups + 1);        // [units][32]
    const uint32_t seq0 = *p.seq;

    for (uint32_t i = tid; i < 32 * B.units; i += nt) {
        const size_t at = 32 * (size_t)B.unit0 + i;
        const uint32_t s = p.slot[at];
        const bool on = s != kCgRowsPad;
        const int2* v = m.bsr_val + 36 * (size_t)(on ? s >> 2 : 0u) + (on ? s & 3u : 0u);
        int2* o = A + 288 * (size_t)(i >> 5) + (i & 31u);
#pragma unroll
        for (int k = 0; k < 9; k++) {
            const int2 w = on ? v[4 * k] : make_int2(0, 0);
            const FxL e = split30((int64_t)((uint64_t)(int64_t)w.y << 32) + w.x);
            o[32 * k] = make_int2(e.l, e.h);
        }
        col[i] = p.col[at];
    }
    for (uint32_t i = tid; i < nn; i += nt)
        rowx[i] = m.bsr_x[bounds_idx(p.node[B.node0 + i] & kCgRowsNode, m.N, kSiteBsrEntry)];
    for (uint32_t i = tid; i < nh; i += nt) {
        rim[i] = bounds_idx(p.halo[B.halo0 + i], m.N, kSiteBsrEntry);
        const uint32_t w = p.owner[B.halo0 + i];  // CTA << 16 | its node
        rimw[i] = w == kCgRowsFar ? w : near_address(myr + 3 * (w & 0xffffu), w >> 16);
    }
    rows_words_start(sums, 2 * C * p.warps, 3 * p.npb, seq0, tid, nt);
    for (uint32_t i = tid; i <= B.ngroups; i += nt) group[i] = p.group[B.group0 + i];
    cluster_sync();  // every CTA's words hold an old number

    // this thread's component, in the first warps; the others have the rim's
    const uint32_t vwarps = p.warps, rim0 = 32 * vwarps;
    const bool vec = warp < vwarps, mine = tid < n3;
    size_t at = 0;
    bool far = false, near = false, live = false;
    double ny = 0.0, nr = 0.0, nd = 0.0, nq = 0.0;
    if (mine) {
        const uint32_t w = p.node[B.node0 + tid / 3], n = bounds_idx(w & kCgRowsNode, m.N, kSiteBsrEntry);
        at = 3 * (size_t)n + tid % 3;
        far = (w & kCgRowsFarShared) != 0;
        near = (w & kCgRowsNearShared) != 0;
        live = !m.fixed[n];
        ny = y[at];
    }
    const double mfm = c.mass * c.factor_M;

    auto put = [&](uint32_t i, double v) {
        const int32_t e = fx_exp(v);
        rec[i / 3].v[i % 3] = fx_align<59>(v, e);
        rec[i / 3].e[i % 3] = (uint16_t)e;
    };
    // K times the records, into ku
    auto product = [&] {
        __syncthreads();
        constexpr uint32_t kRows = 32 / L;  // per warp and turn
        for (uint32_t w = warp; w < B.ngroups; w += nt >> 5) {
            const uint32_t u0 = group[w], u1 = group[w + 1];
            const uint32_t row = kRows * w + lane / L, sub = lane % L;
            int32_t E = 0;
            for (uint32_t u = u0; u < u1; u++) {
                const uint2 e = *reinterpret_cast<const uint2*>(rec[col[32 * u + lane]].e);
                E = max(E, (int32_t)max(max(e.x & 0xffffu, e.x >> 16), e.y & 0xffffu));
            }
#pragma unroll
            for (int o = 1; o < L; o <<= 1) E = max(E, __shfl_xor_sync(0xffffffffu, E, o));
            int64_t hi[3] = {0, 0, 0}, mid[3] = {0, 0, 0};
            auto block = [&](uint32_t u) {
                const longlong2* r2 = reinterpret_cast<const longlong2*>(rec + col[32 * u + lane]);
                const longlong2 v01 = r2[0], v2e = r2[1];
                const FxL x[3] = {split30(v01.x >> fx_min63(E - (int32_t)(v2e.y & 0xffff))),
                                  split30(v01.y >> fx_min63(E - (int32_t)((v2e.y >> 16) & 0xffff))),
                                  split30(v2e.x >> fx_min63(E - (int32_t)((v2e.y >> 32) & 0xffff)))};
                const int2* a = A + 288 * (size_t)u + lane;
#pragma unroll
                for (int r = 0; r < 3; r++)
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        const int2 e = a[32 * (3 * r + k)];
                        fx_mac(hi[r], mid[r], FxL{e.x, e.y}, x[k]);
                    }
            };
            // a block's mid stays below 2^61.2: two between carries
            for (uint32_t u = u0;;) {
                block(u);
                if (++u >= u1) break;
                block(u);
                if (++u >= u1) break;
#pragma unroll
                for (int r = 0; r < 3; r++) {
                    hi[r] += mid[r] >> 30;
                    mid[r] &= (1ll << 30) - 1;
                }
            }
            // the row's lanes add: the first two steps leave a lane one component
            long long v[4] = {0, 0, 0, 0};
#pragma unroll
            for (int r = 0; r < 3; r++) v[r] = hi[r] + ((mid[r] + (1ll << 29)) >> 30);
            const bool b0 = (sub & 1u) != 0, b1 = (sub & 2u) != 0;
            const long long s0 = (b0 ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, b0 ? v[0] : v[2], 1);
            const long long s1 = (b0 ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, b0 ? v[1] : v[3], 1);
            long long t = (b1 ? s1 : s0) + __shfl_xor_sync(0xffffffffu, b1 ? s0 : s1, 2);
#pragma unroll
            for (int o = 4; o < L; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            const uint32_t r = (b0 ? 2u : 0u) + (b1 ? 1u : 0u);
            if (row < nn && sub < 3) {  // r: 0, 2, 1
                const int32_t x = rowx[row];
                ku[3 * row + r] = E == 2047 || x == kFxFp64 ? fx_from_bits(0x7ff8000000000000ull)
                                                              : fx_to_double(t, x + (E - 1081) + 60);
            }
        }
        __syncthreads();
    };
    // The solid's total of every component's acc, in warp 0; bad when a wait
    // gave up. The warps' sums go to every CTA of the cluster, the clusters'
    // totals from each of its CTAs to one CTA of every cluster. meanwhile: what
    // warp 0 does while they come.
    auto total = [&](double acc, int which, uint32_t seq, bool& bad, auto&& meanwhile) -> double {
        ulonglong2* own = sums + (size_t)which * C * vwarps;
        if (vec) {
            const Part v[1] = {part_of(acc)};
            const ulonglong2 w = rows_word<ulonglong2>(part_sum(v), seq);
            if (lane < C) near_put(near_address(own + rank * vwarps + warp, lane), w.x, w.y);
        }
        if (warp != 0) return 0.0;
        meanwhile();
        const uint32_t n = C * vwarps, at = near_address(own, rank);
        auto get = [&](uint32_t i) { return near_get(at + (uint32_t)sizeof(ulonglong2) * i); };
        Part s = n <= 32 ? words_sum<1>(get, n, seq, p.polls, bad) : (n <= 96 ? words_sum<3>(get, n, seq, p.polls, bad) : words_sum<5>(get, n, seq, p.polls, bad));
        if (nrow > 1) {
            ulonglong2* words = p.parts + (size_t)which * G * nrow;
            const ulonglong2 w = rows_word<ulonglong2>(s, seq);
            for (uint32_t i = lane; i < nrow; i += 32) word_put(words + (size_t)(i * C + rank) * nrow + g / C, w.x, w.y);
            words += (size_t)g * nrow;
            auto there = [&](uint32_t i) { return word_get(words + i); };
            s = nrow <= 32 ? words_sum<1>(there, nrow, seq, p.polls, bad) : words_sum<3>(there, nrow, seq, p.polls, bad);
        }
        return part_value(s);
    };
    // r for the neighbours, and theirs
    auto send = [&](uint32_t seq) {
        const ulonglong2 w = rows_word<ulonglong2>(nr, seq);
        if (near) near_put(near_address(myr + tid, rank), w.x, w.y);
        if (far) word_put(p.words + at, w.x, w.y);
    };
    auto receive = [&](uint32_t seq) {  // true when a wait gave up
        int bad = 0;
        if (tid >= rim0)
            for (uint32_t i = tid - rim0; i < h3; i += nt - rim0) {
                const uint32_t k = i / 3, a = i % 3, w = rimw[k];
                const ulonglong2* f = p.words + 3 * (size_t)rim[k] + a;
                uint32_t polls = 0;
                while (!rows_word_is(w == kCgRowsFar ? word_get(f) : near_get(w + (uint32_t)sizeof(ulonglong2) * a), rimr[i], seq))
                    if (++polls > p.polls) {
                        bad = 1;
                        break;
                    }
            }
        return bad;
    };

    // the scalars, in warp 0
    double delta_0 = 0.0, delta = 0.0, delta_old = 0.0, target = 0.0, alpha = 0.0, beta = 0.0, dq = 0.0, rdelta = 0.0;
    const double abs_sq = c.abs_eps_sq;
    uint32_t k = 0, seq = seq0 + 1;
    bool bad = false;
    // comparisons on the bits: an FP64 one holds the pipe as long as a product
    const uint64_t kInf = 0x7ff0000000000000ull, abs_bits = abs_sq == abs_sq ? fx_bits(abs_sq) : 0;
    uint64_t target_bits = 0;
    auto proceeds = [&] {
        const uint64_t v = fx_bits(delta);
        return v > target_bits && v <= kInf && k < c.max_iter;
    };
    auto nothing = [] {};

    if (!kMinres && warp == 0 && nrow > 1)
        // a solve without iterations sends no d.q: the words are renewed, so
        // that none is older than a solve (their numbers wrap at 2^16)
        for (uint32_t i = lane; i < nrow; i += 32) {
            const ulonglong2 w = rows_word<ulonglong2>(Part{0, 0}, seq);
            word_put(p.parts + (size_t)(i * C + rank) * nrow + g / C, w.x, w.y);
        }
    double norm_b = 0.0;
    if constexpr (kMinres) {  // |b|^2, constrained rows too
        const double bi = mine ? b[at] : 0.0;
        norm_b = total(vec ? bi * bi : 0.0, 0, seq, bad, nothing);
    }
    // r = S (b - A y), d = r, |r|^2   (ILSS_CG.h:53-64; ILSS_MINRES.h:66-95: v1 = r)
    if (mine) put(tid, ny);
    if (tid >= rim0)
        for (uint32_t i = tid - rim0; i < h3; i += nt - rim0) {
            put(n3 + i, y[3 * (size_t)rim[i / 3] + i % 3]);
            rimd[i] = 0.0;
        }
    product();
    if (live) nr = b[at] - (c.factor_K * ku[tid] + mfm * ny);
    send(seq);
    {
        const double t = total(vec ? nr * nr : 0.0, 1, seq, bad, nothing);
        if (warp == 0) {
            delta_0 = delta = delta_old = t;
            if constexpr (kMinres) delta_0 = norm_b;
            target = c.rel_eps_sq * delta_0;
            target_bits = target == target && abs_sq == abs_sq ? max(fx_bits(target), abs_bits) : ~(uint64_t)0;
            if (lane == 0) {
                s_scalar = 0.0;
                s_go = bad ? -1 : proceeds();
                if constexpr (kMinres) {
                    s_mr = MinresScalars{};
                    minres_start(s_mr, t);
                    s_mr.norm_b_sq = norm_b;
                }
            }
        }
    }
    int stop = __syncthreads_or(receive(seq));
    int go = stop ? -1 : s_go;
    bool finite = true;  // of the totals, in warp 0
    if constexpr (kMinres) {
        double np = 0.0, np0 = 0.0;
        while (go > 0) {
            // v0 <- v, v <- v1 / beta, v1 = S A v - beta v0, v1.v   (ILSS_MINRES.h:117-123)
            const double inv = s_mr.inv_beta, nb = -s_mr.beta_new;
            double v0 = 0.0, t = 0.0;
            if (vec) {
                v0 = nd;
                nd = nr * inv;
            }
            if (mine) put(tid, nd);
            if (tid >= rim0)
                for (uint32_t i = tid - rim0; i < h3; i += nt - rim0) put(n3 + i, rimr[i] * inv);
            product();
            if (vec) {
                nq = live ? c.factor_K * ku[tid] + mfm * nd : 0.0;
                nr = __fma_rn(nb, v0, nq);
                t = nr * nd;
            }
            seq++;
            t = total(t, 0, seq, bad, nothing);
            if (tid == 0) {
                s_scalar = s_mr.alpha = t;
                s_ok = bad ? -1 : 1;
            }
            __syncthreads();
            if (s_ok < 0) {
                go = -1;
                break;
            }
            // v1 -= alpha v, |v1|^2, the rotation and the loop test, p and y   (:123-156)
            if (vec) {
                nr = __fma_rn(-s_scalar, nd, nr);
                send(seq);
                t = nr * nr;
            }
            t = total(t, 1, seq, bad, nothing);
            if (warp == 0) {
                givens_by_warp(s_mr, t);
                delta_old = delta;
                delta = s_mr.norm_r_sq;
                finite = isfinite(t) && isfinite(delta);
                k++;
                if (lane == 0) s_go = bad ? -1 : proceeds();
            }
            stop = __syncthreads_or(receive(seq));
            go = stop ? -1 : s_go;
            if (vec) {
                double pn = s_mr.neg_r2 * np + nd;
                pn += s_mr.neg_r3 * np0;
                pn *= s_mr.inv_r1;
                np0 = np;
                np = pn;
                ny += s_mr.x_coef * pn;
            }
            __syncthreads();  // before warp 0 writes the scalars again
        }
    }
    while (!kMinres && go > 0) {
        // d = S (beta d + r), q = S A d, d.q   (ILSS_CG.h:90-96,137)
        const double be = s_scalar;
        if (vec) nd = __fma_rn(be, nd, nr);
        if (mine) put(tid, nd);
        if (tid >= rim0)
            for (uint32_t i = tid - rim0; i < h3; i += nt - rim0) {
                const double v = __fma_rn(be, rimd[i], rimr[i]);
                rimd[i] = v;
                put(n3 + i, v);
            }
        product();
        double t = 0.0;
        if (vec) {
            if (live) nq = c.factor_K * ku[tid] + mfm * nd;
            t = nd * nq;
        }
        seq++;
        t = total(t, 0, seq, bad, [&] {
            rdelta = 1.0 / delta;
            asm volatile("" : "+d"(rdelta));  // here, not where it is used
        });
        if (warp == 0) {
            dq = t;
            const bool brk = (fx_bits(t) & ~(1ull << 63)) < abs_bits;  // breakdown: leave before the update (ILSS_CG.h:97)
            if (!brk) alpha = delta / t;
            if (lane == 0) {
                s_scalar = alpha;
                s_ok = bad ? -1 : !brk;
            }
        }
        __syncthreads();
        go = s_ok;
        if (go <= 0) break;
        // y += alpha d, r -= alpha q, |r|^2, beta and the loop test   (ILSS_CG.h:96-137)
        if (vec) {
            const double al = s_scalar;
            nr = __fma_rn(-al, nq, nr);
            send(seq);
            ny = __fma_rn(al, nd, ny);
            t = nr * nr;
        }
        t = total(t, 1, seq, bad, nothing);
        if (warp == 0) {
            delta_old = delta;
            delta = t;
            if (!rows_quotient(t, delta_old, rdelta, beta)) beta = divide(t, delta_old);
            k++;
            if (lane == 0) {
                s_scalar = beta;
                s_go = bad ? -1 : proceeds();
            }
        }
        stop = __syncthreads_or(receive(seq));
        go = stop ? -1 : s_go;
    }
    cluster_sync();  // no CTA leaves while another may still use its shared memory
    if (mine) y[at] = ny;
    if (go < 0 && tid == 0) st->gave_up = 1;  // any block's wait: another one may have seen the loop end
    if (g == 0 && tid == 0) {
        st->delta_0 = delta_0;
        st->delta_new = delta;
        st->delta_old = delta_old;
        st->delta_target = target;
        st->abs_eps_sq = abs_sq;
        st->max_iter = c.max_iter;
        st->k = k;
        st->total_iters += k;
        st->dot_dq = dq;
        st->alpha = alpha;
        st->beta = beta;
        st->status = go < 0 ? 6u : (isfinite(delta) && finite ? 0u : 3u);  // FEM_E_TIMEOUT, FEM_E_NAN
        if constexpr (kMinres) st->mr = st->mr_pend = s_mr;
        st->done = 1;
        st->delta_pend = delta;
        st->done_pend = 1;
        st->rel_residual = kMinres || delta_0 > 0 ? ::sqrt(delta / delta_0) : 0.0;
        st->abs_residual = ::sqrt(delta);
        *p.seq = go < 0 ? seq + 4 : seq;  // past the numbers of blocks that were ahead
    }
}

namespace {
using CgRowsKernel = void (*)(MeshView<double>, StepConsts, CgRowsView, const double*, double*, StepScalars*);
CgRowsKernel cg_rows_kernel(uint32_t lanes, bool minres)
{
    if (minres) return lanes == 4 ? k_cg_rows_fp64<4, true> : (lanes == 8 ? k_cg_rows_fp64<8, true> : k_cg_rows_fp64<16, true>);
    return lanes == 4 ? k_cg_rows_fp64<4, false> : (lanes == 8 ? k_cg_rows_fp64<8, false> : k_cg_rows_fp64<16, false>);
}
}  // namespace

namespace {
void rows_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, const CgRowsPlan& p, cudaStream_t s)
{
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3(p.blocks);
    cfg.blockDim = dim3(p.threads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = s;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = p.cluster;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeCooperative;  // several clusters wait on one another
    at[1].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = p.blocks > p.cluster ? 2 : 1;
}
}  // namespace

uint32_t cg_rows_max_blocks(const CgRowsPlan& p)
{
    if (p.smem > kCgRowsMaxSmem || p.threads > kCgRowsMaxThreads || p.cluster < 1 || p.cluster > 16) return 0;
    int least = 0x7fffffff;
    for (bool minres : {false, true}) {
        auto* k = cg_rows_kernel(p.lanes, minres);
        int n = 0;
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[2];
        rows_config(cfg, at, p, nullptr);
        cfg.gridDim = dim3(p.cluster);
        cfg.numAttrs = 1;
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCgRowsMaxSmem) != cudaSuccess ||
            cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        least = std::min(least, n);
    }
    return std::min((uint32_t)least * p.cluster, kCgRowsMaxBlocks);
}

cudaError_t launch_cg_rows_fp64(const MeshView<double>& m, const StepConsts& c, const CgRowsPlan& plan,
                                const CgRowsView& p, bool minres, const double* b, double* y, StepScalars* st,
                                cudaStream_t s)
{
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[2];
    rows_config(cfg, at, plan, s);
    prof_begin("cg_rows_fp64", s);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, cg_rows_kernel(plan.lanes, minres), m, c, p, b, y, st);
    prof_end("cg_rows_fp64", s);
    launch_counter()++;
    return e;
}

FEMGB_BOUNDS_ACCESSOR(bounds_read_cg_rows)

}  // namespace femgb

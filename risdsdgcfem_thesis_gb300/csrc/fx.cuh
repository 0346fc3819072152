// fx.cuh -- the FP64 path's element products in fixed point, on the integer
// pipe.
//
// GB300 issues one FP64 instruction per 64 clocks on each of an SM's four
// sub-partitions (measured: DFMA 64.1 clocks, DADD 64 to 76, for dependent
// and independent ones alike), and one 32 x 32 + 64 bit integer multiply-add
// (IMAD.WIDE) per 4.3. A product of two 60-bit integers held as two signed
// 32-bit limbs takes three of those (the low x low term is below the last
// bit kept). The element product is therefore one symmetric 9 x 9 matrix per
// element, K9 = the blocks (i, j), i, j = 1..3, of R K0 R^T, baked after each
// evaluation, times the three node differences d_j - d_0 (node 0's output is
// minus the sum of the others'): 81 products, about 1,050 clocks of
// multiplies (1,200 with the rest of the product, 800 for the differences)
// against 8,800 for the 138 FP64 operations of the strain form.
//
// Numbers are block fixed point: the nine differences share one exponent,
// normalised to the largest, K9 one exponent, the twelve outputs one
// exponent. Bounds are stated beside each stage. K9's entries are good to
// about 2^-56 of the largest, the differences to 2^-59 and the sums to 2^-56,
// where FP64 rounds every operation at 2^-53. Elements for which that does
// not hold -- a non-finite or out-of-range operand, a rotation entry above
// 1.125, a rest shape so graded that one exponent for Dm^-1 would cost more
// than the spare bits -- take the FP64 product (elem_math.cuh).
//
// All functions are host callable: the arithmetic is checked on the CPU.
#pragma once
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define FX_HD __host__ __device__ __forceinline__
#else
#define FX_HD inline
#endif

namespace femgb {

// v = h 2^32 + l, l signed.
struct FxL {
    int32_t l, h;
};

FX_HD FxL fx_split(int64_t v)
{
    FxL s;
    s.l = (int32_t)v;
    s.h = (int32_t)(v >> 32) + (int32_t)((uint32_t)s.l >> 31);
#ifdef __CUDA_ARCH__
    // two plain 32-bit values from here on: otherwise the compiler carries the
    // limb as a 64-bit one and multiplies 64 x 64 (four instructions)
    asm("" : "+r"(s.l), "+r"(s.h));
#endif
    return s;
}

// hi += a.h b.h, mid += a.h b.l + a.l b.h: the product in units of 2^64 and 2^32.
FX_HD void fx_mac(int64_t& hi, int64_t& mid, const FxL& a, const FxL& b)
{
    hi += (int64_t)a.h * b.h;
    mid += (int64_t)a.h * b.l;
    mid += (int64_t)a.l * b.h;
}

// The accumulated product in units of 2^(64 - K).
template <int K>
FX_HD int64_t fx_fin(int64_t hi, int64_t mid)
{
    return (int64_t)((uint64_t)hi << K) + (mid >> (32 - K));
}

FX_HD uint64_t fx_bits(double v)
{
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(v);
#else
    uint64_t u;
    memcpy(&u, &v, 8);
    return u;
#endif
}

FX_HD double fx_from_bits(uint64_t u)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double v;
    memcpy(&v, &u, 8);
    return v;
#endif
}

// Biased exponent of a double (0: zero or denormal, 2047: Inf or NaN).
FX_HD int32_t fx_exp(double v) { return (int32_t)(fx_bits(v) >> 52) & 0x7ff; }

// v as an integer in units of 2^(E - 1022 - B), for E >= fx_exp(v), E <=
// 2046: magnitude below 2^B, truncated. Denormals count as zero.
template <int B>
FX_HD int64_t fx_align(double v, int32_t E)
{
    const uint64_t u = fx_bits(v);
    const int32_t e = (int32_t)(u >> 52) & 0x7ff;
    const uint64_t m = ((u & 0xfffffffffffffull) | 0x10000000000000ull) << (B - 53);
    const int32_t sh = e == 0 || E - e > 63 ? 63 : E - e;
    const int64_t s = (int64_t)u >> 63;
    return ((int64_t)(m >> sh) ^ s) - s;
}

// The scale of an element whose product runs in FP64 instead.
constexpr int32_t kFxFp64 = 0x40000000;

// A common exponent x of n values: every |v| < 2^x. False when all are zero
// or one is not finite.
FX_HD bool fx_common(const double* v, int n, int32_t& x)
{
    int32_t e = 0;
    for (int i = 0; i < n; i++) {
        const int32_t ei = fx_exp(v[i]);
        e = ei > e ? ei : e;
    }
    x = e - 1022;
    return e > 0 && e < 2047;
}

FX_HD uint64_t fx_mag(int64_t v) { return (uint64_t)(v ^ (v >> 63)); }  // |v| or |v| - 1

FX_HD int fx_clz(uint64_t v)  // leading zeros, v > 0
{
#ifdef __CUDA_ARCH__
    return __clzll((long long)v);
#else
    return __builtin_clzll(v);
#endif
}

// m 2^x as a double, rounded to nearest (ties away); results below the
// normal range become zero, above it infinity.
FX_HD double fx_to_double(int64_t m, int32_t x)
{
    if (m == 0) return 0.0;
    const uint64_t sign = (uint64_t)m & 0x8000000000000000ull;
    uint64_t a = m < 0 ? 0ull - (uint64_t)m : (uint64_t)m;
    const int lz = fx_clz(a);
    a <<= lz;
    const int32_t e = x + 63 - lz + 1023;  // biased exponent of the leading bit
    if (e <= 0) return fx_from_bits(sign);
    if (e >= 2047) return fx_from_bits(sign | 0x7ff0000000000000ull);
    // the rounding carry moves on into the exponent
    return fx_from_bits(sign | (((uint64_t)(e - 1) << 52) + ((a >> 11) + ((a >> 10) & 1ull))));
}

// A nodal output record: three integers of one element corner, their low four
// bits holding the units' exponent: x + 2048 in 12 bits, low nibble first.
// kFxNan marks a non-finite corner.
constexpr int32_t kFxNan = 4095;
FX_HD int32_t fx_record_exp(int64_t a, int64_t b, int64_t c)
{
    return (int32_t)(a & 15) | ((int32_t)(b & 15) << 4) | ((int32_t)(c & 15) << 8);
}

// Stamps the exponent x of 12 outputs' units into their low bits; false when
// x has no place in a record above (the element takes FP64); far below, the
// outputs become zero.
FX_HD bool fx_stamp(int64_t* out, int32_t x)
{
    const int32_t b = x + 2048;
    if (b >= kFxNan) return false;
    const int32_t c = b < 0 ? 0 : b;
#pragma unroll
    for (int k = 0; k < 12; k++)
        out[k] = b < 0 ? 0 : ((out[k] & ~15ll) | ((c >> (4 * (k % 3))) & 15));
    return true;
}

// 12 FP64 outputs as integers; returns their units' exponent + 2048 (kFxNan
// with zeros when one is not finite).
FX_HD int32_t fx_from_doubles(const double* v, int64_t* out)
{
    int32_t E = 0;
#pragma unroll
    for (int k = 0; k < 12; k++) {
        const int32_t e = fx_exp(v[k]);
        E = e > E ? e : E;
    }
#pragma unroll
    for (int k = 0; k < 12; k++) out[k] = E == 2047 ? 0 : fx_align<61>(v[k], E);
    return E == 2047 ? kFxNan : E - 1022 - 61 + 2048;
}

// The record of 12 FP64 outputs.
FX_HD void fx_stamp_doubles(const double* v, int64_t* out)
{
    const int32_t b = fx_from_doubles(v, out);
#pragma unroll
    for (int k = 0; k < 12; k++) out[k] = (out[k] & ~15ll) | ((b >> (4 * (k % 3))) & 15);
}

// The running sum of a node's records: acc in units of 2^(E - 2048 + guard),
// the guard bits sized so that a node's records cannot overflow.
struct FxSum {
    int64_t acc[3];
    int32_t E;
};
FX_HD int32_t fx_min63(int32_t s) { return s > 63 ? 63 : s; }
FX_HD void fx_add(FxSum& s, int64_t v0, int64_t v1, int64_t v2, int32_t e, int32_t guard)
{
    const int32_t up = fx_min63(e > s.E ? e - s.E : 0), down = fx_min63((e < s.E ? s.E - e : 0) + guard);
    s.acc[0] = (s.acc[0] >> up) + (v0 >> down);
    s.acc[1] = (s.acc[1] >> up) + (v1 >> down);
    s.acc[2] = (s.acc[2] >> up) + (v2 >> down);
    s.E = e > s.E ? e : s.E;
}
FX_HD void fx_add(FxSum& s, int64_t v0, int64_t v1, int64_t v2, int32_t guard)
{
    fx_add(s, v0, v1, v2, fx_record_exp(v0, v1, v2), guard);
}
FX_HD double fx_sum_value(int64_t acc, int32_t E, int32_t guard)
{
    return E == kFxNan ? fx_from_bits(0x7ff8000000000000ull) : fx_to_double(acc, E - 2048 + guard);
}

// K9's packed upper triangle: entry (r, c), r <= c, of the 9 x 9 matrix whose
// index 3 (i - 1) + a is component a of node i.
constexpr int kFxK = 45;
FX_HD constexpr int fx_at(int r, int c)  // r <= c
{
    return 9 * r - r * (r - 1) / 2 + (c - r);
}

// An element's grade max|Dm| max|Dm^-1| (1 for a cube corner): one exponent
// for all of Dm^-1 costs bits of K9 with it, and stiff materials cost bits of
// the shear terms. Measured against 128-bit products (jittered and stretched
// blocks, random rotations; geometric mean over the elements of the ratio to
// the FP64 strain form's error), random fields: 0.6 to 0.8 up to grade 3;
// smooth ones: 0.7 to 0.8 below grade 1.5, 0.9 to 1.0 up to 2, then 1.1 to 1.2
// up to 2.5 and 1.2 to 1.5 up to 3. At nu 0.49 to 0.4999999, grade 1.2: 0.6.
// Blocks of cubic cells jittered by a tenth hold one element in ten thousand
// above grade 2; its FP64 product would be the longest warp of every launch
// (20,480 tets, a step: 515 us with the line at 3, 539 with it at 2). All
// elements in FP64 cost what the strain form did (320,000 tets, 20 iterations:
// 3.2 ms, none 1.8, strain form 3.3).
constexpr float kFxMaxGrade = 3.0f, kFxMaxGradeStiff = 2.0f, kFxMaxGradeRigid = 1.2f;
constexpr double kFxStiff = 2.0, kFxRigid = 9.5;  // lambda / mu

// Whether an element of this rest shape and material may take fx_bake:
// grade = max|Dm| max|Dm^-1|. mu > 0 and 3 lambda + 2 mu >= 0 (a Poisson ratio
// in (-1, 0.5) with E > 0) make K9 positive semidefinite, which its scaling
// by the diagonal needs: with a Poisson ratio of 0.55 its other entries are
// up to several times the diagonal.
FX_HD bool fx_grade_ok(float grade, double kl, double km)
{
    return (int64_t)fx_bits(km) > 0 && ((int64_t)fx_bits(kl) >= 0 || 3.0 * kl + 2.0 * km >= 0.0) &&
           grade <= (kl <= kFxStiff * km ? kFxMaxGrade : (kl <= kFxRigid * km ? kFxMaxGradeStiff : kFxMaxGradeRigid));
}

// Bakes K9 = V (lambda m_i m_j^T + mu m_j m_i^T + mu (g_i . g_j) R R^T) with g_i
// the rows of Dm^-1 and m_i = R g_i (the strain form's product for any R,
// orthonormal or not). kl = V lambda, km = V mu; the caller has checked
// fx_grade_ok. K9 in units of 2^scale (returned), |K9| < 2^60 and its largest
// entry at least 2^59; kFxFp64 when the element takes FP64 (a row of R longer
// than 1.015, a non-finite or extreme operand); put(k, entry) takes the packed
// triangle in order. No FP64 operation.
template <typename FP>
FX_HD int32_t fx_bake(const double* R, const double* Di, double kl, double km, FP&& put)
{
    const double mat[2] = {kl, km};
    int32_t xd = 0, xm = 0;
    bool ok = fx_common(Di, 9, xd) && fx_common(mat, 2, xm) && xd > -400 && xd < 400 && xm > -400 && xm < 400;
#pragma unroll
    for (int i = 0; i < 9; i++)  // |R| < 1.0157 by its high word; false for NaN
        ok = ok && ((uint32_t)(fx_bits(R[i]) >> 32) & 0x7fffffffu) < 0x3ff04000u;
    if (!ok) return kFxFp64;
    FxL r[9], g[9];
#pragma unroll
    for (int i = 0; i < 9; i++) {
        r[i] = fx_split(fx_align<62>(R[i], 1023));        // R 2^61, below 2^61.03
        g[i] = fx_split(fx_align<61>(Di[i], xd + 1022));  // g 2^(61 - xd), below 2^61
    }
    FxL m[9], C[6], W[6];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int a = 0; a < 3; a++) {
            int64_t hi = 0, mid = 0;
#pragma unroll
            for (int b = 0; b < 3; b++) fx_mac(hi, mid, r[3 * a + b], g[3 * i + b]);
            m[3 * i + a] = fx_split(fx_fin<2>(hi, mid));  // m 2^(60 - xd), below 2^60.82
        }
    const int pa[6] = {0, 0, 0, 1, 1, 2}, pb[6] = {0, 1, 2, 1, 2, 2};  // (0,0) (0,1) (0,2) (1,1) (1,2) (2,2)
    const FxL lam = fx_split(fx_align<61>(kl, xm + 1022)), mu = fx_split(fx_align<61>(km, xm + 1022));  // 2^(61 - xm)
#pragma unroll
    for (int k = 0; k < 6; k++) {
        int64_t hi = 0, mid = 0;
#pragma unroll
        for (int b = 0; b < 3; b++) fx_mac(hi, mid, r[3 * pa[k] + b], r[3 * pb[k] + b]);
        const int64_t ck = fx_fin<2>(hi, mid);  // C 2^60, below 2^61.7
        if (pa[k] == pb[k]) ok = ok && ck < (int64_t)(1.03 * 1152921504606846976.0);
        C[k] = fx_split(ck);
        hi = mid = 0;
#pragma unroll
        for (int b = 0; b < 3; b++) fx_mac(hi, mid, g[3 * pa[k] + b], g[3 * pb[k] + b]);
        const FxL G = fx_split(fx_fin<2>(hi, mid));  // G 2^(60 - 2 xd), below 2^61.6
        hi = mid = 0;
        fx_mac(hi, mid, mu, G);
        W[k] = fx_split(fx_fin<2>(hi, mid));  // mu G 2^(59 - xm - 2 xd), below 2^60.6
    }
    FxL L[9], U[9];
#pragma unroll
    for (int k = 0; k < 9; k++) {
        int64_t hi = 0, mid = 0;
        fx_mac(hi, mid, lam, m[k]);
        L[k] = fx_split(fx_fin<2>(hi, mid));  // lambda m 2^(59 - xm - xd), below 2^59.82
        hi = mid = 0;
        fx_mac(hi, mid, mu, m[k]);
        U[k] = fx_split(fx_fin<2>(hi, mid));
    }
    // (mid stays below (2 (2^27.82 + 2^28.82) + 2^28.6 + 2^28.05) 2^31 < 2^63).
    // K9 is positive semidefinite (fx_grade_ok), so its largest entry is on the
    // diagonal: that gives the shift that moves it to [2^59, 2^60). Another
    // entry as large as its row's and column's diagonal belongs to a rotation
    // that moves nodes i and j along m_j and m_i; both diagonals are then V mu
    // |m|^2, at most 3/4 of V (lambda + 2 mu) |m|^2 elsewhere, so truncation
    // cannot lift it above the largest.
    const int sym[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
    auto entry = [&](int r, int c) {
        const int i = r / 3, a = r % 3, j = c / 3, b = c % 3;
        int64_t hi = 0, mid = 0;
        fx_mac(hi, mid, L[3 * i + a], m[3 * j + b]);
        fx_mac(hi, mid, U[3 * j + a], m[3 * i + b]);
        fx_mac(hi, mid, W[sym[3 * i + j]], C[sym[3 * a + b]]);
        return fx_fin<4>(hi, mid);  // K9 2^(59 - xm - 2 xd), below 9.4 2^59
    };
    uint64_t any = 0;
#pragma unroll
    for (int r = 0; r < 9; r++) any |= fx_mag(entry(r, r));
    if (any == 0 || !ok) return kFxFp64;
    const int lz = fx_clz(any);  // 1 at least
#pragma unroll
    for (int r = 0; r < 9; r++)
#pragma unroll
        for (int c = r; c < 9; c++) put(fx_at(r, c), (int64_t)((uint64_t)entry(r, c) << (lz - 1)) >> 3);
    return xm + 2 * xd - 59 - (lz - 1) + 3;
}

// The leading zeros of the largest magnitude of several values, from the
// words fx_top accumulates (31 when all their high words are zero: the values
// are then below 2^32 and moving them up by less is exact).
FX_HD uint32_t fx_top(int64_t v)
{
    const int32_t h = (int32_t)(v >> 32);
    return (uint32_t)(h ^ (h >> 31));
}
FX_HD int fx_clz_top(uint32_t any)
{
#ifdef __CUDA_ARCH__
    return __clz((int)(any | 1u));
#else
    return __builtin_clz(any | 1u);
#endif
}

// The node differences d_j - d_0 (D[3 (j - 1) + a]) in limbs, |D| < 2^59, from
// the four nodes' vectors; returns the exponent x of their units (2^x). False
// when one is not finite (the element takes FP64); all-zero differences give
// zeros. The nine subtractions are FP64's own (the pipe is idle otherwise).
FX_HD bool fx_differences(const double* d, FxL* D, int32_t& x)
{
    double v[9];
    int32_t E = 0;
#pragma unroll
    for (int j = 0; j < 3; j++)
#pragma unroll
        for (int a = 0; a < 3; a++) {
            v[3 * j + a] = d[3 * (j + 1) + a] - d[a];
            const int32_t e = fx_exp(v[3 * j + a]);
            E = e > E ? e : E;
        }
#pragma unroll
    for (int k = 0; k < 9; k++) D[k] = fx_split(fx_align<59>(v[k], E));
    x = E - 1022 - 59;
    return E < 2047;
}

// K9 D: out[3 i + a] for the nodes i = 0..3, normalised (|out| < 2^61, node 0's
// below 3 2^61) in units of 2^(scale + x + the returned shift). K(k) gives
// entry k of the packed triangle, in order. The mid sums stay below
// 9 (2^28 + 2^27) 2^31 < 2^63, the outputs before their normalisation below
// 2^60.2.
template <typename FK>
FX_HD int32_t fx_product(FK&& K, const FxL* D, int64_t* out)
{
    int64_t hi[9], mid[9];
#pragma unroll
    for (int r = 0; r < 9; r++) hi[r] = mid[r] = 0;
#pragma unroll
    for (int r = 0; r < 9; r++)
#pragma unroll
        for (int c = r; c < 9; c++) {  // entry (r, c) goes to rows r and c as it arrives
            const FxL k = K(fx_at(r, c));
            fx_mac(hi[r], mid[r], k, D[c]);
            if (c > r) fx_mac(hi[c], mid[c], k, D[r]);
        }
    uint32_t any = 0;
#pragma unroll
    for (int r = 0; r < 9; r++) {
        out[3 + r] = fx_fin<2>(hi[r], mid[r]);
        any |= fx_top(out[3 + r]);
    }
    const int up = fx_clz_top(any) - 3;
    int64_t sum[3] = {0, 0, 0};
#pragma unroll
    for (int r = 0; r < 9; r++) {
        out[3 + r] = (int64_t)((uint64_t)out[3 + r] << up);
        sum[r % 3] += out[3 + r];
    }
#pragma unroll
    for (int a = 0; a < 3; a++) out[a] = -sum[a];
    return 62 - up;
}

// The 4 x 4 corner blocks of an element's stiffness from K9, as kFxBlockWords
// integers: blocks (p, q), p <= q, in the order 00 01 02 03 11 12 13 22 23 33,
// a diagonal block's upper triangle (6), another block's rows (9). K9 / 2 in
// words 24 + 9 ... : node 0's blocks are minus the sums of the others'.
constexpr int kFxBlockWords = 78;
FX_HD constexpr int fx_block(int p, int q)  // first word of block (p, q), p <= q
{
    return p == 0 ? (q == 0 ? 0 : 6 + 9 * (q - 1))
                  : (p == 1 ? (q == 1 ? 33 : 39 + 9 * (q - 2)) : (p == 2 ? (q == 2 ? 57 : 63) : 72));
}
FX_HD constexpr int fx_tri(int a, int b)  // a, b in a diagonal block's triangle
{
    return a <= b ? 3 * a - a * (a - 1) / 2 + (b - a) : fx_tri(b, a);
}
// Word of entry (a, b) of block (p, q) in either order.
FX_HD int fx_block_word(int p, int q, int a, int b)
{
    if (p == q) return fx_block(p, p) + fx_tri(a, b);
    return p < q ? fx_block(p, q) + 3 * a + b : fx_block(q, p) + 3 * b + a;
}
// w[] holds K9 / 2 (entries (r, c), r <= c, of nodes 1 to 3) in its block words;
// fills in node 0's blocks (below 9 2^59).
FX_HD void fx_node0_blocks(int64_t* w)
{
    int64_t s00[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int j = 1; j < 4; j++)
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int b = 0; b < 3; b++) {
                int64_t v = 0;
#pragma unroll
                for (int i = 1; i < 4; i++) v += w[fx_block_word(i, j, a, b)];
                w[fx_block(0, j) + 3 * a + b] = -v;
                if (a <= b) s00[fx_tri(a, b)] += v;
            }
#pragma unroll
    for (int k = 0; k < 6; k++) w[k] = s00[k];
}

// A sum of 64-bit integers of any number (up to 2^31), in two words.
struct FxWide {
    int64_t hi, lo;  // hi 2^32 + lo
};
FX_HD void fx_wide_add(FxWide& s, int64_t v)
{
    s.hi += v >> 32;
    s.lo += (uint32_t)v;
}
FX_HD double fx_wide_value(const FxWide& s, int32_t x)
{
    const int64_t hi = s.hi + (s.lo >> 32);
    const int32_t bits = 64 - fx_clz(fx_mag(hi) | 1u), r = bits > 30 ? bits - 30 : 0;
    return fx_to_double((int64_t)((uint64_t)hi << (32 - r)) + ((int64_t)(uint32_t)s.lo >> r), x + r);
}

#ifdef __CUDACC__
// The sum of a warp's doubles, the same in every lane: aligned to the largest
// exponent and added exactly in three limbs by integer reductions. About 150
// clocks; five FP64 adds and ten shuffles take about 600. The result is
// within 2^-52 (several terms per lane: 2^-49) of the largest term.
template <int K>
__device__ __forceinline__ double fx_warp_sum(const double (&v)[K])  // K terms per lane
{
    static_assert(K >= 1 && K <= 5, "the limbs' headroom");
    constexpr int kBits = K == 1 ? 57 : 55;
    int32_t E = fx_exp(v[0]);
#pragma unroll
    for (int k = 1; k < K; k++) E = max(E, fx_exp(v[k]));
    E = __reduce_max_sync(0xffffffffu, E);
    if (E == 2047) {  // infinities and NaN add as they do
        double s = v[0];
#pragma unroll
        for (int k = 1; k < K; k++) s += v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        return s;
    }
    int64_t m = 0;
#pragma unroll
    for (int k = 0; k < K; k++) m += fx_align<kBits>(v[k], E);
    const uint32_t l0 = __reduce_add_sync(0xffffffffu, (uint32_t)m & 0xffffffu);
    const uint32_t l1 = __reduce_add_sync(0xffffffffu, (uint32_t)(m >> 24) & 0xffffffu);
    const int32_t l2 = __reduce_add_sync(0xffffffffu, (int32_t)(m >> 48));
    return fx_to_double((int64_t)l0 + ((int64_t)l1 << 24) + ((int64_t)((uint64_t)(int64_t)l2 << 48)), E - 1022 - kBits);
}
__device__ __forceinline__ double fx_warp_sum(double v)
{
    const double t[1] = {v};
    return fx_warp_sum(t);
}
#endif

}  // namespace femgb

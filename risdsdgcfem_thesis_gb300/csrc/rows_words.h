// rows_words.h -- the 128-bit words of the solve on resident rows (cg_rows.cu):
// data, and in the top bits of each half the exchange's number, so that a
// reader knows both halves from the one word. W: ulonglong2. Host callable.
#pragma once
#include <math.h>

#include "fx.cuh"

namespace femgb {

// A value of an exchange, with all 32 bits of its number.
template <typename W>
FX_HD W rows_word(double v, uint32_t seq)
{
    const unsigned long long u = fx_bits(v), s = (unsigned long long)seq << 32;
    W w;
    w.x = (u & 0xffffffffull) | s;
    w.y = (u >> 32) | s;
    return w;
}
template <typename W>
FX_HD bool rows_word_is(const W& w, double& v, uint32_t seq)
{
    v = fx_from_bits((w.x & 0xffffffffull) | (w.y << 32));
    return (uint32_t)(w.x >> 32) == seq && (uint32_t)(w.y >> 32) == seq;
}

// A partial sum: m in units of 2^(e - 1079), |m| <= 2^62; kPartNan: NaN;
// kPartInf: m counts infinities by their sign, 2^56 each (their fraction as
// fx_align leaves it), 2^42 at least after the sums' scaling, so that what
// finite parts leave of m when it is added in their place (-1 at most) is no
// infinity. It stays in integers from the lanes to the solid's total.
struct Part {
    int64_t m;
    int32_t e;
};
constexpr int32_t kPartNan = 0x7fff, kPartInf = 0x7ffe;
FX_HD Part part_of(double v)
{
    const int32_t e = fx_exp(v);
    return Part{fx_align<57>(v, e), e == 2047 ? kPartNan - ((fx_bits(v) << 12) == 0 ? 1 : 0) : e};
}
FX_HD double part_value(const Part& p)
{
    const double v = (double)p.m;
    const int32_t e = fx_exp(v) + p.e - 1079;
    if (p.m == 0 || e < 1 || e > 2046) {  // (kPartInf and kPartNan are far above)
        const int64_t least = 1ll << 39;
        if (p.e == kPartNan || (p.e == kPartInf && p.m < least && p.m > -least)) return fx_from_bits(0x7ff8000000000000ull);
        if (p.e == kPartInf) return fx_from_bits(p.m < 0 ? 0xfff0000000000000ull : 0x7ff0000000000000ull);
        return fx_to_double(p.m, p.e - 1079);
    }
    return fx_from_bits(fx_bits(v) + ((uint64_t)(int64_t)(p.e - 1079) << 52));
}

// A sum, with 16 bits of the exchange's number.
template <typename W>
FX_HD W rows_word(const Part& v, uint32_t seq)
{
    const unsigned long long m = (unsigned long long)v.m, s = (unsigned long long)seq << 48;
    W w;
    w.x = (m & 0xffffffffffffull) | s;
    w.y = (m >> 48) | ((unsigned long long)(v.e & 0xffff) << 16) | s;
    return w;
}
template <typename W>
FX_HD bool rows_word_is(const W& w, Part& v, uint32_t seq)
{
    v.m = (int64_t)((w.x & 0xffffffffffffull) | (w.y << 48));
    v.e = (int32_t)(w.y >> 16) & 0xffff;
    return (uint32_t)(w.x >> 48) == (seq & 0xffffu) && (uint32_t)(w.y >> 48) == (seq & 0xffffu);
}

// t / d from r, 1 / d rounded to nearest: the product t r, corrected once by
// its remainder t - q d, which a fused multiply-add gives exactly (P.
// Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990): within 2^-105 of t / d before the last rounding. False
// where a reciprocal, quotient or remainder may be subnormal or none is
// finite: divide there.
FX_HD bool rows_quotient(double t, double d, double r, double& q)
{
    const double q0 = t * r;
    q = fma(fma(-q0, d, t), r, q0);
    // q0 between 2^-511 and 2^512, r between 2^-959 and 2^389: t is above 2^-900
    return (uint32_t)fx_exp(q0) - 512u < 1024u && (uint32_t)fx_exp(r) - 64u < 1348u;
}

// What the words of a CTA hold when a solve starts after number seq: sums
// words of sums, then values.
template <typename W>
FX_HD void rows_words_start(W* w, uint32_t sums, uint32_t values, uint32_t seq, uint32_t first, uint32_t step)
{
    for (uint32_t i = first; i < sums; i += step) w[i] = rows_word<W>(Part{0, 0}, seq);
    for (uint32_t i = first; i < values; i += step) w[sums + i] = rows_word<W>(0.0, seq);
}

}  // namespace femgb

// fx_device.cuh -- device storage of the element product matrices of fx.cuh,
// shared by the FP64 solid (fem_kernels.cu) and the FP64 batch
// (batch_kernels.cu): kFxGroups 16-byte groups of two entries per element,
// [T / 32][kFxGroups][32], the last group's second half the scale.
#pragma once
#include "fem_device.cuh"
#include "fx.cuh"

namespace femgb {

// Element e's groups: 32 apart.
template <typename P>
__device__ __forceinline__ P* fx_matrix(P* K, size_t e)
{
    return K + (size_t)kFxGroups * (e & ~(size_t)31) + (e & 31);
}

// Bakes element e's matrix (kl = V lambda, km = V mu; grade: fx_grade_ok).
__device__ __forceinline__ void fx_store_matrix(int4* K, size_t e, const double* R, const double* Di, double kl,
                                                double km, float grade)
{
    FxL even{0, 0};
    int4* Kp = fx_matrix(K, e);
    auto put = [&](int k, int64_t w) {  // two entries per 16-byte group
        const FxL v = fx_split(w);
        if ((k & 1) == 0) even = v;
        else Kp[32 * (k >> 1)] = make_int4(even.l, even.h, v.l, v.h);
    };
    const int32_t scale = fx_grade_ok(grade, kl, km) ? fx_bake(R, Di, kl, km, put) : kFxFp64;
    Kp[32 * (kFxGroups - 1)] = make_int4(even.l, even.h, scale, 0);
}

// Element e's matrix times its differences, as fx_product's outputs; x becomes
// the exponent of their units.
__device__ __forceinline__ void fx_load_product(const int4* K, size_t e, const int4& last, const FxL* D, int64_t* out,
                                                int32_t& x)
{
    const int4* Kp = fx_matrix(K, e);
    int4 cur;
    x += last.z + fx_product([&](int k) {
        if (k == kFxK - 1) cur = last;
        else if ((k & 1) == 0) cur = Kp[32 * (k >> 1)];
        return (k & 1) ? FxL{cur.z, cur.w} : FxL{cur.x, cur.y};
    }, D, out);
}

}  // namespace femgb

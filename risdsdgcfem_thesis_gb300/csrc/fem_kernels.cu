// fem_kernels.cu -- FP64 element products, node gathers and CG vector
// kernels of the corotational linear-tet implicit-Euler step.
//
// Element products use K0 = V B^T E B (TetrahedronElement3::Compute_K,
// TetrahedronElement3.h:157-173) through the shape-function gradients (rows of
// Dm^-1; node 0's the negative sum) instead of the reference's 16 stored 3x3
// blocks: the C_WRP differential as one 9 x 9 matrix per element in fixed
// point (fx.cuh), the forces and energies in the strain form
// (elem_math.cuh).
//
// Scatter is atomics-free: each element writes its four nodal vectors to
// eout, and four lanes per node sum its entries in a fixed order. Reductions are
// deterministic: integer warp sums (fx_warp_sum), one partial per block, and
// every block of the kernel that uses the sum adds them all (grid_total); norms
// and energies end in one block (k_finalize).
#include "bounds.cuh"
#include "lcm.cuh"
#include "fem_device.cuh"
#include "msvd.cuh"
#include "elem_math.cuh"
#include "fx_device.cuh"

#include <map>
#include <mutex>
#include <string>
#include <vector>

namespace femgb {

// ---- kernel timing (events on the launching stream) ----
namespace {
struct ProfSlot {
    std::vector<cudaEvent_t> starts, stops;
    double done_ms = 0.0;
    unsigned long long done_count = 0;
};
std::mutex g_prof_mu;
bool g_prof_on = false;
std::map<std::string, ProfSlot> g_prof;
std::vector<cudaEvent_t> g_event_pool;

cudaEvent_t pool_event()
{
    if (!g_event_pool.empty()) {
        cudaEvent_t e = g_event_pool.back();
        g_event_pool.pop_back();
        return e;
    }
    cudaEvent_t e;
    cudaEventCreate(&e);
    return e;
}
}  // namespace

bool prof_enabled() { return g_prof_on; }

void prof_begin(const char* name, cudaStream_t s)
{
    if (!g_prof_on) return;
    std::lock_guard<std::mutex> lk(g_prof_mu);
    cudaEvent_t e = pool_event();
    cudaEventRecord(e, s);
    g_prof[name].starts.push_back(e);
}

void prof_end(const char* name, cudaStream_t s)
{
    if (!g_prof_on) return;
    std::lock_guard<std::mutex> lk(g_prof_mu);
    cudaEvent_t e = pool_event();
    cudaEventRecord(e, s);
    g_prof[name].stops.push_back(e);
}

// Folds completed event pairs into the totals (synchronises on the events).
static void prof_collect()
{
    for (auto& kv : g_prof) {
        ProfSlot& sl = kv.second;
        const size_t n = sl.stops.size() < sl.starts.size() ? sl.stops.size() : sl.starts.size();
        for (size_t i = 0; i < n; i++) {
            float ms = 0.f;
            cudaEventSynchronize(sl.stops[i]);
            cudaEventElapsedTime(&ms, sl.starts[i], sl.stops[i]);
            sl.done_ms += ms;
            sl.done_count++;
            g_event_pool.push_back(sl.starts[i]);
            g_event_pool.push_back(sl.stops[i]);
        }
        sl.starts.erase(sl.starts.begin(), sl.starts.begin() + n);
        sl.stops.erase(sl.stops.begin(), sl.stops.begin() + n);
    }
}

}  // namespace femgb

extern "C" int fem_profile_enable(int on)
{
    std::lock_guard<std::mutex> lk(femgb::g_prof_mu);
    femgb::prof_collect();
    femgb::g_prof_on = on != 0;
    if (on) femgb::g_prof.clear();
    return 0;
}

extern "C" int fem_profile_read(const char* kernel, double* total_ms, unsigned long long* launches)
{
    std::lock_guard<std::mutex> lk(femgb::g_prof_mu);
    femgb::prof_collect();
    auto it = femgb::g_prof.find(kernel ? kernel : "");
    if (total_ms) *total_ms = it == femgb::g_prof.end() ? 0.0 : it->second.done_ms;
    if (launches) *launches = it == femgb::g_prof.end() ? 0ull : it->second.done_count;
    return 0;
}

namespace femgb {

uint64_t& launch_counter()
{
    static uint64_t n = 0;
    return n;
}

// Block sum, valid in every thread (two rounds of fx_warp_sum).
__device__ __forceinline__ double block_sum(double v)
{
    __shared__ double sh[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    v = fx_warp_sum(v);
    if (blockDim.x == 32) return v;
    __syncthreads();
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    return fx_warp_sum(lane < (int)((blockDim.x + 31) >> 5) ? sh[lane] : 0.0);
}

// The total of the previous kernel's block partials, valid in every thread
// and the same in every block.
__device__ __forceinline__ double grid_total(const double* __restrict__ partials, uint32_t count)
{
    double acc = 0.0;
    for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) acc += partials[i];
    return block_sum(acc);
}

template <typename S>
__device__ __forceinline__ void load_elem(const MeshView<S>& m, uint32_t e, S* R, S* Di, S& k1, S& knu, S& k2)
{
    const size_t T = m.T;
#pragma unroll
    for (int c = 0; c < 9; c++) R[c] = m.R[c * T + e];
#pragma unroll
    for (int c = 0; c < 9; c++) Di[c] = m.Dinv[c * T + e];
    k1 = m.mat[e];
    knu = m.mat[T + e];
    k2 = m.mat[2 * T + e];
}

// ---- C_LCM element kernels (csrc/lcm.cuh): the material's force from the
// stored F of the last evaluation (T x 9, row-major per element), its
// truncated differential, its energy. Same eout convention as the C_WRP
// kernels below. ----

__device__ __forceinline__ void load_R_Dinv(const MeshView<double>& m, uint32_t e, double* R, double* Di)
{
    const size_t T = m.T;
#pragma unroll
    for (int c = 0; c < 9; c++) {
        R[c] = m.R[c * T + e];
        Di[c] = m.Dinv[c * T + e];
    }
}

__global__ void k_elem_lcm_force_fp64(MeshView<double> m, const double* __restrict__ F, PkMaterial mat,
                                      int write_out, double* energy_partials)
{
    double energy = 0.0;
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < m.T; e += gridDim.x * blockDim.x) {
        double R[9], Di[9], Fl[9];
        load_R_Dinv(m, e, R, Di);
#pragma unroll
        for (int c = 0; c < 9; c++) Fl[c] = F[9 * (size_t)e + c];
        if (write_out) {
            double out[12];
            pk_force(mat, R, Fl, Di, m.vol[e], out);
            double* o = m.eout + 12 * (size_t)e;
#pragma unroll
            for (int c = 0; c < 12; c++) o[c] = out[c];
        }
        if (energy_partials) energy += pk_energy(mat, R, Fl, m.vol[e]);
    }
    if (energy_partials) {
        double s = block_sum(energy);
        if (threadIdx.x == 0) energy_partials[blockIdx.x] = s;
    }
}

__global__ void k_elem_lcm_spmv_fp64(MeshView<double> m, const double* __restrict__ d, const double* __restrict__ F,
                                     PkMaterial mat, const StepScalars* st, int check_done)
{
    if (check_done && st->done_pend) return;
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < m.T; e += gridDim.x * blockDim.x) {
        const int4 t = m.tets[e];
        const int ids[4] = {(int)bounds_idx((uint32_t)t.x, m.N, kSiteElemNode),
                            (int)bounds_idx((uint32_t)t.y, m.N, kSiteElemNode),
                            (int)bounds_idx((uint32_t)t.z, m.N, kSiteElemNode),
                            (int)bounds_idx((uint32_t)t.w, m.N, kSiteElemNode)};
        double R[9], Di[9], dl[12];
        load_R_Dinv(m, e, R, Di);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            dl[3 * i] = d[3 * (size_t)ids[i]];
            dl[3 * i + 1] = d[3 * (size_t)ids[i] + 1];
            dl[3 * i + 2] = d[3 * (size_t)ids[i] + 2];
        }
        double Fl[9];
        if (mat.kind != 1) {  // C_LCMH and C_CCM read F (and C_CCM det F)
#pragma unroll
            for (int c = 0; c < 9; c++) Fl[c] = F[9 * (size_t)e + c];
        }
        double out[12];
        pk_dforce(mat, R, Fl, mat.kind == 3 ? m.detF[e] : 0.0, Di, m.vol[e], dl, out);
        double* o = m.eout + 12 * (size_t)e;
#pragma unroll
        for (int c = 0; c < 12; c++) o[c] = out[c];
    }
}

// ---- element kernels ----

// Element e's fixed-point product matrix (fx.cuh) from R, Dm^-1 and the
// material scalars: 45 entries and the scale, 368 bytes, written once per
// evaluation. Integer-bound: about 250 products of three multiplies (224 us
// for 1,080,000 tets, a sixth of their rotations).
__global__ void __launch_bounds__(128, 3) k_elem_bake_fp64(MeshView<double> m)
{
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < m.T; e += gridDim.x * blockDim.x) {
        double R[9], Di[9], k1, knu, k2;
        load_elem(m, e, R, Di, k1, knu, k2);
        fx_store_matrix(m.Kfx, e, R, Di, knu, k2, m.grade[e]);
    }
}

// The FP64 product of an element fx.cuh leaves out, from its nodes' vectors,
// as records in o. Out of line and from pointers, so that the fixed-point
// path keeps its values in registers.
__device__ __noinline__ void elem_record_fp64(const double* Rp, const double* Dp, const double* mat, size_t T, const double* p0,
                                              const double* p1, const double* p2, const double* p3, longlong2* o)
{
    double R[9], Di[9], d[12], f[12];
    int64_t out[12];
#pragma unroll
    for (int c = 0; c < 9; c++) {
        R[c] = Rp[c * T];
        Di[c] = Dp[c * T];
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
        d[a] = p0[a];
        d[3 + a] = p1[a];
        d[6 + a] = p2[a];
        d[9 + a] = p3[a];
    }
    elem_RKRt(R, Di, mat[0], mat[T], mat[2 * T], d, f);
    fx_stamp_doubles(f, out);
#pragma unroll
    for (int c = 0; c < 6; c++) o[c] = make_longlong2(out[2 * c], out[2 * c + 1]);
}

// Element e's product from its nodes' vectors into six 16-byte words of
// records. K(k): the matrix entries, in order.
template <typename FK>
__device__ __forceinline__ void elem_records(const MeshView<double>& m, uint32_t e, int32_t scale, FK&& K,
                                             const double* const* p, longlong2* o)
{
    double dl[12];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int a = 0; a < 3; a++) dl[3 * i + a] = p[i][a];
    FxL D[9];
    int64_t out[12];
    int32_t x;
    bool ok = fx_differences(dl, D, x) && scale != kFxFp64;
    x += scale + fx_product(K, D, out);
    ok = ok && fx_stamp(out, x);
    if (ok) {
#pragma unroll
        for (int c = 0; c < 6; c++) o[c] = make_longlong2(out[2 * c], out[2 * c + 1]);
    } else {
        elem_record_fp64(m.R + e, m.Dinv + e, m.mat + e, m.T, p[0], p[1], p[2], p[3], o);
    }
}

// R K0 R^T d per element as fixed-point records in eout. 368 bytes of matrix
// per element: bound by the integer pipe while the matrices stay in L2 (up to
// about 300k tets) and by HBM beyond. The FP64 strain form held the FP64 pipe
// at 90 %: 7,215 tets 11.4 -> 3.6 us, 20,480 tets 11.7 -> 4.8 us, 1,080,000
// tets 273 -> 91 us (540 MB, 5.9 TB/s).
__global__ void __launch_bounds__(128, 3) k_elem_spmv_fp64(MeshView<double> m, const double* __restrict__ d,
                                                           const StepScalars* st, int check_done)
{
    if (check_done && st->done_pend) return;
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < m.T; e += gridDim.x * blockDim.x) {
        const int4 t = m.tets[e];
        const double* p[4] = {d + 3 * (size_t)bounds_idx((uint32_t)t.x, m.N, kSiteElemNode),
                              d + 3 * (size_t)bounds_idx((uint32_t)t.y, m.N, kSiteElemNode),
                              d + 3 * (size_t)bounds_idx((uint32_t)t.z, m.N, kSiteElemNode),
                              d + 3 * (size_t)bounds_idx((uint32_t)t.w, m.N, kSiteElemNode)};
        if (!m.Kfx) {
            elem_record_fp64(m.R + e, m.Dinv + e, m.mat + e, m.T, p[0], p[1], p[2], p[3],
                             reinterpret_cast<longlong2*>(m.eout + 12 * (size_t)e));
            continue;
        }
        const int4* Kp = fx_matrix(m.Kfx, e);
        const int4 last = Kp[32 * (kFxGroups - 1)];
        int4 cur;
        elem_records(m, e, last.z, [&](int k) {
            if (k == kFxK - 1) cur = last;
            else if ((k & 1) == 0) cur = Kp[32 * (k >> 1)];
            return (k & 1) ? FxL{cur.z, cur.w} : FxL{cur.x, cur.y};
        }, p, reinterpret_cast<longlong2*>(m.eout + 12 * (size_t)e));
    }
}

// R K0 (R^T x - r) per element (C_f_e's product); optional eout write and
// per-block elastic-energy partial 0.5 * u^T K0 u (C_V).
__global__ void k_elem_force_fp64(MeshView<double> m, const double* __restrict__ x, int write_out,
                                  double* energy_partials)
{
    double energy = 0.0;
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < m.T; e += gridDim.x * blockDim.x) {
        const int4 t = m.tets[e];
        double R[9], Di[9], k1, knu, k2;
        load_elem(m, e, R, Di, k1, knu, k2);
        const int ids[4] = {(int)bounds_idx((uint32_t)t.x, m.N, kSiteElemNode),
                            (int)bounds_idx((uint32_t)t.y, m.N, kSiteElemNode),
                            (int)bounds_idx((uint32_t)t.z, m.N, kSiteElemNode),
                            (int)bounds_idx((uint32_t)t.w, m.N, kSiteElemNode)};
        double u[12];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const size_t n = ids[i];
            const double xa = x[3 * n], xb = x[3 * n + 1], xc = x[3 * n + 2];
            // u_i = R^T x_i - r_i (accumulator from zero, as the reference)
#pragma unroll
            for (int a = 0; a < 3; a++) {
                double acc = 0.0;
                acc += R[a] * xa;
                acc += R[3 + a] * xb;
                acc += R[6 + a] * xc;
                u[3 * i + a] = acc - m.rest[3 * n + a];
            }
        }
        double D[9];
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int j = 0; j < 3; j++) D[3 * a + j] = u[3 * (j + 1) + a] - u[a];
        double H[9];
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int b = 0; b < 3; b++) H[3 * a + b] = D[3 * a] * Di[b] + D[3 * a + 1] * Di[3 + b] + D[3 * a + 2] * Di[6 + b];
        double P[9], es;
        stress_forces(H, Di, k1, knu, k2, P, es);
        energy += 0.5 * es;
        if (write_out) {
            double out[12];
            rotate_out(R, P, out);
            double* o = m.eout + 12 * (size_t)e;
#pragma unroll
            for (int c = 0; c < 12; c++) o[c] = out[c];
        }
    }
    if (energy_partials) {
        double s = block_sum(energy);
        if (threadIdx.x == 0) energy_partials[blockIdx.x] = s;
    }
}

// Potential energy term of RecomputeEnergy (LeafDSH_Solid3D_FEM.cpp:1554-1584):
// sum_e (rho V_e / 4) (x0+x1+x2+x3) . (-g)
__global__ void k_potential_fp64(MeshView<double> m, StepConsts c, const double* __restrict__ x, double* partials)
{
    double acc = 0.0;
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < m.T; e += gridDim.x * blockDim.x) {
        const int4 t = m.tets[e];
        const int ids[4] = {(int)bounds_idx((uint32_t)t.x, m.N, kSiteElemNode),
                            (int)bounds_idx((uint32_t)t.y, m.N, kSiteElemNode),
                            (int)bounds_idx((uint32_t)t.z, m.N, kSiteElemNode),
                            (int)bounds_idx((uint32_t)t.w, m.N, kSiteElemNode)};
        double s[3] = {0, 0, 0};
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int a = 0; a < 3; a++) s[a] += x[3 * (size_t)ids[i] + a];
        double em = c.density * m.vol[e];
        acc += (em / 4.0) * (s[0] * -c.gravity[0] + s[1] * -c.gravity[1] + s[2] * -c.gravity[2]);
    }
    double v = block_sum(acc);
    if (threadIdx.x == 0) partials[blockIdx.x] = v;
}

// ---- node kernels ----

// The sums at a node are taken by four lanes of a warp (eight nodes per
// warp): lanes 0 to 2 return the components, lane 3 zero. Every lane of a
// warp calls them (on: the node exists). One thread per node left most of the
// chip idle at 20,480 tets (node_q: 20 blocks, 15.9 us; now 5.6) and took
// three FP64 adds per corner (1,080,000 tets: 74 us; now 40).

// Element outputs in FP64 (forces, and the products of the P-K materials):
// lane a adds component a of the node's corners in element order.
__device__ __forceinline__ double gather_fp64(const MeshView<double>& m, uint32_t n, uint32_t a, bool on)
{
    double s = 0.0;
    if (!on || a == 3) return s;
    const uint32_t beg = m.csr_ptr[n], end = m.csr_ptr[n + 1];
#pragma unroll 4
    for (uint32_t j = beg; j < end; j++)
        s += m.eout[3 * (size_t)bounds_idx(m.csr_idx[j], 4ull * m.T, kSiteCsrEntry) + a];
    return s;
}

// The four lanes' record sums of a node brought to the largest exponent and added: lane a's component.
__device__ __forceinline__ double fx_quad_sum(const FxSum& s, uint32_t a, int32_t guard)
{
    int32_t E = s.E;
    E = max(E, __shfl_xor_sync(0xffffffffu, E, 1));
    E = max(E, __shfl_xor_sync(0xffffffffu, E, 2));
    const int32_t sh = fx_min63(E - s.E);
    int64_t t = 0;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        long long v = s.acc[c] >> sh;
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        if ((int)a == c) t = v;
    }
    return fx_sum_value(t, E, guard);
}

// Fixed-point records: lane l adds the corners beg + l, beg + l + 4, ... in
// all three components (integer sums in block exponents, fx.cuh).
__device__ __forceinline__ double gather_fx(const MeshView<double>& m, uint32_t n, uint32_t a, bool on)
{
    constexpr int kBatch = 3;  // records in flight per lane
    const int32_t guard = (int32_t)m.fx_guard;
    FxSum s{{0, 0, 0}, 0};
    if (on) {
        const uint32_t beg = m.csr_ptr[n], end = m.csr_ptr[n + 1];
        const long long* rec = reinterpret_cast<const long long*>(m.eout);
        for (uint32_t j = beg + a; j < end; j += 4 * kBatch) {
            // loaded without a branch, past the end the last one again
            int64_t v[kBatch][3];
            uint32_t at[kBatch];
#pragma unroll
            for (int k = 0; k < kBatch; k++)
                at[k] = bounds_idx(m.csr_idx[min(j + 4 * k, end - 1)], 4ull * m.T, kSiteCsrEntry);
#pragma unroll
            for (int k = 0; k < kBatch; k++) {
                const long long* r = rec + 3 * (size_t)at[k];
                const bool in = j + 4 * k < end;
                v[k][0] = r[0];
                v[k][1] = r[1];
                v[k][2] = r[2];
                if (!in) v[k][0] = v[k][1] = v[k][2] = 0;  // an empty record: the lowest exponent
            }
#pragma unroll
            for (int k = 0; k < kBatch; k++) fx_add(s, v[k][0], v[k][1], v[k][2], guard);
        }
    }
    return fx_quad_sum(s, a, guard);
}

// The assembled row times the vector's records: lane l takes the blocks l,
// l + 4, ...; the vector's entries are brought to the largest exponent among
// the row's columns. The first four groups' records (rows of up to 16 blocks
// whole) are loaded once, ahead of everything that waits for them. A block's
// nine products keep mid below 3 (2^28 + 2^27) 2^31 + 2^32; the row's exponent
// holds bits free for its length.
__device__ __forceinline__ double bsr_row_fx(const MeshView<double>& m, uint32_t n, uint32_t a, bool on)
{
    constexpr int kHeld = 4;
    const uint32_t beg = on ? m.bsr_row[n] : 0u, end = on ? m.bsr_row[n + 1] : 0u;
    const int32_t xr = on ? m.bsr_x[n] : 0;
    auto column = [&](uint32_t g) { return (size_t)bounds_idx(m.bsr_col[4 * (size_t)g + a], m.N, kSiteBsrEntry); };
    longlong2 u01[kHeld], u2e[kHeld];
    int32_t E = 0;
#pragma unroll
    for (int h = 0; h < kHeld; h++) {
        u01[h] = u2e[h] = make_longlong2(0, 0);
        if (beg + h < end) {
            const size_t j = column(beg + h);
            u01[h] = m.bsr_u[2 * j];
            u2e[h] = m.bsr_u[2 * j + 1];
        }
    }
#pragma unroll
    for (int h = 0; h < kHeld; h++) E = max(E, (int32_t)u2e[h].y);
    for (uint32_t g = beg + kHeld; g < end; g++) E = max(E, (int32_t)m.bsr_u[2 * column(g) + 1].y);
    E = max(E, __shfl_xor_sync(0xffffffffu, E, 1));
    E = max(E, __shfl_xor_sync(0xffffffffu, E, 2));
    int64_t hi[3] = {0, 0, 0}, mid[3] = {0, 0, 0};
    auto block = [&](uint32_t g, const longlong2& v01, const longlong2& v2e) {
        const int32_t sh = fx_min63(E - (int32_t)v2e.y);
        const FxL u[3] = {fx_split(v01.x >> sh), fx_split(v01.y >> sh), fx_split(v2e.x >> sh)};
        const int2* A = m.bsr_val + 36 * (size_t)g + a;
#pragma unroll
        for (int r = 0; r < 3; r++) {
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const int2 k = A[4 * (3 * r + c)];
                fx_mac(hi[r], mid[r], FxL{k.x, k.y}, u[c]);
            }
            hi[r] += mid[r] >> 32;
            mid[r] &= 0xffffffffll;
        }
    };
#pragma unroll
    for (int h = 0; h < kHeld; h++)
        if (beg + h < end) block(beg + h, u01[h], u2e[h]);
    for (uint32_t g = beg + kHeld; g < end; g++) {
        const size_t j = column(g);
        block(g, m.bsr_u[2 * j], m.bsr_u[2 * j + 1]);
    }
    int64_t t = 0;
#pragma unroll
    for (int r = 0; r < 3; r++) {
        long long v = fx_fin<4>(hi[r], mid[r]) >> 2;
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        if ((int)a == r) t = v;
    }
    if (E == 2047 || xr == kFxFp64) return fx_from_bits(0x7ff8000000000000ull);
    return a == 3 ? 0.0 : fx_to_double(t, xr + (E - 1081) + 62);
}

// A node's record: its components in units of its own largest.
__device__ __forceinline__ void bsr_record(const MeshView<double>& m, uint32_t n, double v0, double v1, double v2)
{
    const int32_t E = max(fx_exp(v0), max(fx_exp(v1), fx_exp(v2)));
    m.bsr_u[2 * (size_t)n] = make_longlong2(fx_align<59>(v0, E), fx_align<59>(v1, E));
    m.bsr_u[2 * (size_t)n + 1] = make_longlong2(fx_align<59>(v2, E), E);
}
__global__ void k_bsr_vector_fp64(MeshView<double> m, const double* __restrict__ u, const StepScalars* st,
                                  int check_done)
{
    if (check_done && st->done_pend) return;
    for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n < m.N; n += gridDim.x * blockDim.x)
        bsr_record(m, n, u[3 * (size_t)n], u[3 * (size_t)n + 1], u[3 * (size_t)n + 2]);
}

// K u at node n for the solvers' node kernels: the assembled row when the
// solid has one, else the sum of the element outputs of the product launched
// before.
enum NodeKu { kKuRecords = 0, kKuFp64 = 1, kKuBsr = 2 };
template <int kKu>
__device__ __forceinline__ double node_Ku(const MeshView<double>& m, uint32_t n, uint32_t a, bool on)
{
    if constexpr (kKu == kKuBsr) return bsr_row_fx(m, n, a, on);
    else if constexpr (kKu == kKuRecords) return gather_fx(m, n, a, on);
    else return gather_fp64(m, n, a, on);
}

// An element fx.cuh leaves out: K9 / 2 from FP64 (V (lambda m_i m_j^T +
// mu m_j m_i^T + mu (g_i . g_j) R R^T), m = R g) in the block words; returns
// the units' exponent, kFxFp64 when an entry is not finite.
__device__ __noinline__ int32_t elem_blocks_fp64(const double* Rp, const double* Dp, double kl, double km, size_t T, int64_t* w)
{
    double R[9], g[9], mm[9], C[9], K[45];
    for (int c = 0; c < 9; c++) {
        R[c] = Rp[c * T];
        g[c] = Dp[c * T];
    }
    for (int i = 0; i < 3; i++)
        for (int a = 0; a < 3; a++) {
            mm[3 * i + a] = R[3 * a] * g[3 * i] + R[3 * a + 1] * g[3 * i + 1] + R[3 * a + 2] * g[3 * i + 2];
            C[3 * i + a] = R[3 * i] * R[3 * a] + R[3 * i + 1] * R[3 * a + 1] + R[3 * i + 2] * R[3 * a + 2];
        }
    int32_t E = 0;
    for (int r = 0; r < 9; r++)
        for (int c = r; c < 9; c++) {
            const int i = r / 3, a = r % 3, j = c / 3, b = c % 3;
            const double G = g[3 * i] * g[3 * j] + g[3 * i + 1] * g[3 * j + 1] + g[3 * i + 2] * g[3 * j + 2];
            const double v = kl * mm[3 * i + a] * mm[3 * j + b] + km * mm[3 * j + a] * mm[3 * i + b] + km * G * C[3 * a + b];
            K[fx_at(r, c)] = v;
            E = max(E, fx_exp(v));
        }
    for (int r = 0; r < 9; r++)
        for (int c = r; c < 9; c++) {
            const int i = r / 3 + 1, j = c / 3 + 1;
            if (E < 2047) w[fx_block_word(i, j, r % 3, c % 3)] = fx_align<59>(K[fx_at(r, c)], E);
        }
    return E < 2047 ? E - 1022 - 59 : kFxFp64;
}

// The elements' corner blocks: one element per thread, its words staged in
// shared memory (rows of an odd number of words) and written out in whole
// lines. Bound by the integer products of fx_bake and by the writes (632
// bytes per element).
constexpr int kBsrElemBlock = 64, kBsrElemRow = 79;
__global__ void __launch_bounds__(kBsrElemBlock) k_bsr_elements_fp64(MeshView<double> m, BsrBuild a)
{
    extern __shared__ long long el_smem[];
    int64_t* w = reinterpret_cast<int64_t*>(el_smem) + kBsrElemRow * threadIdx.x;
    for (uint32_t e0 = blockIdx.x * kBsrElemBlock; e0 < m.T; e0 += gridDim.x * kBsrElemBlock) {
        const uint32_t e = e0 + threadIdx.x;
        if (e < m.T) {
            double R[9], Di[9], k1, knu, k2;
            load_elem(m, e, R, Di, k1, knu, k2);
            int32_t scale = kFxFp64;
            if (fx_grade_ok(m.grade[e], knu, k2)) {
                int r = 0, c = 0;
                scale = fx_bake(R, Di, knu, k2, [&](int, int64_t v) {
                    w[fx_block_word(r / 3 + 1, c / 3 + 1, r % 3, c % 3)] = v >> 1;
                    if (++c == 9) c = ++r;
                });
            }
            scale = scale != kFxFp64 ? scale + 1 : elem_blocks_fp64(m.R + e, m.Dinv + e, knu, k2, m.T, w);
            fx_node0_blocks(w);
            a.ex[e] = scale;
        }
        __syncthreads();
        const uint32_t words = kBsrElemWords * min((uint32_t)kBsrElemBlock, m.T - e0);
        for (uint32_t i = threadIdx.x; i < words; i += kBsrElemBlock)
            a.eblk[kBsrElemWords * (size_t)e0 + i] = el_smem[kBsrElemRow * (i / kBsrElemWords) + i % kBsrElemWords];
        __syncthreads();
    }
}

// One block slot per thread: the contributions at the largest exponent among
// them, added exactly, as nine doubles in the slot's entries (the rows' kernel
// converts them in place). Diagonal blocks have four times the contributions
// of the others; they come from the row instead.
__global__ void __launch_bounds__(128) k_bsr_slots_fp64(MeshView<double> m, BsrBuild b)
{
    const uint32_t count = 4 * b.groups;
    double* val = reinterpret_cast<double*>(b.val);
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < count; s += gridDim.x * blockDim.x) {
        const uint32_t beg = b.cptr[s], end = b.cptr[s + 1];
        int32_t X = INT32_MIN;
        for (uint32_t k = beg; k < end; k++) X = max(X, b.ex[bounds_idx(b.contrib[k] >> 4, m.T, kSiteBsrEntry)]);
        FxWide acc[9];
#pragma unroll
        for (int c = 0; c < 9; c++) acc[c] = FxWide{0, 0};
        for (uint32_t k = beg; k < end; k++) {
            const uint32_t cb = b.contrib[k], e = bounds_idx(cb >> 4, m.T, kSiteBsrEntry);
            const uint32_t li = (cb >> 2) & 3u, lj = cb & 3u, p = min(li, lj), q = max(li, lj);
            const int32_t sh = fx_min63(X - b.ex[e]);
            const long long* w = b.eblk + kBsrElemWords * (size_t)e + fx_block(p, q);
            int64_t v[9];
#pragma unroll
            for (int c = 0; c < 9; c++) v[c] = w[c] >> sh;
#pragma unroll
            for (int r = 0; r < 3; r++)
#pragma unroll
                for (int c = 0; c < 3; c++) fx_wide_add(acc[3 * r + c], li < lj ? v[3 * r + c] : v[3 * c + r]);
        }
        double* o = val + 36 * (size_t)(s >> 2) + (s & 3u);
#pragma unroll
        for (int c = 0; c < 9; c++)
            o[4 * c] = beg == end ? 0.0
                                  : (X == kFxFp64 ? fx_from_bits(0x7ff8000000000000ull) : fx_wide_value(acc[c], X));
    }
}

// Each row to one exponent, in place, and its diagonal block as minus the sum
// of the others (an element's blocks sum to zero along a row), exactly as the
// row now holds them: rigid translations have no force. Entries below 2^60,
// their magnitudes along a matrix row below 2^62 (the products' headroom).
__global__ void k_bsr_rows_fp64(MeshView<double> m, BsrBuild b)
{
    const uint32_t a = threadIdx.x & 3u, step = (gridDim.x * blockDim.x) >> 2;
    const double* val = reinterpret_cast<const double*>(b.val);
    for (uint32_t n = (blockIdx.x * blockDim.x + threadIdx.x) >> 2; (n & ~7u) < m.N; n += step) {
        const bool on = n < m.N;
        const uint32_t beg = on ? m.bsr_row[n] : 0u, end = on ? m.bsr_row[n + 1] : 0u;
        int32_t E = 0;
        uint32_t diag = 0xffffffffu;  // the first slot of column n (pads follow it)
        for (uint32_t g = beg; g < end; g++) {
            if (m.bsr_col[4 * (size_t)g + a] == n) diag = min(diag, 4 * g + a);
#pragma unroll
            for (int k = 0; k < 9; k++) E = max(E, fx_exp(val[36 * (size_t)g + 4 * k + a]));
        }
        int32_t room = 0;  // bits for the sums of a row
        while ((2u << room) < end - beg) room++;
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
            E = max(E, __shfl_xor_sync(0xffffffffu, E, o));
            diag = min(diag, __shfl_xor_sync(0xffffffffu, diag, o));
        }
        long long sum[9];
        unsigned long long mag[3] = {0, 0, 0};  // eighths
#pragma unroll
        for (int k = 0; k < 9; k++) sum[k] = 0;
        for (uint32_t g = beg; g < end; g++)
#pragma unroll
            for (int k = 0; k < 9; k++) {
                const int64_t v = fx_align<60>(val[36 * (size_t)g + 4 * k + a], E) >> room;
                sum[k] += v;
                mag[k / 3] += fx_mag(v) >> 3;
            }
        uint64_t top = 1;
#pragma unroll
        for (int k = 0; k < 9; k++) {
            sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], 1);
            sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], 2);
            top |= fx_mag(sum[k]);
        }
#pragma unroll
        for (int r = 0; r < 3; r++) {
            mag[r] += __shfl_xor_sync(0xffffffffu, mag[r], 1);
            mag[r] += __shfl_xor_sync(0xffffffffu, mag[r], 2);
#pragma unroll
            for (int c = 0; c < 3; c++) mag[r] += fx_mag(sum[3 * r + c]) >> 3;
        }
        const int32_t bits = 64 - fx_clz(top), bits3 = 67 - fx_clz((mag[0] | mag[1] | mag[2]) + 1);
        const int32_t down = max(0, max(bits - 60, bits3 - 62));
#pragma unroll
        for (int k = 0; k < 9; k++) sum[k] = 0;
        for (uint32_t g = beg; g < end; g++)
#pragma unroll
            for (int k = 0; k < 9; k++) {
                const size_t i = 36 * (size_t)g + 4 * k + a;
                const int64_t v = (fx_align<60>(val[i], E) >> room) >> down;
                sum[k] += v;
                const FxL l = fx_split(v);
                b.val[i] = make_int2(l.l, l.h);
            }
#pragma unroll
        for (int k = 0; k < 9; k++) {
            sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], 1);
            sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], 2);
            if (on && (diag & 3u) == a) {
                const FxL l = fx_split(-sum[k]);
                b.val[36 * (size_t)(diag >> 2) + 4 * k + a] = make_int2(l.l, l.h);
            }
        }
        if (on && a == 0) b.x[n] = E < 2047 ? E - 1082 + room + down : kFxFp64;
    }
}

// b = dt (m g + f_e) + m v ; y = v   (Step_QuasiImplicitEuler_v, :1211-1231)
__global__ void k_node_b_fp64(MeshView<double> m, StepConsts c, const double* __restrict__ v, double* b, double* y)
{
    const uint32_t a = threadIdx.x & 3u, step = (gridDim.x * blockDim.x) >> 2;
    for (uint32_t n = (blockIdx.x * blockDim.x + threadIdx.x) >> 2; (n & ~7u) < m.N; n += step) {
        const bool on = n < m.N;
        const double f = gather_fp64(m, n, a, on);
        if (!on || a == 3) continue;
        const size_t i = 3 * (size_t)n + a;
        const double vi = v[i];
        const double g = a == 0 ? c.gravity[0] : (a == 1 ? c.gravity[1] : c.gravity[2]);
        b[i] = (c.mass * g - f) * c.dt + c.mass * vi;
        y[i] = vi;
    }
}

// Position constraints -> clamped velocity, written to b and y
// (Step_QuasiImplicitEuler_v, LeafDSH_Solid3D_FEM.cpp:1268-1295).
__global__ void k_knc_fp64(uint32_t N, uint32_t count, const uint32_t* __restrict__ nodes,
                           const double* __restrict__ targets, const double* __restrict__ x, StepConsts c, double* b,
                           double* y)
{
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
        const size_t n = bounds_idx(nodes[k], N, kSiteKncNode);
        V3<double> vk = mk<double>(c.inv_dt * (targets[3 * k] - x[3 * n]), c.inv_dt * (targets[3 * k + 1] - x[3 * n + 1]),
                                   c.inv_dt * (targets[3 * k + 2] - x[3 * n + 2]));
        double norm_vk = ::sqrt(dot0(vk, vk));
        V3<double> vel = mk<double>(0.0, 0.0, 0.0);
        if (norm_vk > (double)0.001f) {
            double cl = (norm_vk < 50.0) ? norm_vk : 50.0;
            vel = scale(cl, normalized(vk));
        }
        b[3 * n] = vel.x; b[3 * n + 1] = vel.y; b[3 * n + 2] = vel.z;
        y[3 * n] = vel.x; y[3 * n + 1] = vel.y; y[3 * n + 2] = vel.z;
    }
}

// r = S (b - A y) ; d = r ; partial |r|^2   (ILSS_CG.h:53-64)
template <int kKu>
__global__ void k_node_residual_fp64(MeshView<double> m, StepConsts c, const double* __restrict__ b,
                                     const double* __restrict__ y, double* r, double* d, double* partials)
{
    double acc = 0.0;
    const double mfm = c.mass * c.factor_M;
    const uint32_t a = threadIdx.x & 3u, step = (gridDim.x * blockDim.x) >> 2;
    for (uint32_t n = (blockIdx.x * blockDim.x + threadIdx.x) >> 2; (n & ~7u) < m.N; n += step) {
        const bool on = n < m.N;
        const double s = node_Ku<kKu>(m, n, a, on);
        if (!on || a == 3) continue;
        const size_t i = 3 * (size_t)n + a;
        const double ri = m.fixed[n] ? 0.0 : b[i] - (c.factor_K * s + mfm * y[i]);
        r[i] = ri;
        d[i] = ri;
        acc += ri * ri;
    }
    double s = block_sum(acc);
    if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

// q = S A d ; partial d.q   (ILSS_CG.h:90-96)
template <int kKu>
__global__ void k_node_q_fp64(MeshView<double> m, StepConsts c, const double* __restrict__ d, double* q, double* pq,
                              const StepScalars* st)
{
    if (st->done_pend) return;
    double acc = 0.0;
    const double mfm = c.mass * c.factor_M;
    const uint32_t a = threadIdx.x & 3u, step = (gridDim.x * blockDim.x) >> 2;
    for (uint32_t n = (blockIdx.x * blockDim.x + threadIdx.x) >> 2; (n & ~7u) < m.N; n += step) {
        const bool on = n < m.N;
        const double s = node_Ku<kKu>(m, n, a, on);
        if (!on || a == 3) continue;
        const size_t i = 3 * (size_t)n + a;
        const double di = d[i], qi = m.fixed[n] ? 0.0 : c.factor_K * s + mfm * di;
        q[i] = qi;
        acc += di * qi;
    }
    const double total = block_sum(acc);
    if (threadIdx.x == 0) pq[blockIdx.x] = total;
}

// alpha = |r|^2 / d.q ; y += alpha d ; r -= alpha q ; partial |r|^2
// (ILSS_CG.h:96-117). One thread per block takes the division (a dozen FP64
// instructions, each 64 clocks of its sub-partition per warp that runs it).
__global__ void k_node_xr_fp64(uint32_t N, double* y, double* r, const double* __restrict__ d,
                               const double* __restrict__ q, const double* __restrict__ pq, uint32_t npq, double* pr,
                               StepScalars* st)
{
    if (st->done_pend) {
        if (blockIdx.x == 0 && threadIdx.x == 0) st->done = 1;
        return;
    }
    const uint32_t n3 = 3 * N, i0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    double y0 = 0.0, r0 = 0.0, d0 = 0.0, q0 = 0.0;  // the first component, loaded ahead of alpha
    if (i0 < n3) {
        y0 = y[i0];
        r0 = r[i0];
        d0 = d[i0];
        q0 = q[i0];
    }
    __shared__ double sh_alpha;
    const double dq = grid_total(pq, npq), delta = st->delta_pend;
    const bool brk = ::fabs(dq) < st->abs_eps_sq;  // breakdown: leave before the update (ILSS_CG.h:97)
    if (threadIdx.x == 0) {
        sh_alpha = delta / dq;
        if (blockIdx.x == 0) {
            st->dot_dq = dq;
            st->delta_new = delta;
            st->done = brk ? 1u : 0u;
            if (!brk) st->alpha = sh_alpha;
        }
    }
    if (brk) return;
    __syncthreads();
    const double alpha = sh_alpha, na = -alpha;
    double acc = 0.0;
    for (uint32_t i = i0; i < n3;) {
        y[i] = y0 + alpha * d0;
        const double ri = r0 + na * q0;
        r[i] = ri;
        acc += ri * ri;
        i += step;
        if (i < n3) {
            y0 = y[i];
            r0 = r[i];
            d0 = d[i];
            q0 = q[i];
        }
    }
    const double total = block_sum(acc);
    if (threadIdx.x == 0) pr[blockIdx.x] = total;
}

// beta = |r_new|^2 / |r|^2 and the loop test ; d = S (beta d + r)
// (ILSS_CG.h:117-137)
template <bool kBsr>
__global__ void k_node_d_fp64(MeshView<double> m, double* d, const double* __restrict__ r,
                              const double* __restrict__ pr, uint32_t npr, StepScalars* st,
                              cudaGraphConditionalHandle cond, int set_cond)
{
    const bool first = blockIdx.x == 0 && threadIdx.x == 0;
    if (st->done) {
        if (first) {
            st->done_pend = 1;
            if (set_cond) cudaGraphSetConditional(cond, 0u);
        }
        return;
    }
    // one component per thread, or (kBsr) one node; the first loaded ahead of beta
    constexpr int kW = kBsr ? 3 : 1;
    const uint32_t count = kBsr ? m.N : 3 * m.N, i0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    double d0[kW], r0[kW];
    bool f0 = false;
    auto load = [&](uint32_t i) {
#pragma unroll
        for (int k = 0; k < kW; k++) {
            d0[k] = d[kW * (size_t)i + k];
            r0[k] = r[kW * (size_t)i + k];
        }
        f0 = m.fixed[kBsr ? i : i / 3];
    };
    if (i0 < count) load(i0);
    __shared__ double sh_beta;
    const double total = grid_total(pr, npr);
    if (threadIdx.x == 0) {
        sh_beta = total / st->delta_new;
        if (blockIdx.x == 0) {
            st->delta_old = st->delta_new;
            st->beta = sh_beta;
            st->delta_pend = total;
            st->k += 1;
            st->total_iters += 1;
            const bool go = total > st->abs_eps_sq && total > st->delta_target && st->k < st->max_iter;
            st->done_pend = go ? 0u : 1u;
            if (!isfinite(total)) st->status = 3;
            if (set_cond) cudaGraphSetConditional(cond, go ? 1u : 0u);
        }
    }
    __syncthreads();
    const double beta = sh_beta;
    for (uint32_t i = i0; i < count;) {
        double v[kW];
#pragma unroll
        for (int k = 0; k < kW; k++) d[kW * (size_t)i + k] = v[k] = f0 ? 0.0 : beta * d0[k] + r0[k];
        if constexpr (kBsr) bsr_record(m, i, v[0], v[1], v[2]);
        i += step;
        if (i < count) load(i);
    }
}

// v = y ; x += dt y   (Step_QuasiImplicitEuler_v, :1322-1327)
__global__ void k_integrate_fp64(uint32_t N, double dt, double* x, double* v, const double* __restrict__ y,
                                 const StepScalars* st)
{
    if (st->gave_up) return;
    const uint32_t n3 = 3 * N;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += gridDim.x * blockDim.x) {
        const double yi = y[i];
        v[i] = yi;
        x[i] = x[i] + dt * yi;
    }
}

// ---- fully-implicit Euler, Delta x form (LeafDSH_Solid3D_FEM.cpp:1357-1552) ----
// x holds the Newton iterate x_k, xn and vn the step's x^n and v^n; eout holds
// the element forces at x_k (k_elem_force_fp64 with the rotations of x_k).

// b = m g + f_e(x_k) + (inv_dt m) (v^n - inv_dt (x_k - x^n)) with f_p = 0 and
// f_d left out as in the reference (:1382-1401); y = dt v^n on the first
// Newton iteration (the warm start, :1406-1407), else 0.
__global__ void k_node_b_fie_fp64(MeshView<double> m, StepConsts c, const double* __restrict__ x,
                                  const double* __restrict__ xn, const double* __restrict__ vn, int warm,
                                  double* b, double* y)
{
    const double im = c.inv_dt * c.mass;
    const uint32_t a = threadIdx.x & 3u, step = (gridDim.x * blockDim.x) >> 2;
    for (uint32_t n = (blockIdx.x * blockDim.x + threadIdx.x) >> 2; (n & ~7u) < m.N; n += step) {
        const bool on = n < m.N;
        const double f = gather_fp64(m, n, a, on);
        if (!on || a == 3) continue;
        const size_t i = 3 * (size_t)n + a;
        const double g = a == 0 ? c.gravity[0] : (a == 1 ? c.gravity[1] : c.gravity[2]);
        const double bf = c.mass * g - f;
        b[i] = bf + im * (vn[i] - c.inv_dt * (x[i] - xn[i]));
        y[i] = warm ? c.dt * vn[i] : 0.0;
    }
}

// Position constraints as Delta x rows: b = y = target - x_k (:1441-1465).
__global__ void k_knc_fie_fp64(uint32_t N, uint32_t count, const uint32_t* __restrict__ nodes,
                               const double* __restrict__ targets, const double* __restrict__ x, double* b,
                               double* y)
{
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
        const size_t n = bounds_idx(nodes[k], N, kSiteKncNode);
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const double dx = targets[3 * k + a] - x[3 * n + a];
            b[3 * n + a] = dx;
            y[3 * n + a] = dx;
        }
    }
}

// partial sum of v_i^2 (real_array::sq_norm_2)
__global__ void k_sq_norm_fp64(uint32_t n, const double* __restrict__ v, double* partials)
{
    double acc = 0.0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) acc += v[i] * v[i];
    double s = block_sum(acc);
    if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

// x_k += y ; v_k = inv_dt (x_k - x^n) ; partial |y|^2   (:1500-1512)
__global__ void k_fie_update_fp64(uint32_t N, double inv_dt, double* x, double* v, const double* __restrict__ xn,
                                  const double* __restrict__ y, double* partials)
{
    double acc = 0.0;
    const uint32_t n3 = 3 * N;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += gridDim.x * blockDim.x) {
        const double yi = y[i];
        const double xi = x[i] + yi;
        x[i] = xi;
        v[i] = inv_dt * (xi - xn[i]);
        acc += yi * yi;
    }
    double s = block_sum(acc);
    if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

// ---- MINRES (ILSS_MINRES::Solve, ILSS_MINRES.h:51-168), no preconditioner:
// w == v, w1 == v1. The host rotates the v0/v/v1 and p0/p buffers between
// iterations; every kernel is a no-op once the loop has ended.

// v1 = S (b - A y) ; partial |v1|^2   (:66-74)
template <int kKu>
__global__ void k_mr_init_fp64(MeshView<double> m, StepConsts c, const double* __restrict__ b,
                               const double* __restrict__ y, double* v1, double* partials)
{
    double acc = 0.0;
    const double mfm = c.mass * c.factor_M;
    const uint32_t a = threadIdx.x & 3u, step = (gridDim.x * blockDim.x) >> 2;
    for (uint32_t n = (blockIdx.x * blockDim.x + threadIdx.x) >> 2; (n & ~7u) < m.N; n += step) {
        const bool on = n < m.N;
        const double f = node_Ku<kKu>(m, n, a, on);
        if (!on || a == 3) continue;
        const size_t i = 3 * (size_t)n + a;
        const double r = m.fixed[n] ? 0.0 : b[i] - (c.factor_K * f + mfm * y[i]);
        v1[i] = r;
        acc += r * r;
    }
    double s = block_sum(acc);
    if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

// v1 *= 1/beta_new ; v = p = p0 = 0   (:82-95)
__global__ void k_mr_start_fp64(uint32_t N, double* v1, double* v, double* p, double* p0, const StepScalars* st)
{
    const double inv = 1.0 / st->mr_pend.beta_new;
    const uint32_t n3 = 3 * N;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += gridDim.x * blockDim.x) {
        v1[i] *= inv;
        v[i] = 0.0;
        p[i] = 0.0;
        p0[i] = 0.0;
    }
}

// v1 = S A v - beta v0 ; partial v1.v   (:117-123)
template <int kKu>
__global__ void k_mr_q_fp64(MeshView<double> m, StepConsts c, const double* __restrict__ v,
                            const double* __restrict__ v0, double* v1, double* pq, StepScalars* st)
{
    const bool first = blockIdx.x == 0 && threadIdx.x == 0;
    if (st->done_pend) {
        if (first) st->done = 1;
        return;
    }
    const double mfm = c.mass * c.factor_M;
    const double nb = -st->mr_pend.beta_new;
    if (first) {
        st->done = 0;
        st->mr = st->mr_pend;
        st->mr.beta = st->mr_pend.beta_new;
    }
    double acc = 0.0;
    const uint32_t a = threadIdx.x & 3u, step = (gridDim.x * blockDim.x) >> 2;
    for (uint32_t n = (blockIdx.x * blockDim.x + threadIdx.x) >> 2; (n & ~7u) < m.N; n += step) {
        const bool on = n < m.N;
        const double f = node_Ku<kKu>(m, n, a, on);
        if (!on || a == 3) continue;
        const size_t i = 3 * (size_t)n + a;
        const double vi = v[i], qi = m.fixed[n] ? 0.0 : c.factor_K * f + mfm * vi;
        const double w1 = qi + nb * v0[i];
        v1[i] = w1;
        acc += w1 * vi;
    }
    const double total = block_sum(acc);
    if (threadIdx.x == 0) pq[blockIdx.x] = total;
}

// alpha = v1.v ; v1 -= alpha v ; partial |v1|^2   (:123-129)
__global__ void k_mr_v1_fp64(uint32_t N, double* v1, const double* __restrict__ v, const double* __restrict__ pq,
                             uint32_t npq, double* pr, StepScalars* st)
{
    if (st->done_pend) return;
    const double alpha = grid_total(pq, npq), na = -alpha;
    if (blockIdx.x == 0 && threadIdx.x == 0) st->mr.alpha = alpha;
    double acc = 0.0;
    const uint32_t n3 = 3 * N;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += gridDim.x * blockDim.x) {
        const double r = v1[i] + na * v[i];
        v1[i] = r;
        acc += r * r;
    }
    const double total = block_sum(acc);
    if (threadIdx.x == 0) pr[blockIdx.x] = total;
}

// The Givens rotation and the loop test (:131-144) ; v1 *= 1/beta_new ;
// p_new = ((-r2) p + w + (-r3) p0) / r1 into p0's buffer ;
// y += beta_one c eta p_new   (:146-156)
__global__ void k_mr_update_fp64(uint32_t N, double* v1, const double* __restrict__ v,
                                 const double* __restrict__ p, double* p0, double* y, const double* __restrict__ pr,
                                 uint32_t npr, StepScalars* st, cudaGraphConditionalHandle cond, int set_cond)
{
    if (st->done) {
        if (set_cond && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(cond, 0u);
        return;
    }
    __shared__ MinresScalars sh;
    const double total = grid_total(pr, npr);
    if (threadIdx.x == 0) {
        MinresScalars mr = st->mr;
        minres_givens(mr, total);
        sh = mr;
        if (blockIdx.x == 0) {
            st->mr_pend = mr;
            st->delta_new = mr.norm_r_sq;
            st->k += 1;
            st->total_iters += 1;
            const bool go =
                mr.norm_r_sq > st->abs_eps_sq && mr.norm_r_sq > st->delta_target && st->k < st->max_iter;
            st->done_pend = go ? 0u : 1u;
            if (!isfinite(total) || !isfinite(mr.norm_r_sq)) st->status = 3;
            if (set_cond) cudaGraphSetConditional(cond, go ? 1u : 0u);
        }
    }
    __syncthreads();
    const double inv_beta = sh.inv_beta, neg_r2 = sh.neg_r2, neg_r3 = sh.neg_r3, inv_r1 = sh.inv_r1, x_coef = sh.x_coef;
    const uint32_t n3 = 3 * N;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += gridDim.x * blockDim.x) {
        v1[i] *= inv_beta;
        double pn = neg_r2 * p[i] + v[i];
        pn += neg_r3 * p0[i];
        pn *= inv_r1;
        p0[i] = pn;
        y[i] += x_coef * pn;
    }
}

// q = S (factor_M M d + factor_K sum R K R^T d) using a fresh eout
__global__ void k_apply_A_fp64(MeshView<double> m, double factor_M, double factor_K, double mass,
                               const double* __restrict__ d, double* q)
{
    const double mfm = mass * factor_M;
    const uint32_t a = threadIdx.x & 3u, step = (gridDim.x * blockDim.x) >> 2;
    for (uint32_t n = (blockIdx.x * blockDim.x + threadIdx.x) >> 2; (n & ~7u) < m.N; n += step) {
        const bool on = n < m.N;
        const double s = m.records ? gather_fx(m, n, a, on) : gather_fp64(m, n, a, on);
        if (!on || a == 3) continue;
        const size_t i = 3 * (size_t)n + a;
        q[i] = m.fixed[n] ? 0.0 : factor_K * s + mfm * d[i];
    }
}

// Material triple of every element from one E, nu (k_c = a (1 - nu), a nu,
// a (0.5 - nu), formed on the host): mat[c][e] = V_e k_c, the product
// EditableTetrahedronElementSet3::SetParams re-bakes for every element
// (TetrahedronElementSet3.cpp:2168-2200).
__global__ void k_rebake_material_fp64(uint32_t T, const double* __restrict__ vol, double k0, double k1, double k2,
                                       double* mat)
{
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < T; e += gridDim.x * blockDim.x) {
        const double V = vol[e];
        mat[e] = V * k0;
        mat[(size_t)T + e] = V * k1;
        mat[2 * (size_t)T + e] = V * k2;
    }
}

// R = I, det F = 1 until the first evaluation (CreateCache,
// TetrahedronElementSet3.cpp:190-209).
__global__ void k_rest_rotations_fp64(uint32_t T, double* R, double* detF)
{
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < T; e += gridDim.x * blockDim.x) {
#pragma unroll
        for (int c = 0; c < 9; c++) R[c * (size_t)T + e] = c % 4 == 0 ? 1.0 : 0.0;
        detF[e] = 1.0;
    }
}

void launch_rest_rotations_fp64(uint32_t T, double* R, double* detF, cudaStream_t s)
{
    k_rest_rotations_fp64<<<vec_grid(T), row_block(T), 0, s>>>(T, R, detF);
    launch_counter()++;
}

void launch_rebake_material_fp64(uint32_t T, const double* vol, double k0, double k1, double k2, double* mat,
                                 cudaStream_t s)
{
    k_rebake_material_fp64<<<vec_grid(T), row_block(T), 0, s>>>(T, vol, k0, k1, k2, mat);
    launch_counter()++;
}

// f += sign * sum(eout) per node; records: eout holds those of a product
__global__ void k_gather_sum_fp64(MeshView<double> m, double sign, double* f, int records)
{
    const uint32_t a = threadIdx.x & 3u, step = (gridDim.x * blockDim.x) >> 2;
    for (uint32_t n = (blockIdx.x * blockDim.x + threadIdx.x) >> 2; (n & ~7u) < m.N; n += step) {
        const bool on = n < m.N;
        const double s = records ? gather_fx(m, n, a, on) : gather_fp64(m, n, a, on);
        if (on && a < 3) f[3 * (size_t)n + a] += sign * s;
    }
}

// ---- finalizers (one block) ----

__device__ __forceinline__ bool cg_continue(const StepScalars* st)
{
    return st->delta_new > st->abs_eps_sq && st->delta_new > st->delta_target && st->k < st->max_iter;
}

// ILSS_CG::Solve's scalar steps outside its loop (ILSS_CG.h:53-73,146-151) on a
// reduced total: the start, and the statistics at the end. The loop's are in
// the kernels that use them (k_node_xr_fp64, k_node_d_fp64).
__device__ __forceinline__ void fin_init(StepScalars* st, const StepConsts& c, double total)
{
    st->delta_0 = total;
    st->delta_new = total;
    st->delta_old = total;
    st->delta_target = c.rel_eps_sq * total;
    st->abs_eps_sq = c.abs_eps_sq;
    st->max_iter = c.max_iter;
    st->k = 0;
    st->status = 0;
    st->alpha = 0.0;
    st->beta = 0.0;
    st->done = cg_continue(st) ? 0u : 1u;
    st->delta_pend = total;
    st->done_pend = st->done;
    if (!isfinite(total)) st->status = 3;  // FEM_E_NAN
}
__device__ __forceinline__ void fin_stats(StepScalars* st)
{
    st->rel_residual = (st->delta_0 > 0) ? ::sqrt(st->delta_new / st->delta_0) : 0.0;
    st->abs_residual = ::sqrt(st->delta_new);
}

__global__ void k_finalize(int kind, const double* __restrict__ partials, uint32_t count, StepConsts c,
                           StepScalars* st, cudaGraphConditionalHandle cond, int set_cond)
{
    double acc = 0.0;
    for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) acc += partials[i];
    const double total = block_sum(acc);
    if (threadIdx.x != 0) return;
    switch (kind) {
    case FIN_INIT:
        fin_init(st, c, total);
        break;
    case FIN_ENERGY_E:
        st->elastic_energy = total;
        break;
    case FIN_ENERGY_P:
        st->potential_energy = total;
        break;
    case FIN_SUM:
        st->host_sum = total;
        break;
    case FIN_MR_INIT: {
        // |r0|^2 (sq_norm_2 and dot(v1, w1) are the same sum); |b|^2 from the
        // FIN_SUM before; beta_one = |r0| (:74-107)
        MinresScalars& mr = st->mr;
        minres_start(mr, total);
        mr.norm_b_sq = st->host_sum;
        st->delta_0 = mr.norm_b_sq;
        st->delta_target = c.rel_eps_sq * mr.norm_b_sq;
        st->abs_eps_sq = c.abs_eps_sq;
        st->max_iter = c.max_iter;
        st->k = 0;
        st->status = 0;
        st->done = (mr.norm_r_sq > st->abs_eps_sq && mr.norm_r_sq > st->delta_target && st->k < st->max_iter) ? 0u : 1u;
        st->mr_pend = mr;
        st->done_pend = st->done;
        if (!isfinite(total)) st->status = 3;
        break;
    }
    case FIN_MR_STATS:
        st->rel_residual = ::sqrt(st->mr_pend.norm_r_sq / st->mr_pend.norm_b_sq);
        st->abs_residual = ::sqrt(st->mr_pend.norm_r_sq);
        break;
    case FIN_STATS:
        st->delta_new = st->delta_pend;
        fin_stats(st);
        break;
    }
    if (set_cond && (kind == FIN_INIT || kind == FIN_MR_INIT))
        cudaGraphSetConditional(cond, st->done ? 0u : 1u);
}

// ---- launchers ----

// A node kernel in the form of the solid's operator (MeshView).
#define FEMGB_LAUNCH_KU(kernel, m, ...)                                                                              \
    do {                                                                                                             \
        const bool bsr_ = (m).bsr_val != nullptr;                                                                    \
        const uint32_t g_ = node_grid((m).N, bsr_), b_ = node_block((m).N, bsr_);                                    \
        if (bsr_) kernel<kKuBsr><<<g_, b_, 0, s>>>(m, __VA_ARGS__);                                                  \
        else if ((m).records) kernel<kKuRecords><<<g_, b_, 0, s>>>(m, __VA_ARGS__);                                      \
        else kernel<kKuFp64><<<g_, b_, 0, s>>>(m, __VA_ARGS__);                                                      \
        launch_counter()++;                                                                                          \
    } while (0)
#define FEMGB_LAUNCH(kernel, grid, block, ...)                            \
    do {                                                                  \
        kernel<<<(grid), (block), 0, s>>>(__VA_ARGS__);                   \
        launch_counter()++;                                               \
    } while (0)

void launch_elem_bake_fp64(const MeshView<double>& m, cudaStream_t s)
{
    FEMGB_LAUNCH(k_elem_bake_fp64, elem_grid(m.T), elem_block(m.T), m);
}
void launch_elem_spmv_fp64(const MeshView<double>& m, const double* d, const StepScalars* st, int check_done,
                           cudaStream_t s)
{
    prof_begin("elem_spmv_fp64", s);
    FEMGB_LAUNCH(k_elem_spmv_fp64, elem_grid(m.T), elem_block(m.T), m, d, st, check_done);
    prof_end("elem_spmv_fp64", s);
}
void launch_elem_force_fp64(const MeshView<double>& m, const double* x, int write_out, double* energy_partials,
                            cudaStream_t s)
{
    FEMGB_LAUNCH(k_elem_force_fp64, elem_grid(m.T), elem_block(m.T), m, x, write_out, energy_partials);
}
void launch_node_b_fp64(const MeshView<double>& m, const StepConsts& c, const double* v, double* b, double* y,
                        cudaStream_t s)
{
    FEMGB_LAUNCH(k_node_b_fp64, node_grid(m.N, false), node_block(m.N, false), m, c, v, b, y);
}
void launch_knc_fp64(uint32_t N, uint32_t count, const uint32_t* nodes, const double* targets, const double* x,
                     const StepConsts& c, double* b, double* y, cudaStream_t s)
{
    if (count == 0) return;
    FEMGB_LAUNCH(k_knc_fp64, vec_grid(count), row_block(count), N, count, nodes, targets, x, c, b, y);
}
void launch_node_residual_fp64(const MeshView<double>& m, const StepConsts& c, const double* b, const double* y,
                               double* r, double* d, double* partials, cudaStream_t s)
{
    FEMGB_LAUNCH_KU(k_node_residual_fp64, m, c, b, y, r, d, partials);
}
void launch_node_q_fp64(const MeshView<double>& m, const StepConsts& c, const double* d, double* q, double* pq,
                        const StepScalars* st, cudaStream_t s)
{
    prof_begin("node_q_fp64", s);
    FEMGB_LAUNCH_KU(k_node_q_fp64, m, c, d, q, pq, st);
    prof_end("node_q_fp64", s);
}
void launch_node_xr_fp64(const MeshView<double>& m, double* y, double* r, const double* d, const double* q,
                         const double* pq, double* pr, StepScalars* st, cudaStream_t s)
{
    FEMGB_LAUNCH(k_node_xr_fp64, vec_grid(3 * m.N), row_block(3 * m.N), m.N, y, r, d, q, pq,
                 node_grid(m.N, m.bsr_val != nullptr), pr, st);
}
void launch_node_d_fp64(const MeshView<double>& m, double* d, const double* r, const double* pr, StepScalars* st,
                        cudaStream_t s, cudaGraphConditionalHandle cond, int set_cond)
{
    const uint32_t npr = vec_grid(3 * m.N);
    if (m.bsr_val)
        FEMGB_LAUNCH(k_node_d_fp64<true>, vec_grid(m.N), row_block(m.N), m, d, r, pr, npr, st, cond, set_cond);
    else
        FEMGB_LAUNCH(k_node_d_fp64<false>, npr, row_block(3 * m.N), m, d, r, pr, npr, st, cond, set_cond);
}
void launch_integrate_fp64(uint32_t N, double dt, double* x, double* v, const double* y, const StepScalars* st,
                           cudaStream_t s)
{
    FEMGB_LAUNCH(k_integrate_fp64, vec_grid(3 * N), row_block(3 * N), N, dt, x, v, y, st);
}
void launch_node_b_fie_fp64(const MeshView<double>& m, const StepConsts& c, const double* x, const double* xn,
                            const double* vn, int warm, double* b, double* y, cudaStream_t s)
{
    FEMGB_LAUNCH(k_node_b_fie_fp64, node_grid(m.N, false), node_block(m.N, false), m, c, x, xn, vn, warm, b, y);
}
void launch_knc_fie_fp64(uint32_t N, uint32_t count, const uint32_t* nodes, const double* targets, const double* x,
                         double* b, double* y, cudaStream_t s)
{
    if (count == 0) return;
    FEMGB_LAUNCH(k_knc_fie_fp64, vec_grid(count), row_block(count), N, count, nodes, targets, x, b, y);
}
void launch_sq_norm_fp64(uint32_t n, const double* v, double* partials, cudaStream_t s)
{
    FEMGB_LAUNCH(k_sq_norm_fp64, vec_grid(n), row_block(n), n, v, partials);
}
void launch_fie_update_fp64(uint32_t N, double inv_dt, double* x, double* v, const double* xn, const double* y,
                            double* partials, cudaStream_t s)
{
    FEMGB_LAUNCH(k_fie_update_fp64, vec_grid(3 * N), row_block(3 * N), N, inv_dt, x, v, xn, y, partials);
}
void launch_bsr_assemble_fp64(const MeshView<double>& m, const BsrBuild& a, cudaStream_t s)
{
    static_assert(kBsrElemWords == kFxBlockWords, "an element's block words");
    prof_begin("bsr_assemble_fp64", s);
    const uint32_t blocks = capped((m.T + kBsrElemBlock - 1) / kBsrElemBlock, 65535u);
    k_bsr_elements_fp64<<<blocks, kBsrElemBlock, sizeof(long long) * kBsrElemRow * kBsrElemBlock, s>>>(m, a);
    launch_counter()++;
    FEMGB_LAUNCH(k_bsr_slots_fp64, capped((4 * a.groups + 127) / 128, 65535u), 128u, m, a);
    FEMGB_LAUNCH(k_bsr_rows_fp64, capped((node_rows(m.N) + 127) / 128, 65535u), 128u, m, a);
    prof_end("bsr_assemble_fp64", s);
}
void launch_bsr_vector_fp64(const MeshView<double>& m, const double* u, const StepScalars* st, int check_done,
                            cudaStream_t s)
{
    FEMGB_LAUNCH(k_bsr_vector_fp64, vec_grid(m.N), row_block(m.N), m, u, st, check_done);
}
void launch_mr_init_fp64(const MeshView<double>& m, const StepConsts& c, const double* b, const double* y,
                         double* v1, double* partials, cudaStream_t s)
{
    FEMGB_LAUNCH_KU(k_mr_init_fp64, m, c, b, y, v1, partials);
}
void launch_mr_start_fp64(uint32_t N, double* v1, double* v, double* p, double* p0, const StepScalars* st,
                          cudaStream_t s)
{
    FEMGB_LAUNCH(k_mr_start_fp64, vec_grid(3 * N), row_block(3 * N), N, v1, v, p, p0, st);
}
void launch_mr_q_fp64(const MeshView<double>& m, const StepConsts& c, const double* v, const double* v0,
                      double* v1, double* pq, StepScalars* st, cudaStream_t s)
{
    FEMGB_LAUNCH_KU(k_mr_q_fp64, m, c, v, v0, v1, pq, st);
}
void launch_mr_v1_fp64(const MeshView<double>& m, double* v1, const double* v, const double* pq, double* pr,
                       StepScalars* st, cudaStream_t s)
{
    FEMGB_LAUNCH(k_mr_v1_fp64, vec_grid(3 * m.N), row_block(3 * m.N), m.N, v1, v, pq,
                 node_grid(m.N, m.bsr_val != nullptr), pr, st);
}
void launch_mr_update_fp64(uint32_t N, double* v1, const double* v, const double* p, double* p0, double* y,
                           const double* pr, StepScalars* st, cudaStream_t s, cudaGraphConditionalHandle cond,
                           int set_cond)
{
    FEMGB_LAUNCH(k_mr_update_fp64, vec_grid(3 * N), row_block(3 * N), N, v1, v, p, p0, y, pr, vec_grid(3 * N), st,
                 cond, set_cond);
}
void launch_elem_lcm_force_fp64(const MeshView<double>& m, const double* F, const PkMaterial& mat, int write_out,
                                double* energy_partials, cudaStream_t s)
{
    FEMGB_LAUNCH(k_elem_lcm_force_fp64, elem_grid(m.T), elem_block(m.T), m, F, mat, write_out, energy_partials);
}
void launch_elem_lcm_spmv_fp64(const MeshView<double>& m, const double* d, const double* F, const PkMaterial& mat,
                               const StepScalars* st, int check_done, cudaStream_t s)
{
    FEMGB_LAUNCH(k_elem_lcm_spmv_fp64, elem_grid(m.T), elem_block(m.T), m, d, F, mat, st, check_done);
}
void launch_potential_fp64(const MeshView<double>& m, const StepConsts& c, const double* x, double* partials,
                           cudaStream_t s)
{
    FEMGB_LAUNCH(k_potential_fp64, elem_grid(m.T), elem_block(m.T), m, c, x, partials);
}
void launch_apply_A_fp64(const MeshView<double>& m, double factor_M, double factor_K, double mass,
                         const double* d, double* q, cudaStream_t s)
{
    FEMGB_LAUNCH(k_apply_A_fp64, node_grid(m.N, false), node_block(m.N, false), m, factor_M, factor_K, mass, d, q);
}
void launch_gather_sum_fp64(const MeshView<double>& m, double sign, double* f, bool records, cudaStream_t s)
{
    FEMGB_LAUNCH(k_gather_sum_fp64, node_grid(m.N, false), node_block(m.N, false), m, sign, f, records ? 1 : 0);
}
void launch_finalize(int kind, const double* partials, uint32_t count, const StepConsts& c, StepScalars* st,
                     cudaStream_t s, cudaGraphConditionalHandle cond, int set_cond)
{
    k_finalize<<<1, kFinalizeThreads, 0, s>>>(kind, partials, count, c, st, cond, set_cond);
    launch_counter()++;
}

FEMGB_BOUNDS_ACCESSOR(bounds_read_fem_kernels)

}  // namespace femgb

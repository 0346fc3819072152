// fem_device.cuh -- device-side data layout and launcher declarations shared
// by the kernels (fem_kernels.cu, rotation.cu) and the host runtime (solid.cu).
//
// Layout in HBM for one solid (T tets, N nodes):
//   tets      int4[T]          node ids of each tet
//   Dinv      S[9][T]          Dm^-1 of each tet, row-major, component-major
//                              arrays (coalesced per component)
//   mat       S[3][T]          V*(lambda+2mu), V*lambda, V*mu of each tet (the
//                              entries a_k1, a_nu, a_k2 of the reference's E
//                              matrix, TetrahedronElement3.h:141-156, times V)
//   R         S[9][T]          cached rotation, detF double[T]
//   node vectors (x, v, y, b, r, d, q, rest): AoS xyz, 3N scalars, the
//                              reference's Vec3 array layout
//   eout      S[T][4][3]       per-element nodal products, gathered per node
//   csr_ptr/csr_idx            node -> (4*e + slot) entries in element order,
//                              the order the reference scatters in
//   fixed     uint8[N]         1 where a kinematic node constraint zeroes the row
// S is double on the FP64 path and float on the mixed path.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "lcm.cuh"
#include "rows_plan.h"

namespace femgb {

// MINRES recurrence scalars (ILSS_MINRES::Solve, ILSS_MINRES.h:51-168).
struct MinresScalars {
    double norm_r_sq, norm_b_sq;     // |r|^2 carried by the Givens sines; |b|^2
    double beta, beta_new, beta_one;  // Lanczos norms (beta_one: of the initial residual)
    double alpha;
    double c, c_old, s, s_old, eta;   // Givens rotation state
    double inv_beta, neg_r2, neg_r3, inv_r1, x_coef;  // this iteration's update coefficients
};

// Device-resident CG and step scalars of one solid.
struct StepScalars {
    double delta_new, delta_old, delta_0, delta_target, abs_eps_sq;
    double alpha, beta, dot_dq;
    double elastic_energy, potential_energy;
    double rel_residual, abs_residual;
    uint32_t k, max_iter, done, status;
    uint32_t inverted, fp64_resolved, refresh_every;
    float beta_f;       // beta rounded to FP32 (mixed path)
    uint32_t finished;      // batch: the CG loop ended during this launch (cleared at launch start)
    uint32_t refresh_next;  // mixed: the next iteration recomputes r = b - A y in FP64
    double delta_refresh;   // mixed: |r|^2 right after the last FP64 residual
    uint32_t k_refresh;
    uint32_t confirm;       // mixed: this iteration only measures the FP64 residual (exit test)
    float alpha_f;          // mixed: this iteration's alpha in FP32 (0 on a confirm iteration)
    uint32_t brk;           // mixed: this iteration breaks down (|d.q| < abs^2) and leaves the loop
    uint32_t mr_pending;    // batch MINRES: 1 = this iteration's vector and iterate update is due,
                            // 2 = the start (or restart) residual is to be normalised
    // batch: the step's Newton level (QIE meshes make one pass of it)
    uint32_t nr_go;         // takes part in the next start section (b, constraints, r0)
    uint32_t nr_k;          // FIE: Newton iterations of this step so far
    uint32_t nr_solved;     // FIE: some linear solve ran in this step
    uint32_t step_done;     // the step ended during this launch (energy, completion flag)
    uint32_t fie_cg;        // FIE: linear-solver iterations summed over this step's Newton iterations
    double nr_delta0;       // FIE: |b_0| of this step
    double nr_abs;          // FIE: the last |b_k| or |y_k|
    unsigned long long total_iters;
    double host_sum;        // FIE: the last FIN_SUM total (|b_k|^2 or |y_k|^2), read by the host
    MinresScalars mr;       // MINRES solver state (FP64 solid)
    // mixed: rotations of this step by cause of their double-precision
    // re-solve: det F <= degenerate_det_F (FP64 MSVD), a nearly isotropic
    // F^T F (FP64 MSVD in place of double-float), and with FP32 rotations an
    // MSVD branch near a tie or a failed sensitivity check
    uint32_t res_det_F, res_isotropic, res_tie, res_check;
    // FP64 solid's step loops: the state after the running iteration. An
    // iteration's kernels read either the committed fields above or these,
    // never ones that another block of the same kernel writes: the last
    // kernel of an iteration writes these, an early kernel of the next one
    // commits them.
    double delta_pend;
    MinresScalars mr_pend;
    uint32_t done_pend;
    // FP64 solid: a wait of the resident solve gave up; stays until the host
    // has read it, and no step is integrated in the meantime
    uint32_t gave_up;
};

// One MINRES iteration's Givens rotation and update coefficients from
// |v1|^2 after the Lanczos step (ILSS_MINRES.h:131-156): beta_new, the
// rotation (c, s), the coefficients of the direction and iterate updates,
// and the residual norm carried by the sines.
__device__ __forceinline__ void minres_givens(MinresScalars& mr, double beta_new_sq)
{
    mr.beta_new = ::sqrt(beta_new_sq);
    mr.inv_beta = 1.0 / mr.beta_new;
    const double r2 = mr.s * mr.alpha + mr.c * mr.c_old * mr.beta;
    const double r3 = mr.s_old * mr.beta;
    const double r1_hat = mr.c * mr.alpha - mr.c_old * mr.s * mr.beta;
    const double r1 = ::sqrt(r1_hat * r1_hat + beta_new_sq);
    mr.c_old = mr.c;
    mr.s_old = mr.s;
    mr.c = r1_hat / r1;
    mr.s = mr.beta_new / r1;
    mr.neg_r2 = -r2;
    mr.neg_r3 = -r3;
    mr.inv_r1 = 1.0 / r1;
    mr.x_coef = mr.beta_one * mr.c * mr.eta;
    mr.norm_r_sq *= mr.s * mr.s;
    mr.eta = -mr.s * mr.eta;
}

// MINRES start from the residual r0 (ILSS_MINRES.h:74-107): |r0|^2 and the
// Givens state of an empty Lanczos basis.
__device__ __forceinline__ void minres_start(MinresScalars& mr, double r0_sq)
{
    mr.norm_r_sq = r0_sq;
    mr.beta_new = ::sqrt(r0_sq);
    mr.beta_one = mr.beta_new;
    mr.inv_beta = 1.0 / mr.beta_new;
    mr.c = 1.0; mr.c_old = 1.0; mr.s = 0.0; mr.s_old = 0.0; mr.eta = 1.0;
}

template <typename S>
struct MeshView {
    uint32_t N, T;
    const int4* tets;
    const S* Dinv;     // [9][T]
    const S* mat;      // [3][T]
    S* R;              // [9][T]
    double* detF;      // [T]
    const double* vol; // [T]
    const double* rest;          // [3N] (double)
    const uint32_t* csr_ptr;     // [N+1]
    const uint32_t* csr_idx;     // [4T]
    const uint8_t* fixed;        // [N]
    S* eout;                     // [12T]
    // FP64 solid: the assembled stiffness K = sum_e R K0 R^T as 3x3 blocks of
    // fixed-point entries (fx.cuh), rows padded to groups of four blocks: the
    // groups' row starts [N+1], columns [4 groups] (a pad: the row itself with
    // a zero block), entries [group][9][4], each row's exponent [N] (units
    // 2^x); and the vector a product reads, a 32-byte record per node (three
    // integers in units of 2^(e - 1081), e). When set, the solvers' node
    // kernels take K u from it instead of gathering the element outputs.
    const uint32_t* bsr_row = nullptr;
    const uint32_t* bsr_col = nullptr;
    const int2* bsr_val = nullptr;
    const int32_t* bsr_x = nullptr;
    longlong2* bsr_u = nullptr;  // [2 N]
    // FP64 solid, C_WRP: each element's fixed-point product matrix (fx.cuh),
    // kFxGroups 16-byte groups of two entries, the last group's second half
    // the scale, [T / 32][kFxGroups][32] (a warp's groups at fixed offsets);
    // null without the memory for them (every element then runs in FP64).
    // records: eout holds fixed-point records of the product instead of
    // doubles. fx_guard: log2 of the largest
    // number of element corners at a node, rounded up.
    int4* Kfx = nullptr;
    uint32_t records = 0;
    uint32_t fx_guard = 0;
    const float* grade = nullptr;  // [T] max|Dm| max|Dm^-1| of the rest shape
};
constexpr uint32_t kFxGroups = 23;

struct StepConsts {
    double dt, inv_dt, mass, factor_M, factor_K;
    double gravity[3];
    double density;
    double rel_eps_sq, abs_eps_sq;
    uint32_t max_iter;
};

constexpr int kBlock = 256;
constexpr int kFinalizeThreads = 512;

// ---- launchers (fem_kernels.cu / rotation.cu) ----
void launch_begin_eval_fp64(const MeshView<double>& m, const double* x, double* F_out, StepScalars* st,
                            cudaStream_t s);
struct DapdParams;
void launch_begin_eval_dapd_fp64(const MeshView<double>& m, const double* xprev, const double* x, uchar2* doc,
                                 const DapdParams& p, double* F_out, StepScalars* st, cudaStream_t s);
// Bakes every element's fixed-point product matrix (m.Kfx) from its rotation,
// shape gradients and material.
void launch_elem_bake_fp64(const MeshView<double>& m, cudaStream_t s);
void launch_elem_spmv_fp64(const MeshView<double>& m, const double* d, const StepScalars* st, int check_done,
                           cudaStream_t s);
void launch_elem_force_fp64(const MeshView<double>& m, const double* x, int write_out, double* energy_partials,
                            cudaStream_t s);
void launch_node_b_fp64(const MeshView<double>& m, const StepConsts& c, const double* v, double* b, double* y,
                        cudaStream_t s);
void launch_knc_fp64(uint32_t N, uint32_t count, const uint32_t* nodes, const double* targets, const double* x,
                     const StepConsts& c, double* b, double* y, cudaStream_t s);
void launch_node_residual_fp64(const MeshView<double>& m, const StepConsts& c, const double* b, const double* y,
                               double* r, double* d, double* partials, cudaStream_t s);
// The solvers' reductions are added where they are used: a kernel leaves one
// partial per block, and every block of the next kernel adds them all (the
// same sum in each) and takes the scalar step (alpha; beta and the loop
// test). Against a last-block finish (fence, ticket, a second round trip)
// that took 3.5 us off node_q and 3 us off node_xr at 20,480 tets. pq, pr:
// the partials of d.q and |r|^2 (node_grid(N) and vec_grid(3 N) of them).
// With set_cond the iteration's last kernel sets the step graph's WHILE
// condition.
void launch_node_q_fp64(const MeshView<double>& m, const StepConsts& c, const double* d, double* q, double* pq,
                        const StepScalars* st, cudaStream_t s);
void launch_node_xr_fp64(const MeshView<double>& m, double* y, double* r, const double* d, const double* q,
                         const double* pq, double* pr, StepScalars* st, cudaStream_t s);
// (with the assembled stiffness also the records of d)
void launch_node_d_fp64(const MeshView<double>& m, double* d, const double* r, const double* pr, StepScalars* st,
                        cudaStream_t s, cudaGraphConditionalHandle cond = 0, int set_cond = 0);
// (nothing once a solve has given up)
void launch_integrate_fp64(uint32_t N, double dt, double* x, double* v, const double* y, const StepScalars* st,
                           cudaStream_t s);
// Fully-implicit Euler (Newton on Delta x) pieces, FP64 solid path.
void launch_node_b_fie_fp64(const MeshView<double>& m, const StepConsts& c, const double* x, const double* xn,
                            const double* vn, int warm, double* b, double* y, cudaStream_t s);
void launch_knc_fie_fp64(uint32_t N, uint32_t count, const uint32_t* nodes, const double* targets, const double* x, double* b,
                         double* y, cudaStream_t s);
void launch_sq_norm_fp64(uint32_t n, const double* v, double* partials, cudaStream_t s);
void launch_fie_update_fp64(uint32_t N, double inv_dt, double* x, double* v, const double* xn, const double* y,
                            double* partials, cudaStream_t s);
// C_LCM material (FP64 solid): element force and/or energy from the stored F,
// and the truncated differential of d.
void launch_elem_lcm_force_fp64(const MeshView<double>& m, const double* F, const PkMaterial& mat, int write_out,
                                double* energy_partials, cudaStream_t s);
void launch_elem_lcm_spmv_fp64(const MeshView<double>& m, const double* d, const double* F, const PkMaterial& mat,
                               const StepScalars* st, int check_done, cudaStream_t s);
// MINRES (FP64 solid). v1 = S (b - A y) and partial |v1|^2 from a fresh eout of y.
void launch_mr_init_fp64(const MeshView<double>& m, const StepConsts& c, const double* b, const double* y,
                         double* v1, double* partials, cudaStream_t s);
// v1 *= 1/beta_new ; v = p = p0 = 0
void launch_mr_start_fp64(uint32_t N, double* v1, double* v, double* p, double* p0, const StepScalars* st,
                          cudaStream_t s);
// v1 = S A w - beta v0 (w = v, eout of v) ; partial v1.v
void launch_mr_q_fp64(const MeshView<double>& m, const StepConsts& c, const double* v, const double* v0,
                      double* v1, double* pq, StepScalars* st, cudaStream_t s);
// alpha = v1.v ; v1 -= alpha v ; partial |v1|^2
void launch_mr_v1_fp64(const MeshView<double>& m, double* v1, const double* v, const double* pq, double* pr,
                       StepScalars* st, cudaStream_t s);
// |v1|^2, the Givens rotation and the loop test, then
// v1 /= beta_new ; p0 <- (w - r2 p - r3 p0) / r1 (the new p, in p0's buffer) ; y += coef p_new
void launch_mr_update_fp64(uint32_t N, double* v1, const double* v, const double* p, double* p0, double* y,
                           const double* pr, StepScalars* st, cudaStream_t s, cudaGraphConditionalHandle cond = 0,
                           int set_cond = 0);
void launch_potential_fp64(const MeshView<double>& m, const StepConsts& c, const double* x, double* partials,
                           cudaStream_t s);
void launch_apply_A_fp64(const MeshView<double>& m, double factor_M, double factor_K, double mass,
                         const double* d, double* q, cudaStream_t s);
void launch_gather_sum_fp64(const MeshView<double>& m, double sign, double* f, bool records, cudaStream_t s);
void launch_rest_rotations_fp64(uint32_t T, double* R, double* detF, cudaStream_t s);
void launch_rebake_material_fp64(uint32_t T, const double* vol, double k0, double k1, double k2, double* mat,
                                 cudaStream_t s);

// finalizers: one block, fixed-order sums of `count` block partials
enum FinalizeKind {
    FIN_INIT = 0, FIN_ENERGY_E = 3, FIN_ENERGY_P = 4, FIN_STATS = 5,
    FIN_SUM = 6,  // host_sum = total
    // MINRES: init (|r0|^2 = total, |b|^2 from host_sum), stats
    FIN_MR_INIT = 7, FIN_MR_STATS = 8
};
// set_cond: the solvers' starts also set the step graph's WHILE condition `cond` to
// "the loop goes on"
void launch_finalize(int kind, const double* partials, uint32_t count, const StepConsts& c, StepScalars* st,
                     cudaStream_t s, cudaGraphConditionalHandle cond = 0, int set_cond = 0);

// The assembled stiffness (MeshView::bsr_*) of the current rotations. The
// elements' corner blocks go to eblk ([T][kBsrElemWords], their exponents to
// ex); block slot s then sums, in element order, its contributions
// contrib[cptr[s] .. cptr[s+1]) = element << 4 | li << 2 | lj; last the rows
// are brought to one exponent each and get their diagonal blocks.
constexpr uint32_t kBsrElemWords = 78;
struct BsrBuild {
    uint32_t groups;
    const uint32_t *cptr, *contrib;
    long long* eblk;
    int32_t* ex;
    int2* val;
    int32_t* x;
};
void launch_bsr_assemble_fp64(const MeshView<double>& m, const BsrBuild& a, cudaStream_t s);
// The records (bsr_u) of the vector the next product multiplies.
void launch_bsr_vector_fp64(const MeshView<double>& m, const double* u, const StepScalars* st, int check_done,
                            cudaStream_t s);

// The tables of both made on the device (rows_build.cu). most: entries of the
// longest row (kRowEntries at most); launch_row_lengths gives each row's columns
// and, in groups of four, the row starts.
struct LayoutShape;
struct LayoutRows;
struct LayoutOut;
void launch_row_lengths(const MeshView<double>& m, uint32_t most, uint32_t* used, uint32_t* row, cudaStream_t s);
void launch_row_write(const MeshView<double>& m, uint32_t most, const uint32_t* used, const uint32_t* row, uint32_t* col,
                      uint32_t* cptr, uint32_t* contrib, cudaStream_t s);
void launch_layout_count(const LayoutShape& s, uint32_t blocks, const LayoutRows& m, CgRowsCount* count, cudaStream_t st);
void launch_layout_write(const LayoutShape& s, uint32_t blocks, const LayoutRows& m, const LayoutOut& o, cudaStream_t st);

// The solve on resident rows (cg_rows.cu): the layout's tables (rows_plan.h).
struct CgRowsView {
    const CgRowsBlock* blk;
    const uint32_t *node, *group, *slot, *halo, *owner;
    const uint16_t* col;
    ulonglong2* words;  // [3 N]: r for other clusters
    ulonglong2* parts;  // [2][blocks][clusters]: the clusters' sums
    uint32_t cluster, warps, npb, units, records;  // CgRowsPlan's
    uint32_t* seq;  // the last number used
    uint32_t polls;  // of a word that is not there yet, before the wait gives up
};
// The blocks of the plan's shape that are resident together; 0 when it does not launch.
uint32_t cg_rows_max_blocks(const CgRowsPlan& p);
cudaError_t launch_cg_rows_fp64(const MeshView<double>& m, const StepConsts& c, const CgRowsPlan& plan,
                                const CgRowsView& p, bool minres, const double* b, double* y, StepScalars* st,
                                cudaStream_t s);

// Launch shapes of the grid-stride kernels. One FP64 instruction of a warp
// holds its sub-partition for 64 clocks, so small launches spread one warp
// per block until every sub-partition of the 152 SMs has one.
constexpr uint32_t kSubPartitions = 608;
inline uint32_t elem_block(uint32_t T) { return T <= 32 * kSubPartitions ? 32u : (T <= 64 * kSubPartitions ? 64u : 128u); }
inline uint32_t capped(uint32_t g, uint32_t cap) { return g < 1 ? 1 : (g > cap ? cap : g); }
inline uint32_t elem_grid(uint32_t T) { return capped((T + elem_block(T) - 1) / elem_block(T), 4096u); }
// Node kernels (four lanes per node) and vector kernels (one per component):
// 128 threads until every SM has two blocks, then 512 (the assembled rows'
// kernels, which hold more registers, 256); at most three, two or four blocks
// per SM, so that a block adds few of the previous kernel's partials per
// thread.
inline uint32_t row_block(uint32_t n) { return n <= 304u * 128u ? 128u : 512u; }
inline uint32_t vec_grid(uint32_t n) { return capped((n + row_block(n) - 1) / row_block(n), 304u); }
inline uint32_t node_rows(uint32_t N) { return 4u * (N < (1u << 29) ? N : (1u << 29)); }
inline uint32_t node_block(uint32_t N, bool bsr) { return bsr ? (row_block(node_rows(N)) == 128u ? 128u : 256u) : row_block(node_rows(N)); }
inline uint32_t node_grid(uint32_t N, bool bsr)
{
    const uint32_t b = node_block(N, bsr);
    return capped((node_rows(N) + b - 1) / b, bsr ? 608u : 456u);
}
uint64_t& launch_counter();       // kernels launched by this library

// Optional per-kernel timing with CUDA events recorded on the launching
// stream around each launch of a named kernel (off unless enabled).
void prof_begin(const char* name, cudaStream_t s);
void prof_end(const char* name, cudaStream_t s);
bool prof_enabled();
}  // namespace femgb

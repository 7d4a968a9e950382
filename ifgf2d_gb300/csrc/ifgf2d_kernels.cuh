// ifgf2d_kernels.cuh -- device data layouts and kernel launchers of the forward map.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace ifgf {

// Curve on the device (twin of HostCurve, Geometry/Curve.hpp:106-161)
struct DevCurve {
    int type;
    int pad;
    double p[16];
};

// One rectangular-polar column: a target point (singular or near-singular) on a patch
struct RPColumn {
    int patch;
    int pad;
    double tsing, xs, ys;
};

struct DevPatch {
    double t1, t2;
    int curve, ist1, ist2, pad;
};

// Leaf cone interpolation node: position and 1/(e^{ikr}/sqrt r) at the node radius
struct LeafNode {
    double x, y;
    double ir, ii;
};

// complex vector type of a real type
template <typename R> struct Cx;
template <> struct Cx<double> { using V = double2; };
template <> struct Cx<float> { using V = float2; };
template <typename R> using V2 = typename Cx<R>::V;

// one (target, level, cousin) interpolation term: cone id, Chebyshev (s, theta), e^{ikr}/sqrt r
template <typename R> struct InterpE;
template <> struct InterpE<double> { int cone; int pad; double s, th, fr, fi; };
template <> struct InterpE<float> { int cone; float s, th, fr, fi; };
// batched complex64 interpolation term, grouped by leaf box and cone: cone id, Morton target,
// (s, theta), factor
struct InterpG { int cone; int t; float s, th, fr, fi; };
// the FP64 form of the same, (s, theta) as fixed-point weights (fixpoint.cuh)
struct InterpX { int cone; int pad; long long s, th; double fr, fi; };
// cone coefficients of the single-vector apply: complex64, or fixed-point limbs (re.h, re.l, im.h,
// im.l) with one exponent per cone (fixpoint.cuh) in the FP64 form; and the terms that read them
template <typename R> struct CoefOf;
template <> struct CoefOf<double> { using T = int4; };
template <> struct CoefOf<float> { using T = float2; };
template <typename R> using CoefT = typename CoefOf<R>::T;
// one (parent cone, child, node) propagation term: child cone id, (s, theta), factor ratio
template <typename R> struct PropE;
template <> struct PropE<float> { int child_cone; float s, th, wr, wi; };
// batched propagation term: the parent node pt it feeds, then as PropE.  A parent's terms are
// sorted by child cone, so a warp loads each child cone's coefficients once per parent.
template <typename R> struct PropB;
template <> struct PropB<float> { int child_cone; int pt; float s, th, wr, wi; };
using InterpEntryD = InterpE<double>;
// the FP64 propagation plan, array by array (each lane's loads are whole vectors, coalesced): child
// cone, its slot in its group's staged list (launch_stage_plan), (s, theta) as fixed-point weights,
// factor ratio
struct PlanX { int* child; unsigned short* slot; longlong2* st; double2* w; };

constexpr int kMaxP = 64;          // Ps * Pang limit of the device interpolator

// ---------------- setup kernels ----------------
// keta, when given, holds (k, eta) per item (per column, leaf box or leaf cone) and overrides the
// scalar k and eta: a group of obstacles with their own wavenumbers sets up in one launch.
void launch_rp_precompute(const RPColumn* cols, int ncols, const DevPatch* patches, const DevCurve* curves,
                          const double* ns_nodes, const double* ns_weights, int Np, double p, double k,
                          int form, double eta, double2* M, cudaStream_t s, const double2* keta = nullptr);
void launch_rp_fold(const double2* M, const RPColumn* cols, int ncols, const double* edge_jac, const DevPatch* patches,
                    int Np, double2* W, cudaStream_t s);
void launch_near_setup(const int* leaf_start, const int* leaf_count, const int* nbr_ptr, const int* nbr_box,
                       const long long* near_off, int nleaf, const double* xs, const double* ys,
                       const double* nxs, const double* nys, const int* patch_s, const int* nsp_ptr,
                       const int* nsp, double k, int form, double eta, double2* near, cudaStream_t s,
                       const double2* keta = nullptr);
// leaf-cone tables: Green values at the cone nodes times 1/factorization, mapped to Chebyshev
// coefficients with the separable map Gsep (Ps x Ps radial, then Pang x Pang angular);
// Ps * Pang <= 64
void launch_leaf_setup(const int* cone_box, int ncones, const int* leaf_start, const int* leaf_count,
                       const long long* leaf_off, const LeafNode* nodes, const double* xs, const double* ys,
                       const double* nxs, const double* nys, int Ps, int Pang, double k, int form, double eta,
                       const double* Gsep, double2* L, cudaStream_t s, const double2* keta = nullptr);

// ---------------- per-apply kernels ----------------
// y = singular correction (+ half * x: the jump term of the combined formulation)
void launch_sing_apply(const double2* x, const double2* W, const int* row_ptr, const int* row_col,
                       const RPColumn* cols, int N, int Np, double half, double2* y, cudaStream_t s);
// the same, also writing the quadrature-weighted density to rho64 or rho32 at inv[o] (or o)
void launch_sing_intens(const double2* x, const double2* W, const int* row_ptr, const int* row_col,
                        const RPColumn* cols, int N, int Np, double half, double2* y, const double* wq,
                        const long long* inv, double2* rho64, float2* rho32, cudaStream_t s);
// sources with unit normals snx, sny (NULL for the single layer); form 0 single layer, 2 combined
void launch_direct_far(const double* tx, const double* ty, int ntarget, const int* t_patch, const int* t_nsp_ptr,
                       const int* t_nsp, const double* sx, const double* sy, const double* snx, const double* sny,
                       const int* s_patch, const double2* rho, int nsource, double k, int form, double eta, double2* y,
                       int accumulate, cudaStream_t s);

// precision-templated IFGF apply (ifgf_apply.cu); R = double (plain) or float (mixed)
template <typename R>
void launch_intensities_t(const double2* x, const double* wq, const long long* perm, int N, V2<R>* rho, cudaStream_t s);
// leaf cones; chunks: the threads that share a coefficient's sum.  complex64: per cone its table offset
// (two ints), first source and sources.  An item of the FP64 form is up to leaf_item_cones cones of one
// leaf box: the table offset of the first, its local index, how many, and the box's sources.
struct LeafItem { long long off; int cone, cones, first, n; };
int leaf_item_cones(int P);
void launch_leaf_apply_t(const int4* cones, int ncones, int cone_base, const float2* L, const float2* rho, int P, float2* coef,
                         cudaStream_t s, int chunks = 5);
// the FP64 form in fixed point (fixpoint.cuh): the table and its exponents [cone][coefficient] from
// launch_leaf_fix (in place of the FP64 table; l32, when not null, receives the complex64 copy)
void launch_leaf_fx(const LeafItem* items, int nitems, int cone_base, const int4* L, const int* lexp, const double2* rho, int P, int Ps,
                    int4* coef, int* cexp, cudaStream_t s, int chunks);
void launch_leaf_fix(const int* cone_box, int ncones, const int* leaf_count, const long long* leaf_off, int P, int4* L, int* lexp,
                     float2* l32, cudaStream_t s);
// complex64 leaf cones with the table streamed through shared memory by TMA bulk copies
// (P = 25); false when not launched (other P, or leaf_tma_init not run).  *err is set when a
// completion wait runs out.  leaf_tma_init sets the kernel's shared-memory attribute (outside
// stream capture).  The table array must carry 16 bytes of padding after its end.
bool launch_leaf_tma(const int* cone_box, int ncones, int cone_base, const int* leaf_start, const int* leaf_count,
                     const long long* leaf_off, const float2* L, const float2* rho, int P, float2* coef, int* err, int nsm,
                     cudaStream_t s);
cudaError_t leaf_tma_init();
// the propagation variant that stages child coefficient blocks in shared memory (k_propagate_st);
// other values of cones_per_block: 2, 4, or 0 for the most that fit 256 threads
constexpr int kPropStaged = 1;
void launch_propagate_t(int pbegin, int pend, const long long* pp_ptr, const int* pp_nchild, const PropE<float>* pp, int Ps,
                        int Pang, const float* Gsep, float2* coef, cudaStream_t s, int cones_per_block = 0);
// the FP64 form in fixed point: GsepX the separable map's entries as limbs, cexp the cones' exponents,
// stage the records of the level's groups of parents, which launch_stage_plan fills for all levels together
// with pp.slot
struct StageLevels {
    static constexpr int most = 24;             // the deepest tree
    int n = 0, begin[most] = {}, end[most] = {}, group[most + 1] = {};     // parents, first group of each level
    size_t add(int b, int e, int Ps, int Pang);       // one more level, parents [b, e): where its records start
    size_t size(int Ps, int Pang) const;              // ints of all records
};
void launch_stage_plan(const StageLevels& L, const long long* pp_ptr, PlanX pp, int Ps, int Pang, int* stage, cudaStream_t s);
void launch_propagate_fx(int pbegin, int pend, PlanX pp, const int* stage, int Ps, int Pang, const int2* GsepX, int4* coef, int* cexp,
                         cudaStream_t s);
// n doubles in [-1, 1] as fixed-point limbs; the interpolation plan with (s, theta) as weights
void launch_fx_weights(const double* in, int n, int2* out, cudaStream_t s);
void launch_interp_fx(const InterpE<double>* in, long long n, InterpX* out, cudaStream_t s);
void launch_final_t(int N, const int* point_leaf, const int* leaf_start, const int* near_src_off, const int* near_src,
                    const int* near_rowlen, const long long* near_off, const float2* near, const float2* rho, const int* ip_ptr,
                    const InterpE<float>* ip, const float2* coef, int Ps, int Pang, const long long* sorting, double2* y,
                    cudaStream_t s);
// the FP64 form in fixed point, near field and interpolation by leaf box: a record per box and up to
// kFinTargets of its targets, the near table and its exponents per target from launch_near_fix (in place
// of the FP64 table, with the complex64 copy n32), the plan box-transposed (launch_interp_transpose)
constexpr int kFinTargets = 20;
struct FinItem {
    long long near;            // first near-field table entry of the item's first target
    int first, cnt, n;         // first Morton target, targets, targets of the box
    int ip, nt;                // plan: the box's first entry plus the first target's place in it; terms per target
    int rl, src, pad;          // near-field row: sources, their list
};
void launch_final_fx(const FinItem* items, int nitems, const int* near_src, const int4* near, const int* nexp, const double2* rho,
                     PlanX ip, const int4* coef, const int* cexp, int Ps, int Pang, const long long* sorting, double2* y,
                     cudaStream_t s);
void launch_near_fix(int N, const int* point_leaf, const int* leaf_start, const int* near_rowlen, const long long* near_off, int4* near,
                     int* nexp, float2* n32, cudaStream_t s);
// the complex64 form: pieces of kIbPiece terms, near-field sums by kNearChunk sources, fin_targets of a
// box's targets (nt terms each) to an item
constexpr int kIbPiece = 8, kNearChunk = 1024, kFinTargetsMax = 32, kFinParts = 1024;
inline int fin_targets(int nt) {
    const int npc = (nt + kIbPiece - 1) / kIbPiece, t = npc ? kFinParts / npc : kFinTargetsMax;
    return t < 1 ? 1 : t > kFinTargetsMax ? kFinTargetsMax : t;
}
void launch_final_q(const FinItem* items, int nitems, const int* near_src, const float2* near, const float2* rho,
                    const InterpE<float>* ipT, const float2* coef, int Ps, int Pang, const long long* sorting, double2* y, cudaStream_t s);
// the interpolation plan box-transposed (term j of box target t at the box's first entry + j n + t), in
// complex64 and as px (child the cone, w the factor)
void launch_interp_transpose(int N, const int* point_leaf, const int* leaf_start, const int* leaf_count, const int* ip_ptr,
                             const InterpE<double>* in, InterpE<float>* out, PlanX px, cudaStream_t s);
void launch_d2f(const double2* a, long long n, float2* b, cudaStream_t s);
// Load the direct map's kernels (singular correction, FP64 intensities, both far-sum shapes) into
// the current device's context now.  Under lazy module loading a kernel is otherwise loaded,
// with a device allocation for its code, on its first launch.
cudaError_t preload_direct_kernels();
cudaError_t preload_intensities_kernel();
// direct path intensities (patch order), as in ForwardMap::compute_intensities
inline void launch_intensities(const double2* x, const double* wq, const long long* perm, int N, double2* rho, cudaStream_t s) {
    launch_intensities_t<double>(x, wq, perm, N, rho, s);
}

// terms of the batched FP64 form, sorted by cone within a list: cone and node (or target of the work
// item), factor, and the Chebyshev values T_1.. of s, then of theta, as fixed-point limbs
// (batch_x_rows int4 per term)
struct TermsX { int2* id; double2* w; int4* rows; };

// ---------------- batched apply (ifgf_batch.cu) ----------------
// A batch of B right-hand sides is held interleaved, [N][B] (RHS index fastest); cone
// coefficients likewise [cone][P][B].  One warp serves 32 right-hand sides of one row, cone or
// target, so every table entry is read once per 32 right-hand sides.
constexpr int kMaxBatch = 64;      // right-hand sides per batched apply (larger batches are chunked)
void launch_interleave(const double2* x, long long N, int B, double2* xt, cudaStream_t s);     // [B][N] -> [N][B]
void launch_deinterleave(const double2* xt, long long N, int B, double2* x, cudaStream_t s);   // [N][B] -> [B][N]
// rho32 given: the mixed form (complex64 densities xt32 and weights W32, FP32 sums); else FP64
// with xt and W.  The jump term and the intensities use xt.
void launch_sing_b(const double2* xt, const float2* xt32, const double2* W, const float2* W32, const int* row_ptr,
                   const int* row_col, const RPColumn* cols, int N, int Np, int B, double half, double2* yt,
                   const double* wq, const long long* inv, double2* rho64, float2* rho32, cudaStream_t s);
void launch_leaf_b(const int* cone_box, int ncones, int cone_base, const int* leaf_start, const int* leaf_count,
                   const long long* leaf_off, const float2* L, const float2* rho, int Ps, int Pang, int B, float2* coef,
                   cudaStream_t s);
// the FP64 form in fixed point: table as launch_leaf_fx's, densities and exponents [box][B] from launch_rho_bx;
// most: the sources of the largest leaf box
void launch_rho_bx(const int* leaf_start, const int* leaf_count, int nleaf, const double2* rho, int B, int4* out, int* rexp,
                   cudaStream_t s);
void launch_leaf_bx(const int* cone_box, int ncones, int cone_base, const int* leaf_start, const int* leaf_count,
                    const long long* leaf_off, const int4* L, const int* lexp, const int4* rho, const int* rexp, int Ps, int Pang, int B,
                    int most, int4* coef, int* cexp, cudaStream_t s);
void launch_prop_b(int pbegin, int pend, const long long* pp_ptr, const int* pp_nchild, const PropB<float>* pb, int Ps, int Pang,
                   const float* Gsep, int B, float2* coef, cudaStream_t s);
// the FP64 form in fixed point (fixpoint.cuh): coefficients [cone][P][B] as limbs with one exponent per
// cone and right-hand side, cexp [cone][B].  launch_sort_plan_x fills the propagation's terms, sorted by
// child cone within a parent; launch_group_terms_x the interpolation's from the plan ip: term i is
// ip[src[i]] of target tgt[i] (within its work item)
int batch_x_rows(int Ps, int Pang);
void launch_sort_plan_x(const long long* pp_ptr, int ncones, PlanX px, int Ps, int Pang, TermsX out, cudaStream_t s);
void launch_group_terms_x(const InterpX* ip, const int2* src_tgt, long long n, int Ps, int Pang, TermsX out, cudaStream_t s);
void launch_prop_bx(int pbegin, int pend, const long long* pp_ptr, TermsX terms, int Ps, int Pang, const int2* GsepX, int B, int4* coef,
                    int* cexp, cudaStream_t s);
// yt[sorting[t]] += the interpolation of work items (first term, end term, first Morton target, targets)
void launch_interp_bx(const int4* items, int nitems, TermsX terms, const int4* coef, const int* cexp, int Ps, int Pang,
                      const long long* sorting, int B, double2* yt, cudaStream_t s);
// the complex64 propagation on the tcgen05 tensor cores in 3xTF32 (batch_tcgen05.cu); false when
// the shape is not supported (Ps x Pang other than 5 x 5, more than 64 right-hand sides) and
// nothing was launched.  *err is set when a completion wait runs out.  The kernel's shared-memory
// attribute must be set once per device (prop_t5_init_attributes), outside stream capture.
bool launch_prop_t5(int pbegin, int pend, const long long* pp_ptr, const int* pp_nchild, const PropB<float>* pb, int Ps, int Pang,
                    const float* Gsep, int B, float2* coef, int* err, int nsm, cudaStream_t s);
// the complex64 leaf-cone sums on the tcgen05 tensor cores in 3xTF32: items[i] = (leaf box, first
// cone, end cone, 0), at most kLeafT5Cones cones, indices local to the leaf level; coef offset to
// the level's first cone
constexpr int kLeafT5Cones = 5;
// terms = 2: 3xTF32 (each operand hi + lo, 3 products); terms = 3: three TF32 terms per operand
// and 6 products, FP32-level operands
bool launch_leaf_t5(const int4* items, int nitems, const int* leaf_start, const int* leaf_count, const long long* leaf_off,
                    const float2* L, const float2* rho, int Ps, int Pang, int B, float2* coef, int* err, int nsm, int terms,
                    cudaStream_t s);
cudaError_t prop_t5_init_attributes();
// the complex64 FMA propagation with each child cone's coefficient block staged in shared memory
// by a TMA bulk copy one group ahead; false when the shape is not supported (Ps x Pang other
// than 5 x 5, B odd or above 64) and nothing was launched
// yt[sorting[t]] += the cousin-cone interpolation of the targets of each work item
// items[i] = (first term, end term, first Morton target, targets <= kInterpGrpTargets), terms
// sorted by cone within an item; complex64 coefficients [cone][P][B], B <= 64
constexpr int kInterpGrpTargets = 8;
bool launch_interp_grp(const int4* items, int nitems, const InterpG* terms, const float2* coef, int Ps, int Pang,
                       const long long* sorting, int B, double2* yt, cudaStream_t s);
bool launch_prop_bk(int pbegin, int pend, const long long* pp_ptr, const int* pp_nchild, const PropB<float>* pb, int Ps, int Pang,
                    const float* Gsep, int B, float2* coef, int* err, cudaStream_t s);
void launch_final_b(int N, const int* point_leaf, const int* leaf_start, const int* leaf_count, const int* nbr_ptr,
                    const int* nbr_box, const int* near_rowlen, const long long* near_off, const float2* near,
                    const float2* rho, const int* ip_ptr, const InterpE<float>* ip, const float2* coef, int Ps, int Pang,
                    const long long* sorting, int B, double2* yt, cudaStream_t s);
// the FP64 near field in fixed point (tables as launch_final_fx's, densities as launch_leaf_bx's)
void launch_near_b(const FinItem* items, int nitems, const int* near_src, const float2* near, const float2* rho,
                   const long long* sorting, int B, double2* yt, cudaStream_t s);
void launch_near_bx(int N, const int* point_leaf, const int* leaf_start, const int* leaf_count, const int* nbr_ptr, const int* nbr_box,
                    const int* near_rowlen, const long long* near_off, const int4* near, const int* nexp, const int4* rho,
                    const int* rexp, const long long* sorting, int B, double2* yt, cudaStream_t s);
// batched GMRES helpers on interleaved [N][B] vectors; column c of a basis starts at V + c * ldc
int bdot_chunks(long long N);
// h[c][r] = sum_i conj(V_c[i][r]) w[i][r] for c < ncols; Hcol[c][r] = h (add: +=).  With
// sqrt_row >= 0 (ncols = 1, V = w): Hcol[sqrt_row][r] = sqrt(sum_i |w[i][r]|^2) instead.
void launch_bdot(const double2* V, long long ldc, int ncols, const double2* w, long long N, int B, double2* part,
                 double2* h, double2* Hcol, int add, int sqrt_row, cudaStream_t s);
// w[i][r] += sign * sum_{c < ncols} V_c[i][r] h[c][r]
void launch_bupdate(const double2* V, long long ldc, int ncols, const double2* h, double sign, long long N, int B, double2* w,
                    cudaStream_t s);
// out[i][r] = w[i][r] / hn[r].x, 0 where hn[r] = 0
void launch_bscale(const double2* w, const double2* hn, long long N, int B, double2* out, cudaStream_t s);

// ---------------- tests / GMRES helpers ----------------
void launch_hankel(int order, const double* x, int n, double2* out, cudaStream_t s);
void launch_multidot(const double2* V, long long ldv, int ncols, const double2* w, long long n, double2* h, cudaStream_t s);
void launch_multi_axpy(const double2* V, long long ldv, int ncols, const double2* h, double sign, long long n, double2* w, cudaStream_t s);
void launch_scale(const double2* w, double2 a, long long n, double2* out, cudaStream_t s);
void launch_sub(const double2* a, const double2* b, long long n, double2* out, cudaStream_t s);
// out[i][j] = in[i][act[j]] for an interleaved in [N][B] and a compact out [N][Bc], and back
// (out[i][act[j]] (+)= in[i][j])
void launch_gather_cols(const double2* in, int B, const int* act, int Bc, long long N, double2* out, cudaStream_t s);
void launch_scatter_cols(const double2* in, int Bc, const int* act, int B, long long N, bool add, double2* out, cudaStream_t s);
void launch_nonfinite_check(const double2* v, long long n, int* flag, cudaStream_t s);
// ---------------- GMRES least squares on the device (gmres_device.cu) ----------------
// One right-hand side: R (ldh x m, column-major) the Hessenberg columns rotated to upper
// triangular form, g (m + 1) the rotated right-hand side, gc / gs (m) the rotations, st the
// cycle state [stopped, columns, iteration limit, iterations], sc [estimate, ||r0||, tol].
struct LsqDev {
    double2* R; double2* g; double* gc; double2* gs; int* st; double* sc; int m;
};
// B right-hand sides, each with the arrays of LsqDev at offsets r * ldh * m (R), r * (m + 1) (g),
// r * m (gc, gs), 4 r (st), 3 r (sc)
struct LsqBatchDev {
    double2* R; double2* g; double* gc; double2* gs; int* st; double* sc; int m; int B;
};
// a restart cycle starts: g = beta e_1, j = 0, limit iterations allowed
void launch_lsq_init(LsqDev L, int* jp, double beta, double r0n, double tol, int limit, cudaStream_t s);
// after the Arnoldi step of column j = *jp: rotate it into R, update g and the estimate
// |g_{j+1}| / ||r0||, stop on convergence, the limit or a breakdown, j += 1; set
// the condition of the graph while-loop around the iteration (0 ends the cycle); *nrm2 = 0
void launch_lsq_givens(const double2* H, int ldh, int* jp, LsqDev L, cudaGraphConditionalHandle cond, double* nrm2,
                       cudaStream_t s);
// y = R^{-1} g over the cycle's columns (st[1])
void launch_lsq_solve(LsqDev L, int ldh, double2* y, cudaStream_t s);
// w += sum_{c < *ncols} V[:, c] y[c]
void launch_multi_axpy_dyn(const double2* V, long long ldv, const int* ncols, const double2* y, long long n, double2* w,
                           cudaStream_t s);
// batched: init from per-RHS norms beta[r].x and par[3 r ..] = (||r0||, tol, iteration limit; <= 0 frozen)
void launch_lsq_init_batch(LsqBatchDev L, const double2* beta, const double* par, cudaStream_t s);
// column j (host index) of every running right-hand side, Hcol[i * B + r]; active[j] = how many still run
void launch_lsq_givens_batch(const double2* Hcol, int j, LsqBatchDev L, int* active, cudaStream_t s);
// Y[i * B + r] = (R_r^{-1} g_r)_i, zero from the right-hand side's own column count up to ncols
void launch_lsq_solve_batch(LsqBatchDev L, int ncols, double2* Y, cudaStream_t s);
// the same Givens step with j = *jp read on the device (H: columns of (m + 1) * B entries), for a
// captured iteration: active[j] = the right-hand sides still running, j += 1, and the while-loop
// condition set to 0 once none runs or the cycle is full
void launch_lsq_givens_batch_dev(const double2* H, int* jp, LsqBatchDev L, int* active, cudaGraphConditionalHandle cond,
                                 cudaStream_t s);
// Segmented vectors: B segments side by side in vectors of n entries (one per obstacle of a
// group).  Chunk c covers [chunk_lo[c], chunk_lo[c + 1]) inside one segment; segment s owns
// chunks [seg_chunk[s], seg_chunk[s + 1]); seg_of[i] is the segment of entry i; part holds
// (m + 1) * nchunk partial sums.
struct SegDesc {
    long long n; int B; int nchunk;
    const long long* chunk_lo; const int* seg_chunk; const int* seg_of; double2* part;
};
// one Arnoldi step per segment after w = A v_j (j = *jp): classical Gram-Schmidt `passes`
// times with per-segment coefficients into H column j (layout [row][segment]), the per-segment
// norms into nrm and H's subdiagonal, V[:, j + 1] = w / norm
void launch_seg_arnoldi(const SegDesc& S, double2* V, int m, int* jp, double2* w, double2* hh, double2* H, double2* nrm,
                        int passes, cudaStream_t s);
// nrm[s] = (||v_s||, 0)
void launch_seg_norms(const SegDesc& S, const double2* v, double2* nrm, cudaStream_t s);
// V[:, 0] = w / nrm per segment
void launch_seg_scale0(const SegDesc& S, const double2* w, const double2* nrm, double2* V, cudaStream_t s);
// x += V[:, 0..ncols) Y per segment (Y[c * B + s])
void launch_seg_axpy(const SegDesc& S, const double2* V, int ncols, const double2* Y, double2* x, cudaStream_t s);

// one Arnoldi step after w = A v_j, with j read from *jp (for a captured iteration graph):
// classical Gram-Schmidt against V[:, 0..j], `passes` times (2: CGS2), into the Hessenberg
// column j, ||w||^2 into *nrm2 (zeroed by launch_copy_col and the Givens step), h_{j+1,j} and
// V[:, j+1] = w / h_{j+1,j}, also into vin; then the Givens step of launch_lsq_givens, which advances j.
// h: m + 1 entries of scratch
void launch_arnoldi_step(double2* V, long long n, int m, int* jp, double2* w, double2* vin, double2* h, double2* H, double* nrm2,
                         double2* part, cudaStream_t s, int passes, LsqDev lsq, cudaGraphConditionalHandle cond);
// Its dot products are sums over chunks of kDotChunk rows.  Every block of the update (64 rows) adds up to
// kDotBlockChunks chunks of each column for itself; a longer vector's are added up once by a kernel of their own,
// as that work of the blocks together grows with the square of the length.  An iteration's time beyond the
// apply, us over 20 / 80 columns, by the blocks and by a kernel of its own: N = 81920 86 / 158 and 80 / 144,
// 131072 130 / 262 and 112 / 219, 524288 873 / 1706 and 396 / 820; at 65536 63 / 117 by the blocks.
constexpr int kDotChunk = 2048, kDotBlockChunks = 32;
constexpr long long dot_chunks(long long n) { return (n + kDotChunk - 1) / kDotChunk; }
constexpr long long dot_block_terms(long long n) { return dot_chunks(n) <= kDotBlockChunks ? dot_chunks(n) : 1; }
// size (double2 entries) of the partial-sum buffer launch_arnoldi_step needs
int arnoldi_part_size(long long n, int m);
// Z[:, *jp] = z
void launch_store_col(const double2* z, long long n, const int* jp, double2* Z, cudaStream_t s);
// out = V[:, *jp]; zeroes *nrm2 when given
void launch_copy_col(const double2* V, long long n, const int* jp, double2* out, double* nrm2, cudaStream_t s);
// FP64 FMA throughput (TFLOP/s) of the current device; false on a CUDA error
bool launch_fp64_peak(double* tflops);

}  // namespace ifgf

// ifgf_batch.cu -- the IFGF forward map applied to a batch of right-hand sides at once.
//
// Every table of the single-vector apply (near-field Green values, leaf-cone values,
// propagation and interpolation plans) depends on the geometry and k only, so B right-hand
// sides (plane waves of different incidence, ForwardMap::solve called B times) can share one
// pass over them.  The batch lives interleaved, [N][B] with the RHS index fastest, and one warp
// serves 32 right-hand sides: table entries become warp-uniform broadcast loads and the
// density / coefficient accesses are 256-byte coalesced rows.
//
//   k_sing_b   singular correction + jump term + intensities     ForwardMap.tpp:425-435, 481-515
//              (FP32 weights in the mixed form)
//   k_leaf_b   leaf cone coefficients, table rows staged in shared
//              memory by cp.async, 25 accumulators per RHS          BoxTree.h:685-762
//   k_leaf_bx  the same in fixed point (FP64 form, fixpoint.cuh)
//   k_prop_b   child -> parent, per parent cone one warp; the
//              parent's terms sorted by child cone so each child
//              cone's coefficients are loaded once                 BoxTree.h:767-868, Interpolator.h:81-120
//   k_prop_bx, k_interp_bx  the FP64 propagation and interpolation
//              in fixed point (fixpoint.cuh)
//   k_near_b, k_interp_grp  near field by four targets, cousin
//              interpolation grouped by cone; k_final_b both by
//              target; k_near_bx the FP64 near field               BoxTree.h:614-683, 876-937
//
// plus the batched GMRES vector kernels (per-RHS dot products, CGS updates, scaling).
#include "fixpoint.cuh"
#include "tcgen05.cuh"
#include <type_traits>

namespace ifgf {

static inline unsigned nblk_b(long long n, int b) { return (unsigned)((n + b - 1) / b); }

// ------------------------------------------------------------------ layout changes
__global__ void k_interleave(const double2* __restrict__ x, long long N, int B, double2* __restrict__ xt) {
    __shared__ double2 t[32][33];
    const long long i0 = (long long)blockIdx.x * 32;
    const int r0 = blockIdx.y * 32;
    for (int k = threadIdx.y; k < 32; k += 8) {
        const int r = r0 + k;
        const long long i = i0 + threadIdx.x;
        if (r < B && i < N) t[k][threadIdx.x] = x[(long long)r * N + i];
    }
    __syncthreads();
    for (int k = threadIdx.y; k < 32; k += 8) {
        const long long i = i0 + k;
        const int r = r0 + threadIdx.x;
        if (r < B && i < N) xt[i * B + r] = t[threadIdx.x][k];
    }
}
__global__ void k_deinterleave(const double2* __restrict__ xt, long long N, int B, double2* __restrict__ x) {
    __shared__ double2 t[32][33];
    const long long i0 = (long long)blockIdx.x * 32;
    const int r0 = blockIdx.y * 32;
    for (int k = threadIdx.y; k < 32; k += 8) {
        const long long i = i0 + k;
        const int r = r0 + threadIdx.x;
        if (r < B && i < N) t[k][threadIdx.x] = xt[i * B + r];
    }
    __syncthreads();
    for (int k = threadIdx.y; k < 32; k += 8) {
        const int r = r0 + k;
        const long long i = i0 + threadIdx.x;
        if (r < B && i < N) x[(long long)r * N + i] = t[threadIdx.x][k];
    }
}

// ------------------------------------------------------------------ singular correction
// warp = one output row, lane = one right-hand side.  WT = double2: FP64 weights, densities and
// arithmetic (the plain form; xw = xt); WT = float2: complex64 copies of the FP64-computed
// weights and of the densities (xw), FP32 sums (the mixed form).  The jump term and the
// intensities take the FP64 densities xt.
template <typename WT, typename RhoT>
__global__ void __launch_bounds__(256) k_sing_b(const double2* __restrict__ xt, const WT* __restrict__ xw,
                                                const WT* __restrict__ W, const int* __restrict__ row_ptr,
                                                const int* __restrict__ row_col, const RPColumn* __restrict__ cols, int N,
                                                int Np, int B, double half, double2* __restrict__ yt,
                                                const double* __restrict__ wq, const long long* __restrict__ inv,
                                                RhoT* __restrict__ rho) {
    using A = decltype(WT{}.x);
    const int o = blockIdx.x * 8 + (threadIdx.x >> 5);
    const int r = blockIdx.y * 32 + (threadIdx.x & 31);
    if (o >= N || r >= B) return;
    A ax = A(0), ay = A(0);
    for (int q = row_ptr[o]; q < row_ptr[o + 1]; ++q) {
        const int col = row_col[q];
        const WT* w = W + (long long)col * Np;
        const WT* d = xw + (long long)cols[col].patch * Np * B + r;
        int kk = 0;
        for (; kk + 4 <= Np; kk += 4) {         // four nodes' loads in flight at once
            WT a[4], bw[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) { a[u] = d[(long long)(kk + u) * B]; bw[u] = w[kk + u]; }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                ax = fma(a[u].x, bw[u].x, fma(-a[u].y, bw[u].y, ax));
                ay = fma(a[u].x, bw[u].y, fma(a[u].y, bw[u].x, ay));
            }
        }
        for (; kk < Np; ++kk) {
            const WT a = d[(long long)kk * B], b = w[kk];
            ax = fma(a.x, b.x, fma(-a.y, b.y, ax));
            ay = fma(a.x, b.y, fma(a.y, b.x, ay));
        }
    }
    const double2 v = xt[(long long)o * B + r];
    double2 acc = make_double2((double)ax, (double)ay);
    if (half != 0.0) { acc.x += half * v.x; acc.y += half * v.y; }   // jump term
    yt[(long long)o * B + r] = acc;
    if (rho) {
        const double wv = wq[o];
        RhoT q; q.x = v.x * wv; q.y = v.y * wv;
        rho[inv[o] * B + r] = q;
    }
}

// ------------------------------------------------------------------ asynchronous copies
// cp.async (global -> shared without a register round trip) of one 4-, 8- or 16-byte element
template <int BYTES>
__device__ __forceinline__ void cp_async_el(void* smem, const void* gmem) {
    static_assert(BYTES == 4 || BYTES == 8 || BYTES == 16, "the element sizes of cp.async");
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    if (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(sa), "l"(gmem), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int NPEND>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(NPEND) : "memory"); }

// right-hand sides per lane of the complex64 kernels: two (a warp covers a 64-wide batch, so every table
// entry is read once per batch)
constexpr int kRpl = 2;

// ------------------------------------------------------------------ leaf cones
// complex64: warp = one leaf cone x 32*RPL right-hand sides, P accumulators per (lane, RHS).  The cone's
// table rows stream through shared memory in tiles of TS sources (cp.async, double-buffered)
// and every lane reads them as broadcasts; densities are prefetched one source ahead.
constexpr int kLeafWarps = 4;
template <int P, int RPL>
__global__ void __launch_bounds__(kLeafWarps * 32) k_leaf_b(const int* __restrict__ cone_box, int ncones, int cone_base,
                                                            const int* __restrict__ leaf_start,
                                                            const int* __restrict__ leaf_count,
                                                            const long long* __restrict__ leaf_off,
                                                            const float2* __restrict__ L, const float2* __restrict__ rho, int B,
                                                            float2* __restrict__ coef) {
    using R = float;
    constexpr int TS = 16;
    __shared__ V2<R> tile[kLeafWarps][2][TS * P];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blockIdx.x * kLeafWarps + w;
    if (c >= ncones) return;                 // warps are independent: no block-wide barrier below
    int rr[RPL];
    bool act[RPL];
#pragma unroll
    for (int k = 0; k < RPL; ++k) {
        const int r = blockIdx.y * 32 * RPL + 32 * k + lane;
        act[k] = r < B;
        rr[k] = act[k] ? r : 0;
    }
    const int b = cone_box[c];
    const int n = leaf_count[b], s0 = leaf_start[b];
    const V2<R>* Lc = L + leaf_off[c];
    auto load_tile = [&](int t) {
        const int sb = t * TS;
        const int cnt = (n - sb < TS ? n - sb : TS) * P;
        const V2<R>* src = Lc + (long long)sb * P;
        V2<R>* dst = tile[w][t & 1];
        for (int q = lane; q < cnt; q += 32) cp_async_el<(int)sizeof(V2<R>)>(dst + q, src + q);
        cp_async_commit();
    };
    V2<R> acc[RPL][P];
#pragma unroll
    for (int k = 0; k < RPL; ++k)
#pragma unroll
        for (int m = 0; m < P; ++m) { acc[k][m].x = R(0); acc[k][m].y = R(0); }
    const V2<R>* rh = rho + (long long)s0 * B;
    V2<R> vn[RPL];
#pragma unroll
    for (int k = 0; k < RPL; ++k) vn[k] = rh[rr[k]];
    const int nt = (n + TS - 1) / TS;
    load_tile(0);
    for (int t = 0; t < nt; ++t) {
        if (t + 1 < nt) { load_tile(t + 1); cp_async_wait<1>(); }
        else cp_async_wait<0>();
        __syncwarp();
        const V2<R>* Lt = tile[w][t & 1];
        const int sb = t * TS;
        const int cnt = n - sb < TS ? n - sb : TS;
        for (int s = 0; s < cnt; ++s) {
            V2<R> v[RPL];
#pragma unroll
            for (int k = 0; k < RPL; ++k) v[k] = vn[k];
            if (sb + s + 1 < n) {
#pragma unroll
                for (int k = 0; k < RPL; ++k) vn[k] = rh[(long long)(sb + s + 1) * B + rr[k]];
            }
#pragma unroll
            for (int m = 0; m < P; ++m) {
                const V2<R> l = Lt[s * P + m];
#pragma unroll
                for (int k = 0; k < RPL; ++k) cmac<R>(acc[k][m], l, v[k]);
            }
        }
        __syncwarp();                        // the buffer is refilled two tiles later
    }
#pragma unroll
    for (int k = 0; k < RPL; ++k) {
        if (!act[k]) continue;
        float2* out = coef + (long long)(cone_base + c) * P * B + rr[k];
#pragma unroll
        for (int m = 0; m < P; ++m) out[(long long)m * B] = acc[k][m];
    }
}

// FP64 in fixed point (fixpoint.cuh): the densities of a leaf box as limbs with one exponent per box and
// right-hand side (a block per box, a thread per right-hand side)
__global__ void k_rho_bx(const int* __restrict__ leaf_start, const int* __restrict__ leaf_count, const double2* __restrict__ rho, int B,
                         int4* __restrict__ out, int* __restrict__ rexp) {
    const int b = blockIdx.x, r = threadIdx.x;
    if (r >= B) return;
    const int n = leaf_count[b], T = kFxSumTop;
    const long long s0 = leaf_start[b];
    int mx = 0;
    for (int i = 0; i < n; ++i) { const double2 v = rho[(s0 + i) * B + r]; mx = max(mx, fx_absmax_hi(v.x, v.y)); }
    const int E = fx_expo(mx);
    rexp[(long long)b * B + r] = E;
    for (int i = 0; i < n; ++i) {
        const double2 v = rho[(s0 + i) * B + r];
        out[(s0 + i) * B + r] = E == kFxBad ? make_int4(0, 0, 0, 0) : fx_pack_sum(fx_from(v.x, E, T), fx_from(v.y, E, T));
    }
}
// block = one leaf cone x NT right-hand sides x MS parts of the coefficients (blockDim.y), PM
// coefficients a thread: their integer sums (eight registers each) stay in registers.  The table streams
// through shared memory kLeafBxTile sources at a time (cp.async, double-buffered), read as broadcasts.
// Bound by the wide multiply-adds (12 an entry); kite k = 500, 64 right-hand sides 4.0 -> 1.2 ms.
// BIG (launched for trees with a box of more than kFxSumMost sources): such a box's sums of kFxSumMost
// sources each are added up in FP64, in the place of the coefficients.
constexpr int kLeafBxTile = 8;
// With 6 x 6 cones BIG's loads for all coefficients at once took 237 registers and one block an SM; one at a time and held
// to two blocks, 64 right-hand sides of kite k = 200 take 3.33 ms instead of 3.65.  The other orders keep two and
// three blocks without, and lose 3 % with it.
template <int P, int MS, int NT, bool BIG>
__global__ void __launch_bounds__(NT * MS, BIG && P == 36 ? 65536 / (NT * MS * 160) : 0)
                                           k_leaf_bx(const int* __restrict__ cone_box, int cone_base, const int* __restrict__ leaf_start,
                                                     const int* __restrict__ leaf_count, const long long* __restrict__ leaf_off,
                                                     const int4* __restrict__ L, const int* __restrict__ lexp,
                                                     const int4* __restrict__ rho, const int* __restrict__ rexp, int B, int Ps,
                                                     int4* __restrict__ coef, int* __restrict__ cexp) {
    constexpr int PM = (P + MS - 1) / MS, TS = kLeafBxTile;
    static_assert(kFxSumFold % TS == 0 && kFxSumMost % kFxSumFold == 0, "folds between tiles, parts of whole folds");
    __shared__ int4 tile[2][TS * P];
    __shared__ int stop[NT];
    const int c = blockIdx.x, lt = threadIdx.x, part = threadIdx.y, tid = part * NT + lt;
    const int r = blockIdx.y * NT + lt;
    const bool act = r < B;
    const int rr = act ? r : 0;
    const int b = cone_box[c], n = leaf_count[b];
    const int4* Lc = L + leaf_off[c];
    if (part == 0) stop[lt] = kFxMinExp;
    auto load_tile = [&](int t) {
        const int cnt = min(TS, n - t * TS) * P;
        for (int q = tid; q < cnt; q += NT * MS) cp_async_el<16>(&tile[t & 1][q], Lc + (long long)t * TS * P + q);
        cp_async_commit();
    };
    FxSum re[PM], im[PM];
#pragma unroll
    for (int m = 0; m < PM; ++m) re[m] = im[m] = FxSum{0, 0};
    const int4* rh = rho + (long long)leaf_start[b] * B + rr;
    int Er = BIG ? rexp[(long long)b * B + rr] : 0;
    double2* sums = reinterpret_cast<double2*>(coef + (long long)(cone_base + c) * P * B + r);
    const int nt = (n + TS - 1) / TS;
    int4 dn = n > 0 ? rh[0] : make_int4(0, 0, 0, 0);
    if (nt > 0) load_tile(0);
    for (int t = 0; t < nt; ++t) {
        if (t + 1 < nt) { load_tile(t + 1); cp_async_wait<1>(); }
        else cp_async_wait<0>();
        __syncthreads();
        const int4* Lt = tile[t & 1] + part * PM;
        const int cnt = min(TS, n - t * TS);
        for (int s = 0; s < cnt; ++s) {
            const int4 d = dn;
            if (t * TS + s + 1 < n) dn = rh[(long long)(t * TS + s + 1) * B];
            const int nh = -d.z, nl = -d.w;
#pragma unroll
            for (int m = 0; m < PM; ++m) {
                if (P % MS && part * PM + m >= P) break;
                const int4 l = Lt[s * P + m];
                fx_sum_mac(re[m], l.x, l.y, d.x, d.y);
                fx_sum_mac(re[m], l.z, l.w, nh, nl);
                fx_sum_mac(im[m], l.x, l.y, d.z, d.w);
                fx_sum_mac(im[m], l.z, l.w, d.x, d.y);
            }
        }
        if ((t + 1) % (kFxSumFold / TS) == 0 || t + 1 == nt)
#pragma unroll
            for (int m = 0; m < PM; ++m) { fx_sum_fold(re[m]); fx_sum_fold(im[m]); }
        if (BIG && n > kFxSumMost && ((t + 1) % (kFxSumMost / TS) == 0 || t + 1 == nt)) {
#pragma unroll
            for (int m = 0; m < PM; ++m) {
                const int q = part * PM + m;
                if (q < P && act) {
                    const int El = lexp[(long long)c * P + q], E0 = Er == kFxBad || El == kFxBad ? 0 : El + Er - 2 * kFxSumTop;
                    int ea, eb;
                    const long long ya = fx_sum_value(re[m], E0, ea), yb = fx_sum_value(im[m], E0, eb);
                    double2* o = sums + (long long)q * B;
                    const double2 a = t < kFxSumMost / TS ? make_double2(0.0, 0.0) : *o;
                    *o = make_double2(a.x + fx_scaled(ya, ea), a.y + fx_scaled(yb, eb));
                }
                re[m] = im[m] = FxSum{0, 0};
                if (P == 36) asm volatile("" ::: "memory");   // one coefficient's loads at a time
            }
        }
        __syncthreads();                        // the buffer is refilled two tiles later
    }
    const int T = fx_top(P);
    if (BIG && n > kFxSumMost) {
        int mx = 0;
        for (int m = 0; m < PM; ++m) {
            const int q = part * PM + m;
            if (q >= P || !act) break;
            const double2 v = sums[(long long)q * B];
            mx = max(mx, lexp[(long long)c * P + q] == kFxBad || Er == kFxBad ? 0x7ff00000 : fx_absmax_hi(v.x, v.y));
        }
        if (MS > 1) {
            atomicMax(&stop[lt], mx);
            __syncthreads();
            mx = stop[lt];
        }
        if (!act) return;
        const int E = fx_expo(max(mx, 0));
        for (int m = 0; m < PM; ++m) {
            const int q = part * PM + m;
            if (q >= P) break;
            const double2 v = sums[(long long)q * B];
            const long long xr = E == kFxBad ? 0 : fx_from(v.x, E, T), xi = E == kFxBad ? 0 : fx_from(v.y, E, T);
            reinterpret_cast<int4*>(sums)[(long long)q * B] = q % Ps ? fx_pack(xr, xi) : fx_pack_raw(xr, xi);
        }
        if (part == 0) cexp[(long long)(cone_base + c) * B + r] = E;
        return;
    }
    if (!BIG) Er = rexp[(long long)b * B + rr];
    int top = kFxMinExp;                        // the sums in place as y = .h, e = .m of y 2^e
#pragma unroll
    for (int m = 0; m < PM; ++m) {
        const int q = part * PM + m;
        if (q >= P) continue;
        const int El = lexp[(long long)c * P + q];
        if (Er == kFxBad || El == kFxBad) { top = kFxBad; continue; }
        const int E0 = El + Er - 2 * kFxSumTop;
        int ea, eb;
        const long long ya = fx_sum_value(re[m], E0, ea), yb = fx_sum_value(im[m], E0, eb);
        re[m].h = ya; im[m].h = yb; re[m].m = ea; im[m].m = eb;
        top = max(top, max(fx_top_of(ya, ea), fx_top_of(yb, eb)));
    }
    if (MS > 1) {
        if (nt == 0) __syncthreads();
        atomicMax(&stop[lt], top);
        __syncthreads();
        top = stop[lt];
    }
    if (!act) return;
    const int E = top > kFxMaxExp ? kFxBad : top;
    int4* out = coef + (long long)(cone_base + c) * P * B + r;
#pragma unroll
    for (int m = 0; m < PM; ++m) {
        const int q = part * PM + m;
        if (q >= P) continue;
        const long long xr = E == kFxBad ? 0 : fx_align(re[m].h, (int)re[m].m, E, T), xi = E == kFxBad ? 0 : fx_align(im[m].h, (int)im[m].m, E, T);
        out[(long long)q * B] = q % Ps ? fx_pack(xr, xi) : fx_pack_raw(xr, xi);
    }
    if (part == 0) cexp[(long long)(cone_base + c) * B + r] = E;
}

// ------------------------------------------------------------------ propagation
// complex64: warp = one parent cone x 32*RPL right-hand sides.  Node values accumulate in the lane's own
// shared-memory columns; the values -> coefficients map then runs in the lane's registers.  The parent's
// terms (at most 4 P, uniform over the warp) come into shared memory with one round of copies, and a term is
// read during the one before: read one by one from global memory, a term ahead, their latency was what three
// warps a scheduler waited for.  Kite k = 2000, 64 right-hand sides, all levels: 2438 -> 1897 us (issue 56 ->
// 72 % of the slots; bound by the FP32 multiply-adds).  Prefetching the next child's rows: slower by 10 %.
template <int P, int RPL>
struct PropBlock {
    static constexpr int bytes_per_warp = P * 32 * RPL * (int)sizeof(float2);
    static constexpr int W = 32768 / bytes_per_warp >= 4 ? 4 : (32768 / bytes_per_warp >= 2 ? 2 : 1);
};
template <int PS, int PA, int WPB, int RPL>
__global__ void __launch_bounds__(WPB * 32) k_prop_b(int pbegin, int pend, const long long* __restrict__ pp_ptr,
                                                     const int* __restrict__ pp_nchild, const PropB<float>* __restrict__ pb,
                                                     const float* __restrict__ Gsep, int B, float2* __restrict__ coef) {
    using R = float;
    constexpr int P = PS * PA;
    __shared__ V2<R> sv[WPB][P][32 * RPL];
    __shared__ alignas(16) PropB<R> plan[WPB][4 * P];
    __shared__ R sG[PS * PS + PA * PA];
    for (int i = threadIdx.x; i < PS * PS + PA * PA; i += blockDim.x) sG[i] = Gsep[i];
    __syncthreads();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pc = pbegin + blockIdx.x * WPB + w;
    if (pc >= pend) return;
    // the parent's terms, all on their way at once
    const long long e0 = pp_ptr[pc];
    const int ne = pp_nchild[pc] * P;
    for (int i = lane; i < ne * (int)sizeof(PropB<R>) / 8; i += 32)
        cp_async_el<8>(reinterpret_cast<char*>(plan[w]) + 8 * i, reinterpret_cast<const char*>(pb + e0) + 8 * i);
    cp_async_commit();
    int rr[RPL];
    bool act[RPL];
#pragma unroll
    for (int k = 0; k < RPL; ++k) {
        const int r = blockIdx.y * 32 * RPL + 32 * k + lane;
        act[k] = r < B;
        rr[k] = act[k] ? r : 0;
    }
#pragma unroll
    for (int q = 0; q < P; ++q)
#pragma unroll
        for (int k = 0; k < RPL; ++k) { sv[w][q][32 * k + lane].x = R(0); sv[w][q][32 * k + lane].y = R(0); }
    V2<R> cc[RPL][P];
    int cur = -1;
    cp_async_wait<0>();
    __syncwarp();
    PropB<R> En{};
    if (ne > 0) En = plan[w][0];
    for (int e = 0; e < ne; ++e) {
        const PropB<R> E = En;
        if (e + 1 < ne) En = plan[w][e + 1];
        if (E.child_cone != cur) {             // warp-uniform: E is the same for every lane
            cur = E.child_cone;
            const V2<R>* src = coef + (long long)cur * P * B;
#pragma unroll
            for (int k = 0; k < RPL; ++k)
#pragma unroll
                for (int q = 0; q < P; ++q) cc[k][q] = src[(long long)q * B + rr[k]];
        }
        R Ts[PS], Tt[PA];
        cheb_row<R, PS>(E.s, Ts);
        cheb_row<R, PA>(E.th, Tt);
        V2<R> wv; wv.x = E.wr; wv.y = E.wi;
#pragma unroll
        for (int k = 0; k < RPL; ++k) {
            const V2<R> it = interp_eval_tt<R, PS, PA>(cc[k], Ts, Tt);
            V2<R> a = sv[w][E.pt][32 * k + lane];
            cmac<R>(a, it, wv);
            sv[w][E.pt][32 * k + lane] = a;
        }
    }
    // u[l][m] = sum_k Gs[m][k] v[l][k];  c[n][m] = sum_l Ga[n][l] u[l][m], stored at n*PS + m
#pragma unroll
    for (int k = 0; k < RPL; ++k) {
        V2<R> u[P];
#pragma unroll
        for (int l = 0; l < PA; ++l) {
            V2<R> v[PS];
#pragma unroll
            for (int q = 0; q < PS; ++q) v[q] = sv[w][l * PS + q][32 * k + lane];
#pragma unroll
            for (int m = 0; m < PS; ++m) {
                V2<R> a; a.x = R(0); a.y = R(0);
#pragma unroll
                for (int q = 0; q < PS; ++q) { const R g = sG[m * PS + q]; a.x = rfma(g, v[q].x, a.x); a.y = rfma(g, v[q].y, a.y); }
                u[l * PS + m] = a;
            }
        }
        if (!act[k]) continue;
        V2<R>* out = coef + (long long)pc * P * B + rr[k];
#pragma unroll
        for (int n = 0; n < PA; ++n)
#pragma unroll
            for (int m = 0; m < PS; ++m) {
                V2<R> a; a.x = R(0); a.y = R(0);
#pragma unroll
                for (int l = 0; l < PA; ++l) {
                    const R g = sG[PS * PS + n * PA + l];
                    a.x = rfma(g, u[l * PS + m].x, a.x); a.y = rfma(g, u[l * PS + m].y, a.y);
                }
                out[(long long)(n * PS + m) * B] = a;
            }
    }
}

// ------------------------------------------------------------------ FP64 cone sums in fixed point
// fixpoint.cuh's arithmetic, one right-hand side per thread.  A block's threads share one list of terms
// sorted by cone: the list is staged in shared memory kTermsChunk terms at a time, with the Chebyshev
// values computed at set-up (they are the same for every right-hand side), and a cone's block stays in
// registers for all its terms (about 14).  A term takes some 140 wide multiply-adds a thread, the bound,
// and 6 FP64 operations (conversion and factor) beside them, against 56 FP64 operations before.  Kite
// k = 500, 64 right-hand sides: propagation 11.0 -> 3.2 ms, interpolation 1.6 -> 0.48 ms.
constexpr int kTermsChunk = 64;
template <int PS, int PA>
struct StageX {
    int4 rows[kTermsChunk * fx_rows4(PS, PA)];
    double2 w[kTermsChunk];
    int2 id[kTermsChunk];
};
// add(node, value) for the terms [e0, e0 + n)
template <int PS, int PA, int NT, typename Add>
__device__ __forceinline__ void terms_x(StageX<PS, PA>& S, TermsX terms, long long e0, int n, const int4* __restrict__ coef,
                                        const int* __restrict__ cexp, int B, int rr, Add&& add) {
    constexpr int P = PS * PA, N4 = fx_rows4(PS, PA), T = fx_top(P);
    int4 cc[P];
    int cur = -1;
    FxScale scale{};
    for (int c0 = 0; c0 < n; c0 += kTermsChunk) {
        const int cnt = min(kTermsChunk, n - c0);
        __syncthreads();                       // the previous chunk has been read
        for (int i = threadIdx.x; i < cnt * N4; i += NT) cp_async_el<16>(&S.rows[i], terms.rows + (e0 + c0) * N4 + i);
        for (int i = threadIdx.x; i < cnt; i += NT) {
            cp_async_el<16>(&S.w[i], terms.w + e0 + c0 + i);
            cp_async_el<8>(&S.id[i], terms.id + e0 + c0 + i);
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        for (int i = 0; i < cnt; ++i) {
            const int2 id = S.id[i];
            if (id.x != cur) {                 // uniform over the block
                cur = id.x;
                const int4* src = coef + (long long)cur * P * B + rr;
#pragma unroll
                for (int q = 0; q < P; ++q) cc[q] = src[(long long)q * B];
                scale = fx_scale(cexp[(long long)cur * B + rr], T);
            }
            FxLimb t[2 * N4];
#pragma unroll
            for (int q = 0; q < N4; ++q) {
                const int4 a = S.rows[i * N4 + q];
                t[2 * q] = FxLimb{a.x, a.y}; t[2 * q + 1] = FxLimb{a.z, a.w};
            }
            long long re, im;
            fx_interp<PS, PA>(t, t + PS - 1, [&](int q) { return cc[q]; }, re, im);
            const double2 w = S.w[i];
            add(id.y, fx_value(re, im, scale), w);
        }
    }
}

// block = one parent cone x NT right-hand sides.  Node values accumulate in the thread's own column of
// shared memory; then the cone's exponent, the values->coefficients map and the normalisation, all
// within the column.
template <int PS, int PA, int NT>
__global__ void __launch_bounds__(NT) k_prop_bx(int pbegin, const long long* __restrict__ pp_ptr, TermsX terms,
                                                const int2* __restrict__ Gsep, int B, int4* __restrict__ coef, int* __restrict__ cexp) {
    constexpr int P = PS * PA, T = fx_top(P);
    __shared__ StageX<PS, PA> S;
    __shared__ int4 sv[P][NT];                 // FP64 node values, then limbs
    __shared__ int2 sG[PS * PS + PA * PA];
    const int tid = threadIdx.x;
    for (int i = tid; i < PS * PS + PA * PA; i += NT) sG[i] = Gsep[i];
    const int pc = pbegin + blockIdx.x;
    const int r = blockIdx.y * NT + tid;
    const bool act = r < B;
    const int rr = act ? r : 0;
    auto node = [&](int q) -> double2& { return *reinterpret_cast<double2*>(&sv[q][tid]); };
#pragma unroll
    for (int q = 0; q < P; ++q) node(q) = make_double2(0.0, 0.0);
    const long long e0 = pp_ptr[pc];
    terms_x<PS, PA, NT>(S, terms, e0, (int)(pp_ptr[pc + 1] - e0), coef, cexp, B, rr, [&](int pt, double2 it, double2 w) {
        double2 a = node(pt);
        cmac<double>(a, it, w);
        node(pt) = a;
    });
    __syncthreads();
    if (!act) return;
    int mx = 0;
    for (int q = 0; q < P; ++q) { const double2 a = node(q); mx = max(mx, fx_absmax_hi(a.x, a.y)); }
    const int E = fx_expo(mx);
    for (int l = 0; l < PA; ++l) {             // u[l][m] = sum_k Gs[m][k] v[l][k]
        int4 v[PS];
#pragma unroll
        for (int q = 0; q < PS; ++q) {
            const double2 a = node(l * PS + q);
            v[q] = E == kFxBad ? make_int4(0, 0, 0, 0) : fx_pack(fx_from(a.x, E, T), fx_from(a.y, E, T));
        }
#pragma unroll
        for (int m = 0; m < PS; ++m) {
            long long ur, ui;
            fx_map<PS>([&](int k) { return sG[m * PS + k]; }, [&](int k) { return v[k]; }, ur, ui);
            sv[l * PS + m][tid] = fx_pack(ur, ui);
        }
    }
    int lz = 64;
    for (int m = 0; m < PS; ++m) {             // c[n][m] = sum_l Ga[n][l] u[l][m], stored at n*PS + m
        int4 u[PA];
#pragma unroll
        for (int l = 0; l < PA; ++l) u[l] = sv[l * PS + m][tid];
#pragma unroll
        for (int n = 0; n < PA; ++n) {
            long long cr, ci;
            fx_map<PA>([&](int l) { return sG[PS * PS + n * PA + l]; }, [&](int l) { return u[l]; }, cr, ci);
            lz = min(lz, min(__clzll(cr < 0 ? -cr : cr), __clzll(ci < 0 ? -ci : ci)));
            sv[n * PS + m][tid] = fx_pack_raw(cr, ci);
        }
    }
    int sh = lz - (63 - T);                    // left shift that brings the largest to [2^(T-1), 2^T)
    sh = E == kFxBad ? 0 : min(sh, E - kFxMinExp);
    int4* out = coef + (long long)pc * P * B + r;
    for (int q = 0; q < P; ++q) {
        const int4 a = sv[q][tid];
        const long long x = fx_shift(fx_raw(a.x, a.y), sh), y = fx_shift(fx_raw(a.z, a.w), sh);
        out[(long long)q * B] = q % PS ? fx_pack(x, y) : fx_pack_raw(x, y);
    }
    cexp[(long long)pc * B + r] = E == kFxBad ? kFxBad : E - sh;
}

// block = one work item (up to kInterpGrpTargets targets of one leaf box) x NT right-hand sides; the
// targets' sums accumulate in the thread's column of shared memory, then are added into yt
template <int PS, int PA, int NT>
__global__ void __launch_bounds__(NT) k_interp_bx(const int4* __restrict__ items, TermsX terms, const int4* __restrict__ coef,
                                                  const int* __restrict__ cexp, const long long* __restrict__ sorting, int B,
                                                  double2* __restrict__ yt) {
    __shared__ StageX<PS, PA> S;
    __shared__ double2 acc[kInterpGrpTargets][NT];
    const int4 I = items[blockIdx.x];          // terms [x, y), targets [z, z + w)
    const int r = blockIdx.y * NT + threadIdx.x;
    const bool act = r < B;
    for (int t = 0; t < I.w; ++t) acc[t][threadIdx.x] = make_double2(0.0, 0.0);
    terms_x<PS, PA, NT>(S, terms, I.x, I.y - I.x, coef, cexp, B, act ? r : 0, [&](int t, double2 it, double2 f) {
        double2 a = acc[t][threadIdx.x];
        cmac<double>(a, it, f);
        acc[t][threadIdx.x] = a;
    });
    if (!act) return;
    for (int t = 0; t < I.w; ++t) {
        double2* yo = yt + sorting[I.z + t] * B + r;
        const double2 a = acc[t][threadIdx.x];
        double2 v = *yo;
        v.x += a.x; v.y += a.y;
        *yo = v;
    }
}

// ------------------------------------------------------------------ propagation, TMA-staged
// k_prop_b (complex64) with its loads taken off the FMA loop: the parent's terms are staged in
// shared memory at the start, and the child cones' coefficient blocks by the tensor memory
// accelerator.  When the block starts a group of terms, thread 0 issues a bulk copy
// (cp.async.bulk, completion counted on an mbarrier) of the NEXT group's 25 x B block into
// shared memory, so it has landed by the time the FMA loop needs it.  Two warps share one parent
// cone and one staging buffer, 32 right-hand sides each (half the shared memory per warp of a
// warp per cone, twice the resident warps).  B must be even (the block is a multiple of 16
// bytes).  Waits are bounded; one that runs out sets *err and the block stops.
constexpr int kPropBkWarps = 2;
template <int PS, int PA>
__global__ void __launch_bounds__(32 * kPropBkWarps) k_prop_bk(int pbegin, int pend, const long long* __restrict__ pp_ptr,
                                                               const int* __restrict__ pp_nchild, const PropB<float>* __restrict__ pb,
                                                               const float* __restrict__ Gsep, int B, float2* __restrict__ coef,
                                                               int* __restrict__ err) {
    constexpr int P = PS * PA;
    __shared__ __align__(128) float2 buf[P * 32 * kPropBkWarps];
    __shared__ float2 sv[P][32 * kPropBkWarps];
    __shared__ float sG[PS * PS + PA * PA];
    __shared__ PropB<float> st[4 * P];
    __shared__ __align__(8) unsigned long long mbar;
    const int tid = threadIdx.x, lane = tid & 31;
    const int pc = pbegin + blockIdx.x;
    if (pc >= pend) return;
    for (int i = tid; i < PS * PS + PA * PA; i += blockDim.x) sG[i] = Gsep[i];
    const uint32_t bar = tc5::smem_u32(&mbar), sbuf = tc5::smem_u32(buf);
    const int r = tid;                        // this thread's right-hand side
    const bool act = r < B;
    const int rr = act ? r : 0;
#pragma unroll
    for (int q = 0; q < P; ++q) sv[q][tid] = make_float2(0.f, 0.f);
    const long long e0 = pp_ptr[pc];
    const int ne = pp_nchild[pc] * P;   // at most four children
    const uint32_t bytes = (uint32_t)(P * B * sizeof(float2));
    if (tid == 0) {
        tc5::mbar_init(bar, 1);
        if (ne > 0) tc5::bulk_g2s(sbuf, coef + (long long)pb[e0].child_cone * P * B, bytes, bar);
    }
    for (int i = tid; i < ne; i += blockDim.x) st[i] = pb[e0 + i];   // the parent's terms
    __syncthreads();
    uint32_t phase = 0;
    bool ok = true;
    float2 cc[P];
    int cur = -1;
    for (int e = 0; e < ne; ++e) {
        const PropB<float> E = st[e];
        if (E.child_cone != cur) {             // block-uniform
            cur = E.child_cone;
            ok = __syncthreads_and(tc5::mbar_wait(bar, phase & 1u, 2000000000ll));
            ++phase;
            if (!ok) break;
#pragma unroll
            for (int q = 0; q < P; ++q) cc[q] = buf[q * B + rr];
            __syncthreads();                   // every thread has read the block before it is overwritten
            if (tid < 32) {                    // the next group: the first later term with another child cone
                int nxt = -1;
                for (int base = e + 1; base < ne && nxt < 0; base += 32) {
                    const int idx = base + lane;
                    const int cn = idx < ne ? st[idx].child_cone : cur;
                    const unsigned m = __ballot_sync(0xffffffffu, cn != cur);
                    if (m) nxt = __shfl_sync(0xffffffffu, cn, __ffs(m) - 1);
                }
                if (nxt >= 0 && tid == 0) tc5::bulk_g2s(sbuf, coef + (long long)nxt * P * B, bytes, bar);
            }
        }
        float Ts[PS], Tt[PA];
        cheb_row<float, PS>(E.s, Ts);
        cheb_row<float, PA>(E.th, Tt);
        const float2 it = interp_eval_tt<float, PS, PA>(cc, Ts, Tt);
        float2 a = sv[E.pt][tid];
        cmac<float>(a, it, make_float2(E.wr, E.wi));
        sv[E.pt][tid] = a;
    }
    if (!ok) {   // the copy of the group that timed out may still land: one more bounded wait
        if (tid == 0) { atomicExch(err, 1); tc5::mbar_wait(bar, (phase - 1u) & 1u, 2000000000ll); }
        return;
    }
    // u[l][m] = sum_k Gs[m][k] v[l][k];  c[n][m] = sum_l Ga[n][l] u[l][m], stored at n*PS + m
    float2 u[P];
#pragma unroll
    for (int l = 0; l < PA; ++l) {
        float2 v[PS];
#pragma unroll
        for (int q = 0; q < PS; ++q) v[q] = sv[l * PS + q][tid];
#pragma unroll
        for (int m = 0; m < PS; ++m) {
            float2 a = make_float2(0.f, 0.f);
#pragma unroll
            for (int q = 0; q < PS; ++q) { const float g = sG[m * PS + q]; a.x = fmaf(g, v[q].x, a.x); a.y = fmaf(g, v[q].y, a.y); }
            u[l * PS + m] = a;
        }
    }
    if (!act) return;
    float2* out = coef + (long long)pc * P * B + r;
#pragma unroll
    for (int n = 0; n < PA; ++n)
#pragma unroll
        for (int m = 0; m < PS; ++m) {
            float2 a = make_float2(0.f, 0.f);
#pragma unroll
            for (int l = 0; l < PA; ++l) {
                const float g = sG[PS * PS + n * PA + l];
                a.x = fmaf(g, u[l * PS + m].x, a.x); a.y = fmaf(g, u[l * PS + m].y, a.y);
            }
            out[(long long)(n * PS + m) * B] = a;
        }
}

// ------------------------------------------------------------------ near field + interpolation
// complex64: warp = one Morton-sorted target x 32*RPL right-hand sides; y accumulated at the original index
template <int PS, int PA, int RPL>
__global__ void __launch_bounds__(256) k_final_b(int N, const int* __restrict__ point_leaf, const int* __restrict__ leaf_start,
                                                 const int* __restrict__ leaf_count, const int* __restrict__ nbr_ptr,
                                                 const int* __restrict__ nbr_box, const int* __restrict__ near_rowlen,
                                                 const long long* __restrict__ near_off, const float2* __restrict__ near,
                                                 const float2* __restrict__ rho, const int* __restrict__ ip_ptr,
                                                 const InterpE<float>* __restrict__ ip, const float2* __restrict__ coef,
                                                 const long long* __restrict__ sorting, int B, double2* __restrict__ yt) {
    using R = float;
    constexpr int P = PS * PA;
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= N) return;
    int rr[RPL];
    bool act[RPL];
#pragma unroll
    for (int k = 0; k < RPL; ++k) {
        const int r = blockIdx.y * 32 * RPL + 32 * k + lane;
        act[k] = r < B;
        rr[k] = act[k] ? r : 0;
    }
    const int b = point_leaf[i];
    const int t = i - leaf_start[b];
    const V2<R>* row = near + near_off[b] + (long long)t * near_rowlen[b];
    V2<R> acc[RPL];
#pragma unroll
    for (int k = 0; k < RPL; ++k) { acc[k].x = R(0); acc[k].y = R(0); }
    int sg = 0;
    for (int q = nbr_ptr[b]; q < nbr_ptr[b + 1]; ++q) {
        const int bb = nbr_box[q];
        const int c = leaf_count[bb];
        const V2<R>* rh = rho + (long long)leaf_start[bb] * B;
        int s = 0;
        for (; s + 4 <= c; s += 4) {           // four sources' loads in flight at once
            V2<R> nv[4], rv[4][RPL];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                nv[u] = row[sg + s + u];
#pragma unroll
                for (int k = 0; k < RPL; ++k) rv[u][k] = rh[(long long)(s + u) * B + rr[k]];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int k = 0; k < RPL; ++k) cmac<R>(acc[k], nv[u], rv[u][k]);
        }
        for (; s < c; ++s) {
            const V2<R> nv = row[sg + s];
#pragma unroll
            for (int k = 0; k < RPL; ++k) cmac<R>(acc[k], nv, rh[(long long)s * B + rr[k]]);
        }
        sg += c;
    }
    for (int e = ip_ptr[i]; e < ip_ptr[i + 1]; ++e) {
        const InterpE<R> E = ip[e];
        R Ts[PS], Tt[PA];
        cheb_row<R, PS>(E.s, Ts);
        cheb_row<R, PA>(E.th, Tt);
        V2<R> f; f.x = E.fr; f.y = E.fi;
        const V2<R>* src = coef + (long long)E.cone * P * B;
#pragma unroll
        for (int k = 0; k < RPL; ++k) {
            V2<R> cc[P];
#pragma unroll
            for (int q = 0; q < P; ++q) cc[q] = src[(long long)q * B + rr[k]];
            cmac<R>(acc[k], interp_eval_tt<R, PS, PA>(cc, Ts, Tt), f);
        }
    }
    const long long o = sorting[i];
#pragma unroll
    for (int k = 0; k < RPL; ++k) {
        if (!act[k]) continue;
        double2* yo = yt + o * B + rr[k];
        double2 v = *yo;
        v.x += (double)acc[k].x; v.y += (double)acc[k].y;
        *yo = v;
    }
}

// complex64 near field alone (the interpolation is grouped, k_interp_grp): an item is up to 32 targets of
// one leaf box, a warp four of them x 32 RPL right-hand sides, so that a source's density row serves four
// targets.  The four table rows and the source list come through shared memory, kNearTile sources at a
// time, by the warp's own copies.  Each target's sum runs over its row in order, as in k_final_b.  Bound by
// the latency of the density rows: eight sources' are in flight (four: twice the time; the next eight in
// registers as well: 128 registers, 5 % slower at k = 2000).  Kite k = 500 / 2000, 64 right-hand sides: 102 /
// 384 us with a warp per target, 54 / 202 us so.
constexpr int kNearTile = 32;
template <int RPL>
__global__ void __launch_bounds__(256) k_near_b(const FinItem* __restrict__ items, const int* __restrict__ near_src,
                                                const float2* __restrict__ near, const float2* __restrict__ rho,
                                                const long long* __restrict__ sorting, int B, double2* __restrict__ yt) {
    __shared__ float4 rows[8][2][kNearTile][2];       // [source][targets 0, 1 | 2, 3]
    __shared__ int srcs[8][2][kNearTile];
    const FinItem I = items[blockIdx.x];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, t0 = 4 * w;
    if (t0 >= I.cnt) return;
    const int nt = min(4, I.cnt - t0);
    const float2* row = near + I.near + (long long)t0 * I.rl;
    auto fetch = [&](int c0, int b) {
        const int e = c0 + lane;
        if (e < I.rl) {
            cp_async_el<4>(&srcs[w][b][lane], near_src + I.src + e);
            float2* to = reinterpret_cast<float2*>(rows[w][b][lane]);
#pragma unroll
            for (int u = 0; u < 4; ++u) cp_async_el<8>(to + u, row + (long long)(u < nt ? u : 0) * I.rl + e);
        }
        cp_async_commit();
    };
    int rr[RPL];
    bool act[RPL];
    float2 acc[4][RPL];
#pragma unroll
    for (int k = 0; k < RPL; ++k) {
        const int r = blockIdx.y * 32 * RPL + 32 * k + lane;
        act[k] = r < B;
        rr[k] = act[k] ? r : 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[u][k] = make_float2(0.f, 0.f);
    }
    if (I.rl > 0) fetch(0, 0);
    for (int c0 = 0, b = 0; c0 < I.rl; c0 += kNearTile, b ^= 1) {
        cp_async_wait<0>();
        __syncwarp();                                 // the tile is there, the other one has been used
        if (c0 + kNearTile < I.rl) fetch(c0 + kNearTile, b ^ 1);
        const int n = min(kNearTile, I.rl - c0);
#pragma unroll 8
        for (int e = 0; e < n; ++e) {
            const float2* rh = rho + (long long)srcs[w][b][e] * B;
            const float4 v01 = rows[w][b][e][0], v23 = rows[w][b][e][1];
#pragma unroll
            for (int k = 0; k < RPL; ++k) {
                const float2 d = rh[rr[k]];
                cmac<float>(acc[0][k], make_float2(v01.x, v01.y), d);
                cmac<float>(acc[1][k], make_float2(v01.z, v01.w), d);
                cmac<float>(acc[2][k], make_float2(v23.x, v23.y), d);
                cmac<float>(acc[3][k], make_float2(v23.z, v23.w), d);
            }
        }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        if (u >= nt) break;
        const long long o = sorting[I.first + t0 + u];
#pragma unroll
        for (int k = 0; k < RPL; ++k) {
            if (!act[k]) continue;
            double2* yo = yt + o * B + rr[k];
            double2 v = *yo;
            v.x += (double)acc[u][k].x; v.y += (double)acc[u][k].y;
            *yo = v;
        }
    }
}

// FP64 in fixed point (fixpoint.cuh): warp = one Morton-sorted target x 32 right-hand sides.  The
// neighbour boxes' densities have an exponent per box, so each box's integer sum is added up in FP64.
__global__ void __launch_bounds__(256) k_near_bx(int N, const int* __restrict__ point_leaf, const int* __restrict__ leaf_start,
                                                 const int* __restrict__ leaf_count, const int* __restrict__ nbr_ptr,
                                                 const int* __restrict__ nbr_box, const int* __restrict__ near_rowlen,
                                                 const long long* __restrict__ near_off, const int4* __restrict__ near,
                                                 const int* __restrict__ nexp, const int4* __restrict__ rho,
                                                 const int* __restrict__ rexp, const long long* __restrict__ sorting, int B,
                                                 double2* __restrict__ yt) {
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
    const int r = blockIdx.y * 32 + (threadIdx.x & 31);
    if (i >= N || r >= B) return;
    const int b = point_leaf[i], En = nexp[i];
    const int4* row = near + near_off[b] + (long long)(i - leaf_start[b]) * near_rowlen[b];
    double2 acc = make_double2(0.0, 0.0);
    for (int q = nbr_ptr[b]; q < nbr_ptr[b + 1]; ++q) {
        const int bb = nbr_box[q], c = leaf_count[bb];
        const int4* rh = rho + (long long)leaf_start[bb] * B + r;
        const int Er = rexp[(long long)bb * B + r];
        for (int p0 = 0; p0 < c; p0 += kFxSumMost) {            // the sum of the box, or of kFxSumMost of its sources
            const int p1 = min(c, p0 + kFxSumMost);
            FxSum rr{0, 0}, ii{0, 0}, im{0, 0};
            for (int f0 = p0; f0 < p1; f0 += kFxSumFold) {
                const int f1 = min(p1, f0 + kFxSumFold);
#pragma unroll 4
                for (int s = f0; s < f1; ++s) {
                    const int4 a = row[s], d = rh[(long long)s * B];
                    fx_sum_mac(rr, a.x, a.y, d.x, d.y);
                    fx_sum_mac(ii, a.z, a.w, d.z, d.w);
                    fx_sum_mac(im, a.x, a.y, d.z, d.w);
                    fx_sum_mac(im, a.z, a.w, d.x, d.y);
                }
                fx_sum_fold(rr); fx_sum_fold(ii); fx_sum_fold(im);
            }
            rr.h -= ii.h; rr.m -= ii.m;
            fx_sum_fold(rr);
            if (En == kFxBad || Er == kFxBad) {
                acc.x = acc.y = __hiloint2double(0x7ff80000, 0);
            } else {
                const int E0 = En + Er - 2 * kFxSumTop;
                int er, ei;
                const long long yr = fx_sum_value(rr, E0, er), yi = fx_sum_value(im, E0, ei);
                acc.x += fx_scaled(yr, er); acc.y += fx_scaled(yi, ei);
            }
        }
        row += c;
    }
    double2* yo = yt + sorting[i] * B + r;
    double2 v = *yo;
    v.x += acc.x; v.y += acc.y;
    *yo = v;
}

// ------------------------------------------------------------------ interpolation grouped by cone
// Two warps = one work item (up to kInterpGrpTargets targets of one leaf box), 32 right-hand
// sides each.  The item's terms are sorted by cone, so each cone's 25 x B coefficient block is
// loaded once for every target of the item that reads it (k_final_b loads it once per target);
// per-target sums accumulate in shared memory, then are added into yt.  The terms come in tiles of
// kInterpGrpTile by cp.async: k = 500 / 2000, 64 right-hand sides, 117 / 353 -> 99 / 334 us.
constexpr int kInterpGrpTile = 64;
template <int PS, int PA>
__global__ void __launch_bounds__(64) k_interp_grp(const int4* __restrict__ items, int nitems, const InterpG* __restrict__ terms,
                                                   const float2* __restrict__ coef, const long long* __restrict__ sorting, int B,
                                                   double2* __restrict__ yt) {
    constexpr int P = PS * PA;
    __shared__ float2 acc[kInterpGrpTargets][64];
    __shared__ alignas(16) InterpG tile[2][kInterpGrpTile];
    const int it = blockIdx.x;
    if (it >= nitems) return;
    const int4 I = items[it];   // terms [x, y), targets [z, z + w)
    const int r = threadIdx.x;  // this thread's right-hand side
    const bool act = r < B;
    const int rr = act ? r : 0;
    for (int t = 0; t < I.w; ++t) acc[t][r] = make_float2(0.f, 0.f);   // each thread its own column
    auto fetch = [&](int e0, int b) {           // terms [e0, e0 + kInterpGrpTile) into tile b
        const int n8 = min(kInterpGrpTile, I.y - e0) * ((int)sizeof(InterpG) / 8);
        for (int i = r; i < n8; i += 64)
            cp_async_el<8>(reinterpret_cast<char*>(tile[b]) + 8 * i, reinterpret_cast<const char*>(terms + e0) + 8 * i);
        cp_async_commit();
    };
    float2 cc[P];
    int cur = -1;
    InterpG En{};
    if (I.x < I.y) fetch(I.x, 0);
    for (int e = I.x; e < I.y; ++e) {
        const int q = (e - I.x) % kInterpGrpTile, b = (e - I.x) / kInterpGrpTile & 1;
        if (q == 0) {                           // the tile has arrived, the other one has been used
            cp_async_wait<0>();
            __syncthreads();
            if (e + kInterpGrpTile < I.y) fetch(e + kInterpGrpTile, b ^ 1);
            En = tile[b][0];
        }
        const InterpG E = En;
        if (q + 1 < kInterpGrpTile) En = tile[b][q + 1];     // the next term's, before this one's sums
        if (E.cone != cur) {                    // uniform over the block
            cur = E.cone;
            const float2* src = coef + (long long)cur * P * B;
#pragma unroll
            for (int q = 0; q < P; ++q) cc[q] = src[(long long)q * B + rr];
        }
        float Ts[PS], Tt[PA];
        cheb_row<float, PS>(E.s, Ts);
        cheb_row<float, PA>(E.th, Tt);
        float2 a = acc[E.t - I.z][r];
        cmac<float>(a, interp_eval_tt<float, PS, PA>(cc, Ts, Tt), make_float2(E.fr, E.fi));
        acc[E.t - I.z][r] = a;
    }
    if (!act) return;
    for (int t = 0; t < I.w; ++t) {
        double2* yo = yt + sorting[I.z + t] * B + r;
        const float2 a = acc[t][r];
        double2 v = *yo;
        v.x += (double)a.x; v.y += (double)a.y;
        *yo = v;
    }
}

// ------------------------------------------------------------------ batched GMRES vector kernels
constexpr int kRowsPerChunk = 512;
int bdot_chunks(long long N) { return (int)((N + kRowsPerChunk - 1) / kRowsPerChunk); }

// block (chunk, column c): partial sums of conj(V_c) w over the chunk's rows, per RHS
__global__ void __launch_bounds__(256) k_bdot_part(const double2* __restrict__ V, long long ldc, const double2* __restrict__ w,
                                                   long long N, int B, double2* __restrict__ part) {
    __shared__ double2 sm[256];
    const int c = blockIdx.y, chunk = blockIdx.x, nchunk = gridDim.x;
    const int RP = 256 / B;
    const int t = threadIdx.x, g = t / B, r = t - g * B;
    double2 acc = make_double2(0.0, 0.0);
    if (g < RP) {
        const long long i0 = (long long)chunk * kRowsPerChunk;
        const long long i1 = i0 + kRowsPerChunk < N ? i0 + kRowsPerChunk : N;
        const double2* v = V + (long long)c * ldc;
        for (long long i = i0 + g; i < i1; i += RP) {
            const double2 a = v[i * B + r], b = w[i * B + r];
            acc.x = fma(a.x, b.x, fma(a.y, b.y, acc.x));
            acc.y = fma(a.x, b.y, fma(-a.y, b.x, acc.y));
        }
    }
    sm[t] = acc;
    __syncthreads();
    if (t < B) {
        double2 s = sm[t];
        for (int q = 1; q < RP; ++q) { s.x += sm[q * B + t].x; s.y += sm[q * B + t].y; }
        part[((long long)c * nchunk + chunk) * B + t] = s;
    }
}
__global__ void k_bdot_reduce(const double2* __restrict__ part, int nchunk, int ncols, int B, double2* __restrict__ h,
                              double2* __restrict__ Hcol, int add, int sqrt_row) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= ncols * B) return;
    const int c = idx / B, r = idx - c * B;
    double2 s = make_double2(0.0, 0.0);
    const double2* p = part + (long long)c * nchunk * B + r;
    for (int q = 0; q < nchunk; ++q) { s.x += p[(long long)q * B].x; s.y += p[(long long)q * B].y; }
    if (sqrt_row >= 0) {
        Hcol[(long long)sqrt_row * B + r] = make_double2(sqrt(s.x > 0.0 ? s.x : 0.0), 0.0);
        return;
    }
    if (h) h[idx] = s;
    if (Hcol) {
        double2 v = s;
        if (add) { v.x += Hcol[idx].x; v.y += Hcol[idx].y; }
        Hcol[idx] = v;
    }
}
__global__ void __launch_bounds__(256) k_bupdate(const double2* __restrict__ V, long long ldc, int ncols,
                                                 const double2* __restrict__ h, double sign, long long n, int B,
                                                 double2* __restrict__ w) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    const int r = (int)(e % B);
    double2 acc = make_double2(0.0, 0.0);
    for (int c = 0; c < ncols; ++c) {
        const double2 a = V[(long long)c * ldc + e], b = h[c * B + r];
        acc.x = fma(a.x, b.x, fma(-a.y, b.y, acc.x));
        acc.y = fma(a.x, b.y, fma(a.y, b.x, acc.y));
    }
    double2 v = w[e];
    v.x = fma(sign, acc.x, v.x); v.y = fma(sign, acc.y, v.y);
    w[e] = v;
}
__global__ void k_bscale(const double2* __restrict__ w, const double2* __restrict__ hn, long long n, int B,
                         double2* __restrict__ out) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    const double h = hn[e % B].x;
    const double s = h > 0.0 ? 1.0 / h : 0.0;
    const double2 v = w[e];
    out[e] = make_double2(v.x * s, v.y * s);
}

// columns act[0..Bc) of an interleaved [N][B] array <-> a compact [N][Bc] one
__global__ void k_gather_cols(const double2* __restrict__ in, int B, const int* __restrict__ act, int Bc, long long N,
                              double2* __restrict__ out) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= N * Bc) return;
    const long long i = e / Bc;
    out[e] = in[i * B + act[e - i * Bc]];
}
__global__ void k_scatter_cols(const double2* __restrict__ in, int Bc, const int* __restrict__ act, int B, long long N, int add,
                               double2* __restrict__ out) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= N * Bc) return;
    const long long i = e / Bc;
    double2& o = out[i * B + act[e - i * Bc]];
    const double2 v = in[e];
    if (add) { o.x += v.x; o.y += v.y; } else o = v;
}

// ------------------------------------------------------------------ launchers
void launch_gather_cols(const double2* in, int B, const int* act, int Bc, long long N, double2* out, cudaStream_t s) {
    if (N * Bc > 0) k_gather_cols<<<nblk_b(N * Bc, 256), 256, 0, s>>>(in, B, act, Bc, N, out);
}
void launch_scatter_cols(const double2* in, int Bc, const int* act, int B, long long N, bool add, double2* out, cudaStream_t s) {
    if (N * Bc > 0) k_scatter_cols<<<nblk_b(N * Bc, 256), 256, 0, s>>>(in, Bc, act, B, N, add ? 1 : 0, out);
}
void launch_interleave(const double2* x, long long N, int B, double2* xt, cudaStream_t s) {
    if (N <= 0 || B <= 0) return;
    k_interleave<<<dim3(nblk_b(N, 32), nblk_b(B, 32)), dim3(32, 8), 0, s>>>(x, N, B, xt);
}
void launch_deinterleave(const double2* xt, long long N, int B, double2* x, cudaStream_t s) {
    if (N <= 0 || B <= 0) return;
    k_deinterleave<<<dim3(nblk_b(N, 32), nblk_b(B, 32)), dim3(32, 8), 0, s>>>(xt, N, B, x);
}
void launch_sing_b(const double2* xt, const float2* xt32, const double2* W, const float2* W32, const int* row_ptr,
                   const int* row_col, const RPColumn* cols, int N, int Np, int B, double half, double2* yt,
                   const double* wq, const long long* inv, double2* rho64, float2* rho32, cudaStream_t s) {
    const dim3 grid(nblk_b(N, 8), nblk_b(B, 32));
    if (rho32)
        k_sing_b<float2, float2><<<grid, 256, 0, s>>>(xt, xt32, W32, row_ptr, row_col, cols, N, Np, B, half, yt, wq, inv, rho32);
    else
        k_sing_b<double2, double2><<<grid, 256, 0, s>>>(xt, xt, W, row_ptr, row_col, cols, N, Np, B, half, yt, wq, inv, rho64);
}
void launch_leaf_b(const int* cone_box, int ncones, int cone_base, const int* leaf_start, const int* leaf_count,
                   const long long* leaf_off, const float2* L, const float2* rho, int Ps, int Pang, int B, float2* coef,
                   cudaStream_t s) {
    if (ncones <= 0) return;
    constexpr int RPL = kRpl;
    const dim3 grid(nblk_b(ncones, kLeafWarps), nblk_b(B, 32 * RPL));
    IFGF_DISPATCH_P(Ps, Pang, (k_leaf_b<PS * PA, RPL><<<grid, kLeafWarps * 32, 0, s>>>(
                                   cone_box, ncones, cone_base, leaf_start, leaf_count, leaf_off, L, rho, B, coef)));
}
void launch_rho_bx(const int* leaf_start, const int* leaf_count, int nleaf, const double2* rho, int B, int4* out, int* rexp,
                   cudaStream_t s) {
    if (nleaf > 0 && B > 0) k_rho_bx<<<nleaf, (B + 31) / 32 * 32, 0, s>>>(leaf_start, leaf_count, rho, B, out, rexp);
}
void launch_leaf_bx(const int* cone_box, int ncones, int cone_base, const int* leaf_start, const int* leaf_count,
                    const long long* leaf_off, const int4* L, const int* lexp, const int4* rho, const int* rexp, int Ps, int Pang, int B,
                    int most, int4* coef, int* cexp, cudaStream_t s) {
    if (ncones <= 0 || B <= 0) return;
    IFGF_DISPATCH_P(Ps, Pang, {
        constexpr int P = PS * PA, MS = (P + 12) / 13;   // at most 13 coefficients (104 registers of sums) a thread
        auto go = [&](auto nt, auto big) {
            constexpr int NT = decltype(nt)::value;
            k_leaf_bx<P, MS, NT, decltype(big)::value><<<dim3(ncones, nblk_b(B, NT)), dim3(NT, MS), 0, s>>>(
                cone_box, cone_base, leaf_start, leaf_count, leaf_off, L, lexp, rho, rexp, B, Ps, coef, cexp);
        };
        using N32 = std::integral_constant<int, 32>;
        using N64 = std::integral_constant<int, 64>;
        if (most <= kFxSumMost) B <= 32 ? go(N32{}, std::false_type{}) : go(N64{}, std::false_type{});
        else B <= 32 ? go(N32{}, std::true_type{}) : go(N64{}, std::true_type{});
    });
}
void launch_prop_b(int pbegin, int pend, const long long* pp_ptr, const int* pp_nchild, const PropB<float>* pb, int Ps, int Pang,
                   const float* Gsep, int B, float2* coef, cudaStream_t s) {
    if (pend <= pbegin) return;
    constexpr int RPL = kRpl;
    IFGF_DISPATCH_P(Ps, Pang, {
        constexpr int WPB = PropBlock<PS * PA, RPL>::W;
        const dim3 grid(nblk_b(pend - pbegin, WPB), nblk_b(B, 32 * RPL));
        k_prop_b<PS, PA, WPB, RPL><<<grid, WPB * 32, 0, s>>>(pbegin, pend, pp_ptr, pp_nchild, pb, Gsep, B, coef);
    });
}
// threads (right-hand sides) of a block of the FP64 kernels: 64 share a list of terms where its shared
// memory allows (up to 36 nodes); 32 for batches that fit one warp
template <int P> struct BatchXThreads { static constexpr int v = P <= 36 ? 64 : 32; };
void launch_prop_bx(int pbegin, int pend, const long long* pp_ptr, TermsX terms, int Ps, int Pang, const int2* GsepX, int B, int4* coef,
                    int* cexp, cudaStream_t s) {
    if (pend <= pbegin || B <= 0) return;
    IFGF_DISPATCH_P(Ps, Pang, {
        constexpr int NT = BatchXThreads<PS * PA>::v;
        const dim3 grid(pend - pbegin, nblk_b(B, B <= 32 ? 32 : NT));
        if (B <= 32) k_prop_bx<PS, PA, 32><<<grid, 32, 0, s>>>(pbegin, pp_ptr, terms, GsepX, B, coef, cexp);
        else k_prop_bx<PS, PA, NT><<<grid, NT, 0, s>>>(pbegin, pp_ptr, terms, GsepX, B, coef, cexp);
    });
}
void launch_interp_bx(const int4* items, int nitems, TermsX terms, const int4* coef, const int* cexp, int Ps, int Pang,
                      const long long* sorting, int B, double2* yt, cudaStream_t s) {
    if (nitems <= 0 || B <= 0) return;
    IFGF_DISPATCH_P(Ps, Pang, {
        constexpr int NT = BatchXThreads<PS * PA>::v;
        const dim3 grid(nitems, nblk_b(B, B <= 32 ? 32 : NT));
        if (B <= 32) k_interp_bx<PS, PA, 32><<<grid, 32, 0, s>>>(items, terms, coef, cexp, sorting, B, yt);
        else k_interp_bx<PS, PA, NT><<<grid, NT, 0, s>>>(items, terms, coef, cexp, sorting, B, yt);
    });
}
bool launch_interp_grp(const int4* items, int nitems, const InterpG* terms, const float2* coef, int Ps, int Pang,
                       const long long* sorting, int B, double2* yt, cudaStream_t s) {
    if (Ps != 5 || Pang != 5 || B > 64 || B <= 0) return false;
    if (nitems <= 0) return true;
    k_interp_grp<5, 5><<<nitems, 64, 0, s>>>(items, nitems, terms, coef, sorting, B, yt);
    return true;
}
bool launch_prop_bk(int pbegin, int pend, const long long* pp_ptr, const int* pp_nchild, const PropB<float>* pb, int Ps, int Pang,
                    const float* Gsep, int B, float2* coef, int* err, cudaStream_t s) {
    if (Ps != 5 || Pang != 5 || B > 64 || B <= 0 || (B & 1)) return false;
    if (pend <= pbegin) return true;
    k_prop_bk<5, 5><<<pend - pbegin, 32 * kPropBkWarps, 0, s>>>(pbegin, pend, pp_ptr, pp_nchild, pb, Gsep, B, coef, err);
    return true;
}
void launch_final_b(int N, const int* point_leaf, const int* leaf_start, const int* leaf_count, const int* nbr_ptr,
                    const int* nbr_box, const int* near_rowlen, const long long* near_off, const float2* near,
                    const float2* rho, const int* ip_ptr, const InterpE<float>* ip, const float2* coef, int Ps, int Pang,
                    const long long* sorting, int B, double2* yt, cudaStream_t s) {
    constexpr int RPL = kRpl;
    const dim3 grid(nblk_b(N, 8), nblk_b(B, 32 * RPL));
    IFGF_DISPATCH_P(Ps, Pang, (k_final_b<PS, PA, RPL><<<grid, 256, 0, s>>>(N, point_leaf, leaf_start, leaf_count,
                                                                          nbr_ptr, nbr_box, near_rowlen, near_off, near,
                                                                          rho, ip_ptr, ip, coef, sorting, B, yt)));
}
void launch_near_b(const FinItem* items, int nitems, const int* near_src, const float2* near, const float2* rho,
                   const long long* sorting, int B, double2* yt, cudaStream_t s) {
    if (nitems > 0 && B > 0)
        k_near_b<kRpl><<<dim3(nitems, nblk_b(B, 32 * kRpl)), 256, 0, s>>>(items, near_src, near, rho, sorting, B, yt);
}
void launch_near_bx(int N, const int* point_leaf, const int* leaf_start, const int* leaf_count, const int* nbr_ptr, const int* nbr_box,
                    const int* near_rowlen, const long long* near_off, const int4* near, const int* nexp, const int4* rho,
                    const int* rexp, const long long* sorting, int B, double2* yt, cudaStream_t s) {
    if (N > 0 && B > 0)
        k_near_bx<<<dim3(nblk_b(N, 8), nblk_b(B, 32)), 256, 0, s>>>(N, point_leaf, leaf_start, leaf_count, nbr_ptr, nbr_box, near_rowlen,
                                                                   near_off, near, nexp, rho, rexp, sorting, B, yt);
}
void launch_bdot(const double2* V, long long ldc, int ncols, const double2* w, long long N, int B, double2* part,
                 double2* h, double2* Hcol, int add, int sqrt_row, cudaStream_t s) {
    if (ncols <= 0) return;
    const int nchunk = bdot_chunks(N);
    k_bdot_part<<<dim3(nchunk, ncols), 256, 0, s>>>(V, ldc, w, N, B, part);
    k_bdot_reduce<<<nblk_b((long long)ncols * B, 256), 256, 0, s>>>(part, nchunk, ncols, B, h, Hcol, add, sqrt_row);
}
void launch_bupdate(const double2* V, long long ldc, int ncols, const double2* h, double sign, long long N, int B, double2* w,
                    cudaStream_t s) {
    if (ncols <= 0) return;
    k_bupdate<<<nblk_b(N * B, 256), 256, 0, s>>>(V, ldc, ncols, h, sign, N * B, B, w);
}
void launch_bscale(const double2* w, const double2* hn, long long N, int B, double2* out, cudaStream_t s) {
    k_bscale<<<nblk_b(N * B, 256), 256, 0, s>>>(w, hn, N * B, B, out);
}

}  // namespace ifgf

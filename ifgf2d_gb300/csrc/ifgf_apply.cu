// ifgf_apply.cu -- per-apply IFGF kernels, in two forms.
//
// FP64 (..._fx): tables, cone coefficients and sums in block fixed point of FP64 accuracy
//                (fixpoint.cuh), the factor ratios in FP64.
// complex64    : complex64 copies of the same FP64-computed tables, FP32 arithmetic; the
//                rectangular-polar correction stays FP64.
//
//   k_intensities_t                density * quadrature weight, Morton permutation  ForwardMap.tpp:425-435, BoxTree.h:954-963
//   k_leaf_fx, k_leaf_apply_t      leaf cone coefficients                          BoxTree.h:685-762
//   k_propagate_fx, k_propagate_t  child -> parent coefficients, separable
//                                  values->coefficients map                        BoxTree.h:767-868, Interpolator.h:81-120
//   k_final_fx, k_final_q          near field + every level's cousin interpolants by leaf box (k_final_t by
//                                  target), added to y at the target's original index
//                                                                                  BoxTree.h:614-683, 876-937, 1063-1069
#include "fixpoint.cuh"
#include "tcgen05.cuh"
#include <type_traits>
#include <algorithm>
#include <atomic>

namespace ifgf {

template <typename R>
__global__ void k_intensities_t(const double2* __restrict__ x, const double* __restrict__ wq, const long long* __restrict__ perm,
                                int N, V2<R>* __restrict__ rho) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const long long o = perm ? perm[i] : i;
    const double2 v = x[o];
    const double w = wq[o];
    V2<R> r; r.x = (R)(v.x * w); r.y = (R)(v.y * w);
    rho[i] = r;
}

// complex64 leaf cones, thread = (cone, source chunk, coefficient).  CH threads share one (cone,
// coefficient): chunk ch takes the sources s = ch, ch + CH, ..., by turns into two sums; the CH partial sums
// meet in shared memory.  Boxes hold 10-100 points, so splitting the source walk shortens the latency
// chain of the longest boxes by CH.  cones: a cone's table offset (two ints), first source and sources, one
// load ahead of the table's.  Bound by the loads in flight: 1536 threads an SM, each with the next four table
// entries on their way while it uses four; the table, read once, is marked to leave the caches first.  Kite
// k = 500 / 2000 (72 / 600 MB): 22 / 113 us; 24 / 119 with 2048 threads and four loads at a time, 28 / 129 with
// two and the box looked up first.  Six loads at a time in 61 registers, half the threads: 30 / 147.
constexpr int kLeafAhead = 4;                  // even: the two sums take the entries by turns
template <int CH>
__global__ void __launch_bounds__(256, 6) k_leaf_apply_t(const int4* __restrict__ cones, int ncones, int cone_base,
                                                      const float2* __restrict__ L, const float2* __restrict__ rho, int P,
                                                      float2* __restrict__ coef) {
    __shared__ float2 part[256];
    const int per_cone = P * CH;
    const int cpb = blockDim.x / per_cone;
    const int local = threadIdx.x / per_cone, r = threadIdx.x - local * per_cone;
    const int ch = r / P, m = r - ch * P;
    const int c = blockIdx.x * cpb + local;
    const bool active = local < cpb && c < ncones;
    float2 a0 = make_float2(0.f, 0.f), a1 = a0;
    if (active) {
        const int4 D = cones[c];
        const int n = D.w;
        const float2* Lc = L + ((long long)D.y << 32 | (unsigned)D.x) + m;
        const float2* rh = rho + D.z;
        float2 l[kLeafAhead];
        int s = ch;
#pragma unroll
        for (int u = 0; u < kLeafAhead; ++u) if (s + u * CH < n) l[u] = __ldcs(&Lc[(long long)(s + u * CH) * P]);
        while (s < n) {
            float2 now[kLeafAhead];
            const int next = s + kLeafAhead * CH;
#pragma unroll
            for (int u = 0; u < kLeafAhead; ++u) {             // the next entries on their way before these are used
                now[u] = l[u];
                if (next + u * CH < n) l[u] = __ldcs(&Lc[(long long)(next + u * CH) * P]);
            }
#pragma unroll
            for (int u = 0; u < kLeafAhead; ++u) if (s + u * CH < n) cmac<float>(u % 2 ? a1 : a0, now[u], rh[s + u * CH]);
            s = next;
        }
        a0.x += a1.x; a0.y += a1.y;
    }
    part[threadIdx.x] = a0;
    __syncthreads();
    if (active && ch == 0) {
        float2 acc = a0;
        for (int q = 1; q < CH; ++q) { const float2 v = part[local * per_cone + q * P + m]; acc.x += v.x; acc.y += v.y; }
        coef[(long long)(cone_base + c) * P + m] = acc;
    }
}

// The FP64 form of the same in fixed point (fixpoint.cuh): table and densities as 27-bit limbs, 12 wide
// multiply-adds an entry where FP64 took 4 of the FP64 pipe's operations.  A block takes up to
// 256 / (P CH) cones of one leaf box (items: table offset, first cone, cones, first source,
// sources): it brings the box's densities to their exponent in shared memory once, while its threads'
// first table entries are in flight; the chunks' integer sums meet in shared memory; then the cone's
// coefficients, whose entries have an exponent per coefficient, are brought to the cone's exponent.
// Bound by the table's loads in flight: a thread has the next three entries on their way while it uses
// three, and three are ahead of the barriers; the table, read once, is marked to leave the caches first.
// Kite k = 500 / 2000, 145 MB / 1.2 GB of table: 90 / 580 us with FP64 multiply-adds, 43 / 229 us so (3.4 / 5.2
// TB/s); without the next entries on their way 53 / 281; two or five at a time 49 / 246, 43 / 227.  The kernel is
// held to the 64 registers that let 4 blocks share an SM: left alone it took 68, and the apply 6 / 35 us
// longer.  CH = 2 keeps blocks of 5 cones, which amortises the conversion; without the
// look-ahead 5 took 67 / 350 us, 1 took 65 / 272.
// BIG, a box of more than kFxSumMost sources: a thread's sums of a chunk go to parts in shared memory that
// add up without loss.
constexpr int kLeafFxAhead = 3;
template <int CH>
struct LeafFx {
    static constexpr int chunk = CH > 1 ? 256 : 128;   // sources staged at a time, at most kFxSumMost a thread
    int4 sr[chunk];
    FxSum part[256][2];
    int stop[256], smax;
};
template <int CH, bool BIG>
__device__ __forceinline__ void leaf_fx(LeafFx<CH>& S, const LeafItem& I, int split, int cone_base, const int4* __restrict__ L,
                                        const int* __restrict__ lexp, const double2* __restrict__ rho, int P, int Ps,
                                        int4* __restrict__ coef, int* __restrict__ cexp) {
    constexpr int CHUNK = LeafFx<CH>::chunk;
    static_assert(CHUNK <= CH * kFxSumMost, "a thread's share of a chunk fits its sums");
    const int per_cone = P * CH, cpb = blockDim.x / per_cone, tid = threadIdx.x;
    const int local = tid / per_cone, r = tid - local * per_cone;
    const int ch = CH > 1 ? r / P : 0, m = r - ch * P;
    const int q = (blockIdx.x % split) * cpb + local;         // cone of the item
    const bool active = q < I.cones;
    const int n = I.n, c = I.cone + q, K = BIG ? fx_sum_wide(n) : 0;
    const int4* Lc = L + I.off + (long long)q * n * P + m;
    const double2* rh = rho + I.first;
    int4 ahead[kLeafFxAhead];
    int El = 0;
    if (active) {
#pragma unroll
        for (int u = 0; u < kLeafFxAhead; ++u) if (ch + u * CH < n) ahead[u] = __ldcs(&Lc[(long long)(ch + u * CH) * P]);
        El = lexp[(long long)c * P + m];
    }
    S.stop[tid] = kFxMinExp;
    if (BIG) S.part[tid][0] = S.part[tid][1] = FxSum{0, 0};
    if (tid == 0) S.smax = 0;
    __syncthreads();
    int mx = 0;
    for (int i = tid; i < n; i += blockDim.x) { const double2 v = rh[i]; mx = max(mx, fx_absmax_hi(v.x, v.y)); }
    if (mx) atomicMax(&S.smax, mx);
    __syncthreads();
    const int Er = fx_expo(S.smax);
    constexpr int T = kFxSumTop;
    FxSum rr{0, 0}, ii{0, 0}, im{0, 0};
    auto add = [&](int4 l, int4 d) {
        fx_sum_mac(rr, l.x, l.y, d.x, d.y);
        fx_sum_mac(ii, l.z, l.w, d.z, d.w);
        fx_sum_mac(im, l.x, l.y, d.z, d.w);
        fx_sum_mac(im, l.z, l.w, d.x, d.y);
    };
    for (int c0 = 0; c0 < (BIG ? n : 1); c0 += CHUNK) {
        const int c1 = BIG ? min(n, c0 + CHUNK) : n;
        if (c0) __syncthreads();               // the previous chunk has been read
        for (int i = c0 + tid; i < c1; i += blockDim.x) {
            const double2 v = rh[i];
            S.sr[i - c0] = Er == kFxBad ? make_int4(0, 0, 0, 0) : fx_pack_sum(fx_from(v.x, Er, T), fx_from(v.y, Er, T));
        }
        __syncthreads();
        if (active) {
            int s = c0 + (ch + CH - c0 % CH) % CH, terms = 0;
            if (c0) {
#pragma unroll
                for (int u = 0; u < kLeafFxAhead; ++u) if (s + u * CH < n) ahead[u] = __ldcs(&Lc[(long long)(s + u * CH) * P]);
            }
            while (s < c1) {
                int4 now[kLeafFxAhead];
                const int next = s + kLeafFxAhead * CH;
#pragma unroll
                for (int u = 0; u < kLeafFxAhead; ++u) {      // the next entries on their way before these are used
                    now[u] = ahead[u];
                    if (next + u * CH < c1) ahead[u] = __ldcs(&Lc[(long long)(next + u * CH) * P]);
                }
#pragma unroll
                for (int u = 0; u < kLeafFxAhead; ++u) if (s + u * CH < c1) add(now[u], S.sr[s + u * CH - c0]);
                s = next;
                terms += kLeafFxAhead;
                if (terms + kLeafFxAhead > kFxSumFold) { fx_sum_fold(rr); fx_sum_fold(ii); fx_sum_fold(im); terms = 0; }
            }
            fx_sum_fold(rr); fx_sum_fold(ii); fx_sum_fold(im);
            if (BIG) {
                fx_sum_part(S.part[tid][0], FxSum{rr.h - ii.h, rr.m - ii.m}, K);
                fx_sum_part(S.part[tid][1], im, K);
                rr = ii = im = FxSum{0, 0};
            }
        }
    }
    FxSum re{rr.h - ii.h, rr.m - ii.m};
    if (BIG) { re = S.part[tid][0]; im = S.part[tid][1]; }
    if constexpr (CH > 1) {
        if (!BIG) { S.part[tid][0] = re; S.part[tid][1] = im; }
        __syncthreads();
    }
    long long yr = 0, yi = 0;
    int er = 0, ei = 0;
    if (active && ch == 0) {
        for (int k = 1; k < CH; ++k) {
            const FxSum a = S.part[tid + k * P][0], b = S.part[tid + k * P][1];
            re.h += a.h; re.m += a.m; im.h += b.h; im.m += b.m;
        }
        fx_sum_fold(re, K); fx_sum_fold(im, K);
        const bool bad = Er == kFxBad || El == kFxBad;
        const int E0 = bad ? 0 : El + Er - kFxSumTop - T;
        yr = fx_sum_value(re, E0, er, K);
        yi = fx_sum_value(im, E0, ei, K);
        atomicMax(&S.stop[local], bad ? kFxBad : max(fx_top_of(yr, er), fx_top_of(yi, ei)));
    }
    __syncthreads();
    if (active && ch == 0) {
        const int E = S.stop[local] > kFxMaxExp ? kFxBad : S.stop[local], Tc = fx_top(P);
        const long long xr = E == kFxBad ? 0 : fx_align(yr, er, E, Tc), xi = E == kFxBad ? 0 : fx_align(yi, ei, E, Tc);
        coef[(long long)(cone_base + c) * P + m] = m % Ps ? fx_pack(xr, xi) : fx_pack_raw(xr, xi);
        if (m == 0) cexp[cone_base + c] = E;
    }
}
template <int CH>
__global__ void __launch_bounds__(256, CH > 1 ? 4 : 0) k_leaf_fx(const LeafItem* __restrict__ items, int split, int cone_base,
                                                 const int4* __restrict__ L, const int* __restrict__ lexp,
                                                 const double2* __restrict__ rho, int P, int Ps, int4* __restrict__ coef,
                                                 int* __restrict__ cexp) {
    __shared__ LeafFx<CH> S;
    const LeafItem I = items[blockIdx.x / split];
    if (I.n <= kFxSumMost) leaf_fx<CH, false>(S, I, split, cone_base, L, lexp, rho, P, Ps, coef, cexp);
    else leaf_fx<CH, true>(S, I, split, cone_base, L, lexp, rho, P, Ps, coef, cexp);
}

// set-up: a leaf cone's FP64 table in place as 27-bit limbs, an exponent per coefficient; l32 (may be
// null) receives the complex64 copy
__global__ void __launch_bounds__(256) k_leaf_fix(const int* __restrict__ cone_box, const int* __restrict__ leaf_count,
                                                  const long long* __restrict__ leaf_off, int P, double2* __restrict__ L,
                                                  int* __restrict__ lexp, float2* __restrict__ l32) {
    __shared__ int smax[kMaxP];
    const int c = blockIdx.x;
    const long long o = leaf_off[c];
    const int n = leaf_count[cone_box[c]] * P;
    for (int m = threadIdx.x; m < P; m += blockDim.x) smax[m] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) { const double2 v = L[o + i]; atomicMax(&smax[i % P], fx_absmax_hi(v.x, v.y)); }
    __syncthreads();
    for (int m = threadIdx.x; m < P; m += blockDim.x) lexp[(long long)c * P + m] = fx_expo(smax[m]);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double2 v = L[o + i];
        const int E = fx_expo(smax[i % P]);
        if (l32) l32[o + i] = make_float2((float)v.x, (float)v.y);
        reinterpret_cast<int4*>(L)[o + i] =
            E == kFxBad ? make_int4(0, 0, 0, 0) : fx_pack_sum(fx_from(v.x, E, kFxSumTop), fx_from(v.y, E, kFxSumTop));
    }
}
// complex64 leaf cones with the table streamed by the tensor memory accelerator.  A persistent
// CTA walks its cones (blockIdx.x, + gridDim.x, ...) in pieces of at most kLtSrc sources; thread 0
// keeps kLtStages pieces in flight, each two cp.async.bulk copies (the piece's table rows and its
// densities) into a shared-memory ring, counted on the stage's mbarrier.  Each copy starts at the
// 16-byte boundary at or below its data (the table and density arrays carry 16 bytes of padding
// at their ends).  Threads (chunk, m) sum L[s][m] rho[s] over the piece's sources s = chunk mod kLtChunks,
// and a cone's chunk partials are reduced in shared memory.  Waits are bounded: one that runs
// out sets *err, waits once more for the copies in flight and stops the CTA.
constexpr int kLtSrc = 64, kLtStages = 4, kLtChunks = 5, kLtThreads = 128;
template <int P>
struct LeafTma {
    static constexpr int table = (kLtSrc * P * 8 + 16 + 127) / 128 * 128;   // table rows, then the densities
    static constexpr int stage = table + (kLtSrc * 8 + 16 + 127) / 128 * 128;
    static constexpr int part_off = kLtStages * stage;
    static constexpr int bar_off = part_off + kLtChunks * P * 8;
    static constexpr int smem = bar_off + 8 * kLtStages;
};
template <int P>
__global__ void __launch_bounds__(kLtThreads) k_leaf_tma(const int* __restrict__ cone_box, int ncones, int cone_base,
                                                         const int* __restrict__ leaf_start, const int* __restrict__ leaf_count,
                                                         const long long* __restrict__ leaf_off, const float2* __restrict__ L,
                                                         const float2* __restrict__ rho, float2* __restrict__ coef,
                                                         int* __restrict__ err) {
    static_assert(kLtChunks * P <= kLtThreads, "a thread per (chunk, coefficient)");
    using LT = LeafTma<P>;
    extern __shared__ __align__(128) unsigned char sm[];
    const int tid = threadIdx.x;
    const bool comp = tid < kLtChunks * P;
    const int ch = tid / P, m = tid - (tid / P) * P;
    float2* part = reinterpret_cast<float2*>(sm + LT::part_off);
    auto bar = [&](int st) { return tc5::smem_u32(sm + LT::bar_off + 8 * st); };
    // producer cursor (thread 0): the next piece to fetch
    int fc = blockIdx.x, fq = 0;
    auto piece_src = [&](int c, int q, int& n, int& len) {
        n = leaf_count[cone_box[c]];
        len = min(kLtSrc, n - q * kLtSrc);
        return reinterpret_cast<unsigned long long>(L + leaf_off[c] + (long long)q * kLtSrc * P);
    };
    auto fetch = [&](int st) {
        if (fc >= ncones) return;
        int n, len;
        const unsigned long long a = piece_src(fc, fq, n, len);
        const unsigned long long a0 = a & ~15ull;
        const uint32_t bytes = (uint32_t)(((a - a0) + (unsigned long long)len * P * 8 + 15) & ~15ull);
        const unsigned long long r = reinterpret_cast<unsigned long long>(rho + leaf_start[cone_box[fc]] + fq * kLtSrc);
        const unsigned long long r0 = r & ~15ull;
        const uint32_t rbytes = (uint32_t)(((r - r0) + (unsigned long long)len * 8 + 15) & ~15ull);
        tc5::mbar_expect_tx(bar(st), bytes + rbytes);
        tc5::bulk_g2s_counted(tc5::smem_u32(sm + st * LT::stage), reinterpret_cast<const void*>(a0), bytes, bar(st));
        tc5::bulk_g2s_counted(tc5::smem_u32(sm + st * LT::stage + LT::table), reinterpret_cast<const void*>(r0), rbytes, bar(st));
        if (++fq * kLtSrc >= n) { fq = 0; fc += gridDim.x; }
    };
    if (tid == 0) {
        for (int st = 0; st < kLtStages; ++st) tc5::mbar_init(bar(st), 1);
        for (int st = 0; st < kLtStages; ++st) fetch(st);
    }
    __syncthreads();
    long long piece = 0;
    int c = blockIdx.x, q = 0;
    float2 acc = make_float2(0.f, 0.f);
    bool ok = true;
    while (c < ncones) {
        const int st = (int)(piece % kLtStages);
        ok = __syncthreads_and(tc5::mbar_wait(bar(st), (uint32_t)((piece / kLtStages) & 1), 2000000000ll));
        if (!ok) break;
        int n, len;
        const unsigned long long a = piece_src(c, q, n, len);
        const float2* data = reinterpret_cast<const float2*>(sm + st * LT::stage + (a & 15ull));
        if (comp) {
            const unsigned long long r = reinterpret_cast<unsigned long long>(rho + leaf_start[cone_box[c]] + q * kLtSrc);
            const float2* rh = reinterpret_cast<const float2*>(sm + st * LT::stage + LT::table + (r & 15ull));
            for (int s2 = ch; s2 < len; s2 += kLtChunks) cmac<float>(acc, data[s2 * P + m], rh[s2]);
        }
        __syncthreads();                        // the stage has been read
        if (tid == 0) fetch(st);                // refill it with the piece kLtStages ahead
        ++piece;
        if (++q * kLtSrc >= n) {                // the cone is complete
            if (comp) part[ch * P + m] = acc;
            __syncthreads();
            if (comp && ch == 0) {
                float2 t = part[m];
                for (int k2 = 1; k2 < kLtChunks; ++k2) { t.x += part[k2 * P + m].x; t.y += part[k2 * P + m].y; }
                coef[(long long)(cone_base + c) * P + m] = t;
            }
            acc = make_float2(0.f, 0.f);
            q = 0;
            c += gridDim.x;
        }
    }
    if (!ok && tid == 0) {   // the pieces fetched ahead may still land: one more bounded wait each
        atomicExch(err, 1);
        for (int i = 0; i < kLtStages; ++i) {
            const long long p2 = piece + i;
            tc5::mbar_wait(bar((int)(p2 % kLtStages)), (uint32_t)((p2 / kLtStages) & 1), 2000000000ll);
        }
    }
}

// complex64: thread = (parent cone, interpolation node); CPB cones per block.  Gsep = [PS x PS radial
// map | PA x PA angular map] of the values->coefficients transform, normalisation included.
template <int PS, int PA, int CPB>
__global__ void __launch_bounds__(256) k_propagate_t(int pbegin, int pend, const long long* __restrict__ pp_ptr,
                                                     const int* __restrict__ pp_nchild, const PropE<float>* __restrict__ pp,
                                                     const float* __restrict__ Gsep, float2* __restrict__ coef) {
    using R = float;
    constexpr int P = PS * PA;
    __shared__ V2<R> sv[CPB][P];
    __shared__ V2<R> su[CPB][P];
    __shared__ R sGs[PS * PS], sGa[PA * PA];
    for (int i = threadIdx.x; i < PS * PS; i += blockDim.x) sGs[i] = Gsep[i];
    for (int i = threadIdx.x; i < PA * PA; i += blockDim.x) sGa[i] = Gsep[PS * PS + i];
    const int local = threadIdx.x / P, pt = threadIdx.x - local * P;
    const int pc = pbegin + blockIdx.x * CPB + local;
    const bool active = local < CPB && pc < pend;
    if (active) {
        const long long e0 = pp_ptr[pc];
        const int nch = pp_nchild[pc];
        V2<R> v; v.x = R(0); v.y = R(0);
        // all plan entries first, then two children's coefficient gathers before any arithmetic
        PropE<R> E[4];
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) if (ch < nch) E[ch] = pp[e0 + (long long)ch * P + pt];
#pragma unroll
        for (int c0 = 0; c0 < 4; c0 += 2) {
            if (c0 >= nch) break;
            V2<R> ca[P], cb[P];
            const V2<R>* pa = coef + (long long)E[c0].child_cone * P;
            const bool two = c0 + 1 < nch;
            const int cb_cone = two ? E[c0 + 1].child_cone : E[c0].child_cone;
            const V2<R>* pb = coef + (long long)cb_cone * P;
#pragma unroll
            for (int q = 0; q < P; ++q) { ca[q] = pa[q]; cb[q] = pb[q]; }
            V2<R> w; w.x = E[c0].wr; w.y = E[c0].wi;
            cmac<R>(v, interp_eval<R, PS, PA>(ca, E[c0].s, E[c0].th), w);
            if (two) {
                w.x = E[c0 + 1].wr; w.y = E[c0 + 1].wi;
                cmac<R>(v, interp_eval<R, PS, PA>(cb, E[c0 + 1].s, E[c0 + 1].th), w);
            }
        }
        sv[local][pt] = v;
    }
    __syncthreads();
    const int m = pt % PS, l = pt / PS;
    if (active) {            // u[l][m] = sum_k Gs[m][k] v[l*PS + k]
        V2<R> u; u.x = R(0); u.y = R(0);
#pragma unroll
        for (int k = 0; k < PS; ++k) {
            const R g = sGs[m * PS + k];
            const V2<R> v = sv[local][l * PS + k];
            u.x = rfma(g, v.x, u.x); u.y = rfma(g, v.y, u.y);
        }
        su[local][l * PS + m] = u;
    }
    __syncthreads();
    if (active) {            // c[n][m] = sum_l Ga[n][l] u[l][m], stored at n*PS + m
        const int n = l;
        V2<R> c; c.x = R(0); c.y = R(0);
#pragma unroll
        for (int q = 0; q < PA; ++q) {
            const R g = sGa[n * PA + q];
            const V2<R> u = su[local][q * PS + m];
            c.x = rfma(g, u.x, c.x); c.y = rfma(g, u.y, c.y);
        }
        coef[(long long)pc * P + n * PS + m] = c;
    }
}

// k_propagate_fx's blocks: parent cones (a thread per node), child blocks held in shared memory, and
// the block's record: first plan entry (two ints), staged children, the cones' first entries from it
// (cones + 1), the children
constexpr int kPropFxThreads = 128;
template <int P>
struct PropFx {
    static constexpr int cones = kPropFxThreads / P;
    static constexpr int slots = 12000 / (16 * P);
    static constexpr int list = 4 + cones;
    static constexpr int record = list + slots;
    static constexpr int terms = cones * 4 * P;
};
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// FP64 in fixed point (fixpoint.cuh).  A block takes a group of PropFx::cones parent cones.  The group's
// terms are one contiguous range of the plan; the range and the distinct child blocks it reads (listed
// at set-up, k_stage_plan; about four per parent cone, each read by some 14 terms) are copied into
// shared memory, all copies in flight together behind the group's one record.  Every term gets a thread
// (no lane waits for a cone with more children); then a thread per node sums its children in order.  A
// term interpolates in integers (about 160 wide multiply-adds) and takes 6 FP64 operations for its
// conversion and factor ratio, against 60 with FP64 interpolation.  The node values get their cone's
// common exponent, the values->coefficients map runs in integers again, and the coefficients are
// normalised to the top bits of the cone's largest.  Kite, all levels: k = 500 290 -> 96 us, k = 2000
// 1287 -> 381 us (the FP64 kernel before it ran at 91-95 % of the FP64 pipe).  What bounds it: the wide
// multiply-adds and 64-bit shifts take two issue slots each; some 41 % of the slots issue.  Measured
// slower: a thread per node gathering from L1 (110 us), a warp per parent cone (131 us: 25 of 32
// lanes), persistent blocks that fetch ahead (111-125 us).
template <int PS, int PA>
__global__ void __launch_bounds__(kPropFxThreads) k_propagate_fx(int pbegin, int pend, PlanX pp, const int* __restrict__ stage,
                                                                 const int2* __restrict__ Gsep, int4* __restrict__ coef,
                                                                 int* __restrict__ cexp) {
    constexpr int P = PS * PA, T = fx_top(P), NT = kPropFxThreads;
    using F = PropFx<P>;
    constexpr int CPB = F::cones, CAP = F::slots;
    static_assert(CPB * P <= NT && F::terms <= 4 * NT, "a thread per node, at most four terms a thread");
    __shared__ int4 blk[CAP * P];
    __shared__ longlong2 sst[F::terms];
    __shared__ double2 val[F::terms];          // the terms' factor ratios, then their values
    __shared__ int4 sv[CPB * P];
    __shared__ int2 sGs[PS * PS], sGa[PA * PA];
    __shared__ int rec[F::record], sE[CAP], smax[CPB], slz[CPB];
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    for (int i = tid; i < F::record; i += NT) rec[i] = stage[(long long)blockIdx.x * F::record + i];
    for (int i = tid; i < PS * PS; i += NT) sGs[i] = Gsep[i];
    for (int i = tid; i < PA * PA; i += NT) sGa[i] = Gsep[PS * PS + i];
    if (tid < CPB) { smax[tid] = 0; slz[tid] = 64; }
    __syncthreads();
    const long long e0 = ((long long)rec[1] << 32) | (unsigned)rec[0];
    const int ns = rec[2], nt = rec[3 + CPB];
    for (int k = wp; k < ns; k += NT / 32) {
        const int4* src = coef + (long long)rec[F::list + k] * P;
#pragma unroll
        for (int i = 0; i < P; i += 32) if (lane + i < P) cp_async16(&blk[k * P + lane + i], src + lane + i);
    }
    int slot[4] = {0, 0, 0, 0};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int t = tid + k * NT;
        if (t < nt) {
            cp_async16(&sst[t], pp.st + e0 + t);
            cp_async16(&val[t], pp.w + e0 + t);
            slot[k] = pp.slot[e0 + t];
        }
    }
    for (int i = tid; i < ns; i += NT) sE[i] = cexp[rec[F::list + i]];
    cp_async_wait_all();
    __syncthreads();
#pragma unroll 1
    for (int k = 0; k < 4; ++k) {
        const int t = tid + k * NT, sl = k == 0 ? slot[0] : (k == 1 ? slot[1] : (k == 2 ? slot[2] : slot[3]));
        if (t >= nt) break;
        double2 it;
        if (sl < CAP) {
            it = fx_interp_value<PS, PA>([&](int i) { return blk[sl * P + i]; }, sE[sl], sst[t]);
        } else {   // more distinct children than slots
            const int c = pp.child[e0 + t];
            const int4* src = coef + (long long)c * P;
            it = fx_interp_value<PS, PA>([&](int i) { return src[i]; }, cexp[c], sst[t]);
        }
        const double2 w = val[t];
        val[t] = make_double2(it.x * w.x - it.y * w.y, it.x * w.y + it.y * w.x);
    }
    __syncthreads();
    const int local = tid / P, pt = tid - local * P, m = pt % PS, l = pt / PS;
    const int pc = pbegin + blockIdx.x * CPB + local;
    const bool active = local < CPB && pc < pend;
    double2 v = make_double2(0.0, 0.0);
    if (active) {
        for (int t = rec[3 + local] + pt; t < rec[4 + local]; t += P) { v.x += val[t].x; v.y += val[t].y; }
        atomicMax(&smax[local], fx_absmax_hi(v.x, v.y));
    }
    __syncthreads();
    const int E = active ? fx_expo(smax[local]) : 0;
    if (active) sv[tid] = E == kFxBad ? make_int4(0, 0, 0, 0) : fx_pack(fx_from(v.x, E, T), fx_from(v.y, E, T));
    __syncthreads();
    int4* su = blk;          // the child blocks have been read
    if (active) {            // u[l][m] = sum_k Gs[m][k] v[l*PS + k]
        long long ur, ui;
        fx_map<PS>([&](int k) { return sGs[m * PS + k]; }, [&](int k) { return sv[local * P + l * PS + k]; }, ur, ui);
        su[tid] = fx_pack(ur, ui);
    }
    __syncthreads();
    long long cr = 0, ci = 0;
    if (active) {            // c[n][m] = sum_l Ga[n][l] u[l][m], stored at n*PS + m
        fx_map<PA>([&](int q) { return sGa[l * PA + q]; }, [&](int q) { return su[local * P + q * PS + m]; }, cr, ci);
        atomicMin(&slz[local], min(__clzll(cr < 0 ? -cr : cr), __clzll(ci < 0 ? -ci : ci)));
    }
    __syncthreads();
    if (active) {
        int sh = slz[local] - (63 - T);      // left shift that brings the largest to [2^(T-1), 2^T)
        sh = E == kFxBad ? 0 : min(sh, E - kFxMinExp);
        cr = fx_shift(cr, sh); ci = fx_shift(ci, sh);
        coef[(long long)pc * P + pt] = m ? fx_pack(cr, ci) : fx_pack_raw(cr, ci);
        if (pt == 0) cexp[pc] = E == kFxBad ? kFxBad : E - sh;
    }
}

// set-up of k_propagate_fx: a group's record with the first PropFx::slots of its distinct child cones
// in ascending order, and per term its slot (PropFx::slots: not staged).  All levels in one launch: a level by
// itself takes the latency of one group's searches, 24 to 29 us at k = 500 however few its groups.
template <int P>
__global__ void __launch_bounds__(kPropFxThreads) k_stage_plan(const __grid_constant__ StageLevels L, const long long* __restrict__ pp_ptr,
                                                               PlanX pp, int* __restrict__ stage) {
    using F = PropFx<P>;
    constexpr int CPB = F::cones, CAP = F::slots, NT = kPropFxThreads;
    __shared__ int kid[F::terms], uniq[F::terms];
    __shared__ int nu;
    const int tid = threadIdx.x;
    int l = 0;
    while (l + 1 < L.n && (int)blockIdx.x >= L.group[l + 1]) ++l;
    const int c0 = L.begin[l] + ((int)blockIdx.x - L.group[l]) * CPB, nc = min(CPB, L.end[l] - c0);
    const long long e0 = pp_ptr[c0];
    const int nt = min((int)(pp_ptr[c0 + nc] - e0), F::terms);
    if (tid == 0) nu = 0;
    for (int t = tid; t < nt; t += NT) kid[t] = pp.child[e0 + t];
    __syncthreads();
    for (int t = tid; t < nt; t += NT) {       // a child's first term lists it (neighbouring terms mostly share a child)
        const int c = kid[t];
        bool first = true;
        for (int q = t - 1; q >= 0 && first; --q) first = kid[q] != c;
        if (first) uniq[atomicAdd(&nu, 1)] = c;
    }
    __syncthreads();
    int* rec = stage + (long long)blockIdx.x * F::record;
    const int n = nu;
    if (tid == 0) { rec[0] = (int)e0; rec[1] = (int)(e0 >> 32); rec[2] = min(n, CAP); }
    if (tid <= CPB) rec[3 + tid] = (int)(pp_ptr[c0 + min(tid, nc)] - e0);
    for (int i = n + tid; i < CAP; i += NT) rec[F::list + i] = 0;
    for (int t = tid; t < nt; t += NT) {
        const int c = kid[t];
        int r = 0;
        for (int q = 0; q < n; ++q) r += uniq[q] < c;
        pp.slot[e0 + t] = (unsigned short)min(r, CAP);
        if (r < CAP) rec[F::list + r] = c;
    }
}

// k_propagate_t with the child coefficient blocks staged in shared memory.  A parent cone's 25
// nodes read 1-4 children's blocks each, but the block's ten parent cones touch only about 40
// distinct child cones (3.4-4.3 per parent cone on the kite trees), so the per-thread gathers
// of k_propagate_t read each block about twelve times.  Here the block first collects its
// distinct child cones in a shared hash table (open addressing, at most kStageKeys probes),
// copies each one's block once with coalesced loads, and evaluates from shared memory.  A child
// cone that finds no free key or no data slot is read from global memory.  Each thread's
// arithmetic is that of k_propagate_t in the same order, so the results are bit-identical.
// On the kite trees the 25 shared-memory reads per term cost as much as the L1 hits they replace.
constexpr int kStageKeys = 128;
template <typename R, int P>
struct PropStage {
    static constexpr int cap = (size_t)P * sizeof(V2<R>) * 64 <= 26000 ? 64 : (int)(26000 / ((size_t)P * sizeof(V2<R>)));
};
template <int PS, int PA, int CPB>
__global__ void __launch_bounds__(256) k_propagate_st(int pbegin, int pend, const long long* __restrict__ pp_ptr,
                                                      const int* __restrict__ pp_nchild, const PropE<float>* __restrict__ pp,
                                                      const float* __restrict__ Gsep, float2* __restrict__ coef) {
    using R = float;
    constexpr int P = PS * PA;
    constexpr int CAP = PropStage<R, P>::cap;
    __shared__ int key[kStageKeys], slot_of[kStageKeys], ulist[CAP];
    __shared__ int nused;
    __shared__ V2<R> blk[CAP][P];
    __shared__ V2<R> sv[CPB][P];
    __shared__ V2<R> su[CPB][P];
    __shared__ R sGs[PS * PS], sGa[PA * PA];
    for (int i = threadIdx.x; i < PS * PS; i += blockDim.x) sGs[i] = Gsep[i];
    for (int i = threadIdx.x; i < PA * PA; i += blockDim.x) sGa[i] = Gsep[PS * PS + i];
    for (int i = threadIdx.x; i < kStageKeys; i += blockDim.x) key[i] = -1;
    if (threadIdx.x == 0) nused = 0;
    const int local = threadIdx.x / P, pt = threadIdx.x - local * P;
    const int pc = pbegin + blockIdx.x * CPB + local;
    const bool active = local < CPB && pc < pend;
    PropE<R> E[4];
    int nch = 0, pos[4] = {-1, -1, -1, -1};
    if (active) {
        const long long e0 = pp_ptr[pc];
        nch = min(pp_nchild[pc], 4);
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) if (ch < nch) E[ch] = pp[e0 + (long long)ch * P + pt];
    }
    __syncthreads();
    // the distinct child cones of the block: lanes of a warp that share a cone elect one leader,
    // which claims (or finds) the cone's key; the thread that claims a key appends the cone
    const int lane = threadIdx.x & 31;
    const int wsize = min(32, (int)blockDim.x - (int)(threadIdx.x & ~31u));   // the block's last warp may be partial
    const unsigned wmask = wsize == 32 ? 0xffffffffu : (1u << wsize) - 1u;
#pragma unroll
    for (int ch = 0; ch < 4; ++ch) {
        const int c = ch < nch ? E[ch].child_cone : -1;
        const unsigned peers = __match_any_sync(wmask, c);
        const int leader = __ffs(peers) - 1;
        int h = -1;
        if (c >= 0 && lane == leader) {
            int q = (int)(((unsigned)c * 2654435761u) >> 25) & (kStageKeys - 1);
            for (int probe = 0; probe < kStageKeys; ++probe) {
                const int old = atomicCAS(&key[q], -1, c);
                if (old == -1) {
                    const int id = atomicAdd(&nused, 1);
                    slot_of[q] = id < CAP ? id : -1;
                    if (id < CAP) ulist[id] = c;
                    h = q;
                    break;
                }
                if (old == c) { h = q; break; }
                q = (q + 1) & (kStageKeys - 1);
            }
        }
        h = __shfl_sync(wmask, h, leader);
        if (c >= 0) pos[ch] = h;
    }
    __syncthreads();
    // one coalesced copy of each distinct child block
    {
        const int n = min(nused, CAP) * P;
        for (int i0 = threadIdx.x; i0 < n; i0 += 4 * blockDim.x) {
            V2<R> v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = i0 + u * blockDim.x;
                if (i < n) v[u] = coef[(long long)ulist[i / P] * P + i % P];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = i0 + u * blockDim.x;
                if (i < n) blk[i / P][i % P] = v[u];
            }
        }
    }
    __syncthreads();
    if (active) {
        V2<R> v; v.x = R(0); v.y = R(0);
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
            if (ch >= nch) break;
            const int slot = pos[ch] >= 0 ? slot_of[pos[ch]] : -1;
            const V2<R> it = slot >= 0 ? interp_eval<R, PS, PA>(blk[slot], E[ch].s, E[ch].th)
                                       : interp_eval<R, PS, PA>(coef + (long long)E[ch].child_cone * P, E[ch].s, E[ch].th);
            V2<R> w; w.x = E[ch].wr; w.y = E[ch].wi;
            cmac<R>(v, it, w);
        }
        sv[local][pt] = v;
    }
    __syncthreads();
    const int m = pt % PS, l = pt / PS;
    if (active) {            // u[l][m] = sum_k Gs[m][k] v[l*PS + k]
        V2<R> u; u.x = R(0); u.y = R(0);
#pragma unroll
        for (int k = 0; k < PS; ++k) {
            const R g = sGs[m * PS + k];
            const V2<R> vv = sv[local][l * PS + k];
            u.x = rfma(g, vv.x, u.x); u.y = rfma(g, vv.y, u.y);
        }
        su[local][l * PS + m] = u;
    }
    __syncthreads();
    if (active) {            // c[n][m] = sum_l Ga[n][l] u[l][m], stored at n*PS + m
        const int n = l;
        V2<R> c; c.x = R(0); c.y = R(0);
#pragma unroll
        for (int q = 0; q < PA; ++q) {
            const R g = sGa[n * PA + q];
            const V2<R> u = su[local][q * PS + m];
            c.x = rfma(g, u.x, c.x); c.y = rfma(g, u.y, c.y);
        }
        coef[(long long)pc * P + n * PS + m] = c;
    }
}

// complex64: near field and interpolation of a leaf box's targets, a block per (box, share of its targets)
// with one record (FinItem).  Near field: the neighbour boxes' densities are staged in shared memory
// kNearChunk at a time, each warp streams two targets' table rows against them; a target's chunk sums add
// up in chunk order.  Interpolation: a thread takes kIbPiece terms of a target, the targets fastest.  The
// targets of a box share their ancestors, hence the same cousin lists in the same order: their j-th terms
// read the same cousin box, mostly the same cone (2.5-3 distinct cones in 32 targets on the kite trees), so
// the gathers are broadcasts; the plan is stored in that order.  The warps take the row pairs and then 32
// pieces at a time from one counter, so that none waits at a barrier between the two; the pieces' sums are
// added in order to the near sum.  Bound by the latency of the plan's and the coefficients' loads; a term's
// plan entry is loaded during the term before.  Kite k = 100 / 500 / 2000: 25 / 37 / 64 us as two
// kernels, 12 / 18 / 53 so; without the counter 12 / 21 / 55; two or four blocks an SM: 14 / 21 / 55 or slower.
template <int PS, int PA>
__global__ void __launch_bounds__(256, 3) k_final_q(const FinItem* __restrict__ items, const int* __restrict__ near_src,
                                                 const float2* __restrict__ near, const float2* __restrict__ rho,
                                                 const InterpE<float>* __restrict__ ipT, const float2* __restrict__ coef,
                                                 const long long* __restrict__ sorting, double2* __restrict__ y) {
    constexpr int P = PS * PA;
    __shared__ float2 srho[kNearChunk];
    __shared__ float2 sacc[kFinTargetsMax], part[kFinParts];
    __shared__ int next;
    const FinItem I = items[blockIdx.x];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cnt = I.cnt, rl = I.rl;
    const int* src = near_src + I.src;
    if (tid == 0) next = 0;
    if (tid < cnt) sacc[tid] = make_float2(0.f, 0.f);
    auto rows = [&](int q, int c0, int cn) {   // targets q and q + 1 against the staged densities
        const float2* r0 = near + I.near + (long long)q * rl + c0;
        const float2* r1 = q + 1 < cnt ? r0 + rl : r0;
        float2 a = make_float2(0.f, 0.f), b = a;
#pragma unroll 4
        for (int e = lane; e < cn; e += 32) {
            const float2 u = r0[e], v = r1[e], r = srho[e];
            cmac<float>(a, u, r); cmac<float>(b, v, r);
        }
        a.x = warp_sum_r<float>(a.x); a.y = warp_sum_r<float>(a.y);
        b.x = warp_sum_r<float>(b.x); b.y = warp_sum_r<float>(b.y);
        if (lane == 0) {
            sacc[q].x += a.x; sacc[q].y += a.y;
            if (q + 1 < cnt) { sacc[q + 1].x += b.x; sacc[q + 1].y += b.y; }
        }
    };
    const int npc = (I.nt + kIbPiece - 1) / kIbPiece, pairs = rl > 0 ? (cnt + 1) / 2 : 0;
    int c0 = 0, cn;
    for (;; c0 += kNearChunk) {
        cn = min(kNearChunk, rl - c0);
        for (int e = tid; e < cn; e += 256) srho[e] = rho[src[c0 + e]];
        __syncthreads();
        if (c0 + kNearChunk >= rl) break;
        for (int q = 2 * warp; q < cnt; q += 16) rows(q, c0, cn);
        __syncthreads();                       // the chunk has been read
    }
    // the last chunk's rows and the pieces, each warp the next when it is done with one
    for (;;) {
        int u = 0;
        if (lane == 0) u = atomicAdd(&next, 1);
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u < pairs) { rows(2 * u, c0, cn); continue; }
        if ((u - pairs) * 32 >= npc * cnt) break;
        const int w = (u - pairs) * 32 + lane, pc = w / cnt, t = w - pc * cnt;
        if (pc < npc) {
            const InterpE<float>* e = ipT + I.ip + t;
            const int z = min(I.nt, (pc + 1) * kIbPiece);
            float2 acc = make_float2(0.f, 0.f);
            InterpE<float> En = e[(long long)(pc * kIbPiece) * I.n];
            for (int j = pc * kIbPiece; j < z; ++j) {
                const InterpE<float> E = En;
                if (j + 1 < z) En = e[(long long)(j + 1) * I.n];             // in flight during this term
                cmac<float>(acc, interp_eval<float, PS, PA>(coef + (long long)E.cone * P, E.s, E.th), make_float2(E.fr, E.fi));
            }
            part[w] = acc;
        }
    }
    __syncthreads();
    float2 sum = make_float2(0.f, 0.f);
    if (tid < cnt) {
        sum = sacc[tid];
        for (int q = 0; q < npc; ++q) { const float2 v = part[q * cnt + tid]; sum.x += v.x; sum.y += v.y; }
    }
    if (tid < cnt) {
        const long long o = sorting[I.first + tid];
        double2 v = y[o];
        v.x += (double)sum.x; v.y += (double)sum.y;
        y[o] = v;
    }
}

__device__ __forceinline__ InterpX interp_fx(const InterpE<double>& E) {
    return InterpX{E.cone, E.pad, fx_weight(E.s), fx_weight(E.th), E.fr, E.fi};
}
// the interpolation plan of each leaf box transposed: term j of the box's target t moves from
// ip_ptr[i] + j to ip_ptr[box's first target] + j n + t (every target of a box has as many terms);
// complex64, and the FP64 form array by array
__global__ void k_interp_transpose(int N, const int* __restrict__ point_leaf, const int* __restrict__ leaf_start,
                                   const int* __restrict__ leaf_count, const int* __restrict__ ip_ptr,
                                   const InterpE<double>* __restrict__ in, InterpE<float>* __restrict__ out, PlanX px) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const int b = point_leaf[i], s = leaf_start[b], n = leaf_count[b], t = i - s;
    const int base = ip_ptr[s], nt = ip_ptr[i + 1] - ip_ptr[i];
    for (int j = 0; j < nt; ++j) {
        const InterpE<double> E = in[ip_ptr[i] + j];
        const long long o = base + (long long)j * n + t;
        out[o] = InterpE<float>{E.cone, (float)E.s, (float)E.th, (float)E.fr, (float)E.fi};
        px.child[o] = E.cone;
        px.st[o] = make_longlong2(fx_weight(E.s), fx_weight(E.th));
        px.w[o] = make_double2(E.fr, E.fi);
    }
}
__global__ void k_interp_fx(const InterpE<double>* __restrict__ in, long long n, InterpX* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = interp_fx(in[i]);
}
__global__ void k_fx_weights(const double* __restrict__ in, int n, int2* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { const FxLimb t = fx_split(fx_weight(in[i])); out[i] = make_int2(t.h, t.l); }
}

// complex64: one warp per Morton-sorted target; near row layout [target][neighbour sources], and
// near_src[near_src_off[b] + e] the Morton index of entry e's source in leaf box b's rows, so the
// lanes stride over one flat row with independent loads.
template <int PS, int PA>
__global__ void __launch_bounds__(256) k_final_t(int N, const int* __restrict__ point_leaf, const int* __restrict__ leaf_start,
                                                 const int* __restrict__ near_src_off, const int* __restrict__ near_src,
                                                 const int* __restrict__ near_rowlen,
                                                 const long long* __restrict__ near_off, const float2* __restrict__ near,
                                                 const float2* __restrict__ rho, const int* __restrict__ ip_ptr,
                                                 const InterpE<float>* __restrict__ ip, const float2* __restrict__ coef,
                                                 const long long* __restrict__ sorting, double2* __restrict__ y) {
    constexpr int P = PS * PA;
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= N) return;
    const int b = point_leaf[i];
    const int t = i - leaf_start[b];
    const int rl = near_rowlen[b];
    const float2* row = near + near_off[b] + (long long)t * rl;
    const int* src = near_src + near_src_off[b];
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int e = lane; e < rl; e += 32) cmac<float>(acc, row[e], rho[src[e]]);
    for (int e = ip_ptr[i] + lane; e < ip_ptr[i + 1]; e += 32) {
        const InterpE<float> E = ip[e];
        cmac<float>(acc, interp_eval<float, PS, PA>(coef + (long long)E.cone * P, E.s, E.th), make_float2(E.fr, E.fi));
    }
    acc.x = warp_sum_r<float>(acc.x);
    acc.y = warp_sum_r<float>(acc.y);
    if (lane == 0) {
        const long long o = sorting[i];
        double2 v = y[o];
        v.x += (double)acc.x; v.y += (double)acc.y;
        y[o] = v;
    }
}

// FP64 in fixed point (fixpoint.cuh): near field and interpolation of a leaf box's targets, a block per
// (box, up to kFinTargets targets) with one record (FinItem).  Interpolation: a thread per (target, term),
// the targets fastest: the box's targets share their cousin lists, so their j-th terms read the same
// cousin box and mostly the same cone (broadcast gathers), and the plan is stored in that order; each
// thread keeps the sum of its target's terms, the threads of a target add up in shared memory.  Near
// field: the neighbour boxes' densities, loaded while the interpolation runs, are brought to one exponent
// in shared memory; a warp takes a target's table row with its lanes over the sources, and the lanes'
// integer sums add up by shuffles.  Bound by latency at small sizes, by the wide multiply-adds else.
// Kite k = 500 / 2000: 55 / 260 us with FP64 multiply-adds, 33 / 105 us so.  When it took 35 / 114 with 4 blocks
// an SM, 3 took 39 / 119 and 2 41 / 150.
template <int PS, int PA>
__global__ void __launch_bounds__(256, 4) k_final_fx(const FinItem* __restrict__ items, const int* __restrict__ near_src,
                                                  const int4* __restrict__ near, const int* __restrict__ nexp,
                                                  const double2* __restrict__ rho, PlanX ip, const int4* __restrict__ coef,
                                                  const int* __restrict__ cexp, const long long* __restrict__ sorting,
                                                  double2* __restrict__ y) {
    constexpr int P = PS * PA, NS = kNearChunk / 2;
    constexpr int T = kFxSumTop;               // a lane sums at most NS / 32 products
    __shared__ int4 srho[NS];
    __shared__ double2 snear[kFinTargets], part[256];
    __shared__ int smax;
    const FinItem I = items[blockIdx.x];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cnt = I.cnt, rl = I.rl;
    const int* src = near_src + I.src;
    if (tid == 0) smax = 0;
    if (tid < cnt) snear[tid] = make_double2(0.0, 0.0);
    double2 d0 = make_double2(0.0, 0.0);       // this thread's source of the first 256
    if (tid < rl) d0 = rho[src[tid]];
    // interpolation
    const int G = 256 / cnt, g = tid / cnt, t = tid - g * cnt;
    double2 acc = make_double2(0.0, 0.0);
    if (g < G) {
        long long e = I.ip + t + (long long)g * I.n;
        int cn = 0;
        longlong2 sn = make_longlong2(0, 0);
        double2 fn = make_double2(0.0, 0.0);
        if (g < I.nt) { cn = ip.child[e]; sn = ip.st[e]; fn = ip.w[e]; }
        for (int j = g; j < I.nt; j += G) {
            const int c = cn;
            const longlong2 s = sn;
            const double2 f = fn;
            e += (long long)G * I.n;
            if (j + G < I.nt) { cn = ip.child[e]; sn = ip.st[e]; fn = ip.w[e]; }   // in flight during this term
            const int4* blk = coef + (long long)c * P;
            cmac<double>(acc, fx_interp_value<PS, PA>([&](int i) { return blk[i]; }, cexp[c], s), f);
        }
    }
    part[tid] = acc;
    int mx = fx_absmax_hi(d0.x, d0.y);
    for (int q = tid + 256; q < rl; q += 256) { const double2 v = rho[src[q]]; mx = max(mx, fx_absmax_hi(v.x, v.y)); }
    mx = __reduce_max_sync(0xffffffffu, mx);
    __syncthreads();
    if (lane == 0) atomicMax(&smax, mx);
    // the threads of a target: four partial sums
    double2 a4 = make_double2(0.0, 0.0);
    const int q4 = tid / cnt, tt = tid - q4 * cnt;
    if (q4 < 4)
        for (int k = q4; k < G; k += 4) { const double2 v = part[k * cnt + tt]; a4.x += v.x; a4.y += v.y; }
    __syncthreads();
    const int E = fx_expo(smax);
    for (int c0 = 0; c0 < rl; c0 += NS) {
        const int cn = min(NS, rl - c0);
        if (c0) __syncthreads();               // the previous chunk has been read
        for (int e = tid; e < cn; e += 256) {
            const double2 v = c0 + e < 256 ? d0 : rho[src[c0 + e]];
            srho[e] = E == kFxBad ? make_int4(0, 0, 0, 0) : fx_pack_sum(fx_from(v.x, E, T), fx_from(v.y, E, T));
        }
        __syncthreads();
        for (int q = warp; q < cnt; q += 8) {
            const int4* row = near + I.near + (long long)q * rl + c0;
            const int En = nexp[I.first + q];
            FxSum rr{0, 0}, ii{0, 0}, im{0, 0};
#pragma unroll 4
            for (int e = lane; e < cn; e += 32) {
                const int4 a = row[e], d = srho[e];
                fx_sum_mac(rr, a.x, a.y, d.x, d.y);
                fx_sum_mac(ii, a.z, a.w, d.z, d.w);
                fx_sum_mac(im, a.x, a.y, d.z, d.w);
                fx_sum_mac(im, a.z, a.w, d.x, d.y);
            }
            rr.h -= ii.h; rr.m -= ii.m;
            fx_sum_fold(rr); fx_sum_fold(im);
            // one shift for the warp that keeps 32 lanes' sum below 2^62
            const int lz = min(__clzll(rr.h < 0 ? ~rr.h : rr.h), __clzll(im.h < 0 ? ~im.h : im.h));
            const int sh = min(__reduce_min_sync(0xffffffffu, lz) - 8, kFxSumLow);
            long long yr = sh >= 0 ? (rr.h << sh) + (rr.m >> (kFxSumLow - sh)) : rr.h >> -sh;
            long long yi = sh >= 0 ? (im.h << sh) + (im.m >> (kFxSumLow - sh)) : im.h >> -sh;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                yr += __shfl_xor_sync(0xffffffffu, yr, o);
                yi += __shfl_xor_sync(0xffffffffu, yi, o);
            }
            if (lane < 2) {
                const int e = En + E - kFxSumTop - T + 2 * kFxSumLow - sh;
                const double v = En == kFxBad || E == kFxBad ? __hiloint2double(0x7ff80000, 0) : fx_scaled(lane ? yi : yr, e);
                double* o = lane ? &snear[q].y : &snear[q].x;
                *o += v;
            }
        }
    }
    if (q4 < 4) part[tid] = a4;
    __syncthreads();
    if (tid < cnt) {
        double2 v = snear[tid];
        for (int k = 0; k < min(4, G); ++k) { v.x += part[k * cnt + tid].x; v.y += part[k * cnt + tid].y; }
        const long long o = sorting[I.first + tid];
        double2 w = y[o];
        w.x += v.x; w.y += v.y;
        y[o] = w;
    }
}
// set-up: the FP64 near-field table in place as 27-bit limbs, an exponent per target row (a warp per
// Morton-sorted target), and its complex64 copy
__global__ void __launch_bounds__(256) k_near_fix(int N, const int* __restrict__ point_leaf, const int* __restrict__ leaf_start,
                                                  const int* __restrict__ near_rowlen, const long long* __restrict__ near_off,
                                                  double2* __restrict__ near, int* __restrict__ nexp, float2* __restrict__ n32) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= N) return;
    const int b = point_leaf[i], rl = near_rowlen[b];
    const long long o = near_off[b] + (long long)(i - leaf_start[b]) * rl;
    int mx = 0;
    for (int e = lane; e < rl; e += 32) { const double2 v = near[o + e]; mx = max(mx, fx_absmax_hi(v.x, v.y)); }
    const int E = fx_expo(__reduce_max_sync(0xffffffffu, mx));
    if (lane == 0) nexp[i] = E;
    for (int e = lane; e < rl; e += 32) {
        const double2 v = near[o + e];
        n32[o + e] = make_float2((float)v.x, (float)v.y);
        reinterpret_cast<int4*>(near)[o + e] =
            E == kFxBad ? make_int4(0, 0, 0, 0) : fx_pack_sum(fx_from(v.x, E, kFxSumTop), fx_from(v.y, E, kFxSumTop));
    }
}

__global__ void k_d2f(const double2* __restrict__ a, long long n, float2* __restrict__ b) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = make_float2((float)a[i].x, (float)a[i].y);
}

// ------------------------------------------------------------------ launchers
static inline unsigned nblk_a(long long n, int b) { return (unsigned)((n + b - 1) / b); }

template <typename R>
void launch_intensities_t(const double2* x, const double* wq, const long long* perm, int N, V2<R>* rho, cudaStream_t s) {
    k_intensities_t<R><<<nblk_a(N, 256), 256, 0, s>>>(x, wq, perm, N, rho);
}
cudaError_t preload_intensities_kernel() {
    cudaFuncAttributes a;
    return cudaFuncGetAttributes(&a, k_intensities_t<double>);
}
// chunks per coefficient (the tuning variant): 1, 2, 5 or 10; a block holds 256 / (P * CH) cones
template <typename Go>
static void leaf_chunks(int P, int chunks, Go&& go) {
    if (chunks == 10 && 256 / (P * 10) >= 1) go(std::integral_constant<int, 10>{});
    else if (chunks == 2 && 256 / (P * 2) >= 1) go(std::integral_constant<int, 2>{});
    else if (chunks == 1 || 256 / (P * 5) < 1) go(std::integral_constant<int, 1>{});
    else go(std::integral_constant<int, 5>{});
}
int leaf_item_cones(int P) { return 256 / P; }
void launch_leaf_apply_t(const int4* cones, int ncones, int cone_base, const float2* L, const float2* rho, int P, float2* coef,
                         cudaStream_t s, int chunks) {
    if (ncones <= 0) return;
    leaf_chunks(P, chunks, [&](auto tag) {
        constexpr int CH = decltype(tag)::value;
        const int cpb = 256 / (P * CH);
        k_leaf_apply_t<CH><<<nblk_a(ncones, cpb), cpb * P * CH, 0, s>>>(cones, ncones, cone_base, L, rho, P, coef);
    });
}
void launch_leaf_fx(const LeafItem* items, int nitems, int cone_base, const int4* L, const int* lexp, const double2* rho, int P, int Ps,
                    int4* coef, int* cexp, cudaStream_t s, int chunks) {
    if (nitems <= 0) return;
    leaf_chunks(P, chunks, [&](auto tag) {
        constexpr int CH = decltype(tag)::value;
        const int cpb = 256 / (P * CH), split = (leaf_item_cones(P) + cpb - 1) / cpb;
        k_leaf_fx<CH><<<(unsigned)nitems * split, cpb * P * CH, 0, s>>>(items, split, cone_base, L, lexp, rho, P, Ps, coef, cexp);
    });
}
void launch_leaf_fix(const int* cone_box, int ncones, const int* leaf_count, const long long* leaf_off, int P, int4* L, int* lexp,
                     float2* l32, cudaStream_t s) {
    if (ncones > 0) k_leaf_fix<<<ncones, 256, 0, s>>>(cone_box, leaf_count, leaf_off, P, reinterpret_cast<double2*>(L), lexp, l32);
}
static std::atomic<int> g_leaf_tma_ready{0};
cudaError_t leaf_tma_init() {
    if (g_leaf_tma_ready.load()) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(k_leaf_tma<25>, cudaFuncAttributeMaxDynamicSharedMemorySize, LeafTma<25>::smem);
    if (e == cudaSuccess) g_leaf_tma_ready.store(1);
    return e;
}
bool launch_leaf_tma(const int* cone_box, int ncones, int cone_base, const int* leaf_start, const int* leaf_count,
                     const long long* leaf_off, const float2* L, const float2* rho, int P, float2* coef, int* err, int nsm,
                     cudaStream_t s) {
    if (P != 25) return false;
    if (ncones <= 0) return true;
    if (!g_leaf_tma_ready.load()) return false;   // leaf_tma_init not run on this device
    const int grid = std::min(ncones, 4 * std::max(nsm, 1));
    k_leaf_tma<25><<<grid, kLtThreads, LeafTma<25>::smem, s>>>(cone_box, ncones, cone_base, leaf_start, leaf_count, leaf_off, L,
                                                              rho, coef, err);
    return true;
}
void launch_propagate_t(int pbegin, int pend, const long long* pp_ptr, const int* pp_nchild, const PropE<float>* pp, int Ps, int Pang,
                        const float* Gsep, float2* coef, cudaStream_t s, int cones_per_block) {
    if (pend <= pbegin) return;
    // cones per block (the tuning variant): 2, 4 or the most that fit 256 threads; kPropStaged:
    // the most that fit, child blocks staged in shared memory
    IFGF_DISPATCH_P(Ps, Pang, {
        constexpr int CPBMAX = 256 / (PS * PA);
        if (cones_per_block == kPropStaged)
            k_propagate_st<PS, PA, CPBMAX><<<nblk_a(pend - pbegin, CPBMAX), CPBMAX * PS * PA, 0, s>>>(pbegin, pend, pp_ptr,
                                                                                                      pp_nchild, pp, Gsep, coef);
        else if (cones_per_block == 2 && CPBMAX >= 2)
            k_propagate_t<PS, PA, 2><<<nblk_a(pend - pbegin, 2), 2 * PS * PA, 0, s>>>(pbegin, pend, pp_ptr, pp_nchild, pp, Gsep, coef);
        else if (cones_per_block == 4 && CPBMAX >= 4)
            k_propagate_t<PS, PA, 4><<<nblk_a(pend - pbegin, 4), 4 * PS * PA, 0, s>>>(pbegin, pend, pp_ptr, pp_nchild, pp, Gsep, coef);
        else
            k_propagate_t<PS, PA, CPBMAX><<<nblk_a(pend - pbegin, CPBMAX), CPBMAX * PS * PA, 0, s>>>(pbegin, pend, pp_ptr,
                                                                                                     pp_nchild, pp, Gsep, coef);
    });
}
size_t StageLevels::add(int b, int e, int Ps, int Pang) {
    int groups = 0, record = 0;
    IFGF_DISPATCH_P(Ps, Pang, { groups = (int)nblk_a(e - b, PropFx<PS * PA>::cones); record = PropFx<PS * PA>::record; });
    begin[n] = b; end[n] = e;
    const size_t at = (size_t)group[n] * record;
    group[n + 1] = group[n] + groups;
    ++n;
    return at;
}
size_t StageLevels::size(int Ps, int Pang) const {
    size_t record = 0;
    IFGF_DISPATCH_P(Ps, Pang, record = PropFx<PS * PA>::record;);
    return (size_t)group[n] * record;
}
void launch_stage_plan(const StageLevels& L, const long long* pp_ptr, PlanX pp, int Ps, int Pang, int* stage, cudaStream_t s) {
    if (L.group[L.n] <= 0) return;
    IFGF_DISPATCH_P(Ps, Pang, (k_stage_plan<PS * PA><<<L.group[L.n], kPropFxThreads, 0, s>>>(L, pp_ptr, pp, stage)));
}
void launch_propagate_fx(int pbegin, int pend, PlanX pp, const int* stage, int Ps, int Pang, const int2* GsepX, int4* coef, int* cexp,
                         cudaStream_t s) {
    if (pend <= pbegin) return;
    IFGF_DISPATCH_P(Ps, Pang, (k_propagate_fx<PS, PA><<<nblk_a(pend - pbegin, PropFx<PS * PA>::cones), kPropFxThreads, 0, s>>>(
                                   pbegin, pend, pp, stage, GsepX, coef, cexp)));
}
void launch_fx_weights(const double* in, int n, int2* out, cudaStream_t s) {
    if (n > 0) k_fx_weights<<<nblk_a(n, 128), 128, 0, s>>>(in, n, out);
}
void launch_interp_fx(const InterpE<double>* in, long long n, InterpX* out, cudaStream_t s) {
    if (n > 0) k_interp_fx<<<nblk_a(n, 256), 256, 0, s>>>(in, n, out);
}
void launch_final_t(int N, const int* point_leaf, const int* leaf_start, const int* near_src_off, const int* near_src,
                    const int* near_rowlen, const long long* near_off, const float2* near, const float2* rho, const int* ip_ptr,
                    const InterpE<float>* ip, const float2* coef, int Ps, int Pang, const long long* sorting, double2* y,
                    cudaStream_t s) {
    IFGF_DISPATCH_P(Ps, Pang, (k_final_t<PS, PA><<<nblk_a((long long)N * 32, 256), 256, 0, s>>>(
                                   N, point_leaf, leaf_start, near_src_off, near_src, near_rowlen, near_off, near, rho,
                                   ip_ptr, ip, coef, sorting, y)));
}
void launch_final_fx(const FinItem* items, int nitems, const int* near_src, const int4* near, const int* nexp, const double2* rho,
                     PlanX ip, const int4* coef, const int* cexp, int Ps, int Pang, const long long* sorting, double2* y,
                     cudaStream_t s) {
    if (nitems <= 0) return;
    IFGF_DISPATCH_P(Ps, Pang, (k_final_fx<PS, PA><<<nitems, 256, 0, s>>>(items, near_src, near, nexp, rho, ip, coef, cexp, sorting, y)));
}
void launch_near_fix(int N, const int* point_leaf, const int* leaf_start, const int* near_rowlen, const long long* near_off, int4* near,
                     int* nexp, float2* n32, cudaStream_t s) {
    if (N > 0)
        k_near_fix<<<nblk_a((long long)N * 32, 256), 256, 0, s>>>(N, point_leaf, leaf_start, near_rowlen, near_off,
                                                                 reinterpret_cast<double2*>(near), nexp, n32);
}
void launch_final_q(const FinItem* items, int nitems, const int* near_src, const float2* near, const float2* rho,
                    const InterpE<float>* ipT, const float2* coef, int Ps, int Pang, const long long* sorting, double2* y, cudaStream_t s) {
    if (nitems <= 0) return;
    IFGF_DISPATCH_P(Ps, Pang, (k_final_q<PS, PA><<<(unsigned)nitems, 256, 0, s>>>(items, near_src, near, rho, ipT, coef, sorting, y)));
}
void launch_interp_transpose(int N, const int* point_leaf, const int* leaf_start, const int* leaf_count, const int* ip_ptr,
                             const InterpE<double>* in, InterpE<float>* out, PlanX px, cudaStream_t s) {
    if (N > 0) k_interp_transpose<<<nblk_a(N, 256), 256, 0, s>>>(N, point_leaf, leaf_start, leaf_count, ip_ptr, in, out, px);
}
void launch_d2f(const double2* a, long long n, float2* b, cudaStream_t s) {
    if (n > 0) k_d2f<<<nblk_a(n, 256), 256, 0, s>>>(a, n, b);
}

template void launch_intensities_t<double>(const double2*, const double*, const long long*, int, double2*, cudaStream_t);
template void launch_intensities_t<float>(const double2*, const double*, const long long*, int, float2*, cudaStream_t);

}  // namespace ifgf

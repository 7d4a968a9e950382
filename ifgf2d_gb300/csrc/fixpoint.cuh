// fixpoint.cuh -- block fixed-point arithmetic for the FP64 form of the IFGF sums.
//
// GB300 retires about 2 FP64 operations per SM and clock (FMA, add, multiply and every conversion
// from or to a double alike), but 29 wide integer multiply-adds (32 x 32 + 64 bits), both measured.
// The cone interpolants are sums of products of known range, so the FP64 form evaluates them in
// integers:
//   * a block of coefficients (one cone, one right-hand side) shares one binary exponent E: the
//     value X 2^(E - T) is kept as the integer X = x1 2^29 + x0, |x0| <= 2^28 (two int32 limbs),
//     |X| <= 2^T, T = 55 (54 for more than 36 coefficients: headroom for the sum of them all);
//   * a weight t in [-1, 1] (Chebyshev values) is t1 2^29 + t0 over 2^58;
//   * x t = x1 t1 + (x1 t0 + x0 t1) 2^-29 (+ x0 t0 2^-58, below 1/2 unit of X and left out):
//     three wide multiply-adds into two 64-bit accumulators, exact and free of overflow.
// Every value is held to 2^-56 of its block's largest and every weight to 2^-59, an eighth of the
// FP64 rounding unit of the largest value; the sums round once.  So the results are nearer to the
// exact ones than FP64 arithmetic's.  Exponents cover FP64's whole range, subnormal numbers included;
// blocks that hold a NaN or an infinity, or whose values pass FP64's range, carry the exponent kFxBad and
// evaluate to NaN.
#pragma once
#include "ifgf_device.cuh"

namespace ifgf {

constexpr int kFxLow = 29;                    // bits of the low limb
constexpr int kFxOne = 2 * kFxLow;            // fraction bits of a weight
constexpr int kFxMinExp = -1022;              // smallest block exponent: its values' unit is below FP64's smallest number
constexpr int kFxMaxExp = 1024;               // larger (or non-finite) values make the block kFxBad
constexpr int kFxBad = 0x7fffffff;
constexpr int kFxNear0 = -960, kFxNear1 = 1010;   // exponents whose blocks' values are normal numbers
__host__ __device__ constexpr int fx_top(int P) { return P <= 36 ? 55 : 54; }

// limbs of a 64-bit integer, |value| < 2^60: the low one balanced (what is stored), or as the bits
// fall, 0 <= l < 2^29 (fewer instructions, for values used at once)
struct FxLimb { int h, l; };
__device__ __forceinline__ FxLimb fx_split(long long x) {
    FxLimb r;
    r.h = (int)((x + (1ll << (kFxLow - 1))) >> kFxLow);
    r.l = (int)((unsigned)x - ((unsigned)r.h << kFxLow));
    return r;
}
__device__ __forceinline__ FxLimb fx_cut(long long x) {
    return FxLimb{(int)(x >> kFxLow), (int)((unsigned)x & ((1u << kFxLow) - 1u))};
}
// a b + c: one wide multiply-add (as mad.wide it becomes a multiply and a 64-bit add, 10 % slower here)
__device__ __forceinline__ long long fx_wide(int a, int b, long long c) {
    unsigned lo = (unsigned)c;
    int hi = (int)(c >> 32);
    asm("mad.lo.cc.s32 %0, %2, %3, %0; madc.hi.s32 %1, %2, %3, %1;" : "+r"(lo), "+r"(hi) : "r"(a), "r"(b));
    return ((long long)hi << 32) | lo;
}
// the low-order half of a product sum: m += a b without their high limbs' product
__device__ __forceinline__ long long fx_low(FxLimb a, FxLimb b, long long m) { return fx_wide(a.l, b.h, fx_wide(a.h, b.l, m)); }
constexpr long long kFxHalf = 1ll << (kFxLow - 1);   // start of m: its shift by kFxLow then rounds

// a weight in [-1, 1]
__device__ __forceinline__ long long fx_weight(double t) { return __double2ll_rn(t * (double)(1ll << kFxOne)); }
__device__ __forceinline__ double fx_weight_value(long long t) { return (double)t * (1.0 / (double)(1ll << kFxOne)); }

// int4 that hold the Chebyshev values T_1.. of s and theta of a batched term
__host__ __device__ constexpr int fx_rows4(int Ps, int Pang) { return (Ps + Pang - 1) / 2; }

// a block's exponent from the largest high word of its values' magnitudes: |value| < 2^E
__device__ __forceinline__ int fx_expo(int maxhi) {
    const int e = (maxhi >> 20) - 1022;        // kFxMinExp at least
    return e > kFxMaxExp ? kFxBad : e;
}
__device__ __forceinline__ int fx_absmax_hi(double a, double b) {
    return max(__double2hiint(a) & 0x7fffffff, __double2hiint(b) & 0x7fffffff);
}
// round(v 2^(T - E)) for |v| < 2^E, by shifts of the mantissa (an FP64 conversion costs as much as an FMA)
__device__ __forceinline__ long long fx_from(double v, int E, int T) {
    const int hi = __double2hiint(v);
    const int e = max((hi >> 20) & 0x7ff, 1);
    const unsigned top = (hi & 0xfffff) | (((hi >> 20) & 0x7ff) ? 0x100000u : 0u);
    const long long mant = ((long long)top << 32) | (unsigned)__double2loint(v);
    const int s = E + 1078 - T - e;            // of mant 2^3; >= 1 as |v| < 2^E
    const long long x = s > 60 ? 0ll : ((mant << 3) + (1ll << (s - 1))) >> s;
    return hi < 0 ? -x : x;
}
// d 2^e for d = 0 or 1 <= |d| < 2^63, rounded once: subnormal or infinite where FP64's range ends
__device__ __forceinline__ double fx_ldexp(double d, int e) {
    const int a = min(max(e, -1000), 1000), b = min(max(e - a, -1022), 1023);
    return d * __hiloint2double((1023 + a) << 20, 0) * __hiloint2double((1023 + b) << 20, 0);
}
// what a block's exponent E does to its values: added to a double's high word, if near (else by fx_ldexp)
struct FxScale { unsigned add; int e; bool near; };
__device__ __forceinline__ FxScale fx_scale(int E, int T) {
    return FxScale{(unsigned)(E - T) << 20, E == kFxBad ? kFxBad : E - T, (unsigned)(E - kFxNear0) <= (unsigned)(kFxNear1 - kFxNear0)};
}
// (x, y) 2^(E - T) as doubles (x and y integers below 2^62 in magnitude)
__device__ __forceinline__ double2 fx_value(long long x, long long y, FxScale s) {
    double a = (double)x, b = (double)y;
    if (s.near) {
        a = __hiloint2double(x != 0 ? (int)((unsigned)__double2hiint(a) + s.add) : 0, __double2loint(a));
        b = __hiloint2double(y != 0 ? (int)((unsigned)__double2hiint(b) + s.add) : 0, __double2loint(b));
    } else {
        const double nan = __hiloint2double(0x7ff80000, 0);
        a = s.e == kFxBad ? nan : fx_ldexp(a, s.e);
        b = s.e == kFxBad ? nan : fx_ldexp(b, s.e);
    }
    return make_double2(a, b);
}

// T_1..T_{n-1} of a weight (T_0 = 1 is left out), t[i] holding T_{i+1}:
// T_{2j} = 2 T_j^2 - 1, T_{2j+1} = 2 T_j T_{j+1} - T_1
template <int NT>
__device__ __forceinline__ void fx_cheb(long long x, FxLimb* t) {
    t[0] = fx_cut(x);
#pragma unroll
    for (int i = 2; i < NT; ++i) {
        const FxLimb a = t[i / 2 - 1], b = t[(i + 1) / 2 - 1];
        const long long m = i % 2 ? fx_low(a, b, kFxHalf >> 1) >> (kFxLow - 1)
                                  : fx_wide(a.h, a.l, kFxHalf >> 2) >> (kFxLow - 2);
        t[i - 1] = fx_cut(fx_wide(2 * a.h, b.h, m - (i % 2 ? x : 1ll << kFxOne)));
    }
}

// a coefficient of T_0(s), multiplied by no weight, is kept as its 64 bits instead of limbs
__device__ __forceinline__ long long fx_raw(int lo, int hi) { return ((long long)hi << 32) | (unsigned)lo; }
__device__ __forceinline__ int4 fx_pack_raw(long long re, long long im) {
    return make_int4((int)re, (int)(re >> 32), (int)im, (int)(im >> 32));
}
// the cone interpolant sum_a T_a(th) sum_q T_q(s) c[a * PS + q] in units of the block's values;
// at most PS * PA times the largest |X|.  The low halves of a sum are taken first and shifted into
// the start of its high half.
template <int PS, int PA, typename Load>
__device__ __forceinline__ void fx_interp(const FxLimb* Ts, const FxLimb* Tt, Load&& c, long long& re, long long& im) {
    // the left-out products u.l T.l of the outer sums are positive: start as high as keeps zero zero
    long long mr = 2 * kFxHalf - 1, mi = mr, u0r = 0, u0i = 0;
    FxLimb ur[PA], ui[PA];
#pragma unroll
    for (int a = 0; a < PA; ++a) {
        const int4 c0 = c(a * PS);
        long long vr = kFxHalf, vi = kFxHalf;
        int xr[PS], xi[PS];
#pragma unroll
        for (int q = 1; q < PS; ++q) {
            const int4 v = c(a * PS + q);
            vr = fx_low(FxLimb{v.x, v.y}, Ts[q - 1], vr);
            vi = fx_low(FxLimb{v.z, v.w}, Ts[q - 1], vi);
            xr[q] = v.x; xi[q] = v.z;
        }
        vr = fx_raw(c0.x, c0.y) + (vr >> kFxLow); vi = fx_raw(c0.z, c0.w) + (vi >> kFxLow);
#pragma unroll
        for (int q = 1; q < PS; ++q) { vr = fx_wide(xr[q], Ts[q - 1].h, vr); vi = fx_wide(xi[q], Ts[q - 1].h, vi); }
        if (a == 0) {
            u0r = vr; u0i = vi;
        } else {
            ur[a] = fx_cut(vr); ui[a] = fx_cut(vi);
            mr = fx_low(ur[a], Tt[a - 1], mr); mi = fx_low(ui[a], Tt[a - 1], mi);
        }
    }
    re = u0r + (mr >> kFxLow); im = u0i + (mi >> kFxLow);
#pragma unroll
    for (int a = 1; a < PA; ++a) { re = fx_wide(ur[a].h, Tt[a - 1].h, re); im = fx_wide(ui[a].h, Tt[a - 1].h, im); }
}
// the interpolant of a cone's block at (s, th), st = both as weights, as a double
template <int PS, int PA, typename Load>
__device__ __forceinline__ double2 fx_interp_value(Load&& c, int E, longlong2 st) {
    FxLimb Ts[PS], Tt[PA];
    fx_cheb<PS>(st.x, Ts);
    fx_cheb<PA>(st.y, Tt);
    long long re, im;
    fx_interp<PS, PA>(Ts, Tt, c, re, im);
    return fx_value(re, im, fx_scale(E, fx_top(PS * PA)));
}
// ---- table sums (leaf cones): sum_s L[s] rho[s] of complex values, the table entries and the densities
// both as integers of kFxSumTop bits in two 27-bit limbs, X = h 2^27 + l, |l| <= 2^26 (the left-out
// products l l stay below 2^-56 of the largest).  The entries of one coefficient share an exponent, the
// densities of one leaf box another.  kFxSumMost terms fit the 64-bit sums; larger boxes are summed in
// parts of at most so many.
constexpr int kFxSumLow = 27, kFxSumTop = 54, kFxSumFold = 64, kFxSumMost = 128;
__device__ __forceinline__ int4 fx_pack_sum(long long re, long long im) {
    const int rh = (int)((re + (1ll << (kFxSumLow - 1))) >> kFxSumLow), ih = (int)((im + (1ll << (kFxSumLow - 1))) >> kFxSumLow);
    return make_int4(rh, (int)((unsigned)re - ((unsigned)rh << kFxSumLow)), ih, (int)((unsigned)im - ((unsigned)ih << kFxSumLow)));
}
// a sum's value is (h + m 2^-27) 2^54 in units of the two blocks'; kFxSumFold terms after a fold at most
struct FxSum { long long h, m; };
__device__ __forceinline__ void fx_sum_mac(FxSum& s, int ah, int al, int bh, int bl) {
    s.m = fx_wide(ah, bl, s.m);
    s.m = fx_wide(al, bh, s.m);
    s.h = fx_wide(ah, bh, s.h);
}
__device__ __forceinline__ void fx_sum_fold(FxSum& s, int K = 0) {
    s.h += s.m >> (kFxSumLow + K);
    s.m &= (1ll << (kFxSumLow + K)) - 1;
}
// The parts of a sum of n > kFxSumMost terms add up without loss in units of 2^K, K = fx_sum_wide(n): h of 2^K,
// m of 2^-kFxSumLow
__device__ __forceinline__ int fx_sum_wide(int n) { return max(0, 32 - __clz(max(n - 1, 0)) - 7); }
__device__ __forceinline__ void fx_sum_part(FxSum& s, FxSum part, int K) {
    s.h += part.h >> K;
    s.m += ((part.h & ((1ll << K) - 1)) << kFxSumLow) + part.m;
}
// a folded sum's value, or such parts' (K > 0), of blocks with exponent E (table plus density, minus their bits) as
// y 2^e, |y| < 2^62 with at most the sum's own bits lost
__device__ __forceinline__ long long fx_sum_value(FxSum s, int E, int& e, int K = 0) {
    const int low = kFxSumLow + K, lz = __clzll(s.h < 0 ? ~s.h : s.h);
    const int sh = min(max(lz - 3, 0), low);
    e = E + 2 * kFxSumLow + K - sh;
    return (s.h << sh) + (s.m >> (low - sh));
}
// y 2^e as the integer of a block with exponent E and T bits, rounded
__device__ __forceinline__ long long fx_align(long long y, int e, int E, int T) {
    const int sh = e - E + T;
    return sh >= 0 ? y << sh : (sh < -62 ? 0ll : (y + (1ll << (-sh - 1))) >> -sh);
}
// y 2^e as a double, rounded once more where it is subnormal, infinite past the range
__device__ __forceinline__ double fx_scaled(long long y, int e) {
    const double d = (double)y;
    const int hi = __double2hiint(d), x = ((hi >> 20) & 0x7ff) + e;
    if (y == 0 || (unsigned)(x - 1) >= 0x7feu) return fx_ldexp(d, e);
    return __hiloint2double((hi & 0x800fffff) | (x << 20), __double2loint(d));
}
// the exponent that y 2^e stays below
__device__ __forceinline__ int fx_top_of(long long y, int e) { return y ? e + 64 - __clzll(y < 0 ? -y : y) : kFxMinExp; }

// re + i im = sum_k g(k) v(k): a row of the values->coefficients map
template <int N, typename G, typename V>
__device__ __forceinline__ void fx_map(G&& g, V&& v, long long& re, long long& im) {
    long long mr = kFxHalf, mi = kFxHalf;
    int gh[N], xr[N], xi[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const int2 b = g(k);
        const int4 a = v(k);
        mr = fx_low(FxLimb{a.x, a.y}, FxLimb{b.x, b.y}, mr);
        mi = fx_low(FxLimb{a.z, a.w}, FxLimb{b.x, b.y}, mi);
        gh[k] = b.x; xr[k] = a.x; xi[k] = a.z;
    }
    re = mr >> kFxLow; im = mi >> kFxLow;
#pragma unroll
    for (int k = 0; k < N; ++k) { re = fx_wide(xr[k], gh[k], re); im = fx_wide(xi[k], gh[k], im); }
}
// x 2^sh, rounded
__device__ __forceinline__ long long fx_shift(long long x, int sh) {
    return sh >= 0 ? x << sh : (x + (1ll << (-sh - 1))) >> -sh;
}
__device__ __forceinline__ int4 fx_pack(long long re, long long im) {
    const FxLimb a = fx_split(re), b = fx_split(im);
    return make_int4(a.h, a.l, b.h, b.l);
}

}  // namespace ifgf

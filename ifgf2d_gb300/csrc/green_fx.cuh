// green_fx.cuh -- the kernels of the single-layer and combined formulations in fixed point.
//
// A Green value in FP64 arithmetic takes 110-200 operations of a pipe that does two a clock and SM:
// square root, quotients, sine, cosine and four polynomials of degree 9 (or Chebyshev pieces of degree
// 18).  Here all but the distance, d . n and the last product run on the integer pipe, which does a 32 x 32
// + 64 multiply-add 14 times as often:
//   1. |d|^2 = m 16^e, m in [1, 16): m^(-1/4) from two approximate FP32 operations and one cubic Newton
//      step, hence 1/r, r and the amplitude r^(-1/2); 62-bit mantissas.
//   2. k r / (2 pi) from the top 96 bits of k / (2 pi); its fraction in 64 bits; sine and cosine by their
//      power series in the quadrant (z in [-1/2, 1/2) quarter turns).
//   3. H_nu = sqrt(2 / (pi x)) e^{i(x - pi/4 - nu pi/2)} (P_nu + i Q_nu)(1/x) (A&S 9.2.28-31 without the
//      expansion): P_nu, Q_nu have no phase, and on dyadic pieces of w = 1/x a polynomial of degree 6
//      holds them to 2^-61; the terms from t^4 on fit FP32, the t^3 one 32 bits.
//   4. i H1 and H0 share the phase: g = A e^{i(x - pi/4)} (c (P1 + i Q1) + eta/4 (P0 + i Q0)), the
//      bracket with one binary exponent, the larger of the two coefficients'.
// The errors are a few 2^-57 of |g| and x 2^-58 in the phase (r is an integer in units of 2^-58 of a power of
// two: 1e-15 at x = 300, 5e-13 at 10^5) beside those of the FP64 operations that are left (|d|^2, d . n, the
// products by A), against x 2^-53, the rounding of k r, and more before.  Arguments x <= 1, x >= 2^30, r < 1e-14
// and non-finite values take the FP64 form.
#pragma once
#include <cmath>
#include <cstring>
#include "fixpoint.cuh"
#include "hankel.cuh"

namespace ifgf {

namespace gx {
// 16 bytes of the table, one load; the table's element, so that its alignment is the loads'
struct alignas(16) Four { unsigned x, y, z, w; };
#define GX_TABLE __device__ const Four
#include "green_tables.inc"
}  // namespace gx

struct GreenFx {
    unsigned long long kinv, kap_hi;   // 1/k = kinv 2^(kinv_e - 64); k / (2 pi) = (kap_hi 2^32 + kap_lo) 2^(kap_e - 96)
    unsigned long long turn;           // added to the phase, in 2^-64 turns
    long long eta;                     // the coefficient of H0 in units of the scale: eta 2^(eta_e - 61)
    double a;                          // scale: sqrt(2 / (pi k)) k / 4, or / 4 for the single layer
    unsigned kap_lo;
    int kinv_e, kap_e, eta_e;
    unsigned lo, span;                 // high words of |d|^2 taken here: [lo, lo + span)
    int form;
    double k, k4, eta4;                // k, k / 4 and eta / 4 of the FP64 form
};

// value = mantissa 2^(e - 64), mantissa in [2^63, 2^64)
inline unsigned long long gx_split(double v, int& e) {
    const double f = frexp(v, &e);
    return (unsigned long long)ldexp(f, 53) << 11;
}

inline GreenFx green_fx(int form, double k, double eta) {
    GreenFx g{};
    g.form = form; g.k = k; g.k4 = 0.25 * k; g.eta4 = 0.25 * eta;
    if (!(k > 1e-40 && k < 1e40) || (form == 2 && !(fabs(eta) < 1e40))) return g;     // span 0: all by green_form
    int e;
    const unsigned long long m = gx_split(k, e);
    // 1 / (2 pi) = 0xa2f9836e... 2^-66 (the leading bit is 2^-3); the top 96 bits of the product with m
    const unsigned long long c[2] = {0xa2f9836e4e441529ull, 0xfc2757d1f534ddc0ull};
    auto mul = [](unsigned long long a, unsigned long long b, unsigned long long& hi, unsigned long long& lo) {
        const unsigned __int128 p = (unsigned __int128)a * b;
        hi = (unsigned long long)(p >> 64); lo = (unsigned long long)p;
    };
    unsigned long long h0, l0, h1, l1;
    mul(m, c[0], h0, l0);
    mul(m, c[1], h1, l1);
    l0 += h1;
    h0 += l0 < h1;
    g.kap_e = e - 2;
    if (!(h0 >> 63)) { h0 = h0 << 1 | l0 >> 63; l0 <<= 1; --g.kap_e; }
    g.kap_hi = h0; g.kap_lo = (unsigned)(l0 >> 32);
    // 1 / k = 2^-e 2^64 / m: 64 bits of 2^127 / m by long division
    const unsigned __int128 one = (unsigned __int128)1 << 127;
    const unsigned __int128 q = one / m;                       // in (2^63, 2^64]
    g.kinv = q >> 64 ? ~0ull : (unsigned long long)q;
    g.kinv_e = 1 - e;
    const bool cf = form == 2;
    g.turn = cf ? 0xe000000000000000ull : 0x2000000000000000ull;       // -1/8; the single layer's factor i: + 1/4
    g.a = sqrt(kTwoOverPi / k) * (cf ? 0.25 * k : 0.25);
    const double h = cf ? eta / k : 1.0;
    g.eta_e = -300;
    if (h != 0.0) {
        const unsigned long long hm = gx_split(fabs(h), e);
        g.eta = (long long)(hm >> 3);
        if (h < 0.0) g.eta = -g.eta;
        g.eta_e = e;
    }
    auto hiword = [](double v) { unsigned long long b; memcpy(&b, &v, 8); return (unsigned)(b >> 32); };
    g.lo = hiword(fmax(1.0001 / (k * k), 1.0001e-28)) + 1;
    const unsigned top = hiword(0x1p60 / (k * k));
    g.span = top > g.lo ? top - g.lo : 0;
    return g;
}

namespace gx {

__host__ __device__ __forceinline__ unsigned long long mulhi(unsigned long long a, unsigned long long b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (unsigned long long)((unsigned __int128)a * b >> 64);
#endif
}
__host__ __device__ __forceinline__ unsigned long long wide_u(unsigned a, unsigned b) { return (unsigned long long)a * b; }
__host__ __device__ __forceinline__ long long wide(int a, int b, long long c) {
#ifdef __CUDA_ARCH__
    return fx_wide(a, b, c);
#else
    return (long long)a * b + c;
#endif
}
// a number as its high word and the upper 31 bits of the low one
struct Pair { int h, l; };
__host__ __device__ __forceinline__ Pair pair(long long v) { return Pair{(int)(v >> 32), (int)((unsigned)v >> 1)}; }
// v t / 2^64 + c, short of up to two units; the cross products of both factors fit 63 bits together
__host__ __device__ __forceinline__ long long mul(Pair v, Pair t, long long c) {
    const long long m = wide(v.h, t.l, wide(v.l, t.h, 0));
    return wide(v.h, t.h, m >> 31) + c;
}
__host__ __device__ __forceinline__ long long mul2(Pair a, Pair b, Pair c, Pair d) {     // (a b + c d) / 2^64
    const long long m = wide(a.h, b.l, wide(a.l, b.h, wide(c.h, d.l, wide(c.l, d.h, 0))));
    return wide(a.h, b.h, wide(c.h, d.h, m >> 31));
}
__host__ __device__ __forceinline__ int f2i(float v) {
#ifdef __CUDA_ARCH__
    return __float_as_int(v);
#else
    int i; memcpy(&i, &v, 4); return i;
#endif
}
__host__ __device__ __forceinline__ float i2f(int i) {
#ifdef __CUDA_ARCH__
    return __int_as_float(i);
#else
    float v; memcpy(&v, &i, 4); return v;
#endif
}
__host__ __device__ __forceinline__ unsigned long long d2u(double v) {
#ifdef __CUDA_ARCH__
    return (unsigned long long)__double_as_longlong(v);
#else
    unsigned long long u; memcpy(&u, &v, 8); return u;
#endif
}
__host__ __device__ __forceinline__ double u2d(unsigned long long u) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double v; memcpy(&v, &u, 8); return v;
#endif
}
__host__ __device__ __forceinline__ int lz(unsigned long long v) {
#ifdef __CUDA_ARCH__
    return __clzll((long long)v);
#else
    return v ? __builtin_clzll(v) : 64;
#endif
}

constexpr float kMagic = 12582912.0f;      // 1.5 * 2^23: the sum's low bits are the rounded integer
constexpr int kMagicBits = 0x4B400000;

// y = m^(-1/4) 2^63 for m = M 2^-60 in [1, 16), mf its FP32 value
__host__ __device__ __forceinline__ unsigned long long root4(unsigned long long M, float mf) {
    float y;
#ifdef __CUDA_ARCH__
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(mf));
    asm("sqrt.approx.ftz.f32 %0, %0;" : "+f"(y));
#else
    y = sqrtf(1.0f / sqrtf(mf));
#endif
    const int yb = f2i(y);
    const int b = yb < 0x3f000000 ? 0x3f000000 : yb > 0x3f7fffff ? 0x3f7fffff : yb;
    const unsigned Y0 = ((unsigned)b & 0x7fffffu) | 0x800000u;         // 2^24 y0
    const unsigned long long A2 = wide_u(Y0, Y0) << 16;                // 2^64 y0^2
    const long long eps = (1ll << 60) - (long long)mulhi(M, mulhi(A2, A2));    // 2^60 (1 - m y0^4), below 2^41
    const int eh = (int)(eps >> 12);
    const long long c = (eps >> 2) + ((wide(eh, eh, 0) * 5) >> 41);    // 2^60 (eps / 4 + 5/32 eps^2)
    return ((unsigned long long)Y0 << 39) + (unsigned long long)(((long long)(int)Y0 * c) >> 21);
}

// 2^62 (cos, sin) of f 2^-64 turns: the power series of cos and sin of pi z / 2 in u = z^2, coefficients (-1)^j (pi /
// 2)^(2 j) / (2 j)! and (-1)^j (pi / 2)^(2 j + 1) / (2 j + 1)! times 2^62, in the FP32 tails 2^50 (j >= 6) and 2^47 (j >= 5)
__host__ __device__ __forceinline__ void cos_sin(unsigned long long f, long long& C, long long& S) {
    const unsigned long long g = f + (1ull << 61);
    const int quad = (int)(g >> 62);
    const Pair z = pair((long long)((g << 2) ^ (1ull << 63)));          // quarter turns, [-1/2, 1/2)
    const long long u = wide(z.h, z.h, wide(z.h, z.l, 0) >> 30);
    const Pair up = pair(u);
    const float uf = (float)up.h * 0x1p-32f;
    const int v6 = f2i(fmaf(uf, fmaf(uf, fmaf(uf, -596.0964692794682f, 73926.17259487494f), -7190675.817082061f), kMagic)) +
                   (530397347 - kMagicBits);
    long long c = (wide(v6, up.h, 0) >> 20) - 0x69b47ca8812all;
    c = mul(pair(c), up, 0xf0fa83448dd5dll);
    c = mul(pair(c), up, -0x155d3c7e3cbffa0ll);
    c = mul(pair(c), up, 0x103c1f081b5ac3b3ll);
    c = mul(pair(c), up, -0x4ef4f326f9177969ll);
    c = mul(pair(c), up, 0x4000000000000000ll);
    const int v5 = f2i(fmaf(uf, fmaf(uf, fmaf(uf, fmaf(uf, -6.160172002365761f, 853.8452968090816f), -94125.72633871163f), 8011021.203219744f),
                            kMagic)) + (-506492158 - kMagicBits);
    long long s = (wide(v5, up.h, 0) >> 17) + 0x2a0f0690fdcf0ll;
    s = mul(pair(s), up, -0x4cb4b3398af617ll);
    s = mul(pair(s), up, 0x519af19dd6ab875ll);
    s = mul(pair(s), up, -0x295779cc4b7ca57dll);
    s = mul(pair(s), up, 0x6487ed5110b4611all);
    s = mul(pair(s), z, 0);
    const long long a = quad & 1 ? s : c, b = quad & 1 ? c : s;         // quadrants 1, 2: -cos; 2, 3: -sin
    C = (quad + 1) & 2 ? -a : a;
    S = quad & 2 ? -b : b;
}

__host__ __device__ __forceinline__ Four load(const Four* p) {
    static_assert(alignof(Four) == sizeof(uint4), "read as a uint4");
#ifdef __CUDA_ARCH__
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
    return Four{v.x, v.y, v.z, v.w};
#else
    return *p;
#endif
}
__host__ __device__ __forceinline__ long long join(unsigned lo, unsigned hi) { return (long long)((unsigned long long)hi << 32 | lo); }
// 2^62 p(t), t = tp 2^-64 (tf its FP32 value)
__host__ __device__ __forceinline__ long long poly(Four c01, unsigned c2l, unsigned c2h, Four tail, Pair tp, float tf) {
    const int v3 = (int)((unsigned)f2i(fmaf(fmaf(fmaf(i2f((int)tail.w), tf, i2f((int)tail.z)), tf, i2f((int)tail.y)), tf, kMagic)) + tail.x);
    const long long v2 = (wide(v3, tp.h, 0) >> (32 - (62 - GX_Q3))) + join(c2l, c2h);
    const long long v1 = mul(pair(v2), tp, join(c01.z, c01.w));
    return mul(pair(v1), tp, join(c01.x, c01.y));
}

// the value for d = target - source with |d|^2 = d2 in the taken range and dot = d . n
__host__ __device__ __forceinline__ double2 value(const GreenFx& K, const Four* __restrict__ table, double d2, double dot) {
    const unsigned long long db = d2u(d2);
    const int ex = (int)(db >> 52) - 1023, e = ex >> 2, s = ex & 3;
    const unsigned long long M = (db & 0xfffffffffffffull | 1ull << 52) << (8 + s);
    const float mf = i2f((127 + s) << 23 | (int)(db >> 29 & 0x7fffff));
    const unsigned long long Y = root4(M, mf);                         // r^(-1/2) = Y 2^(-63 - e)
    const unsigned long long ri = mulhi(Y, Y);                         // 1 / r = ri 2^(-62 - 2 e)
    const unsigned long long r = mulhi(M, ri);                         // r = r 2^(-58 + 2 e)

    // the phase: r k / (2 pi), bits of weight 2^-1 ... 2^-64
    const unsigned rl = (unsigned)r, rh = (unsigned)(r >> 32), k1 = (unsigned)K.kap_hi, k2 = (unsigned)(K.kap_hi >> 32);
    const unsigned long long t = wide_u(rl, k2);
    const unsigned long long s1 = wide_u(rh, k1) + (wide_u(rl, k1) >> 32) + (wide_u(rh, K.kap_lo) >> 32) + (unsigned)t;
    const unsigned long long hi = wide_u(rh, k2) + (t >> 32) + (s1 >> 32), lo = s1 << 32;
    const int n = 58 - 2 * e - K.kap_e;                                // 27 ... 63 in the taken range
    long long C, S;
    cos_sin((hi << (64 - n) | lo >> n) + K.turn, C, S);

    // the piece of w = 1 / x and the position in it
    const unsigned long long W = mulhi(ri, K.kinv);                    // w = W 2^(-62 + kinv_e - 2 e)
    const int z = lz(W);
    const unsigned long long wm = W << z;
    int o = z - 2 - K.kinv_e + 2 * e;
    o = o < 0 ? 0 : o;
    const bool far = o >= 8;
    const int nb = far ? 0 : (int)(0x01234456u >> (4 * o) & 15);
    const int base = far ? GX_PIECES - 1 : (int)((o < 4 ? 0x70604000u >> (8 * o) : 0x8e8c8880u >> (8 * (o - 4))) & 255);
    const int sub = far ? 0 : (int)(((unsigned)(wm >> 32) & 0x7fffffffu) >> (31 - nb));
    const Four* c = table + (base + sub) * 10;
    const unsigned long long tu = far ? wm >> (o - 8 < 63 ? o - 8 : 63) : wm << (1 + nb);
    const long long ts = (long long)(tu ^ (1ull << 63));
    const Pair tp = pair(ts);
    const float tf = (float)tp.h * 0x1p-32f;

    const Four q0 = load(c + 4);
    const Pair p0 = pair(poly(load(c), q0.x, q0.y, load(c + 6), tp, tf));
    const Pair i0 = pair(poly(load(c + 1), q0.z, q0.w, load(c + 7), tp, tf));
    long long zr, zi;
    int E = K.eta_e;
    if (K.form == 2) {
        const Four q1 = load(c + 5);
        const Pair p1 = pair(poly(load(c + 2), q1.x, q1.y, load(c + 8), tp, tf));
        const Pair i1 = pair(poly(load(c + 3), q1.z, q1.w, load(c + 9), tp, tf));
        // d . n / r, an integer of scale 2^61 and its exponent
        const unsigned long long ob = d2u(dot);
        const int oe = (int)(ob >> 52 & 0x7ff);
        long long B = oe ? (long long)(mulhi((ob & 0xfffffffffffffull | 1ull << 52) << 11, ri) >> 1) : 0;
        if (ob >> 63) B = -B;
        const int eb = oe - 1023 - 2 * e + 1;
        E = E > eb ? E : eb;
        const int sb = E - eb < 63 ? E - eb : 63, sh = E - K.eta_e < 63 ? E - K.eta_e : 63;
        const Pair b = pair(B >> sb), h = pair(K.eta >> sh);
        zr = mul2(b, p1, h, p0);
        zi = mul2(b, i1, h, i0);
    } else {
        const Pair h = pair(K.eta);
        zr = mul(h, p0, 0);
        zi = mul(h, i0, 0);
    }
    const Pair a = pair(zr), b = pair(zi), cp = pair(C), sp = pair(S), sn = pair(-S);
    const long long gr = mul2(a, cp, b, sn), gi = mul2(a, sp, b, cp);  // scale 2^57 2^-E
    const double A = u2d(((unsigned long long)(964 - e + E) << 52) + ((Y + 512) >> 10)) * K.a;
    return make_double2(A * (double)gr, A * (double)gi);
}

}  // namespace gx

// The pairs that are left to the FP64 form pay for no operation twice: |d|^2 is formed once, k / 4 and eta / 4
// before the sum.  A sum whose every argument is below 1 takes what it takes with that form alone (N = 45000,
// k = 0.5: 643 and 402 ms, combined and single layer; out of line, with these formed again, 662 and 411).
__device__ __forceinline__ double2 green(const GreenFx& K, double dx, double dy, double nx, double ny) {
    const double d2 = dx * dx + dy * dy;
    if (__builtin_expect((unsigned)__double2hiint(d2) - K.lo >= K.span, 0)) {
        if (K.form != 2) return green_sl(d2, K.k);
        return green_cfie(d2, dx * nx + dy * ny, K.k, K.k4, K.eta4);
    }
    return gx::value(K, gx::gx_table, d2, K.form == 2 ? dx * nx + dy * ny : 0.0);
}

}  // namespace ifgf

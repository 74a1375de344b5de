// Device-side numerics of the IFGF matvec: complex arithmetic, interpolation
// coordinates, cone lookups, Chebyshev evaluation and the six kernel plug-ins.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstring>

#include <cuda_runtime.h>

#include "common.hpp"

namespace ifgf
{

template <typename R> struct cplx
{
    R re, im;
};

template <typename R> __device__ __forceinline__ cplx<R> cmake(R a, R b) { return {a, b}; }
template <typename R> __device__ __forceinline__ cplx<R> cadd(cplx<R> a, cplx<R> b)
{
    return {a.re + b.re, a.im + b.im};
}
template <typename R> __device__ __forceinline__ cplx<R> cmul(cplx<R> a, cplx<R> b)
{
    return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
template <typename R> __device__ __forceinline__ cplx<R> cscale(cplx<R> a, R s)
{
    return {a.re * s, a.im * s};
}
// acc += a * b
template <typename R> __device__ __forceinline__ void cfma(cplx<R>& acc, cplx<R> a, cplx<R> b)
{
    acc.re = fma(a.re, b.re, fma(-a.im, b.im, acc.re));
    acc.im = fma(a.re, b.im, fma(a.im, b.re, acc.im));
}

constexpr double INV4PI = 1.0 / (4.0 * 3.14159265358979323846);
constexpr double DPI = 3.14159265358979323846;
constexpr double INF64 = __builtin_huge_val();

// Wavenumber and plug-in switches shared by all kernels of one operator.
struct KParams
{
    static constexpr bool NORMAL = false; // squared distances may be zero or subnormal
    double kr, ki; // k = kr + i ki (real kernels use kr)
    int dx;        // GradHelmholtz derivative direction, -1 = plain single layer
    // kr and ki rounded to floats, and the wavenumbers in turns, kr / (2 pi)
    // and -ki / (2 pi), as two floats each (hi + lo), for the mixed pipeline
    float krh, kih;
    float trh, trl, tih, til;
    // FP64 phases and damping in the units their reductions use, as hi + lo
    // pairs: quarter turns 2 kr / pi and -2 ki / pi, octaves -kr / ln 2
    double qrh, qrl, qih, qil, erh, erl;
    // odd_square's range of squares whose damping is a normal number
    unsigned damp_range;
};
constexpr unsigned NORMAL_SQUARES = 0x7fe00000u;

// a (bh + bl) as an unevaluated sum
inline void scaled_pair(double a, double bh, double bl, double* h, double* l)
{
    *h = a * bh;
    *l = fma(a, bh, -*h) + a * bl;
}

// octaves of damping (or growth) that leave a normal number
constexpr double DAMP_OCTAVES = 1020.0;

inline KParams make_kparams(double kr, double ki, int dx)
{
    KParams p;
    p.kr = kr;
    p.ki = ki;
    p.dx = dx;
    p.krh = (float)kr;
    p.kih = (float)ki;
    // 2 / pi and 1 / ln 2 as hi + lo pairs
    constexpr double TWO_PI_H = 0.6366197723675814, TWO_PI_L = -3.935735335036497e-17;
    constexpr double LOG2E_H = 1.4426950408889634, LOG2E_L = 2.0355273740931033e-17;
    scaled_pair(kr, TWO_PI_H, TWO_PI_L, &p.qrh, &p.qrl);
    scaled_pair(-ki, TWO_PI_H, TWO_PI_L, &p.qih, &p.qil);
    scaled_pair(-kr, LOG2E_H, LOG2E_L, &p.erh, &p.erl);
    p.trh = (float)(0.25 * p.qrh);
    p.trl = (float)(0.25 * p.qrh - (double)p.trh);
    p.tih = (float)(0.25 * p.qih);
    p.til = (float)(0.25 * p.qih - (double)p.tih);
    p.damp_range = NORMAL_SQUARES;
    if (p.erh != 0.0)
    {
        const double lim = DAMP_OCTAVES / std::fabs(p.erh), sq = lim * lim;
        unsigned long long bits;
        std::memcpy(&bits, &sq, sizeof bits);
        const unsigned hi = (unsigned)(bits >> 32);
        p.damp_range = hi > 0x00100000u ? std::min(hi - 0x00100000u, NORMAL_SQUARES) : 0u;
    }
    return p;
}

// ---------------------------------------------------------------------------
// FP64 distance, phase and damping of the kernels.  With the library's square
// root, division and sincos a Helmholtz (source, node) pair took about 150
// instructions, 55 of them on the FP64 pipe; the forms below take about 77
// and 44.  The phase k d is never rounded: its reduction is exact through FMA.
// tests/test_kernel_values.py holds single values to bounds derived from the
// roundings (5.5 units for 1 / d); the library's rounded k d misses the phase's.
// ---------------------------------------------------------------------------
struct DistInv
{
    double d, id; // sqrt(d2), 1 / sqrt(d2)
};

// whether a square of a distance is anything but a normal number (zero or
// subnormal, infinity, NaN), or one beyond `range`
__device__ __forceinline__ bool odd_square(double d2, unsigned range = NORMAL_SQUARES)
{
    return (unsigned)(__double2hiint(d2) - 0x00100000) >= range;
}

// Root and reciprocal root together by Goldschmidt's coupled iteration with a
// residual correction (P. Markstein, "Software division and square root using
// Goldschmidt's algorithms", 6th Conference on Real Numbers and Computers,
// 2004).  From the PTX estimate y of 1 / sqrt(x) (about 20 bits), g = x y and
// h = y / 2 approach sqrt(x) and 1 / (2 sqrt(x)) with one relative error
// r = 1/2 - g h in common; g + g r and h + h r square it.  The root then takes
// its residual x - g^2, and the reciprocal i = 2 h its error 1 - i sqrt(x)
// against that root.
// Unless NORMAL (the caller has seen that d2 is a normal number), zero and
// subnormal squares are scaled first; d2 = 0 gives d = 0, id = inf, and
// d2 = inf d = inf, id = 0.
template <bool NORMAL> __device__ __forceinline__ DistInv dist_inv(double d2)
{
    const bool odd = !NORMAL && odd_square(d2);
    double x = d2, y;
    if (odd)
        x = d2 * 0x1p200;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double g = x * y, h = 0.5 * y;
    const double r = fma(-g, h, 0.5);
    g = fma(g, r, g);
    h = fma(h, r, h);
    const double i = h + h;
    DistInv q;
    q.d = fma(fma(-g, g, x), h, g);
    q.id = fma(i, fma(-i, q.d, 1.0), i);
    if (odd)
    {
        const bool end = d2 == 0.0 || d2 == INF64;
        q.d = end ? d2 : q.d * 0x1p-100;
        q.id = d2 == 0.0 ? INF64 : d2 == INF64 ? 0.0 : q.id * 0x1p100;
    }
    return q;
}

// The reciprocal alone by two steps of Newton's iteration y (3/2 - x y^2 / 2)
template <bool NORMAL> __device__ __forceinline__ double dist_inverse(double d2)
{
    const bool odd = !NORMAL && odd_square(d2);
    double x = d2, y;
    if (odd)
        x = d2 * 0x1p200;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double c = 0.5 * x;
    y *= fma(-(c * y), y, 1.5);
    y = fma(y, fma(-(c * y), y, 0.5), y);
    if (odd)
        y = d2 == 0.0 ? INF64 : d2 == INF64 ? 0.0 : y * 0x1p100;
    return y;
}

// Polynomials through Chebyshev points (exact rational arithmetic, rounded):
// sin(pi r / 2) / r in r^2 (the constant term as a hi + lo pair) and
// (cos(pi r / 2) - 1) / r^2 in r^2 for |r| <= 1/2 (truncation 4e-18 and 1e-19
// of the result), (2^f - 1) / f for |f| <= 1/2 (1e-17 of 2^f).
constexpr int TRIG_N = 15, EXP2_N = 11;
#define IFGF_TRIG_C                                                                           \
    1.5707963267948966, 5.628876619455937e-17, -0.6459640975062443, 0.07969262624604301,       \
        -0.004681754132340976, 0.0001604411507421909, -3.598643352982311e-06,                  \
        5.633933781538053e-08, -1.2337005501361697, 0.2536695079010478, -0.020863480763340773, \
        0.0009192602745468447, -2.5202039028029178e-05, 4.7106784055052287e-07,                \
        -6.329396344967619e-09
#define IFGF_EXP2_C                                                                           \
    0.6931471805599453, 0.24022650695910097, 0.0555041086648216, 0.009618129107606888,         \
        0.0013333558146416936, 0.0001540353044173605, 1.525273382983612e-05,                   \
        1.321544258792169e-06, 1.0178062445845774e-07, 7.072585949269187e-09,                  \
        4.454960598186499e-10
struct PolyConst // the coefficients as compile-time constants
{
    __device__ static constexpr double trig(int i)
    {
        constexpr double c[TRIG_N] = {IFGF_TRIG_C};
        return c[i];
    }
    __device__ static constexpr double exp2(int i)
    {
        constexpr double c[EXP2_N] = {IFGF_EXP2_C};
        return c[i];
    }
};
// The same values in memory, for loops that keep them in registers: as
// constants every use in a loop loads its coefficient again (111 instead of
// 78 instructions per leaf evaluation).
static __device__ double poly_mem[TRIG_N + EXP2_N] = {IFGF_TRIG_C, IFGF_EXP2_C};
struct PolyRegs
{
    double t[TRIG_N], e[EXP2_N];
    __device__ __forceinline__ PolyRegs()
    {
#pragma unroll
        for (int i = 0; i < TRIG_N; i++)
            t[i] = poly_mem[i];
#pragma unroll
        for (int i = 0; i < EXP2_N; i++)
            e[i] = poly_mem[TRIG_N + i];
    }
    __device__ __forceinline__ double trig(int i) const { return t[i]; }
    __device__ __forceinline__ double exp2(int i) const { return e[i]; }
};
// KParams of a loop that keeps the coefficients in registers and has seen
// that the squared distances and the damping are normal numbers
struct KParamsRegs : KParams
{
    static constexpr bool NORMAL = true;
    PolyRegs c;
    __device__ __forceinline__ explicit KParamsRegs(const KParams& p) : KParams(p) {}
};
__device__ __forceinline__ PolyConst poly_of(const KParams&) { return {}; }
__device__ __forceinline__ const PolyRegs& poly_of(const KParamsRegs& p) { return p.c; }

// adding 1.5 2^52 rounds to an integer, held in the sum's low bits
constexpr double ROUND_MAGIC = 6755399441055744.0;

// e^{i (pi / 2) (qh + ql) d}: the quarter turns q d less their nearest integer
// are formed exactly by FMA, |r| <= 1/2
template <class C>
__device__ __forceinline__ cplx<double> quarter_turns(double qh, double ql, double d, const C& k)
{
    const double m = fma(qh, d, ROUND_MAGIC);
    const int n = __double2loint(m);
    double r = fma(qh, d, -(m - ROUND_MAGIC));
    r = fma(ql, d, r);
    const double z = r * r;
    double sp = k.trig(7), cp = k.trig(14);
#pragma unroll
    for (int i = 6; i >= 1; i--)
        sp = fma(sp, z, k.trig(i));
#pragma unroll
    for (int i = 13; i >= 8; i--)
        cp = fma(cp, z, k.trig(i));
    const double s = fma(r, k.trig(0), r * sp);
    const double c = fma(cp, z, 1.0);
    // quarter n mod 4: swap for odd n, negate the cosine for 1 and 2, the
    // sine for 2 and 3
    const bool odd = n & 1;
    const double cc = odd ? s : c, ss = odd ? c : s;
    return {__hiloint2double(__double2hiint(cc) ^ (((n + 1) & 2) << 30), __double2loint(cc)),
            __hiloint2double(__double2hiint(ss) ^ ((n & 2) << 30), __double2loint(ss))};
}

// e^{-kr d} as 2^t, t = (erh + erl) d: 2^f scaled through the exponent field.
// Without branches (they would keep the compiler from interleaving a
// thread's evaluations).  Unless NORMAL the scaling takes two products, the
// second of which rounds to a subnormal number, zero or infinity.
template <class KP> __device__ __forceinline__ double damping(const KP& p, double d)
{
    const double m = fma(p.erh, d, ROUND_MAGIC);
    const int n = __double2loint(m), mh = __double2hiint(m);
    const double f = fma(p.erl, d, fma(p.erh, d, -(m - ROUND_MAGIC)));
    const auto& k = poly_of(p);
    double e = k.exp2(EXP2_N - 1);
#pragma unroll
    for (int i = EXP2_N - 2; i >= 0; i--)
        e = fma(e, f, k.exp2(i));
    e = fma(e, f, 1.0);
    if constexpr (KP::NORMAL)
        return __hiloint2double(__double2hiint(e) + (n << 20), __double2loint(e));
    // m's high word is 0x43380000 (0x4337ffff) for 0 <= n (< 0) in 32 bits
    const bool in = (unsigned)(mh - 0x4337ffff) <= 1u;
    const int t = in ? min(max(n, -1200), 1200) : (mh < 0x43380000 ? -1200 : 1200);
    const int half = t >> 1;
    return (in ? e : 1.0) * __hiloint2double((half + 1023) << 20, 0) *
           __hiloint2double((t - half + 1023) << 20, 0);
}

// f e^{-k d} for complex k: f e^{-kr d} (cos(ki d), -sin(ki d))
template <class KP> __device__ __forceinline__ cplx<double> exp_mk(const KP& p, double d, double f)
{
    return cscale(quarter_turns(p.qih, p.qil, d, poly_of(p)), f * damping(p, d));
}
// e^{i k d} for real k
template <class KP> __device__ __forceinline__ cplx<double> exp_ik(const KP& p, double d)
{
    return quarter_turns(p.qrh, p.qrl, d, poly_of(p));
}

// ---------------------------------------------------------------------------
// Interpolation coordinates (util.hpp:96-116, 156-171)
// ---------------------------------------------------------------------------
// (s, theta, phi) of x relative to the centre xc of a box of side H.  Angles
// are clamped into [0, pi] / [-pi, pi], the range of the C library's atan2,
// so that a device atan2 rounding past +-pi cannot push a point out of the
// interpolation domain.
__device__ __forceinline__ void cart_to_interp(double p0, double p1, double p2, double H,
                                               double* s)
{
    const double a = p0 * p0 + p1 * p1;
    s[2] = fmin(fmax(atan2(p1, p0), -DPI), DPI);
    s[1] = fmin(fmax(atan2(sqrt(a), p2), 0.0), DPI);
    s[0] = H / sqrt(a + p2 * p2);
}

__device__ __forceinline__ void interp_to_cart(const double* s, const double* xc, double H,
                                               double* x)
{
    const double r = H / s[0];
    double st, ct, sp, cp;
    sincos(s[1], &st, &ct);
    sincos(s[2], &sp, &cp);
    x[0] = xc[0] + r * cp * st;
    x[1] = xc[1] + r * sp * st;
    x[2] = xc[2] + r * ct;
}

// ConeDomain::elementForPoint (cone_domain.hpp:232-256): element id or -1
// when the point lies outside the interpolation domain.  hinv = 1 / width:
// floor((s - min) * hinv) equals the reference's floor((s - min) / h) except
// within one rounding of an element boundary.
__device__ __forceinline__ int element_for_point(const double* s, const double* dmin,
                                                 const double* dmax, const double* hinv,
                                                 const int* n)
{
    double d2 = 0;
#pragma unroll
    for (int k = 0; k < 3; k++)
    {
        if (dmin[k] > s[k])
        {
            const double a = dmin[k] - s[k];
            d2 += a * a;
        }
        else if (s[k] > dmax[k])
        {
            const double a = s[k] - dmax[k];
            d2 += a * a;
        }
    }
    if (d2 > 0)
        return -1;
    int id = 0, stride = 1;
#pragma unroll
    for (int j = 0; j < 3; j++)
    {
        int q = (int)floor((s[j] - dmin[j]) * hinv[j]);
        q = min(max(q, 0), n[j] - 1);
        id += q * stride;
        stride *= n[j];
    }
    return id;
}

// ConeDomain::transformBackwards (cone_domain.hpp:173-184), with the division
// by the half width replaced by a multiplication with 2 / width
__device__ __forceinline__ void to_local(int el, const double* s, const double* dmin,
                                         const double* h, const double* hinv, const int* n,
                                         double* loc)
{
    int i0 = el % n[0];
    int r = el / n[0];
    int i1 = r % n[1];
    int i2 = r / n[1];
    const int idx[3] = {i0, i1, i2};
#pragma unroll
    for (int d = 0; d < 3; d++)
    {
        const double a2 = 2.0 * hinv[d]; // 1 / (h / 2)
        const double b = dmin[d] + ((double)idx[d] + 0.5) * h[d];
        loc[d] = (s[d] - b) * a2;
    }
}

// ConeDomain::transform (cone_domain.hpp:145-158)
__device__ __forceinline__ void from_local(int el, const double* loc, const double* dmin,
                                           const double* h, const int* n, double* s)
{
    int i0 = el % n[0];
    int r = el / n[0];
    int i1 = r % n[1];
    int i2 = r / n[1];
    const int idx[3] = {i0, i1, i2};
#pragma unroll
    for (int d = 0; d < 3; d++)
    {
        const double a = 0.5 * h[d];
        const double b = dmin[d] + ((double)idx[d] + 0.5) * h[d];
        s[d] = loc[d] * a + b;
    }
}

// Tensor-product Chebyshev series sum_{ijk} c[i + n0 (j + n1 k)] T_i(x0)
// T_j(x1) T_k(x2) (the function ClenshawEvaluator computes,
// chebinterp.hpp:252-346), with T evaluated by the three-term recurrence.
template <int MAXN>
__device__ __forceinline__ cplx<double> cheb_eval3(const double2* __restrict__ c,
                                                   const double* x, const int* n)
{
    double t0[MAXN], t1[MAXN], t2[MAXN];
    const double* xs[3] = {x, x + 1, x + 2};
    double* ts[3] = {t0, t1, t2};
#pragma unroll
    for (int d = 0; d < 3; d++)
    {
        double* t = ts[d];
        const double xv = *xs[d];
        t[0] = 1.0;
        if (n[d] > 1)
            t[1] = xv;
        for (int i = 2; i < n[d]; i++)
            t[i] = 2.0 * xv * t[i - 1] - t[i - 2];
    }
    double ar = 0, ai = 0;
    int q = 0;
    for (int k = 0; k < n[2]; k++)
    {
        double br = 0, bi = 0;
        for (int j = 0; j < n[1]; j++)
        {
            double cr = 0, ci = 0;
            for (int i = 0; i < n[0]; i++, q++)
            {
                const double2 v = __ldg(c + q);
                cr = fma(v.x, t0[i], cr);
                ci = fma(v.y, t0[i], ci);
            }
            br = fma(cr, t1[j], br);
            bi = fma(ci, t1[j], bi);
        }
        ar = fma(br, t2[k], ar);
        ai = fma(bi, t2[k], ai);
    }
    return {ar, ai};
}

// ---------------------------------------------------------------------------
// Kernel plug-ins.  x = x_src - y_tgt throughout, as in the reference's
// evaluateKernel loops (e.g. helmholtz_ifgf.hpp:104-111).
//   kernel4pi  4 pi G
//   cf         centred factor G(y, xc) at distance q
//   transfer   centre shift G(y, x_child) / G(y, x_parent)
//   leaf_add   s += w G(y, x) / G(y, xc) / leaf_scale(dc) with a = x - y and
//              dc = |y - xc|: the factor that depends on the node alone is
//              applied once to the sum
// kernel4pi and leaf_add take KParams, or KParamsRegs where the caller knows
// that |x|^2 (|a|^2) is a normal number, and the damping (of kernels that have
// one: `damped`) over |x| (|a| - dc) too.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double dot3(const double* a, const double* b)
{
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}
// component dx of a (a dynamic index would put a in local memory)
__device__ __forceinline__ double component(const double* a, int dx)
{
    return dx == 0 ? a[0] : (dx == 1 ? a[1] : a[2]);
}

template <int KIND> struct Plugin;

// laplace_ifgf.hpp
template <> struct Plugin<K_LAPLACE>
{
    static constexpr bool damped = false;
    static constexpr bool needs_normals = false;
    template <class KP>
    __device__ static cplx<double> kernel4pi(const double* x, const double*, const KP&)
    {
        const double d2 = dot3(x, x);
        return {!KP::NORMAL && d2 == 0 ? 0.0 : dist_inverse<KP::NORMAL>(d2), 0.0};
    }
    __device__ static cplx<double> cf(const DistInv& q, const KParams&)
    {
        return {q.id * INV4PI, 0.0};
    }
    __device__ static cplx<double> transfer(double d2, double dp2, const KParams&)
    {
        return {sqrt(dp2) / sqrt(d2), 0.0};
    }
    __device__ static double leaf_scale(double dc) { return dc; }
    template <class KP>
    __device__ static void leaf_add(cplx<double>& s, const double* a, const double*,
                                    cplx<double> w, double, const KP&)
    {
        const double d2 = dot3(a, a);
        s.re = fma(w.re, !KP::NORMAL && d2 == 0 ? 0.0 : dist_inverse<KP::NORMAL>(d2), s.re);
    }
};

// helmholtz_ifgf.hpp (real k)
template <> struct Plugin<K_HELMHOLTZ>
{
    static constexpr bool damped = false;
    static constexpr bool needs_normals = false;
    template <class KP>
    __device__ static cplx<double> kernel4pi(const double* x, const double*, const KP& p)
    {
        const DistInv q = dist_inv<KP::NORMAL>(dot3(x, x));
        return cscale(exp_ik(p, q.d), !KP::NORMAL && q.d == 0 ? 0.0 : q.id);
    }
    __device__ static cplx<double> cf(const DistInv& q, const KParams& p)
    {
        return cscale(exp_ik(p, q.d), q.id * INV4PI);
    }
    __device__ static cplx<double> transfer(double d2, double dp2, const KParams& p)
    {
        const double d = sqrt(d2), dp = sqrt(dp2);
        return cscale(exp_ik(p, d - dp), dp / d);
    }
    __device__ static double leaf_scale(double dc) { return dc; }
    template <class KP>
    __device__ static void leaf_add(cplx<double>& s, const double* a, const double*,
                                    cplx<double> w, double dc, const KP& p)
    {
        const DistInv q = dist_inv<KP::NORMAL>(dot3(a, a));
        cfma(s, w, cscale(exp_ik(p, q.d - dc), q.id));
    }
};

// modified_helmholtz_ifgf.hpp (complex k, kernel e^{-kd}/(4 pi d))
template <> struct Plugin<K_MODHELMHOLTZ>
{
    static constexpr bool damped = true;
    static constexpr bool needs_normals = false;
    template <class KP>
    __device__ static cplx<double> kernel4pi(const double* x, const double*, const KP& p)
    {
        const DistInv q = dist_inv<KP::NORMAL>(dot3(x, x));
        return exp_mk(p, q.d, !KP::NORMAL && q.d == 0 ? 0.0 : q.id);
    }
    __device__ static cplx<double> cf(const DistInv& q, const KParams& p)
    {
        return exp_mk(p, q.d, q.id * INV4PI);
    }
    __device__ static cplx<double> transfer(double d2, double dp2, const KParams& p)
    {
        const double d = sqrt(d2), dp = sqrt(dp2);
        return exp_mk(p, d - dp, dp / d);
    }
    __device__ static double leaf_scale(double dc) { return dc; }
    template <class KP>
    __device__ static void leaf_add(cplx<double>& s, const double* a, const double*,
                                    cplx<double> w, double dc, const KP& p)
    {
        const DistInv q = dist_inv<KP::NORMAL>(dot3(a, a));
        cfma(s, w, exp_mk(p, q.d - dc, !KP::NORMAL && q.d == 0 ? 0.0 : q.id));
    }
};

// grad_helmholtz_ifgf.hpp (complex k, derivative along dx, or plain if -1)
template <> struct Plugin<K_GRADHELMHOLTZ>
{
    static constexpr bool damped = true;
    static constexpr bool needs_normals = false;
    template <class KP>
    __device__ static cplx<double> kernel4pi(const double* x, const double*, const KP& p)
    {
        const DistInv q = dist_inv<KP::NORMAL>(dot3(x, x));
        const double id = q.d < 1e-12 ? 0.0 : q.id;
        if (p.dx < 0)
            return exp_mk(p, q.d, id);
        // -(1/d^2) e^{-kd} (-k - 1/d) x[dx]
        const double f = (id * id) * component(x, p.dx);
        return cmul(exp_mk(p, q.d, f), cplx<double>{p.kr + id, p.ki});
    }
    __device__ static cplx<double> cf(const DistInv& q, const KParams& p)
    {
        return exp_mk(p, q.d, q.id * INV4PI);
    }
    __device__ static cplx<double> transfer(double d2, double dp2, const KParams& p)
    {
        const double invd = d2 > 1e-12 ? 1.0 / sqrt(d2) : 0.0;
        const double dp = sqrt(dp2), d = d2 * invd;
        return exp_mk(p, d - dp, dp * invd);
    }
    __device__ static double leaf_scale(double dc) { return dc; }
    template <class KP>
    __device__ static void leaf_add(cplx<double>& s, const double* a, const double*,
                                    cplx<double> w, double dc, const KP& p)
    {
        const double d2 = dot3(a, a);
        const DistInv q = dist_inv<KP::NORMAL>(d2);
        const double id = d2 > 1e-12 ? q.id : 0.0, d = d2 > 1e-12 ? q.d : 0.0;
        if (p.dx < 0)
        {
            cfma(s, w, exp_mk(p, d - dc, id));
            return;
        }
        const double f = (q.id * q.id) * component(a, p.dx);
        cfma(s, w, cmul(exp_mk(p, d - dc, f), cplx<double>{p.kr + id, p.ki}));
    }
};

// double_layer_helmholtz_ifgf.hpp (complex k, source normals)
template <> struct Plugin<K_DOUBLELAYER>
{
    static constexpr bool damped = true;
    static constexpr bool needs_normals = true;
    template <class KP>
    __device__ static cplx<double> kernel4pi(const double* x, const double* n, const KP& p)
    {
        const DistInv q = dist_inv<KP::NORMAL>(dot3(x, x));
        const double id = q.d < 1e-12 ? 0.0 : q.id;
        const double f = (id * id) * dot3(x, n);
        return cmul(exp_mk(p, q.d, f), cplx<double>{p.kr + id, p.ki});
    }
    __device__ static cplx<double> cf(const DistInv& q, const KParams& p)
    {
        return exp_mk(p, q.d, q.id * INV4PI);
    }
    __device__ static cplx<double> transfer(double d2, double dp2, const KParams& p)
    {
        const double invd = 1.0 / sqrt(d2);
        const double dp = sqrt(dp2), d = d2 * invd;
        return exp_mk(p, d - dp, dp * invd);
    }
    __device__ static double leaf_scale(double dc) { return dc; }
    template <class KP>
    __device__ static void leaf_add(cplx<double>& s, const double* a, const double* n,
                                    cplx<double> w, double dc, const KP& p)
    {
        const double d2 = dot3(a, a);
        const DistInv q = dist_inv<KP::NORMAL>(d2);
        const double id = d2 > 1e-12 ? q.id : 0.0, d = d2 > 1e-12 ? q.d : 0.0;
        const double f = (q.id * q.id) * dot3(a, n);
        cfma(s, w, cmul(exp_mk(p, d - dc, f), cplx<double>{p.kr + id, p.ki}));
    }
};

// combined_field_helmholtz_ifgf.hpp (real kappa, source normals):
// e^{i kap d} / d^3 (nxy - i kap (d nxy + d^2)), nxy = -n . x
template <> struct Plugin<K_COMBINEDFIELD>
{
    static constexpr bool damped = false;
    static constexpr bool needs_normals = true;
    template <class KP>
    __device__ static cplx<double> kernel4pi(const double* x, const double* n, const KP& p)
    {
        const double d2 = dot3(x, x);
        const DistInv q = dist_inv<KP::NORMAL>(d2);
        const double id = d2 < 1e-14 ? 0.0 : q.id, d = d2 < 1e-14 ? 0.0 : q.d;
        const double nxy = -dot3(n, x);
        return cmul(cscale(exp_ik(p, d), id * id * id),
                    cplx<double>{nxy, -p.kr * fma(d, nxy, d2)});
    }
    __device__ static cplx<double> cf(const DistInv& q, const KParams& p)
    {
        return cscale(exp_ik(p, q.d), q.id * INV4PI);
    }
    __device__ static cplx<double> transfer(double d2, double dp2, const KParams& p)
    {
        const double invd = 1.0 / sqrt(d2);
        const double dp = sqrt(dp2), d = d2 * invd;
        return cscale(exp_ik(p, d - dp), dp * invd);
    }
    __device__ static double leaf_scale(double dc) { return dc; }
    template <class KP>
    __device__ static void leaf_add(cplx<double>& s, const double* a, const double* n,
                                    cplx<double> w, double dc, const KP& p)
    {
        const double d2 = dot3(a, a);
        const DistInv q = dist_inv<KP::NORMAL>(d2);
        const double id = d2 > 1e-14 ? q.id : 0.0;
        const double nxy = -dot3(a, n);
        cfma(s, w, cmul(cscale(exp_ik(p, q.d - dc), id * id * id),
                        cplx<double>{nxy, -p.kr * fma(q.d, nxy, d2)}));
    }
};

// d/dk of the Helmholtz kernel, i e^{ikr} / (4 pi).  Centred factor
// e^{ik r_c} / (4 pi) (no 1/r_c: the factored kernel i e^{ik(r - r_c)} is then
// as smooth in the cone coordinates as the Helmholtz one), centre shift
// e^{ik(r - r_p)}.
template <> struct Plugin<K_HELMHOLTZ_DK>
{
    static constexpr bool damped = false;
    static constexpr bool needs_normals = false;
    template <class KP>
    __device__ static cplx<double> kernel4pi(const double* x, const double*, const KP& p)
    {
        const double d = dist_inv<KP::NORMAL>(dot3(x, x)).d;
        const cplx<double> e = exp_ik(p, d);
        const bool zero = !KP::NORMAL && d == 0;
        return {zero ? 0.0 : -e.im, zero ? 0.0 : e.re};
    }
    __device__ static cplx<double> cf(const DistInv& q, const KParams& p)
    {
        return cscale(exp_ik(p, q.d), INV4PI);
    }
    __device__ static cplx<double> transfer(double d2, double dp2, const KParams& p)
    {
        return exp_ik(p, sqrt(d2) - sqrt(dp2));
    }
    __device__ static double leaf_scale(double) { return 1.0; }
    template <class KP>
    __device__ static void leaf_add(cplx<double>& s, const double* a, const double*,
                                    cplx<double> w, double dc, const KP& p)
    {
        const cplx<double> e = exp_ik(p, dist_inv<KP::NORMAL>(dot3(a, a)).d - dc);
        cfma(s, w, cplx<double>{-e.im, e.re});
    }
};

// d/dkappa of the combined-field kernel e^{i kap d} / (4 pi d^3)
// (nxy (1 - i kap d) - i kap d^2):  e^{i kap d} / (4 pi d) (kap (nxy + d) - i),
// nxy = -n . x.  Centred factor and centre shift as for K_HELMHOLTZ_DK.
template <> struct Plugin<K_COMBINEDFIELD_DK>
{
    static constexpr bool damped = false;
    static constexpr bool needs_normals = true;
    template <class KP>
    __device__ static cplx<double> kernel4pi(const double* x, const double* n, const KP& p)
    {
        const double d2 = dot3(x, x);
        const DistInv q = dist_inv<KP::NORMAL>(d2);
        const double id = d2 < 1e-14 ? 0.0 : q.id;
        return cmul(cscale(exp_ik(p, q.d), id), cplx<double>{p.kr * (q.d - dot3(n, x)), -1.0});
    }
    __device__ static cplx<double> cf(const DistInv& q, const KParams& p)
    {
        return cscale(exp_ik(p, q.d), INV4PI);
    }
    __device__ static cplx<double> transfer(double d2, double dp2, const KParams& p)
    {
        return exp_ik(p, sqrt(d2) - sqrt(dp2));
    }
    __device__ static double leaf_scale(double) { return 1.0; }
    template <class KP>
    __device__ static void leaf_add(cplx<double>& s, const double* a, const double* n,
                                    cplx<double> w, double dc, const KP& p)
    {
        const double d2 = dot3(a, a);
        const DistInv q = dist_inv<KP::NORMAL>(d2);
        const double id = d2 > 1e-14 ? q.id : 0.0;
        cfma(s, w, cmul(cscale(exp_ik(p, q.d - dc), id),
                        cplx<double>{p.kr * (q.d - dot3(a, n)), -1.0}));
    }
};

// ===========================================================================
// Mixed precision: FP32 arithmetic on coordinates relative to a nearby box
// centre, with the phase k*r formed and reduced modulo 2 pi in FP64 and the
// reduced angle (|r| <= pi) fed to the FP32 sine/cosine unit.
// ===========================================================================
constexpr float INV4PIF = (float)INV4PI;

// (cos, sin) of (qh + ql) r quarter turns, formed and reduced in FP64: the
// nearest multiple of four is taken off exactly by FMA (adding 1.5 2^54 rounds
// to it), |f| <= 2
__device__ __forceinline__ cplx<float> phase_sc(double qh, double ql, double r)
{
    constexpr double MAGIC4 = 4.0 * ROUND_MAGIC;
    const double n = fma(qh, r, MAGIC4) - MAGIC4;
    const double f = fma(ql, r, fma(qh, r, -n));
    float s, c;
    __sincosf((float)f * 1.5707963267948966f, &s, &c);
    return {c, s};
}

// (cos, sin) of (th + tl) r turns for an FP32 distance r: the nearest integer
// is taken off exactly by FMA (adding 1.5 2^23 rounds to it), so the reduced
// angle carries the accuracy of an FP64 reduction without leaving the FP32
// pipes
__device__ __forceinline__ cplx<float> phase_sc_ff(float th, float tl, float r)
{
    constexpr float MAGIC = 12582912.f;
    const float n = fmaf(th, r, MAGIC) - MAGIC;
    const float f = fmaf(tl, r, fmaf(th, r, -n));
    float s, c;
    __sincosf(f * 6.2831853071795865f, &s, &c);
    return {c, s};
}

// e^{-k r} for complex k (FP64 distance): e^{-kr r} (cos(ki r), -sin(ki r))
__device__ __forceinline__ cplx<float> exp_mk_f(const KParams& p, double r)
{
    const cplx<float> e = phase_sc(p.qih, p.qil, r);
    const float m = __expf((float)(-p.kr * r));
    return {m * e.re, m * e.im};
}
__device__ __forceinline__ cplx<float> exp_ik_f(const KParams& p, double r)
{
    return phase_sc(p.qrh, p.qrl, r);
}

// the same for an FP32 distance (double-float phase)
__device__ __forceinline__ cplx<float> exp_ik_ff(const KParams& p, float r)
{
    return phase_sc_ff(p.trh, p.trl, r);
}
__device__ __forceinline__ cplx<float> exp_mk_ff(const KParams& p, float r)
{
    const cplx<float> e = phase_sc_ff(p.tih, p.til, r);
    const float m = __expf(-p.krh * r);
    return {m * e.re, m * e.im};
}

template <typename R> __device__ __forceinline__ void cfmaf(cplx<R>& acc, cplx<R> a, cplx<R> b)
{
    acc.re = fmaf(a.re, b.re, fmaf(-a.im, b.im, acc.re));
    acc.im = fmaf(a.re, b.im, fmaf(a.im, b.re, acc.im));
}

template <int KIND> struct PluginF;

// Near field: kernel(x, n) with x = x_src - y_tgt in FP32.  Kernels with
// normals take x and n in FP64 (kernel_d): for neighbouring points of a
// surface x.n is O(|x|^2) and would cancel in FP32, so x.n and |x|^2 are
// formed in FP64 and only the rest in FP32.
//
// Leaf sampling: factored(a, aa, b, n, w, dc) = w G(y, x)/G(y, xc) with
// a = x - xc, aa = |a|^2, b = y - xc (FP32) and dc = |b|; the difference
// d - dc is formed as (aa - 2 a.b) / (d + dc), free of cancellation.
__device__ __forceinline__ void factored_geom(const float* a, float aa, const float* b, float dc,
                                              float& inv, float& d, float& dd, float& d2)
{
    const float v0 = a[0] - b[0], v1 = a[1] - b[1], v2 = a[2] - b[2];
    d2 = v0 * v0 + v1 * v1 + v2 * v2;
    inv = rsqrtf(d2);
    d = d2 * inv;
    const float ab = a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
    dd = __fdividef(fmaf(-2.f, ab, aa), d + dc);
}

template <> struct PluginF<K_LAPLACE>
{
    static constexpr bool needs_normals = false;
    __device__ static cplx<float> kernel(const float* x, const float*, const KParams&)
    {
        const float d2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
        return {d2 == 0.f ? 0.f : INV4PIF * rsqrtf(d2), 0.f};
    }
    __device__ static cplx<float> factored(const float* a, float, const float* b, const float*,
                                           cplx<float> w, float dc, const KParams&)
    {
        const float v0 = a[0] - b[0], v1 = a[1] - b[1], v2 = a[2] - b[2];
        const float d2 = v0 * v0 + v1 * v1 + v2 * v2;
        return {d2 == 0.f ? 0.f : w.re * dc * rsqrtf(d2), 0.f};
    }
};

template <> struct PluginF<K_HELMHOLTZ>
{
    static constexpr bool needs_normals = false;
    __device__ static cplx<float> kernel(const float* x, const float*, const KParams& p)
    {
        const float d2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
        if (d2 == 0.f)
            return {0.f, 0.f};
        const float inv = rsqrtf(d2);
        const cplx<float> e = exp_ik_ff(p, d2 * inv);
        const float f = inv * INV4PIF;
        return {e.re * f, e.im * f};
    }
    __device__ static cplx<float> factored(const float* a, float aa, const float* b, const float*,
                                           cplx<float> w, float dc, const KParams& p)
    {
        float inv, d, dd, d2;
        factored_geom(a, aa, b, dc, inv, d, dd, d2);
        const cplx<float> e = exp_ik_ff(p, dd);
        const float f = dc * inv;
        return {f * (w.re * e.re - w.im * e.im), f * (w.re * e.im + w.im * e.re)};
    }
};

template <> struct PluginF<K_MODHELMHOLTZ>
{
    static constexpr bool needs_normals = false;
    __device__ static cplx<float> kernel(const float* x, const float*, const KParams& p)
    {
        const float d2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
        if (d2 == 0.f)
            return {0.f, 0.f};
        const float inv = rsqrtf(d2);
        const cplx<float> e = exp_mk_ff(p, d2 * inv);
        const float f = inv * INV4PIF;
        return {e.re * f, e.im * f};
    }
    __device__ static cplx<float> factored(const float* a, float aa, const float* b, const float*,
                                           cplx<float> w, float dc, const KParams& p)
    {
        float inv, d, dd, d2;
        factored_geom(a, aa, b, dc, inv, d, dd, d2);
        if (d2 == 0.f)
            return {0.f, 0.f};
        const cplx<float> e = exp_mk_ff(p, dd);
        const float f = dc * inv;
        return {f * (w.re * e.re - w.im * e.im), f * (w.re * e.im + w.im * e.re)};
    }
};

template <> struct PluginF<K_GRADHELMHOLTZ>
{
    static constexpr bool needs_normals = false;
    __device__ static cplx<float> kernel(const float* x, const float*, const KParams& p)
    {
        const float d2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
        if (!(d2 >= 1e-24f))
            return {0.f, 0.f};
        const float inv = rsqrtf(d2), d = d2 * inv;
        const cplx<float> e = exp_mk_ff(p, d);
        if (p.dx < 0)
            return {e.re * inv * INV4PIF, e.im * inv * INV4PIF};
        // -(1/4pi) (1/d^2) e^{-kd} (-k - 1/d) x[dx]
        const float mr = -p.krh - inv, mi = -p.kih;
        const float s = -INV4PIF * inv * inv * x[p.dx];
        return {s * (e.re * mr - e.im * mi), s * (e.re * mi + e.im * mr)};
    }
    __device__ static cplx<float> factored(const float* a, float aa, const float* b, const float*,
                                           cplx<float> w, float dc, const KParams& p)
    {
        float inv, d, dd, d2;
        factored_geom(a, aa, b, dc, inv, d, dd, d2);
        if (!(d2 > 1e-12f))
            inv = 0.f;
        const cplx<float> e = exp_mk_ff(p, dd);
        const cplx<float> we = {w.re * e.re - w.im * e.im, w.re * e.im + w.im * e.re};
        if (p.dx < 0)
            return {we.re * dc * inv, we.im * dc * inv};
        const float ww = -(inv * inv) * dc * (a[p.dx] - b[p.dx]);
        const float mr = -p.krh - inv, mi = -p.kih;
        return {ww * (we.re * mr - we.im * mi), ww * (we.re * mi + we.im * mr)};
    }
};

template <> struct PluginF<K_DOUBLELAYER>
{
    static constexpr bool needs_normals = true;
    __device__ static cplx<float> kernel_d(const double* x, const double* n, const KParams& p)
    {
        const double d2d = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
        if (!(d2d >= 1e-24))
            return {0.f, 0.f};
        const float xn = (float)(x[0] * n[0] + x[1] * n[1] + x[2] * n[2]);
        const float d2 = (float)d2d;
        const float inv = rsqrtf(d2), d = d2 * inv;
        const cplx<float> e = exp_mk_ff(p, d);
        const float mr = -p.krh - inv, mi = -p.kih;
        const float s = -INV4PIF * inv * inv * xn;
        return {s * (e.re * mr - e.im * mi), s * (e.re * mi + e.im * mr)};
    }
    __device__ static cplx<float> factored(const float* a, float aa, const float* b, const float* n,
                                           cplx<float> w, float dc, const KParams& p)
    {
        float inv, d, dd, d2;
        factored_geom(a, aa, b, dc, inv, d, dd, d2);
        if (!(d2 > 1e-12f))
            inv = 0.f;
        const float an = (a[0] - b[0]) * n[0] + (a[1] - b[1]) * n[1] + (a[2] - b[2]) * n[2];
        const float ww = -(inv * inv) * dc * an;
        const cplx<float> e = exp_mk_ff(p, dd);
        const cplx<float> we = {w.re * e.re - w.im * e.im, w.re * e.im + w.im * e.re};
        const float mr = -p.krh - inv, mi = -p.kih;
        return {ww * (we.re * mr - we.im * mi), ww * (we.re * mi + we.im * mr)};
    }
};

template <> struct PluginF<K_COMBINEDFIELD>
{
    static constexpr bool needs_normals = true;
    __device__ static cplx<float> kernel_d(const double* x, const double* n, const KParams& p)
    {
        const double d2d = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
        if (!(d2d >= 1e-14))
            return {0.f, 0.f};
        const float kap = p.krh;
        const float nxy = (float)-(n[0] * x[0] + n[1] * x[1] + n[2] * x[2]);
        const float d2 = (float)d2d;
        const float inv = rsqrtf(d2), d = d2 * inv;
        const cplx<float> e = exp_ik_ff(p, d);
        const float f = INV4PIF * inv * inv * inv;
        return {f * (e.re * nxy + e.im * kap * (d * nxy + d2)),
                f * (-e.re * kap * (d * nxy + d2) + e.im * nxy)};
    }
    __device__ static cplx<float> factored(const float* a, float aa, const float* b, const float* n,
                                           cplx<float> w, float dc, const KParams& p)
    {
        float inv, d, dd, d2;
        factored_geom(a, aa, b, dc, inv, d, dd, d2);
        if (!(d2 > 1e-14f))
            return {0.f, 0.f};
        const float kap = p.krh;
        // z = y - x = b - a
        const float nxy = (b[0] - a[0]) * n[0] + (b[1] - a[1]) * n[1] + (b[2] - a[2]) * n[2];
        const cplx<float> e = exp_ik_ff(p, dd);
        const float f = dc * inv * inv * inv;
        const float A = w.re * e.re - w.im * e.im, B = w.re * e.im + w.im * e.re;
        return {f * (A * nxy + B * kap * (d * nxy + d2)), f * (-A * kap * (d * nxy + d2) + B * nxy)};
    }
};

template <> struct PluginF<K_HELMHOLTZ_DK>
{
    static constexpr bool needs_normals = false;
    __device__ static cplx<float> kernel(const float* x, const float*, const KParams& p)
    {
        const float d2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
        if (d2 == 0.f)
            return {0.f, 0.f};
        const cplx<float> e = exp_ik_ff(p, d2 * rsqrtf(d2));
        return {-e.im * INV4PIF, e.re * INV4PIF};
    }
    __device__ static cplx<float> factored(const float* a, float aa, const float* b, const float*,
                                           cplx<float> w, float dc, const KParams& p)
    {
        float inv, d, dd, d2;
        factored_geom(a, aa, b, dc, inv, d, dd, d2);
        const cplx<float> e = exp_ik_ff(p, dd);
        return {-(w.re * e.im + w.im * e.re), w.re * e.re - w.im * e.im};
    }
};
template <> struct PluginF<K_COMBINEDFIELD_DK>
{
    static constexpr bool needs_normals = true;
    __device__ static cplx<float> kernel_d(const double* x, const double* n, const KParams& p)
    {
        const double d2d = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
        if (!(d2d >= 1e-14))
            return {0.f, 0.f};
        const float kap = p.krh;
        const float nxy = (float)-(n[0] * x[0] + n[1] * x[1] + n[2] * x[2]);
        const float d2 = (float)d2d;
        const float inv = rsqrtf(d2), d = d2 * inv;
        const cplx<float> e = exp_ik_ff(p, d);
        const float f = INV4PIF * inv, g = kap * (nxy + d);
        return {f * (g * e.re + e.im), f * (g * e.im - e.re)};
    }
    __device__ static cplx<float> factored(const float* a, float aa, const float* b, const float* n,
                                           cplx<float> w, float dc, const KParams& p)
    {
        float inv, d, dd, d2;
        factored_geom(a, aa, b, dc, inv, d, dd, d2);
        if (!(d2 > 1e-14f))
            return {0.f, 0.f};
        const float kap = p.krh;
        // z = y - x = b - a, nxy = z . n
        const float nxy = (b[0] - a[0]) * n[0] + (b[1] - a[1]) * n[1] + (b[2] - a[2]) * n[2];
        const cplx<float> e = exp_ik_ff(p, dd);
        const float vr = w.re * e.re - w.im * e.im, vi = w.re * e.im + w.im * e.re;
        const float g = kap * (nxy + d);
        return {inv * (g * vr + vi), inv * (g * vi - vr)};
    }
};


// Centred factor CF(y - xc) and centre-shift factor G(y, xc)/G(y, pxc) in
// mixed precision: distances in FP64 (d2 given), phases reduced in FP64.
template <int KIND>
__device__ __forceinline__ cplx<float> cf_mixed(double d2, const KParams& p)
{
    const double d = dist_inv<false>(d2).d;
    if (KIND == K_HELMHOLTZ_DK || KIND == K_COMBINEDFIELD_DK)
    {
        const cplx<float> e = exp_ik_f(p, d);
        return {e.re * INV4PIF, e.im * INV4PIF};
    }
    const float id = rsqrtf((float)d2) * INV4PIF;
    if (KIND == K_LAPLACE)
        return {id, 0.f};
    if (KIND == K_HELMHOLTZ || KIND == K_COMBINEDFIELD)
    {
        const cplx<float> e = exp_ik_f(p, d);
        return {e.re * id, e.im * id};
    }
    const cplx<float> e = exp_mk_f(p, d);
    return {e.re * id, e.im * id};
}

template <int KIND>
__device__ __forceinline__ cplx<float> transfer_mixed(double d2, double dp2, const KParams& p)
{
    const double d = sqrt(d2), dp = sqrt(dp2);
    if (KIND == K_HELMHOLTZ_DK || KIND == K_COMBINEDFIELD_DK)
        return exp_ik_f(p, d - dp);
    const float ratio = __fdividef((float)dp, (float)d);
    if (KIND == K_LAPLACE)
        return {ratio, 0.f};
    if (KIND == K_HELMHOLTZ || KIND == K_COMBINEDFIELD)
    {
        const cplx<float> e = exp_ik_f(p, d - dp);
        return {e.re * ratio, e.im * ratio};
    }
    const cplx<float> e = exp_mk_f(p, d - dp);
    return {e.re * ratio, e.im * ratio};
}

// The same factor from a tabulated delta = d - d_parent (FP64 difference
// rounded to FP32) and ratio = d_parent / d: the distance tables of
// multi-wavenumber batches, which serve every wavenumber of the batch.
template <int KIND>
__device__ __forceinline__ cplx<float> transfer_delta(float delta, float ratio, const KParams& p)
{
    if (KIND == K_HELMHOLTZ_DK || KIND == K_COMBINEDFIELD_DK)
        return exp_ik_ff(p, delta);
    if (KIND == K_LAPLACE)
        return {ratio, 0.f};
    const cplx<float> e = (KIND == K_HELMHOLTZ || KIND == K_COMBINEDFIELD) ? exp_ik_ff(p, delta)
                                                                          : exp_mk_ff(p, delta);
    return {e.re * ratio, e.im * ratio};
}

// FP32 coordinates: (s, theta, phi) from an FP32 difference vector.  Roundings
// are spelled out (the compiler could contract products and sums differently
// in every kernel), so that all kernels get the same coordinates.
__device__ __forceinline__ void cart_to_interp_f(float p0, float p1, float p2, float H, float* s)
{
    const float a = __fmaf_rn(p1, p1, __fmul_rn(p0, p0));
    s[2] = fminf(fmaxf(atan2f(p1, p0), -(float)DPI), (float)DPI);
    s[1] = fminf(fmaxf(atan2f(sqrtf(a), p2), 0.f), (float)DPI);
    s[0] = __fmul_rn(H, rsqrtf(__fmaf_rn(p2, p2, a)));
}


// FP32 cone-lookup parameters of one level, made once per CTA in shared
// memory so that the far-field lookups read no level data from global memory.
struct LookupF
{
    float lo[3], hi[3], hinv[3], top[3]; // domain, 1 / fine width, nf - 1
    int nf[3];
};

__device__ __forceinline__ void make_lookupf(const LevelGeom& G, LookupF& L)
{
#pragma unroll
    for (int d = 0; d < 3; d++)
    {
        L.lo[d] = (float)G.dmin[d];
        L.hi[d] = (float)G.dmax[d];
        L.hinv[d] = (float)G.hfi[d];
        L.top[d] = (float)(G.nf[d] - 1);
        L.nf[d] = G.nf[d];
    }
}

// Fine element of the point p in FP32 (-1 outside the domain) and its local
// coordinates: with t = (s - lo) / h the element index is q = floor(t)
// (clamped) and the local coordinate 2 (t - q) - 1, the same quantities as
// (s - centre) / (h / 2), the same in every kernel (roundings spelled out).
__device__ __forceinline__ int lookup_f(const LookupF& L, const double* p, double H, float* loc)
{
    float sf[3];
    cart_to_interp_f((float)p[0], (float)p[1], (float)p[2], (float)H, sf);
    bool inside = true;
    int id = 0, stride = 1;
#pragma unroll
    for (int j = 0; j < 3; j++)
    {
        inside = inside && sf[j] >= L.lo[j] && sf[j] <= L.hi[j];
        const float t = __fmul_rn(__fsub_rn(sf[j], L.lo[j]), L.hinv[j]);
        const float q = fminf(fmaxf(floorf(t), 0.f), L.top[j]);
        loc[j] = __fmaf_rn(2.f, __fsub_rn(t, q), -1.f);
        id += __float2int_rz(q) * stride;
        stride *= L.nf[j];
    }
    return inside ? id : -1;
}

// fine_lookup_mixed with the level's FP32 parameters at hand (lookup_f); the
// FP64 fallback (outside the FP32 domain or an inactive cone) is that of
// fine_lookup_mixed.
__device__ __forceinline__ int fine_lookup_fast(const LookupF& L, const LevelGeom& G,
                                                const int* __restrict__ fm, const double* p,
                                                double H, float* loc, unsigned long long* err)
{
    const int id = lookup_f(L, p, H, loc);
    if (id >= 0)
    {
        const int gf = fm[id];
        if (gf >= 0)
            return gf;
    }
    double s[3], ld[3];
    cart_to_interp(p[0], p[1], p[2], H, s);
    const int fe = element_for_point(s, G.dmin, G.dmax, G.hfi, G.nf);
    if (fe < 0)
        return -1;
    const int gf = fm[fe];
    if (gf < 0)
    {
        atomicAdd(err, 1ull);
        return -1;
    }
    to_local(fe, s, G.dmin, G.hf, G.hfi, G.nf, ld);
    loc[0] = (float)ld[0];
    loc[1] = (float)ld[1];
    loc[2] = (float)ld[2];
    return gf;
}

} // namespace ifgf

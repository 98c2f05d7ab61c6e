// mk_tri.cuh -- the FP64 form's geodesic integrator on the FP32 pipe.
//
// One binary64 warp instruction holds a GB300 sub-partition's FP64 unit 64
// cycles, so an RK4 step in binary64 (four accelerations, ~420 instructions)
// takes ~27 k cycles of a warp however few of its lanes work.  Its precision
// is needed in the state, not in the accelerations: with the step rule dt =
// (r - r_EH) / 40 an acceleration enters k as dt a, at most ~1/40 of k, and x
// as dt^2 a, so an acceleration good to 2^-48 of its largest term moves the
// state by about as much as one binary64 rounding of k near the hole and by
// far less elsewhere.  Hence:
//   * state (x^mu, k^mu), r and the step size: three floats each (72 bits),
//     with no rounding of the state worth counting (binary64 rounds x at
//     1000 M to 1e-13 M, which is most of that form's error at the hole);
//   * accelerations and stage points: float pairs (~48 bits), ~780 FP32
//     instructions an acceleration, ~4.2 k a step.
// Against a 113-bit integration of 400 random rays each at spin 0, 0.5 and
// 0.94 (camera at 1000 M), end states are 0.17-0.24 times as far off as
// those of the binary64 integrator (geometric mean), captured and escaping
// rays alike, if the last approach to the horizon is taken in binary64 (in
// triples it took longer, ~38 k cycles a step against ~31 k):
// there k grows as 1 / (r - r_EH), and E and L, which steer the ray, are
// small differences of its components.  near_distance (mk_geodesic.cu) says
// from where.  The fused render needs no such switch: what a ray emits there
// is redshifted away, and its images do not change with the stopping distance
// from tol 1e-2 to 1e-8.
//
// That holds where binary64's own rounding of the state is large: from afar,
// off the axes, with many short steps.  Few long steps, or a state that
// binary64 rounds little, turn it round, and such rays stay in binary64
// (tri_policy, fixed_range, pair_request, with the measurements).
//
// Error-free steps: TwoSum (Knuth, TAOCP vol. 2, 4.2.2), FastTwoSum (Dekker
// 1971), the product error by one fused multiply-add.  Every product and sum
// is written through f_mul / f_add, which no compiler contracts.
#pragma once

#include <math.h>

#include "mk_kerr.cuh"

namespace mk {

#define MK_HD __host__ __device__ __forceinline__

MK_HD float f_mul(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fmul_rn(a, b);
#else
    volatile float p = a * b;
    return p;
#endif
}
MK_HD float f_add(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fadd_rn(a, b);
#else
    return a + b;
#endif
}
MK_HD float f_sub(float a, float b) { return f_add(a, -b); }

struct pr {   // pair: h + l
    float h, l;
};
struct tri {  // h + m + l
    float h, m, l;
};

MK_HD void two_sum_f(float a, float b, float &s, float &e) {
    s = f_add(a, b);
    const float v = f_sub(s, a);
    e = f_add(f_sub(a, f_sub(s, v)), f_sub(b, v));
}
MK_HD void fast_sum_f(float a, float b, float &s, float &e) {
    s = f_add(a, b);
    e = f_sub(b, f_sub(s, a));
}

// ------------------------------------------------------------------ pairs
// mul and add leave the low word unnormalised (a few ulp of the high one);
// mulr and addr normalise, where the result is a factor of several products
// or a sum that may cancel.
MK_HD pr p_norm(pr x) {
    pr o;
    fast_sum_f(x.h, x.l, o.h, o.l);
    return o;
}
MK_HD pr p_mul(pr x, pr y) {
    const float p = f_mul(x.h, y.h);
    float e = fmaf(x.h, y.h, -p);
    e = fmaf(x.h, y.l, e);
    e = fmaf(x.l, y.h, e);
    return {p, e};
}
MK_HD pr p_mulr(pr x, pr y) { return p_norm(p_mul(x, y)); }
MK_HD pr p_sqr(pr x) {
    const float p = f_mul(x.h, x.h);
    float e = fmaf(x.h, x.h, -p);
    e = fmaf(f_add(x.h, x.h), x.l, e);
    return {p, e};
}
MK_HD pr p_two(pr x, float c) { return {f_mul(x.h, c), f_mul(x.l, c)}; }  // c a power of two
MK_HD pr p_neg(pr x) { return {-x.h, -x.l}; }
MK_HD pr p_add(pr x, pr y) {
    float s, e;
    two_sum_f(x.h, y.h, s, e);
    return {s, f_add(e, f_add(x.l, y.l))};
}
MK_HD pr p_addr(pr x, pr y) { return p_norm(p_add(x, y)); }
MK_HD pr p_sub(pr x, pr y) { return p_add(x, p_neg(y)); }
MK_HD pr p_subr(pr x, pr y) { return p_norm(p_sub(x, y)); }

// 1/sqrt and 1/x: the float unit's approximation, one Newton step in float,
// then a second- (third-) order correction from the pair residual
MK_HD pr p_rsqrt(pr x) {
#ifdef __CUDA_ARCH__
    float y = rsqrt_ftz(x.h);
#else
    float y = 1.0f / sqrtf(x.h);
#endif
    y = fmaf(f_mul(0.5f, y), fmaf(-f_mul(x.h, y), y, 1.0f), y);
    const float t = f_mul(y, y), u = fmaf(y, y, -t);
    const float p = f_mul(x.h, t);
    float e = fmaf(x.h, t, -p);
    e = fmaf(x.h, u, e);
    e = fmaf(x.l, t, e);
    const float d = f_sub(f_sub(1.0f, p), e);  // 1 - x y^2
    return p_norm({y, f_mul(f_mul(y, d), fmaf(0.375f, d, 0.5f))});
}
MK_HD pr p_rcp(pr x) {
#ifdef __CUDA_ARCH__
    float y = rcp_ftz(x.h);
#else
    float y = 1.0f / x.h;
#endif
    y = fmaf(fmaf(-x.h, y, 1.0f), y, y);
    const float p = f_mul(x.h, y);
    float e = fmaf(x.h, y, -p);
    e = fmaf(x.l, y, e);
    const float d = f_sub(f_sub(1.0f, p), e);  // 1 - x y
    return p_norm({y, f_mul(y, fmaf(d, d, d))});
}

// Paired FP32 instructions (each lane rounds as its scalar twin): the pipe
// takes two cycles for one, but half as many are fetched and issued.
__device__ __forceinline__ float2 v_two_sum(float2 a, float2 b, float2 &e) {
    const float2 m1 = make_float2(-1.0f, -1.0f), s = __fadd2_rn(a, b), v = __ffma2_rn(a, m1, s);
    e = __fadd2_rn(__ffma2_rn(__ffma2_rn(v, m1, s), m1, a), __ffma2_rn(v, m1, b));
    return s;
}

// Z^(-1/3): the float unit's estimate, one Newton step in float, a third-order
// correction from the pair residual 1 - Z x^3
__device__ __forceinline__ pr p_rcbrt(pr z) {
    float l, x;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(z.h));
    l *= -0.333333343f;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(x) : "f"(l));
    x = fmaf(f_mul(x, 0.333333343f), fmaf(-f_mul(f_mul(z.h, x), x), x, 1.0f), x);
    const pr x2 = {f_mul(x, x), fmaf(x, x, -f_mul(x, x))};
    const pr x3 = p_mulr(x2, {x, 0.0f});
    const float p = f_mul(z.h, x3.h);
    float e = fmaf(z.h, x3.h, -p);
    e = fmaf(z.h, x3.l, e);
    e = fmaf(z.l, x3.h, e);
    const float d = f_sub(f_sub(1.0f, p), e);
    return p_norm({x, f_mul(f_mul(x, d), fmaf(0.222222222f, d, 0.333333343f))});
}

// ---------------------------------------------------------------- triples
// On the device both conversions keep off the FP64 pipe, where each F2F costs
// as much as an addition (64 cycles a warp instruction): the words are moved
// by bit operations, and only a triple's two additions are binary64.  Values
// outside the formats' common normal range take the ordinary conversions.
MK_HD tri t_from_cvt(double v) {
    tri t;
    t.h = (float)v;
    v -= (double)t.h;
    t.m = (float)v;
    t.l = (float)(v - (double)t.m);
    return t;
}
MK_HD tri t_from(double v) {
#ifdef __CUDA_ARCH__
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    const unsigned sign = hi & 0x80000000u, a = hi & 0x7fffffffu, e = a >> 20;
    if (e - 947u <= 180u) {  // 2^-76 <= |v| < 2^105
        // significand words of 24, 24 and 5 bits (the first truncated)
        tri t;
        t.h = __uint_as_float(sign | (((a - (896u << 20)) << 3) | (lo >> 29)));
        const unsigned low = lo & 0x1fffffffu;
        const float u = __uint_as_float(sign | ((e - 943u) << 23));  // 2^(e - 1023 - 47)
        t.m = f_mul((float)(low >> 5), u);
        t.l = f_mul((float)(low & 31u), f_mul(u, 0.03125f));
        return t;
    }
    if ((a | lo) == 0u) return {v < 0.0 ? -0.0f : 0.0f, 0.0f, 0.0f};
#endif
    return t_from_cvt(v);
}
MK_HD tri t_norm(tri x) {
    float h, t;
    tri o;
    fast_sum_f(x.h, x.m, h, t);
    fast_sum_f(t, x.l, o.m, o.l);
    fast_sum_f(h, o.m, o.h, o.m);
    return o;
}
// t_from cuts its words off; these are rounded to the nearest, as the sums
// below leave theirs: for words that t_less compares, and for constants of
// which a pair is kept (cut off they were up to 2^-48 too small)
MK_HD tri t_near(double v) { return t_norm(t_from(v)); }
MK_HD pr p_near(double v) {
    const tri t = t_near(v);
    return {t.h, t.m};
}
MK_HD double d_from(float x) {
#ifdef __CUDA_ARCH__
    const unsigned u = __float_as_uint(x), a = u & 0x7fffffffu;
    if (a - 0x00800000u < 0x7f000000u || a == 0u) {  // normal or zero
        const unsigned hi = (a >> 3) + (896u << 20);
        return __hiloint2double((int)((a ? hi : 0u) | (u & 0x80000000u)), (int)(a ? u << 29 : 0u));
    }
#endif
    return (double)x;
}
MK_HD double t_to(tri t) { return d_from(t.h) + (d_from(t.m) + d_from(t.l)); }
MK_HD tri t_neg(tri t) { return {-t.h, -t.m, -t.l}; }
MK_HD pr t_pair(tri t) { return {t.h, t.m}; }

MK_HD tri t_add(tri x, tri y) {
    float s1, e1, s2, e2, e3, h, t, m;
    two_sum_f(x.h, y.h, s1, e1);
    two_sum_f(x.m, y.m, s2, e2);
    two_sum_f(s2, e1, s2, e3);
    const float s3 = f_add(f_add(x.l, y.l), f_add(e2, e3));
    tri o;
    fast_sum_f(s1, s2, h, t);
    fast_sum_f(t, s3, m, o.l);
    fast_sum_f(h, m, o.h, o.m);
    return o;
}
// product to ~2^-66, words in order but not normalised
MK_HD tri t_mul(tri x, tri y) {
    const float p = f_mul(x.h, y.h), e = fmaf(x.h, y.h, -p);
    const float c = f_mul(x.h, y.m), ce = fmaf(x.h, y.m, -c);
    const float d = f_mul(x.m, y.h), de = fmaf(x.m, y.h, -d);
    float s, t, u, w;
    two_sum_f(c, d, s, t);
    two_sum_f(e, s, u, w);
    const float lo = fmaf(x.m, y.m, fmaf(x.h, y.l, fmaf(x.l, y.h, f_add(f_add(ce, de), f_add(t, w)))));
    return {p, u, lo};
}
MK_HD tri t_sqr(tri x) {
    const float p = f_mul(x.h, x.h), e = fmaf(x.h, x.h, -p);
    const float g = f_add(x.h, x.h), c = f_mul(g, x.m), ce = fmaf(g, x.m, -c);
    float s, t;
    two_sum_f(e, c, s, t);
    return {p, s, fmaf(x.m, x.m, fmaf(g, x.l, f_add(ce, t)))};
}
MK_HD tri t_mulr(tri x, tri y) { return t_norm(t_mul(x, y)); }

// 1/x: the pair reciprocal and a Newton step from the triple residual
__device__ __forceinline__ tri t_rcp(tri x) {
    const pr y = p_rcp({x.h, x.m});
    const tri p = t_mul(x, {y.h, y.l, 0.0f});
    const float d = f_sub(f_sub(f_sub(1.0f, p.h), p.m), p.l);
    return t_norm({y.h, y.l, f_mul(y.h, d)});
}

__device__ __forceinline__ tri t_rsqrt(tri x) {
    const pr y = p_rsqrt({x.h, x.m});
    const tri y3 = {y.h, y.l, 0.0f}, p = t_mul(t_norm(t_sqr(y3)), x);
    const float d = f_sub(f_sub(f_sub(1.0f, p.h), p.m), p.l);
    return t_norm({y.h, y.l, f_mul(f_mul(0.5f, y.h), d)});
}
static __device__ __noinline__ tri t_dot(tri x1, tri y1, tri x2, tri y2, tri x3, tri y3) {
    return t_add(t_add(t_mul(x1, y1), t_mul(x2, y2)), t_mul(x3, y3));
}
__device__ __forceinline__ tri t_sub(tri x, tri y) { return t_add(x, t_neg(y)); }

// x < y on the two leading words (x and y normalised)
MK_HD bool t_less(tri x, tri y) { return x.h < y.h || (x.h == y.h && x.m < y.m); }

// ----------------------------------------------------------- acceleration
struct SpinTri {
    pr a, aa;     // spin and its square as pairs
    tri aa3;      // the square to 72 bits
};
MK_HD SpinTri spin_tri(double a) {
    SpinTri s;
    const tri t = t_from(a);  // the last word to the pair's low one, not cut off
    s.a = {t.h, f_add(t.m, t.l)};
    s.aa3 = t_from(a * a);
    s.aa = {s.aa3.h, f_add(s.aa3.m, s.aa3.l)};
    return s;
}

// What accel_pair meets on its way and the radius, step rule and sampler use:
// r, f, l3, 1/(r^2 + a^2), and 1/q, 1/r to float.
struct PairPoint {
    pr r, f, l3, ira;
    float iq, ir;
};

// kerr_accel's contraction in pairs.
MK_HD void accel_pair(pr x, pr y, pr z, pr k0, pr k1, pr k2, pr k3, pr a, pr aa, pr A[4], PairPoint &o) {
    const pr zz = p_sqr(z);
    const pr kk = p_two(p_subr(p_add(p_add(p_sqr(x), p_sqr(y)), zz), aa), 0.5f);
    const pr Q = p_addr(p_sqr(kk), p_mul(aa, zz));
    const pr iq = p_rsqrt(Q);
    const pr rr = p_addr(p_mul(Q, iq), kk);
    const pr ir = p_rsqrt(rr);
    const pr r = p_mulr(rr, ir);
    const pr rra = p_addr(rr, aa), ira = p_rcp(rra);
    const pr l3 = p_mulr(z, ir), f = p_mulr(r, iq), rira = p_mulr(r, ira), aira = p_mulr(a, ira);
    const pr P = p_addr(p_mul(x, k1), p_mul(y, k2)), M = p_subr(p_mul(y, k1), p_mul(x, k2));
    const pr c = p_two(f, 0.5f), rz = p_two(p_mulr(l3, p_mulr(rra, iq)), 0.5f);
    const pr Dr = p_addr(p_mul(c, P), p_mul(rz, k3));
    const pr L = p_addr(p_mul(rira, P), p_mul(aira, M));
    const pr lv = p_addr(k0, p_add(L, p_mul(l3, k3)));
    const pr h = p_mulr(l3, ir);
    const pr G = p_subr(p_sub(p_mul(ira, P), p_two(p_mul(rira, L), 2.0f)), p_mul(h, k3));
    const pr T = p_add(p_mul(rira, p_addr(p_sqr(k1), p_sqr(k2))), p_mul(ir, p_sqr(k3)));
    const pr Dlv = p_addr(p_mul(G, Dr), T);
    const pr fc = p_subr(p_add(iq, p_two(iq, 2.0f)), p_two(p_sqr(f), 2.0f));
    const pr ft = p_mulr(p_mul(aa, l3), p_sqr(iq));
    const pr Df = p_subr(p_mul(fc, Dr), p_mul(ft, k3));
    const pr flv = p_mulr(f, lv), hl = p_norm(p_two(p_sqr(lv), 0.5f));
    const pr mF0 = p_addr(p_mul(Df, lv), p_mul(f, Dlv));
    const pr al = p_addr(p_mul(flv, G), p_mul(fc, hl));
    const pr be = p_mulr(flv, Dr), ga = p_two(p_mulr(flv, aira), 2.0f);
    const pr N = p_subr(p_mul(rira, M), p_mul(aira, P));
    const pr lg = p_addr(rira, p_mul(p_mulr(a, aira), p_mulr(h, l3)));
    const pr fth = p_mulr(ft, hl);
    const pr lF = p_subr(p_add(al, p_add(p_mul(be, lg), p_mul(ga, N))), p_mul(l3, fth));
    A[0] = p_addr(p_mul(f, lF), mF0);
    const pr F2 = p_subr(p_two(p_mul(be, rira), 2.0f), A[0]);
    const pr Aa = p_subr(p_add(p_mul(rira, F2), p_mul(al, c)), p_mul(be, ira)), B = p_mulr(aira, F2);
    A[1] = p_sub(p_add(p_mul(x, Aa), p_mul(y, B)), p_mul(ga, k2));
    A[2] = p_add(p_sub(p_mul(y, Aa), p_mul(x, B)), p_mul(ga, k1));
    A[3] = p_sub(p_add(p_mul(l3, p_subr(p_mul(be, ir), A[0])), p_mul(al, rz)), fth);
    o.r = r;
    o.f = f;
    o.l3 = l3;
    o.ira = ira;
    o.iq = iq.h;
    o.ir = ir.h;
}

// The radius to ~2^-60 from its pair r0: one Newton step on r^4 - (x^2 + y^2
// + z^2 - a^2) r^2 - a^2 z^2 = 0 (slope 2 q r^2 / r^2 in r^2), its residual in
// triples.  The step size near the horizon is the small difference r - r_EH.
MK_HD tri t_radius(tri x, tri y, tri z, tri aa, pr r0, float iq, float ir) {
    const tri z2 = t_sqr(z);
    const tri R2 = t_add(t_add(t_sqr(x), t_sqr(y)), z2);
    const tri rr = t_sqr({r0.h, r0.l, 0.0f});
    const tri w = t_add(t_add(rr, t_neg(R2)), aa);
    const tri F = t_add(t_mul(rr, w), t_neg(t_mul(aa, z2)));
    const float d = f_mul(f_mul(f_add(F.h, F.m), f_mul(-0.5f, iq)), f_mul(0.5f, ir));
    return t_add({r0.h, r0.l, 0.0f}, {d, 0.0f, 0.0f});
}

// ---------------------------------------------------------------- RK4 step
struct TriState {
    tri X[4], K[4];
};
MK_HD void tri_state(const double s[8], TriState &o) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
        o.X[i] = t_from(s[i]);
        o.K[i] = t_from(s[4 + i]);
    }
}
MK_HD void tri_doubles(const TriState &o, double s[8]) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
        s[i] = t_to(o.X[i]);
        s[4 + i] = t_to(o.K[i]);
    }
}

// Ranges in which the triples hold every intermediate with all its words
// inside the float range; a ray that leaves them is continued in binary64 from
// the state before, one that starts outside from its start.
constexpr float TRI_MIN_R = 1e-2f, TRI_MAX_R = 1e6f, TRI_MAX_K = 1e12f, TRI_MIN_K = 1e-6f;
// true out of range or at NaN: a step over the horizon toward r = 0 overflows
// floats before doubles; r^4 underflows them, and inside the ring, where r^2
// is a small difference, the pairs lose the radius (1e-11 of r - r_EH at r =
// 1e-6, spin 0.9)
__device__ __forceinline__ float tri_sum_k(const TriState &s) {
    return (fabsf(s.K[0].h) + fabsf(s.K[1].h)) + (fabsf(s.K[2].h) + fabsf(s.K[3].h));
}
__device__ __forceinline__ bool tri_left_range(const TriState &s, float r) {
    return !(r >= TRI_MIN_R && r <= TRI_MAX_R && tri_sum_k(s) <= TRI_MAX_K);
}

// first-stage acceleration, radius and metric data at a state
struct TriPoint {
    pr a1[4];
    tri r;
    PairPoint m;
};

// One RK4 step of size dt from s, where q holds the first-stage acceleration,
// then the same at the new state: x += dt k + dt^2/6 (a1 + a2 + a3), k +=
// dt/6 (a1 + 2 a2 + 2 a3 + a4) (RK4_gen, geodesics.py:317-336, for x'' = a(x,
// x')), the leading dt k to 2^-66.  ready: s is the new state already, only q
// is evaluated.  TIME: advance x^0 too (nothing on the imaging path reads it).
//
// The four accelerations are one copy of the code in a loop: unrolled, a step
// was ~5 k instructions (80 KB) and its warps waited for instruction fetches
// 3 cycles of every 5.
template <bool TIME>
MK_HD void tri_step(TriState &s, TriPoint &q, tri dt, pr a, pr aa, tri aa3, bool ready) {
    const pr d = {dt.h, dt.m}, h = p_two(d, 0.5f);
    pr x[4], k[4], b[4], acc[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        k[i] = t_pair(s.K[i]);
        b[i] = q.a1[i];
        acc[i] = {0.0f, 0.0f};
    }
#pragma unroll 1
    for (int st = ready ? 3 : 0; st < 4; ++st) {
        if (st < 3) {  // the point of stage st + 2
            const pr e = st == 2 ? d : h;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (i) x[i] = p_addr(t_pair(s.X[i]), p_mul(e, k[i]));
                k[i] = p_addr(t_pair(s.K[i]), p_mul(e, b[i]));
            }
        } else {
            if (!ready) {  // the new state
                const pr d6 = p_mulr(d, {0x1.555556p-3f, -0x1.555556p-28f}), c = p_mulr(d, d6);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    if (i || TIME) {
                        const pr u = p_mulr(c, p_addr(q.a1[i], acc[i]));
                        s.X[i] = t_add(s.X[i], t_add(t_mul(dt, s.K[i]), {u.h, u.l, 0.0f}));
                    }
                    const pr g = p_mulr(d6, p_addr(p_addr(q.a1[i], b[i]), p_two(acc[i], 2.0f)));
                    s.K[i] = t_add(s.K[i], {g.h, g.l, 0.0f});
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (i) x[i] = t_pair(s.X[i]);
                k[i] = t_pair(s.K[i]);
            }
        }
        accel_pair(x[1], x[2], x[3], k[0], k[1], k[2], k[3], a, aa, b, q.m);
        if (st < 2)  // a2 + a3
#pragma unroll
            for (int i = 0; i < 4; i++) acc[i] = p_addr(acc[i], b[i]);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) q.a1[i] = b[i];
    q.r = t_radius(s.X[1], s.X[2], s.X[3], aa3, q.m.r, q.m.iq, q.m.ir);
}

// ---------------------------------------------------------------- step rule
// geodesic_step's rule (geodesics.py:249-252) on triples: dt = -(r - r_EH) /
// div; no step (false) below tol, beyond 1500 or at NaN, with the reason.
// d: r - r_EH to float.  For div > 0.
struct RuleTri {
    tri reh, ninv;  // horizon radius, -1/div
    pr tol;
};
MK_HD RuleTri rule_tri(double a, double div, double tol) {
    RuleTri o;
    o.reh = t_from(radius_eh(a));
    o.ninv = t_from(-1.0 / div);
    o.tol = p_near(tol);
    return o;
}
MK_HD bool rule_dt(tri r, const RuleTri &R, tri &dt, float &d_out, int &why) {
    const tri d = t_add(r, t_neg(R.reh));
    const float s = d.h < 0.0f ? -1.0f : 1.0f;
    const tri ad = {s * d.h, s * d.m, 0.0f};
    d_out = d.h;
    why = MK_RAY_ACTIVE;
    if (d.h != d.h) why = MK_RAY_NAN;
    else if (t_less(ad, {R.tol.h, R.tol.l, 0.0f})) why = MK_RAY_CAPTURED;
    else if (t_less({1500.0f, 0.0f, 0.0f}, ad)) why = MK_RAY_ESCAPED;
    dt = t_add(t_mul(d, R.ninv), {0.0f, 0.0f, 0.0f});
    return why == MK_RAY_ACTIVE;
}

}  // namespace mk

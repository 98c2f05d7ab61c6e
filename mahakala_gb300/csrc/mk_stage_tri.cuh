// mk_stage_tri.cuh -- the stage kernels' electron temperature and synchrotron
// coefficients on the FP32 pipe, in triples (mk_tri.cuh).
//
// In binary64 these kernels were bound by the FP64 pipe at 5 % of the HBM
// rate: a coefficient pair is ~130 FP64-pipe instructions of 64-76 cycles a
// warp.  In triples (72 bits, products and sums to ~2^-64) it is ~1 k FP32
// instructions and the sine; results are within an ulp of the formulas'
// values, nearer than the binary64 evaluation's own roundings leave them.
// Inputs outside a range where every word stays a normal float take the
// binary64 code.
#pragma once

#include "mk_fluid.cuh"
#include "mk_tri.cuh"

namespace mk {

// 2^(-j/32), three words each
__device__ const float EXP32[32][3] = {
    {0x1.0000000000000p+0f, 0x0.0p+0f, 0x0.0p+0f}, {0x1.f507660000000p-1f, -0x1.246eb00000000p-27f, 0x1.9d3e120000000p-55f},
    {0x1.ea4afa0000000p-1f, 0x1.52486c0000000p-28f, 0x1.858f740000000p-53f}, {0x1.dfc9740000000p-1f, -0x1.908c940000000p-26f, -0x1.4697360000000p-53f},
    {0x1.d5818e0000000p-1f, -0x1.822dbc0000000p-28f, -0x1.b44bf40000000p-54f}, {0x1.cb720e0000000p-1f, -0x1.8837cc0000000p-28f, 0x1.1503cc0000000p-53f},
    {0x1.c199be0000000p-1f, -0x1.3d56b20000000p-28f, 0x1.1106580000000p-56f}, {0x1.b7f7700000000p-1f, -0x1.a094380000000p-26f, 0x1.baa9ec0000000p-51f},
    {0x1.ae89fa0000000p-1f, -0x1.a94b140000000p-27f, -0x1.50bc660000000p-52f}, {0x1.a5503c0000000p-1f, -0x1.b83b540000000p-26f, -0x1.ba5ede0000000p-52f},
    {0x1.9c49180000000p-1f, 0x1.51f8480000000p-28f, 0x1.c7c46c0000000p-57f}, {0x1.93737c0000000p-1f, -0x1.e647440000000p-26f, 0x1.3d14080000000p-51f},
    {0x1.8ace540000000p-1f, 0x1.15506e0000000p-28f, -0x1.48b0760000000p-54f}, {0x1.82589a0000000p-1f, -0x1.accc7c0000000p-27f, 0x1.4567c40000000p-52f},
    {0x1.7a11480000000p-1f, -0x1.829fd00000000p-26f, 0x1.b5f5440000000p-51f}, {0x1.71f75e0000000p-1f, 0x1.1d8bee0000000p-26f, 0x1.ee91b80000000p-52f},
    {0x1.6a09e60000000p-1f, 0x1.9fcef40000000p-27f, -0x1.b7ba680000000p-52f}, {0x1.6247ec0000000p-1f, -0x1.f8b5500000000p-26f, 0x1.2c7c3e0000000p-51f},
    {0x1.5ab07e0000000p-1f, -0x1.5bd5ec0000000p-28f, 0x1.58c9300000000p-53f}, {0x1.5342b60000000p-1f, -0x1.2c56100000000p-26f, 0x1.df0a840000000p-53f},
    {0x1.4bfdae0000000p-1f, -0x1.593abc0000000p-26f, 0x1.c750e60000000p-51f}, {0x1.44e0860000000p-1f, 0x1.8624b40000000p-31f, 0x1.89b7a00000000p-60f},
    {0x1.3dea640000000p-1f, 0x1.8246840000000p-26f, 0x1.1ada0a0000000p-52f}, {0x1.371a740000000p-1f, -0x1.18aac60000000p-26f, -0x1.563aea0000000p-51f},
    {0x1.306fe00000000p-1f, 0x1.4636e20000000p-26f, 0x1.4b7a360000000p-51f}, {0x1.29e9e00000000p-1f, -0x1.5c04240000000p-26f, 0x1.2c25d20000000p-53f},
    {0x1.2387a60000000p-1f, 0x1.ceac480000000p-26f, -0x1.e64f820000000p-51f}, {0x1.1d48740000000p-1f, -0x1.d2e8ca0000000p-26f, -0x1.61fe920000000p-51f},
    {0x1.172b840000000p-1f, -0x1.c157420000000p-28f, -0x1.2320840000000p-53f}, {0x1.11301e0000000p-1f, -0x1.fdb4960000000p-26f, 0x1.49d77e0000000p-54f},
    {0x1.0b55860000000p-1f, 0x1.9f31220000000p-26f, -0x1.3ace8e0000000p-54f}, {0x1.059b0e0000000p-1f, -0x1.9d4f520000000p-26f, 0x1.0eb9f20000000p-51f}};

// exp(-x) for 0 <= x < 750 as m 2^-e: x = (32 e + j) ln2/32 - r, the table's
// 2^(-j/32) and the series of exp(r), |r| < 0.011, each term in as many words
// as its size calls for
__device__ __forceinline__ tri t_exp_neg(tri x, int &e) {
    const float n = rintf(x.h * 46.166241308446828f);
    const float c1 = 0x1.62e43p-6f, c2 = -0x1.05c61p-34f, c3 = -0x1.950d88p-59f;
    const float p = f_mul(n, c1), pe = fmaf(n, c1, -p), q = f_mul(n, c2), qe = fmaf(n, c3, fmaf(n, c2, -q));
    const tri r = t_add(t_add({p, pe, 0.0f}, {q, qe, 0.0f}), t_neg(x));
    const pr r1 = {r.h, r.m}, r2 = p_mulr(r1, r1);
    const pr c6 = {0x1.555556p-3f, -0x1.555556p-28f}, c24 = {0x1.555556p-5f, -0x1.555556p-30f};
    const pr t3 = p_mul(p_mulr(r2, r1), c6);
    pr t4 = p_mul(p_mulr(r2, r2), c24);
    t4.l = f_add(t4.l, f_mul(f_mul(f_mul(r2.h, r2.h), r.h), fmaf(r.h, 1.0f / 720.0f, 1.0f / 120.0f)));
    const pr s = p_add(p_add(p_two(r2, 0.5f), t3), t4);
    const tri E = t_add({1.0f, 0.0f, 0.0f}, t_add(r, t_norm({s.h, s.l, 0.0f})));
    const int k = (int)n;
    const float *T = EXP32[k & 31];
    e = k >> 5;
    return t_mulr({__ldg(T), __ldg(T + 1), __ldg(T + 2)}, E);
}

// cos and sin of j pi/64, three words each
__device__ const float COSSIN64[33][6] = {
    {0x1.0000000000000p+0f, 0x0.0p+0f, 0x0.0p+0f, 0x0.0p+0f, 0x0.0p+0f, 0x0.0p+0f},
    {0x1.ff621e0000000p-1f, 0x1.bcb6be0000000p-28f, 0x1.e3a8440000000p-53f, 0x1.91f6600000000p-5f, -0x1.de44fe0000000p-30f, 0x1.f376a20000000p-56f},
    {0x1.fd88da0000000p-1f, 0x1.e892920000000p-28f, 0x1.9e08280000000p-53f, 0x1.917a6c0000000p-4f, -0x1.eb25ea0000000p-31f, -0x1.e2718e0000000p-60f},
    {0x1.fa75580000000p-1f, -0x1.eeb5d20000000p-30f, -0x1.7a0a8c0000000p-55f, 0x1.2c81060000000p-3f, 0x1.d1cc280000000p-28f, -0x1.7768000000000p-53f},
    {0x1.f6297c0000000p-1f, 0x1.feeb960000000p-26f, 0x1.5621720000000p-56f, 0x1.8f8b840000000p-3f, -0x1.cb2cfa0000000p-30f, -0x1.49b4660000000p-55f},
    {0x1.f0a7f00000000p-1f, -0x1.1b73ca0000000p-27f, -0x1.ab4e140000000p-54f, 0x1.f19f980000000p-3f, -0x1.37a83a0000000p-29f, 0x1.57a4220000000p-54f},
    {0x1.e9f4160000000p-1f, -0x1.273a440000000p-26f, -0x1.689f4e0000000p-51f, 0x1.2940620000000p-2f, 0x1.dab3e00000000p-27f, 0x1.6a2d720000000p-52f},
    {0x1.e212100000000p-1f, 0x1.3da1ba0000000p-27f, -0x1.a0298e0000000p-52f, 0x1.58f9a80000000p-2f, -0x1.4a9c040000000p-27f, -0x1.80f7ee0000000p-53f},
    {0x1.d906bc0000000p-1f, 0x1.e651a80000000p-26f, 0x1.8a2bf40000000p-51f, 0x1.87de2a0000000p-2f, 0x1.abaa580000000p-28f, 0x1.68d3120000000p-53f},
    {0x1.ced7b00000000p-1f, -0x1.7867120000000p-26f, 0x1.7861260000000p-52f, 0x1.b5d1000000000p-2f, 0x1.3c2b980000000p-27f, 0x1.5b362c0000000p-57f},
    {0x1.c38b300000000p-1f, -0x1.cfe84a0000000p-26f, 0x1.a47d3a0000000p-54f, 0x1.e2b5d40000000p-2f, -0x1.fe42720000000p-28f, 0x1.8f06c40000000p-53f},
    {0x1.b728340000000p-1f, 0x1.465b900000000p-27f, -0x1.378d3e0000000p-52f, 0x1.07387a0000000p-1f, -0x1.b740040000000p-27f, -0x1.34b4020000000p-52f},
    {0x1.a9b6620000000p-1f, 0x1.21d4340000000p-26f, 0x1.819f640000000p-52f, 0x1.1c73b40000000p-1f, -0x1.9465ce0000000p-27f, 0x1.b25dd20000000p-55f},
    {0x1.9b3e040000000p-1f, 0x1.fce1d00000000p-27f, 0x1.6788ec0000000p-54f, 0x1.30ff800000000p-1f, -0x1.8f47e60000000p-28f, 0x1.c206740000000p-54f},
    {0x1.8bc8060000000p-1f, 0x1.62a2e80000000p-26f, 0x1.69d0f60000000p-54f, 0x1.44cf320000000p-1f, 0x1.4247760000000p-27f, -0x1.e7f8960000000p-53f},
    {0x1.7b5df20000000p-1f, 0x1.3557d80000000p-28f, -0x1.21ea700000000p-53f, 0x1.57d6940000000p-1f, -0x1.6e626c0000000p-26f, -0x1.75720a0000000p-55f},
    {0x1.6a09e60000000p-1f, 0x1.9fcef40000000p-27f, -0x1.b7ba680000000p-52f, 0x1.6a09e60000000p-1f, 0x1.9fcef40000000p-27f, -0x1.b7ba680000000p-52f},
    {0x1.57d6940000000p-1f, -0x1.6e626c0000000p-26f, -0x1.75720a0000000p-55f, 0x1.7b5df20000000p-1f, 0x1.3557d80000000p-28f, -0x1.21ea700000000p-53f},
    {0x1.44cf320000000p-1f, 0x1.4247760000000p-27f, -0x1.e7f8960000000p-53f, 0x1.8bc8060000000p-1f, 0x1.62a2e80000000p-26f, 0x1.69d0f60000000p-54f},
    {0x1.30ff800000000p-1f, -0x1.8f47e60000000p-28f, 0x1.c206740000000p-54f, 0x1.9b3e040000000p-1f, 0x1.fce1d00000000p-27f, 0x1.6788ec0000000p-54f},
    {0x1.1c73b40000000p-1f, -0x1.9465ce0000000p-27f, 0x1.b25dd20000000p-55f, 0x1.a9b6620000000p-1f, 0x1.21d4340000000p-26f, 0x1.819f640000000p-52f},
    {0x1.07387a0000000p-1f, -0x1.b740040000000p-27f, -0x1.34b4020000000p-52f, 0x1.b728340000000p-1f, 0x1.465b900000000p-27f, -0x1.378d3e0000000p-52f},
    {0x1.e2b5d40000000p-2f, -0x1.fe42720000000p-28f, 0x1.8f06c40000000p-53f, 0x1.c38b300000000p-1f, -0x1.cfe84a0000000p-26f, 0x1.a47d3a0000000p-54f},
    {0x1.b5d1000000000p-2f, 0x1.3c2b980000000p-27f, 0x1.5b362c0000000p-57f, 0x1.ced7b00000000p-1f, -0x1.7867120000000p-26f, 0x1.7861260000000p-52f},
    {0x1.87de2a0000000p-2f, 0x1.abaa580000000p-28f, 0x1.68d3120000000p-53f, 0x1.d906bc0000000p-1f, 0x1.e651a80000000p-26f, 0x1.8a2bf40000000p-51f},
    {0x1.58f9a80000000p-2f, -0x1.4a9c040000000p-27f, -0x1.80f7ee0000000p-53f, 0x1.e212100000000p-1f, 0x1.3da1ba0000000p-27f, -0x1.a0298e0000000p-52f},
    {0x1.2940620000000p-2f, 0x1.dab3e00000000p-27f, 0x1.6a2d720000000p-52f, 0x1.e9f4160000000p-1f, -0x1.273a440000000p-26f, -0x1.689f4e0000000p-51f},
    {0x1.f19f980000000p-3f, -0x1.37a83a0000000p-29f, 0x1.57a4220000000p-54f, 0x1.f0a7f00000000p-1f, -0x1.1b73ca0000000p-27f, -0x1.ab4e140000000p-54f},
    {0x1.8f8b840000000p-3f, -0x1.cb2cfa0000000p-30f, -0x1.49b4660000000p-55f, 0x1.f6297c0000000p-1f, 0x1.feeb960000000p-26f, 0x1.5621720000000p-56f},
    {0x1.2c81060000000p-3f, 0x1.d1cc280000000p-28f, -0x1.7768000000000p-53f, 0x1.fa75580000000p-1f, -0x1.eeb5d20000000p-30f, -0x1.7a0a8c0000000p-55f},
    {0x1.917a6c0000000p-4f, -0x1.eb25ea0000000p-31f, -0x1.e2718e0000000p-60f, 0x1.fd88da0000000p-1f, 0x1.e892920000000p-28f, 0x1.9e08280000000p-53f},
    {0x1.91f6600000000p-5f, -0x1.de44fe0000000p-30f, 0x1.f376a20000000p-56f, 0x1.ff621e0000000p-1f, 0x1.bcb6be0000000p-28f, 0x1.e3a8440000000p-53f},
    {0x0.0p+0f, 0x0.0p+0f, 0x0.0p+0f, 0x1.0000000000000p+0f, 0x0.0p+0f, 0x0.0p+0f}};

// acos(c), |c| <= 1: the angle t0 = j pi/64 nearest to it, sin(acos(c) - t0) =
// s cos t0 - c sin t0 with s = sqrt((1 - c)(1 + c)), and the arcsine's series,
// |x| < 0.025.  In binary64 the library's acos was a third of the sampling
// kernel's FP64-pipe instructions.
__device__ __forceinline__ tri t_acos(tri c) {
    const tri one = {1.0f, 0.0f, 0.0f};
    const tri s2 = t_mulr(t_sub(one, c), t_add(one, c));
    const tri s = s2.h > 0.0f ? t_mulr(s2, t_rsqrt(s2)) : tri{0.0f, 0.0f, 0.0f};
    const int j = min(64, max(0, (int)rintf(acosf(fminf(fmaxf(c.h, -1.0f), 1.0f)) * 20.371832f)));
    const float *T = COSSIN64[j <= 32 ? j : 64 - j];
    const float g = j <= 32 ? 1.0f : -1.0f;  // cos(pi - t) = -cos t
    const tri c0 = {g * __ldg(T), g * __ldg(T + 1), g * __ldg(T + 2)}, s0 = {__ldg(T + 3), __ldg(T + 4), __ldg(T + 5)};
    const tri x = t_sub(t_mul(s, c0), t_mul(c, s0));
    // x + x^3/6 + 3 x^5/40 + 15 x^7/336 + 105 x^9/3456
    const pr p = {x.h, x.m}, p2 = p_mulr(p, p), p3 = p_mulr(p2, p);
    pr q = p_mul(p_mulr(p3, p2), {0x1.333334p-4f, -0x1.99999ap-29f});
    const float x2 = p2.h;
    q.l = fmaf(f_mul(f_mul(f_mul(p3.h, x2), x2), fmaf(x2, 105.0f / 3456.0f, 15.0f / 336.0f)), 1.0f, q.l);
    const pr r = p_add(p_mul(p3, {0x1.555556p-3f, -0x1.555556p-28f}), q);
    const tri t0 = t_mulr({(float)j, 0.0f, 0.0f}, {0x1.921fb6p-5f, -0x1.777a5cp-30f, -0x1.ee59dap-55f});
    return t_add(t0, t_add(x, t_norm({r.h, r.l, 0.0f})));
}

// Tests and scalings by the bits: a comparison costs the FP64 pipe as much as
// an addition.  Positive doubles order as integers; NaN lies above infinity.
__device__ __forceinline__ bool within(double v, double lo, double hi) {
    const long long b = __double_as_longlong(v);
    return b >= __double_as_longlong(lo) && b <= __double_as_longlong(hi);
}
__device__ __forceinline__ bool is_zero(double v) { return (__double_as_longlong(v) << 1) == 0; }
// v 2^e, v a positive normal number and the result too, or v = 0
__device__ __forceinline__ double scaled(double v, int e) {
    return is_zero(v) ? 0.0 : __hiloint2double(__double2hiint(v) + (int)((unsigned)e << 20), __double2loint(v));
}

// v 2^e for 2^-140 <= v < 2^128, or v = 0: faint to the end of the doubles'
// range, where 2^e is taken in two normal factors with one rounding
__device__ __forceinline__ double pow2_scaled(double v, int e) {
    if (e < -850)
        return v * __hiloint2double((1023 + e / 2) << 20, 0) * __hiloint2double((1023 + (e - e / 2)) << 20, 0);
    return scaled(v, e);
}

// doubles in order as integers (-0 = 0)
__device__ __forceinline__ long long ordered(double v) {
    const long long b = __double_as_longlong(v);
    return (b << 1) == 0 ? 0 : b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}

// sin(x) for 0 <= x <= 100: x = n pi/64 + r, the table's sine and cosine and
// the series of r, |r| < 0.025
__device__ __forceinline__ tri t_sin(tri x) {
    const float n = rintf(x.h * 20.371832f);
    const float c1 = 0x1.921fb6p-5f, c2 = -0x1.777a5cp-30f, c3 = -0x1.ee59dap-55f;
    const float p = f_mul(n, c1), pe = fmaf(n, c1, -p), q = f_mul(n, c2), qe = fmaf(n, c3, fmaf(n, c2, -q));
    const tri r = t_sub(x, t_add({p, pe, 0.0f}, {q, qe, 0.0f}));
    const int k = (int)n & 127, m = k & 63, i = m <= 32 ? m : 64 - m;  // sin and cos of k pi/64 from the first octant pair
    const float *T = COSSIN64[i];
    const float g = k < 64 ? 1.0f : -1.0f, gc = m <= 32 ? g : -g;
    const tri s0 = {g * __ldg(T + 3), g * __ldg(T + 4), g * __ldg(T + 5)};
    const tri c0 = {gc * __ldg(T), gc * __ldg(T + 1), gc * __ldg(T + 2)};
    const pr r1 = {r.h, r.m}, r2 = p_mulr(r1, r1), r3 = p_mulr(r2, r1), r4 = p_mulr(r2, r2);
    const float z = r2.h;
    // sin r - r and cos r - 1
    pr a = p_mul(r3, {-0x1.555556p-3f, 0x1.555556p-28f});
    const pr a5 = p_mul(p_mulr(r4, r1), {0x1.111112p-7f, -0x1.dddddep-32f});
    a = p_add(a, {a5.h, fmaf(f_mul(f_mul(r4.h, r3.h), 1.0f), fmaf(z, 1.0f / 362880.0f, -1.0f / 5040.0f), a5.l)});
    pr b = p_two(r2, -0.5f);
    const pr b4 = p_mul(r4, {0x1.555556p-5f, -0x1.555556p-30f});
    b = p_add(b, {b4.h, fmaf(f_mul(r4.h, z), fmaf(z, 1.0f / 40320.0f, -1.0f / 720.0f), b4.l)});
    const tri sr = t_add(r, t_norm({a.h, a.l, 0.0f})), cr = t_norm({b.h, b.l, 0.0f});
    return t_add(t_add(s0, t_mul(s0, cr)), t_mul(c0, sr));
}

// synchrotron_coefficients (transfer.py:30-86): with Z = nu_s / nu and Y =
// Z^(1/3) the emissivity is K Ne nu (1 + 2^(11/12) Y)^2 exp(-1/Y) / Theta_e^2
// (see mk_sample_pair.cuh).  Frequencies are in units of 2^37 Hz and K carries
// a factor 2^60, so that no word of a constant leaves the float range.
struct SynchroTri {
    tri knus, kem, kbx, kab, resc;
    int ok;
};

inline SynchroTri synchro_tri_consts(bool invariant, double rescale_nu) {
    SynchroTri c;
    const double U = 137438953472.0;  // 2^37
    c.knus = t_from(TWO_NINTHS * EE / TWO_PI_ME_CL / U);
    c.kem = t_from(0.5 * SQRT2 * PI * EE2 / THREE_CL * U * 0x1p60);
    c.kbx = t_from(HPL / ME_CL_CL * U);
    c.kab = t_from(CL2 / (TWO_HPL * U * U * U));
    c.resc = t_from(rescale_nu * U);
    c.ok = !invariant || (rescale_nu * U >= 1e-6 && rescale_nu * U <= 1e12);
    return c;
}

// false: outside the range, nothing computed
__device__ __forceinline__ bool synchro_tri(const SynchroTri &c, double Ne, double Th, double B, double pitch,
                                            double nu, bool invariant, double &em_out, double &ab_out) {
    em_out = ab_out = 0.0;
    // no emission: Theta_e below 0.3 or NaN, no electrons, no field
    if (!within(Th, 0.3, __longlong_as_double(0x7ff0000000000000LL)) || is_zero(Ne) || is_zero(B)) return true;
    // the density's exponent goes to the result (it falls by tens of decades
    // along a torus' poles)
    const unsigned hn = (unsigned)__double2hiint(Ne);
    const int en = (int)(hn >> 20) - 1023;  // of a positive normal number
    if (!(c.ok && en > -400 && en < 400 && within(Th, 0.3, 1e6) && within(B, 1e-20, 1e10) && within(nu, 1e3, 1e16) &&
          within(pitch, 0.0, 100.0)))
        return false;
    const tri ne = t_from(__hiloint2double((int)(hn - ((unsigned)en << 20)), __double2loint(Ne)));
    const tri th = t_from(Th), v = t_from(scaled(nu, -37)), rv = t_rcp(v), rth = t_rcp(th);
    const tri nus = t_mulr(t_mulr(c.knus, t_from(B)), t_mulr(t_mulr(th, th), t_sin(t_from(pitch))));
    const tri Z = t_mulr(nus, rv);
    if (!(Z.h >= 1e-12f)) return true;  // X > 1e12, or a sine that is not positive (X < 0: not a number)
    const pr y0 = p_rcbrt({Z.h, Z.m});
    const tri y = {y0.h, y0.l, 0.0f}, p3 = t_mul(t_mulr(t_mulr(y, y), y), Z);
    const float d = f_sub(f_sub(f_sub(1.0f, p3.h), p3.m), p3.l);
    const tri x3 = t_norm({y0.h, y0.l, f_mul(f_mul(y0.h, d), 0.333333343f)});  // X^(1/3)
    if (!(x3.h < 745.13f)) return true;  // exp(-x3) = 0
    const tri Y = t_mulr(t_mulr(x3, x3), Z);
    const tri t = t_add({1.0f, 0.0f, 0.0f}, t_mulr({0x1.e3437ep+0f, 0x1.c404dp-26f, 0x1.dbca56p-51f}, Y));
    int e;
    const tri E = t_exp_neg(x3, e);
    tri em = t_mulr(t_mulr(t_mulr(c.kem, ne), t_mulr(rth, rth)), t_mulr(t_mulr(t, t), E));  // em_raw / nu
    const tri bx = t_mulr(t_mulr(c.kbx, v), rth);
    tri den;
    if (bx.h < 2.e-3f) {  // bx (1 + bx/2 (1 + bx/3 (1 + bx/4))), as the reference cuts it
        const pr b1 = {bx.h, bx.m}, b2 = p_mulr(b1, b1);
        pr s = p_add(p_two(b2, 0.5f), p_mul(p_mulr(b2, b1), {0x1.555556p-3f, -0x1.555556p-28f}));
        s.l = f_add(s.l, f_mul(f_mul(b2.h, b2.h), 1.0f / 24.0f));
        den = t_add(bx, t_norm({s.h, s.l, 0.0f}));
    } else {
        den = t_from(exp(t_to(bx)) - 1.0);
    }
    // alpha = em_raw / B_nu, B_nu = 2 h nu^3 / (c^2 den)
    tri ab = t_mulr(t_mulr(em, t_mulr(rv, rv)), t_mulr(den, c.kab));
    int ex = en - 60 - e;  // the result's power of two
    if (invariant) {
        // 1/w^2 by w's significand: at rescale_nu = 1 it is 1e-23 at 230 GHz,
        // whose low words no float holds
        const tri w = t_mulr(v, c.resc);
        const int ew = ((int)(__float_as_uint(w.h) >> 23) & 255) - 127;
        const float sw = __uint_as_float((unsigned)(127 - ew) << 23);
        const tri rw = t_rcp({sw * w.h, sw * w.m, sw * w.l});
        em = t_mulr(t_mulr(em, v), t_mulr(rw, rw));
        em_out = pow2_scaled(t_to(em), ex - 2 * ew);
        ab = t_mulr(ab, w);
    } else {
        em_out = pow2_scaled(t_to(t_mulr(em, v)), ex);
    }
    ab_out = pow2_scaled(t_to(ab), ex);
    return true;
}

// rlow_rhigh_model (electrons.py:32-50): Theta_e = C u (1 + beta^2) / (dens
// (g_i (1 + beta^2) + g_e (R_high beta^2 + R_low))), C = (MP/ME) g_e g_i
struct RlowTri {
    tri c, ge, gi, rl, rh;
    int ok;
};

inline RlowTri rlow_tri_consts(double r_low, double r_high, double gem1, double gim1) {
    RlowTri k;
    k.c = t_from(CL2 * MP / ME_CL_CL * gem1 * gim1);
    k.ge = t_from(gem1);
    k.gi = t_from(gim1);
    k.rl = t_from(r_low);
    k.rh = t_from(r_high);
    auto in = [](double v) { return v >= 1e-4 && v <= 1e6; };
    k.ok = in(gem1) && in(gim1) && in(r_low) && in(r_high);
    return k;
}

__device__ __forceinline__ bool rlow_tri(const RlowTri &k, double dens, double u, double beta, double &out) {
    if (is_zero(dens) && is_zero(u)) {  // outside the snapshot: 0 / 0
        out = nan("");
        return true;
    }
    const unsigned hd = (unsigned)__double2hiint(dens), hu = (unsigned)__double2hiint(u);
    const int ed = (int)(hd >> 20) - 1023, eu = (int)(hu >> 20) - 1023;  // of positive normal numbers
    if (!(k.ok && ed > -400 && ed < 400 && eu > -400 && eu < 400 &&
          ((unsigned)__double2hiint(beta) & 0x7fffffffu) <= 0x41cdcd65u))  // |beta| <= 1e9
        return false;
    // significands in [1, 2); the exponents go to the result
    const tri d = t_from(__hiloint2double((int)(hd - ((unsigned)ed << 20)), __double2loint(dens)));
    const tri s = t_from(__hiloint2double((int)(hu - ((unsigned)eu << 20)), __double2loint(u)));
    // 1 and beta^2 over beta's power of two squared where that is above one
    // (the quotient is the same): their products with gammas and R_high, and
    // the reciprocal, would leave the range in which a triple keeps its words
    const unsigned hb = (unsigned)__double2hiint(beta);
    const int eb = max(0, (int)((hb >> 20) & 0x7ffu) - 1023);
    const float sb = __uint_as_float((unsigned)(127 - eb) << 23), o2 = sb * sb;
    const tri b = t_from(__hiloint2double((int)(hb - ((unsigned)eb << 20)), __double2loint(beta)));
    const tri b2 = t_mulr(b, b), ob = t_add({o2, 0.0f, 0.0f}, b2);
    const tri D = t_add(t_mulr(k.gi, ob), t_mulr(k.ge, t_add(t_mulr(k.rh, b2), {k.rl.h * o2, k.rl.m * o2, k.rl.l * o2})));
    const tri th = t_mulr(t_mulr(k.c, s), t_mulr(ob, t_rcp(t_mulr(d, D))));
    if (k.rh.h > 0.0f && !(th.h > 1e-30f)) return false;
    out = scaled(t_to(th), eu - ed);
    return true;
}

// get_fluid_scalars_from_geodesics (athenak.py:639-812) at one point: the cell
// and the frame in triples, the interpolation as eight binary64 weights times
// cells (64 fused multiply-adds, the cells moved to binary64 by bit
// operations), the angle by t_acos.  In binary64 the point was ~500 FP64-pipe
// instructions, also outside the snapshot, where only k.u = -k^t / sqrt(1 + f)
// is needed.  false: the point is left to the binary64 code (not finite or
// beyond 1e6, a wavevector beyond 1e12, next to the ring, or at a face two
// blocks do not share to the bit; velocities beyond 1e6).
struct FluidTri {
    tri a, aa;                // spin and its square
    float lo[3], inv_w[3];    // the block grid
    double fallback;          // the pitch angle where there is no field
};
inline FluidTri fluid_tri_consts(const mk_snapshot_view &sv, double a, double cos_fallback) {
    FluidTri c;
    c.fallback = acos(fabs(cos_fallback) > 1.0 ? copysign(1.0, cos_fallback) : cos_fallback);
    c.a = t_from(a);
    c.aa = t_from(a * a);
    for (int i = 0; i < 3; i++) {
        c.lo[i] = (float)sv.lo[i];
        c.inv_w[i] = (float)(1.0 / sv.width[i]);
    }
    return c;
}

__device__ __forceinline__ bool fluid_point_tri(const mk_snapshot_view &sv, const FluidTri &cst, const double s[8],
                                                double out[5]) {
    const tri a = cst.a, aa = cst.aa;
    tri x[3], k[4];
#pragma unroll
    for (int i = 0; i < 3; i++) x[i] = t_from(s[1 + i]);
#pragma unroll
    for (int i = 0; i < 4; i++) k[i] = t_from(s[4 + i]);
    const float xm = fmaxf(fmaxf(fabsf(x[0].h), fabsf(x[1].h)), fabsf(x[2].h));
    const float ks = (fabsf(k[0].h) + fabsf(k[1].h)) + (fabsf(k[2].h) + fabsf(k[3].h));  // NaN if any is
    if (!(xm <= 1e6f && ks >= 1e-6f && ks <= 1e12f && x[0].h == x[0].h && x[1].h == x[1].h && x[2].h == x[2].h))
        return false;
    // the block and cell
    int c[3], idx[3], near[3], mb = -1;
    tri del[3];
    bool inside = true, beside = false;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const float lo = cst.lo[i], u = (x[i].h - lo) * cst.inv_w[i];
        const float tol = 1e-5f * ((fabsf(lo) + xm) * cst.inv_w[i] + 1.0f);  // of u
        if (u < -tol || u > (float)sv.nb[i] + tol) inside = false;
        if (fabsf(u - rintf(u)) <= tol) beside = true;
        c[i] = max(0, min((int)u, sv.nb[i] - 1));
    }
    if (inside) {
        const float n = (float)sv.n;
        for (int it = 0;; ++it) {
            mb = table_at(sv, c);
            if (mb < 0) {
                // a place without a block: beside a face of the table the
                // point may lie across it, in one that is there
                if (it == 0 && beside) return false;
                break;
            }
            const double *g = sv.geom + 6 * (int64_t)mb;
            bool moved = false;
#pragma unroll
            for (int i = 0; i < 3; i++) {
                const tri left = t_from(__ldg(g + i)), d = t_near(__ldg(g + 3 + i));
                const tri v = t_sub(x[i], left), id = t_rcp(d);
                const pr t = p_mulr({v.h, v.m}, {id.h, id.m});
                // faces at t = -1/2 and n - 1/2; next to one, the block's own
                // face decides (left < x <= right)
                float e0 = f_add(t.h, 0.5f) + t.l, e1 = f_sub(t.h, n - 0.5f) + t.l;
                const bool n0 = !(fabsf(e0) > 1e-6f), n1 = !(fabsf(e1) > 1e-6f);
                if (n0 || n1) {
                    const double *fc = sv.faces + 6 * (int64_t)mb + 2 * i;
                    if (n0) e0 = ordered(s[1 + i]) <= ordered(__ldg(fc)) ? -1.0f : 1.0f;
                    if (n1) e1 = ordered(s[1 + i]) > ordered(__ldg(fc + 1)) ? 1.0f : -1.0f;
                }
                near[i] = n0 ? -1 : (n1 ? 1 : 0);
                if (e0 < 0.0f) { --c[i]; moved = true; }
                else if (e1 > 0.0f) { ++c[i]; moved = true; }
                float fl = floorf(t.h);
                tri u = t_sub(v, t_mul({fl, 0.0f, 0.0f}, d));
                // the quotient may have rounded across a cell's edge: the rest
                // lies in [0, d), and is 0 at a cell centre
                if (u.h < 0.0f) { fl -= 1.0f; u = t_add(u, d); }
                else if (!t_less(u, d)) { fl += 1.0f; u = t_sub(u, d); }
                fl = fminf(fmaxf(fl, -1.0f), n - 1.0f);
                idx[i] = (int)fl + 1;
                del[i] = t_mulr(u, id);
            }
            if (!moved) {
                // two blocks can both hold a point next to a face they do not
                // share to the bit: the binary64 code takes the later one
#pragma unroll
                for (int i = 0; i < 3; i++)
                    if (near[i]) {
                        int o[3] = {c[0], c[1], c[2]};
                        o[i] += near[i];
                        const int nb = table_at(sv, o);
                        const int mine = 2 * i + (near[i] > 0), theirs = 2 * i + (near[i] < 0);
                        if (nb >= 0 && ordered(__ldg(sv.faces + 6 * (int64_t)mb + mine)) !=
                                           ordered(__ldg(sv.faces + 6 * (int64_t)nb + theirs)))
                            return false;
                    }
                break;
            }
            if (it == 3) return false;
        }
    }
    // metric data
    const tri zz = t_norm(t_sqr(x[2]));
    tri kk = t_sub(t_add(t_add(t_sqr(x[0]), t_sqr(x[1])), zz), aa);
    kk = {0.5f * kk.h, 0.5f * kk.m, 0.5f * kk.l};
    const tri Q = t_add(t_sqr(kk), t_mul(aa, zz));
    if (!(Q.h >= 1e-12f)) return false;
    const tri iq = t_rsqrt(Q), rr = t_add(t_mul(Q, iq), kk);
    if (!(rr.h > 1e-4f * fabsf(kk.h))) return false;
    const tri ir = t_rsqrt(rr), r = t_mulr(rr, ir), f = t_mulr(r, iq);
    const tri one = {1.0f, 0.0f, 0.0f};
    const tri alpha = t_rsqrt(t_add(one, f));
    if (mb < 0) {  // primitives zero: u = (1/alpha, -alpha f l), b = 0
        out[0] = out[1] = out[4] = 0.0;
        out[2] = cst.fallback;
        out[3] = -t_to(t_mulr(k[0], alpha));
        return true;
    }
    // blocks whose ghosts average finer cells are kept in binary64
    const int row = sv.blocks64 ? __ldg(sv.block64 + mb) : -1;
    double prim[8];
    {
        const int n2 = sv.n + 2;
        const int64_t sj = (int64_t)n2 * 8, sk = (int64_t)n2 * n2 * 8;
        const int64_t block = n2 * sk, cell = idx[2] * sk + idx[1] * sj + (int64_t)idx[0] * 8;
        // weights rounded to binary64 once
        const tri u0 = t_sub(one, del[0]), u1 = t_sub(one, del[1]), u2 = t_sub(one, del[2]);
        const tri zy[4] = {t_mulr(u2, u1), t_mulr(u2, del[1]), t_mulr(del[2], u1), t_mulr(del[2], del[1])};
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const double w = t_to(t_mul(zy[q >> 1], q & 1 ? del[0] : u0));
            const int64_t at = cell + (q >> 2) * sk + ((q >> 1) & 1) * sj + (q & 1) * 8;
            double v[8];
            if (row < 0) {
                const float4 lo = ldg4(sv.blocks + mb * block + at), hi = ldg4(sv.blocks + mb * block + at + 4);
                const float f[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                for (int i = 0; i < 8; i++) v[i] = d_from(f[i]);
            } else {
#pragma unroll
                for (int i = 0; i < 8; i++) v[i] = __ldg(sv.blocks64 + row * block + at + i);
            }
#pragma unroll
            for (int i = 0; i < 8; i++) prim[i] = q == 0 ? w * v[i] : fma(w, v[i], prim[i]);
        }
    }
    // cells that are not finite: which sums are infinite and which not a number
    // follows from the order of the binary64 code's
    unsigned top = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) top = max(top, (unsigned)__double2hiint(prim[i]) & 0x7fffffffu);
    if (top >= 0x7ff00000u) return false;
    // the field scaled to order one by a power of two: along the poles of a
    // torus it falls by tens of decades
    const unsigned hB = max(max((unsigned)__double2hiint(prim[5]) & 0x7fffffffu, (unsigned)__double2hiint(prim[6]) & 0x7fffffffu),
                            (unsigned)__double2hiint(prim[7]) & 0x7fffffffu);
    const bool noB = hB == 0u;
    const int eB = noB ? 0 : (int)(hB >> 20) - 1023;
    const double sB = __hiloint2double((1023 - eB) << 20, 0);
    tri U[3], B[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        U[i] = t_from(prim[1 + i]);
        B[i] = t_from(prim[5 + i] * sB);
    }
    const float Um = fmaxf(fmaxf(fabsf(U[0].h), fabsf(U[1].h)), fabsf(U[2].h));
    if (!(eB > -500 && eB < 500 && Um <= 1e6f)) return false;
    const tri ira = t_rcp(t_add(rr, aa));
    const tri l1 = t_mulr(t_add(t_mul(r, x[0]), t_mul(a, x[1])), ira);
    const tri l2 = t_mulr(t_sub(t_mul(r, x[1]), t_mul(a, x[0])), ira);
    const tri l3 = t_mulr(x[2], ir);
    // the frame, as in sample_pair
    const tri lU = t_dot(l1, U[0], l2, U[1], l3, U[2]), lB = t_dot(l1, B[0], l2, B[1], l3, B[2]);
    const tri lk = t_dot(l1, k[1], l2, k[2], l3, k[3]), lv = t_add(k[0], lk);
    const tri kU = t_dot(k[1], U[0], k[2], U[1], k[3], U[2]), kB = t_dot(k[1], B[0], k[2], B[1], k[3], B[2]);
    const tri UU = t_dot(U[0], U[0], U[1], U[1], U[2], U[2]), BB = t_dot(B[0], B[0], B[1], B[1], B[2], B[2]);
    const tri BU = t_dot(B[0], U[0], B[1], U[1], B[2], U[2]);
    const tri flU = t_mulr(f, lU), flB = t_mulr(f, lB);
    const tri G = t_add(t_add(UU, t_mul(flU, lU)), one), rG = t_rsqrt(G);
    const tri ga = t_mulr(t_mulr(G, rG), alpha), iut = t_mulr(alpha, rG);
    const tri Bu = t_add(BU, t_mul(flU, lB));
    const tri b2 = t_mulr(t_add(t_add(BB, t_mul(flB, lB)), t_sqr(Bu)), t_norm(t_sqr(iut)));
    const tri ku = t_sub(t_add(kU, t_mul(flU, lv)), t_mul(k[0], ga));
    out[0] = prim[0];
    out[1] = prim[4];
    out[3] = t_to(ku);
    out[2] = cst.fallback;
    out[4] = 0.0;
    if (b2.h > 0.0f) {
        const tri gaf = t_mulr(ga, f);
        const tri lb = t_add(Bu, t_mul(t_add(lB, t_mul(t_sub(lU, gaf), Bu)), iut));
        const tri kb3 = t_mulr(t_add(kB, t_mul(t_sub(kU, t_mul(gaf, lk)), Bu)), iut);
        const tri kb = t_add(t_sub(kb3, t_mul(k[0], Bu)), t_mul(t_mulr(f, lb), lv));
        const tri ib = t_rsqrt(b2);
        out[4] = t_to(t_mulr(b2, ib)) * __hiloint2double((1023 + eB) << 20, 0);
        if (ku.h == 0.0f) return false;
        const float sg = ku.h < 0.0f ? -1.0f : 1.0f;
        tri cp = t_mulr(t_mulr(kb, ib), t_rcp({ku.h * sg, ku.m * sg, ku.l * sg}));
        if (cp.h > 1.0f || (cp.h == 1.0f && cp.m > 0.0f)) cp = {1.0f, 0.0f, 0.0f};
        if (cp.h < -1.0f || (cp.h == -1.0f && cp.m < 0.0f)) cp = {-1.0f, 0.0f, 0.0f};
        out[2] = t_to(t_acos(cp));
    }
    return true;
}

}  // namespace mk

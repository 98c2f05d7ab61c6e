// mk_sample_pair.cuh -- the fused FP64 render's sampling and emission on the
// FP32 pipe, in float pairs (mk_tri.cuh).
//
// In binary64 a sample is ~510 FP64-pipe instructions (64-76 cycles of a warp
// each on GB300, conversions between float and double included): ~35 k
// cycles, eight times an RK4 step on pairs.  Here it is ~1.9 k FP32
// instructions to ~2^-47 of each quantity; the emission's exponential keeps
// its exponent apart, so faint pixels keep their digits, and the transfer
// sums stay binary64.  A sample's error (~1e-14, times x^(1/3) through the
// exponential) is as large as what the pairs' geodesic leaves in the image and
// below what binary64's leaves at the views that pair_request admits; it says
// which, and what was measured.
//
// Identities used (g = eta + f l l, l null): u_i = U_i + f (l.U) l_i, l_mu
// u^mu = gamma alpha + l.U, b^2 = (B.B + f (l.B)^2 + (B.u)^2) / (u^t)^2, so
// the frame needs eight dot products and no vector of its own; with Z =
// nu_s / nu and Y = Z^(1/3) = x^(-1/3) the synchrotron fit (transfer.py:30-86)
// is Ne const (1 + 2^(11/12) Y)^2 exp(-1/Y) / (2 Theta_e^2 nu), without roots.
#pragma once

#include "mk_fluid.cuh"
#include "mk_tri.cuh"

namespace mk {

// A request's constants, one column of shared memory each (registers hold the
// ray itself).
enum PairConst {
    PC_A = 0, PC_AA = 2, PC_AA_L = 4, PC_REH = 5, PC_NINV = 8, PC_TOL = 11, PC_BOX = 13, PC_INVW = 19,
    PC_GAM2 = 22, PC_RHIGH = 24, PC_RLOW = 26, PC_GEM1 = 28, PC_GIM1 = 30, PC_KTH = 32, PC_SIGMA = 34,
    PC_LUNIT = 36, PC_NU = 38,  // per frequency: emissivity, nu_s, bx and 1/B_nu factors, 8 floats
    PC_COUNT = PC_NU + 8 * MK_MAX_NU
};
constexpr int EXP_STEPS = 32;  // table of 2^(-j/32)

template <int STRIDE>
struct PairConsts {
    float *c;  // the request's column
    __device__ __forceinline__ pr p(int i) const { return {c[i * STRIDE], c[(i + 1) * STRIDE]}; }
    __device__ __forceinline__ tri t(int i) const { return {c[i * STRIDE], c[(i + 1) * STRIDE], c[(i + 2) * STRIDE]}; }
    __device__ __forceinline__ float f(int i) const { return c[i * STRIDE]; }
    __device__ __forceinline__ void set(int i, double v, int words) {
        const tri t = t_near(v);
        c[i * STRIDE] = t.h;
        c[(i + 1) * STRIDE] = t.m;
        if (words > 2) c[(i + 2) * STRIDE] = t.l;
    }
};

// the folded constants of the emission at one frequency
struct EmissionFold {
    double kem, knus, kbx, kib;
};
MK_HD EmissionFold emission_fold(const mk_request &R, double nu) {
    EmissionFold e;
    e.kem = (0.5 * SQRT2 * PI * EE2 / THREE_CL) * nu * R.Ne_unit;
    e.knus = (TWO_NINTHS * EE / TWO_PI_ME_CL) * R.B_unit / nu;
    e.kbx = HPL * nu / ME_CL_CL;
    e.kib = CL2 / (TWO_HPL * nu * nu * nu);
    return e;
}

// Requests that the pairs render no less exactly than binary64, and whose
// constants leave every pair's low word inside the float range.  Any other
// request is rendered by the binary64 kernel.
//
// Pairs leave ~6e-14 of a pixel (the geodesic half of it, the sampler the
// other: 48 bits of x^(1/3) in the emission's exponential).  Binary64's state
// rounds by 2^-54 of each coordinate a step, of which the part across the ray
// counts: little for a camera on an axis or near by.  Errors against a
// 64-bit-significand evaluation (48^2 and 40^2 rays, 20 GHz, spins 0 to
// 0.998), pairs and binary64, medians, and their geometric mean ratio:
//   at 1000 M   17-75 deg   0.6-1.1e-13, 1.2-3.4e-13   0.2-0.7
//               10, 80      0.6-0.9e-13, 0.9-1.4e-13   0.6-0.9
//               85          0.8e-13,     0.7e-13       1.0-1.4 (ninth decile 0.5-0.7)
//               86.5, 3     0.6-0.9e-13, 0.3-0.5e-13   1.1-1.6
//               88, 1, 90   0.6-0.9e-13, 0.2-0.4e-13   1.7-5
//   at 60 deg   200 M       0.6-0.9e-13, 0.5-0.8e-13   1.2-1.3
//               150, 100 M  0.6-0.8e-13, 0.3-0.8e-13   1.0-1.8
//   div 1, 2, 4, 7, 10, 20  ratio 19, 3, 1.9, 1.3, 0.7-1.1, 0.5-0.6; tol 1e-2
//   to 1e-8 changes neither.
// The lines: distance |sin i cos i| of 78 M (4.5 to 85.5 deg at 1000 M), div 10.
MK_HD bool pair_request(const mk_request &R) {
    auto in = [](double v, double lo, double hi) { return fabs(v) >= lo && fabs(v) <= hi; };
    bool ok = R.policy.div >= 10.0 && R.policy.div <= 1e6 && R.policy.tol >= 1e-8 && fabs(R.camera.bhspin) <= 1.0 &&
              R.camera.kind == MK_CAMERA_GRID &&
              fabs(R.camera.distance * R.camera.cos_inc * R.camera.sin_inc) >= 78.0 &&
              fabs(R.camera.distance) <= 1e6 && fabs(R.camera.fov_lower) <= 1e6 && fabs(R.camera.fov_upper) <= 1e6;
    ok = ok && in(R.fluid_gamma - 1.0, 1e-6, 1e6) && R.r_low >= 0.0 && R.r_low <= 1e6 && R.r_high >= 0.0 &&
         R.r_high <= 1e6 && R.r_low + R.r_high >= 1e-6 && in(R.electron_gamma_m1, 1e-6, 1e6) &&
         in(R.ion_gamma_m1, 1e-6, 1e6) && in(R.sigma_cut, 1e-12, 1e12) && in(R.L_unit, 1e5, 1e20);
    for (int ch = 0; ch < MK_MAX_NU; ch++)
        if (ch < R.nnu) {
            const EmissionFold e = emission_fold(R, R.nu[ch]);
            ok = ok && in(e.kem, 1e-22, 1e20) && in(e.knus, 1e-20, 1e20) && in(e.kbx, 1e-16, 1e10) &&
                 in(e.kib, 1e-10, 1e25);
        }
    return ok;
}

// the geodesic's part (to PC_TOL) and the sampler's (from PC_BOX)
template <int STRIDE>
__device__ __forceinline__ void pair_consts_geodesic(const mk_request &R, PairConsts<STRIDE> C) {
    const double a = R.camera.bhspin;
    C.set(PC_A, a, 2);
    C.set(PC_AA, a * a, 3);  // the third word is PC_AA_L
    C.set(PC_REH, radius_eh(a), 3);
    C.set(PC_NINV, -1.0 / R.policy.div, 3);
    C.set(PC_TOL, R.policy.tol, 2);
}

template <int STRIDE>
__device__ __forceinline__ void pair_consts_sample(const mk_request &R, const mk_snapshot_view &sv,
                                                   PairConsts<STRIDE> C) {
#pragma unroll
    for (int i = 0; i < 3; i++) {
        // the block grid's box, widened by more than the float's rounding
        const double lo = sv.lo[i], hi = sv.lo[i] + sv.nb[i] * sv.width[i], m = 1e-5 * (fabs(lo) + fabs(hi));
        C.c[(PC_BOX + i) * STRIDE] = (float)(lo - m);
        C.c[(PC_BOX + 3 + i) * STRIDE] = (float)(hi + m);
        C.c[(PC_INVW + i) * STRIDE] = (float)(1.0 / sv.width[i]);
    }
    C.set(PC_GAM2, 2.0 * (R.fluid_gamma - 1.0), 2);
    C.set(PC_RHIGH, R.r_high, 2);
    C.set(PC_RLOW, R.r_low, 2);
    C.set(PC_GEM1, R.electron_gamma_m1, 2);
    C.set(PC_GIM1, R.ion_gamma_m1, 2);
    C.set(PC_KTH, (MP * CL2 / ME_CL_CL) * R.electron_gamma_m1 * R.ion_gamma_m1, 2);
    C.set(PC_SIGMA, R.sigma_cut, 2);
    C.set(PC_LUNIT, R.L_unit, 2);
#pragma unroll
    for (int ch = 0; ch < MK_MAX_NU; ch++)
        if (ch < R.nnu) {
            const EmissionFold e = emission_fold(R, R.nu[ch]);
            C.set(PC_NU + 8 * ch, e.kem, 2);
            C.set(PC_NU + 8 * ch + 2, e.knus, 2);
            C.set(PC_NU + 8 * ch + 4, e.kbx, 2);
            C.set(PC_NU + 8 * ch + 6, e.kib, 2);
        }
}

// The warps, of `warps`, that a block's last rays move into: one a
// sub-partition as long as they fit.  With no ray left there is nothing to
// move, and the block's loop still divides by what it has.
__host__ __device__ constexpr int warps_for(int rays, int warps) {
    const int need = 4 * ((rays + 127) / 128);
    return rays > 0 && need < warps ? need : warps;
}

// The snapshot's fields a sample reads.
struct SampleView {
    const float *blocks;
    const double *geom, *faces;
    const int32_t *table, *block64;  // block64: null if no block is kept in binary64
    int nb[3], n;
};
__device__ __forceinline__ SampleView sample_view(const mk_snapshot_view &sv) {
    return {sv.blocks, sv.geom, sv.faces, sv.table, sv.blocks64 ? sv.block64 : nullptr, {sv.nb[0], sv.nb[1], sv.nb[2]}, sv.n};
}

// Beside face i of block mb at table cell c (0, 1: left and right in x; ...): on
// which side of the block x lies, 0 in it (left < x <= right; the difference of
// triples has its sign to the state's 72 bits).  2: the neighbour there does not
// share the face to the bit, so both or neither may hold the point.
static __device__ __noinline__ int near_face(const SampleView &sv, int mb, int c0, int c1, int c2, int i, tri x) {
    const double face = __ldg(sv.faces + 6 * (int64_t)mb + i);
    const int step = (i & 1) ? 1 : -1, a = i >> 1;
    const int o[3] = {c0 + (a == 0 ? step : 0), c1 + (a == 1 ? step : 0), c2 + (a == 2 ? step : 0)};
    const int nb = table_at(sv, o);
    const float d = t_sub(x, t_from(face)).h;
    if (nb >= 0 && __ldg(sv.faces + 6 * (int64_t)nb + (i ^ 1)) != face) return 2;
    return (i & 1) ? d > 0.0f : -(d <= 0.0f);
}

// The cell of x: the block whose faces enclose it (left < x <= right) and the
// ghost-shifted index and offset in it (locate_fast).  The candidate comes
// from the float coordinate; its own cell coordinate t, faces at -1/2 and n -
// 1/2, decides and moves it across a face it lies beyond, or next to one
// (|e| < 1e-9 of a cell; t is good to 1e-11) the face itself.  -1: outside
// the snapshot; -2: left to the binary64 lookup (beside a place without a
// block, or at a face that two blocks do not share to the bit).
template <int STRIDE>
__device__ __forceinline__ int locate_pair(const SampleView &sv, const PairConsts<STRIDE> &C, const tri x[3],
                                           int idx[3], pr del[3]) {
    int c[3];
    bool beside = false;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const float lo = C.f(PC_BOX + a), hi = C.f(PC_BOX + 3 + a), iw = C.f(PC_INVW + a);
        if (!(x[a].h >= lo && x[a].h <= hi)) return -1;
        // the box's margin is 1e-5 of its coordinates; twice that off, so that a
        // point on a face, which is in the block below, finds that block at once
        const float tol = 2e-5f * (fabsf(lo) + fabsf(hi)) * iw, u = (x[a].h - lo) * iw - tol;
        if (fabsf(u - rintf(u)) <= 1.5f * tol) beside = true;
        c[a] = max(0, min((int)u, sv.nb[a] - 1));
    }
    const float n = (float)sv.n;
    for (int it = 0; it < 4; ++it) {
        const int mb = table_at(sv, c);
        if (mb < 0) return it == 0 && beside ? -2 : -1;
        const double *g = sv.geom + 6 * (int64_t)mb;
        const int at[3] = {c[0], c[1], c[2]};
        bool moved = false;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const tri left = t_from(__ldg(g + a)), d = t_near(__ldg(g + 3 + a));
            const tri s = t_add(x[a], t_neg(left));
            const pr w = {d.h, d.m}, iw = p_rcp(w), t = p_mulr({s.h, s.m}, iw);
            const float e0 = f_add(f_add(t.h, 0.5f), t.l), e1 = f_add(f_sub(t.h, n - 0.5f), t.l);
            int side = e0 < 0.0f ? -1 : (e1 > 0.0f ? 1 : 0);
            if (fminf(fabsf(e0), fabsf(e1)) < 1e-9f) {
                side = near_face(sv, mb, at[0], at[1], at[2], 2 * a + (fabsf(e1) < fabsf(e0)), x[a]);
                if (side == 2) return -2;
            }
            c[a] += side;
            if (side) moved = true;
            float fl = floorf(t.h);
            if (fl == t.h && t.l < 0.0f) fl -= 1.0f;
            fl = fminf(fmaxf(fl, -1.0f), n - 1.0f);
            idx[a] = (int)fl + 1;
            // offset from the cell's own centre, so that it keeps its digits
            const float p = f_mul(fl, d.h), e = fmaf(fl, d.h, -p);
            float uh, ul;
            two_sum_f(s.h, -p, uh, ul);
            const pr u = p_norm({uh, f_add(f_add(ul, fmaf(-fl, d.m, s.m)), -e)});
            del[a] = p_mulr(u, iw);
        }
        if (!moved) return mb;
    }
    return -2;
}

// exp(-x) for x >= 0 as m 2^-e, m in [1/2, 1]: x = (32 e + j) ln2/32 - r, the
// table's 2^(-j/32), and the series of exp(r), |r| < 0.011
__device__ __forceinline__ pr p_exp_neg(pr x, const float2 *tab, int &e) {
    const float n = rintf(x.h * (float)(EXP_STEPS * 1.4426950408889634));
    constexpr double STEP = 0.693147180559945309417 / EXP_STEPS;
    constexpr float c1 = (float)STEP, c2 = (float)(STEP - (double)c1);
    const float p = f_mul(n, c1), pe = fmaf(n, c1, -p);
    float rh, re;
    two_sum_f(p, -x.h, rh, re);
    pr r;
    fast_sum_f(rh, f_add(re, fmaf(n, c2, f_sub(pe, x.l))), r.h, r.l);
    const pr s = p_two(p_sqr(r), 0.5f);
    const float t = f_mul(f_mul(f_mul(r.h, r.h), r.h), fmaf(r.h, fmaf(r.h, 1.0f / 120.0f, 1.0f / 24.0f), 1.0f / 6.0f));
    pr q = p_add(r, {s.h, f_add(s.l, t)});
    float h, l;
    fast_sum_f(1.0f, q.h, h, l);
    const int k = (int)n, j = k & (EXP_STEPS - 1);
    e = k / EXP_STEPS;
    const float2 T = tab[j];
    return p_mulr({T.x, T.y}, {h, f_add(l, q.l)});
}

// m 2^-e as a double, |m| a normal float or 0, by the exponent's bits
__device__ __forceinline__ double p_scaled(pr m, int e) {
    if (e > 1201 || m.h == 0.0f) return 0.0;  // |m| < 2^128: below every double
    const double v = d_from(m.h) + d_from(m.l);
    if (e > 850)  // 2^-e in two normal factors, one rounding
        return v * __hiloint2double((1023 - e / 2) << 20, 0) * __hiloint2double((1023 - (e - e / 2)) << 20, 0);
    return __hiloint2double(__double2hiint(v) - (int)((unsigned)e << 20), __double2loint(v));
}
// A sample's coefficients at one frequency: em 2^-e and ab 2^-e.
struct PairCoeff {
    pr em, ab;
    int e;
};

enum { PS_OUTSIDE = 0, PS_SAMPLED = 1, PS_BINARY64 = 2 };

// One sample at x (triples) for the photon k; a: the spin, m: r, f, l3 and
// 1/(r^2 + a^2) there.  PS_SAMPLED: co holds the
// invariant coefficients of every frequency; PS_BINARY64: the point lies in
// the snapshot, in a block kept in binary64 or at primitives outside the
// pairs' range, or where only the binary64 lookup tells (locate_pair); the
// caller samples it in binary64.
template <int STRIDE>
__device__ __forceinline__ int sample_pair(const SampleView &sv, const PairConsts<STRIDE> &C, int nnu,
                                           const tri x[3], const pr k[4], pr a, const pr m[4], const float2 *tab,
                                           PairCoeff co[MK_MAX_NU]) {
    int idx[3];
    pr del[3];
    const int mb = locate_pair(sv, C, x, idx, del);
    if (mb < 0) return mb == -2 ? PS_BINARY64 : PS_OUTSIDE;
    if (sv.block64 && __ldg(sv.block64 + mb) >= 0) return PS_BINARY64;
    // Each primitive as the sum of eight weights times cells; one copy of the
    // code for the four (z, y) neighbours (see tri_step), a neighbour's cells
    // loaded while the one before it is summed.  Density, energy and field can
    // fall by tens of decades (along a torus' poles): where they leave the
    // floats' comfortable range the sums are taken again with those weights
    // scaled by 2^100.
    const int n2 = sv.n + 2;
    const int64_t sj = (int64_t)n2 * 8, sk = (int64_t)n2 * n2 * 8;
    const float *base = sv.blocks + ((((int64_t)mb * n2 + idx[2]) * n2 + idx[1]) * n2 + idx[0]) * 8;
    const pr one = {1.0f, 0.0f};
    const pr u0 = p_subr(one, del[0]), u1 = p_subr(one, del[1]), u2 = p_subr(one, del[2]);
    pr prim[8];
    float Bm, up = 1.0f;
    for (;;) {
        // primitives two by two (0-1, 2-3, 4-5, 6-7) on paired instructions
        float2 sh[4], sl[4];
#pragma unroll
        for (int i = 0; i < 4; i++) sh[i] = sl[i] = make_float2(0.0f, 0.0f);
        float4 next[4] = {ldg4(base), ldg4(base + 4), ldg4(base + 8), ldg4(base + 12)};
#pragma unroll 1
        for (int q = 0; q < 4; q++) {
            const float4 c[4] = {next[0], next[1], next[2], next[3]};
            if (q < 3) {
                const float *p = base + ((q + 1) >> 1) * sk + ((q + 1) & 1) * sj;
                next[0] = ldg4(p);
                next[1] = ldg4(p + 4);
                next[2] = ldg4(p + 8);
                next[3] = ldg4(p + 12);
            }
            const pr zy = p_mulr((q & 2) ? del[2] : u2, (q & 1) ? del[1] : u1);
#pragma unroll
            for (int x = 0; x < 2; x++) {
                const pr w = p_mulr(zy, x ? del[0] : u0), ws = p_two(w, up);
                const float4 lo = c[2 * x], hi = c[2 * x + 1];
                const float2 v[4] = {make_float2(lo.x, lo.y), make_float2(lo.z, lo.w), make_float2(hi.x, hi.y),
                                     make_float2(hi.z, hi.w)};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    // velocities (1, 2, 3) are not scaled
                    const float2 gh = i == 0 ? make_float2(ws.h, w.h) : (i == 1 ? make_float2(w.h, w.h) : make_float2(ws.h, ws.h));
                    const float2 gl = i == 0 ? make_float2(ws.l, w.l) : (i == 1 ? make_float2(w.l, w.l) : make_float2(ws.l, ws.l));
                    const float2 t = __fmul2_rn(gh, v[i]);
                    const float2 e = __ffma2_rn(gl, v[i], __ffma2_rn(gh, v[i], make_float2(-t.x, -t.y)));
                    float2 r;
                    sh[i] = v_two_sum(sh[i], t, r);
                    sl[i] = __fadd2_rn(sl[i], __fadd2_rn(e, r));
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            prim[2 * i] = p_norm({sh[i].x, sl[i].x});
            prim[2 * i + 1] = p_norm({sh[i].y, sl[i].y});
        }
        Bm = fmaxf(fmaxf(fabsf(prim[5].h), fabsf(prim[6].h)), fabsf(prim[7].h));
        if ((prim[0].h >= 1e-22f && prim[4].h >= 1e-22f && Bm >= 1e-22f) || up != 1.0f) break;
        // excised cells: nothing emits (sigma or Theta_e is not a number)
        if (prim[0].h == 0.0f) break;
        up = 0x1p100f;
    }
#pragma unroll
    for (int ch = 0; ch < MK_MAX_NU; ch++) co[ch] = {{0.0f, 0.0f}, {0.0f, 0.0f}, 0};
    // no energy: Theta_e = 0; no field: beta is infinite and Theta_e not a number
    if (prim[0].h == 0.0f || prim[4].h == 0.0f || Bm == 0.0f) return PS_SAMPLED;
    const float Um = fmaxf(fmaxf(fabsf(prim[1].h), fabsf(prim[2].h)), fabsf(prim[3].h));
    if (!(Bm >= 1e-22f && Bm <= 1e25f && Um <= 1e6f && prim[0].h >= 1e-22f && prim[0].h <= 1e25f &&
          prim[4].h <= 1e12f * prim[0].h && prim[4].h >= 0.0f))
        return PS_BINARY64;
    // density and energy, and the field, scaled to order one by powers of two
    const int shift = up == 1.0f ? 0 : 100;
    const int ed = ((int)(__float_as_uint(prim[0].h) >> 23) & 255) - 127;
    const int eB = ((int)(__float_as_uint(Bm) >> 23) & 255) - 127;
    const int ex = (ed - shift) - 2 * (eB - shift);  // of dens / B^2
    if (ex < -100 || ex > 100) return PS_BINARY64;
    const float sd = __uint_as_float((unsigned)(127 - ed) << 23), sB = __uint_as_float((unsigned)(127 - eB) << 23);
    const pr dens = p_two(prim[0], sd), ue = p_two(prim[4], sd);
    const pr *U = prim + 1;
    const pr B[3] = {p_two(prim[5], sB), p_two(prim[6], sB), p_two(prim[7], sB)};
    const float ratio = __uint_as_float((unsigned)(127 + ex) << 23);  // (dens / B^2) over the scaled one
    // the frame
    const pr r = m[0], f = m[1], l3 = m[2], ira = m[3];
    const pr X = {x[0].h, x[0].m}, Y = {x[1].h, x[1].m};
    const pr l1 = p_mulr(p_addr(p_mul(r, X), p_mul(a, Y)), ira);
    const pr l2 = p_mulr(p_subr(p_mul(r, Y), p_mul(a, X)), ira);
    auto dot = [](pr x1, pr y1, pr x2, pr y2, pr x3, pr y3) {
        return p_addr(p_add(p_mul(x1, y1), p_mul(x2, y2)), p_mul(x3, y3));
    };
    const pr lU = dot(l1, U[0], l2, U[1], l3, U[2]), lB = dot(l1, B[0], l2, B[1], l3, B[2]);
    const pr UU = dot(U[0], U[0], U[1], U[1], U[2], U[2]), BB = dot(B[0], B[0], B[1], B[1], B[2], B[2]);
    const pr BU = dot(B[0], U[0], B[1], U[1], B[2], U[2]);
    const pr kU = dot(k[1], U[0], k[2], U[1], k[3], U[2]), kB = dot(k[1], B[0], k[2], B[1], k[3], B[2]);
    const pr lk = dot(l1, k[1], l2, k[2], l3, k[3]), lv = p_addr(k[0], lk);  // l.k, l_mu k^mu
    const pr flU = p_mulr(f, lU), flB = p_mulr(f, lB);
    const pr G = p_addr(p_add(UU, p_mul(flU, lU)), one);
    const pr alpha = p_rsqrt(p_addr(f, one)), rG = p_rsqrt(G);
    const pr ga = p_mulr(p_mulr(G, rG), alpha);           // gamma alpha
    const pr iut = p_mulr(alpha, rG);                     // 1/u^t
    const pr Bu = p_addr(BU, p_mul(flU, lB));             // b^t = B^i u_i
    const pr b2 = p_mulr(p_addr(p_add(BB, p_mul(flB, lB)), p_sqr(Bu)), p_mulr(iut, iut));
    if (!(b2.h > 0.0f)) return PS_SAMPLED;
    const pr ku = p_subr(p_add(kU, p_mul(flU, lv)), p_mul(k[0], ga));  // k.u
    const pr gaf = p_mulr(ga, f);
    // l_mu b^mu = b^t + (l.B + (l.U - gamma alpha f) b^t) / u^t, and k.b
    const pr lb = p_addr(Bu, p_mul(p_addr(lB, p_mul(p_subr(lU, gaf), Bu)), iut));
    const pr kb3 = p_mulr(p_addr(kB, p_mul(p_subr(kU, p_mul(gaf, lk)), Bu)), iut);
    const pr kb = p_addr(p_subr(kb3, p_mul(k[0], Bu)), p_mul(p_mulr(f, lb), lv));
    const pr ib = p_rsqrt(b2);
    const pr b = p_mulr(b2, ib);
    const pr nup = p_neg(ku);                             // nu'
    if (!(nup.h > 0.0f)) return PS_SAMPLED;               // the fit's roots are not numbers
    const pr inup = p_rcp(nup);
    const pr cp = p_mulr(p_mul(kb, ib), inup);
    const pr s2 = p_mulr(p_subr(one, cp), p_addr(one, cp));
    if (!(s2.h > 0.0f)) return PS_SAMPLED;                // nu_s = 0
    const pr sp = p_mulr(s2, p_rsqrt(s2));
    // sigma cut, electron temperature
    if (p_sub(b2, p_mul(C.p(PC_SIGMA), p_two(dens, ratio))).h > 0.0f) return PS_SAMPLED;
    pr beta = p_mulr(p_mulr(p_two(ue, ratio), C.p(PC_GAM2)), p_mulr(ib, ib));
    if (fabsf(beta.h) > 1e15f) beta = {1e15f, 0.0f};      // T_ratio is r_high to 2^-99
    // 1 and beta^2 over beta's power of two squared, where that is above one
    // (the quotient is the same): beta^2 R_high and its reciprocal would leave
    // the floats' range
    const int ebe = max(0, (int)(__float_as_uint(beta.h) >> 23 & 255u) - 127);
    const float sbe = __uint_as_float((unsigned)(127 - min(ebe, 50)) << 23), one2 = sbe * sbe;
    beta = p_two(beta, sbe);
    const pr be2 = p_mulr(beta, beta), ope = p_addr(be2, {one2, 0.0f});
    const pr gi = C.p(PC_GIM1), ge = C.p(PC_GEM1);
    // Theta_e = K u (1 + beta^2) / (dens (g_i (1 + beta^2) + g_e (R_high beta^2 + R_low)))
    const pr D = p_mulr(dens, p_addr(p_mul(gi, ope), p_mul(ge, p_addr(p_mul(C.p(PC_RHIGH), be2), p_two(C.p(PC_RLOW), one2)))));
    const pr th = p_mulr(p_mulr(C.p(PC_KTH), ue), p_mulr(ope, p_rcp(D)));
    if (p_sub(th, {0.3f, (float)(0.3 - (double)0.3f)}).h < 0.0f) return PS_SAMPLED;
    if (!(th.h < 1e8f)) return PS_BINARY64;               // or not a number
    const pr ith = p_rcp(th);
    const pr base_nus = p_mulr(p_mulr(p_mulr(b, sp), p_mulr(th, th)), inup);
    const pr base_em = p_mulr(p_mulr(dens, inup), p_mulr(ith, ith));
    const pr base_bx = p_mulr(nup, ith);
    if (eB - shift < -120) return PS_SAMPLED;              // X > 1e12 at any temperature
    const float iB = __uint_as_float((unsigned)(127 + eB - shift) << 23);
    if (!(base_nus.h >= 1e-26f && base_nus.h <= 1e26f && base_em.h >= 1e-26f && base_em.h <= 1e26f))
        return PS_BINARY64;
#pragma unroll
    for (int ch = 0; ch < MK_MAX_NU; ch++) {
        if (ch >= nnu) break;
        const int at = PC_NU + 8 * ch;
        const pr Z = p_mulr(C.p(at + 2), p_two(base_nus, iB));  // nu_s / nu'
        if (!(Z.h >= 1e-12f)) continue;                   // X > 1e12: no emission
        const pr x3 = p_rcbrt(Z);
        const pr Yc = p_mulr(p_mulr(x3, x3), Z);
        constexpr pr C211 = {(float)C2_11_12, (float)(C2_11_12 - (double)(float)C2_11_12)};
        const pr t = p_addr(one, p_mul(C211, Yc));
        int e;
        const pr E = p_exp_neg(x3, tab, e);
        e -= ed - shift;
        // the low word of a product below 1e-28 starts to fall among the floats'
        // last digits, before t^2 lifts it again
        const pr e0 = p_mulr(C.p(at), base_em);
        if (!(e0.h >= 1e-28f)) return PS_BINARY64;
        const pr em_m = p_mulr(e0, p_mulr(p_mulr(t, t), E));
        if (!(em_m.h >= 1e-28f && em_m.h <= 1e15f)) return PS_BINARY64;
        const pr bx = p_mulr(C.p(at + 4), base_bx);
        pr den;
        if (bx.h < 2.e-3f) {
            // bx (1 + bx/2 (1 + bx/3 (1 + bx/4))), as the reference cuts it
            const pr q = p_sqr(bx);
            const float c3 = f_mul(f_mul(f_mul(bx.h, bx.h), bx.h), fmaf(bx.h, 1.0f / 24.0f, 1.0f / 6.0f));
            den = p_addr(bx, {f_mul(0.5f, q.h), fmaf(0.5f, q.l, c3)});
        } else {
            if (!(bx.h < 60.0f)) return PS_BINARY64;
            den = p_near(exp((double)bx.h + (double)bx.l) - 1.0);
        }
        const pr dk = p_mulr(den, C.p(at + 6)), ab_m = p_mulr(em_m, dk);
        if (!(bx.h >= 1e-28f && dk.h >= 1e-28f && ab_m.h >= 1e-30f && ab_m.h <= 1e15f)) return PS_BINARY64;
        co[ch] = {em_m, ab_m, e};
    }
    return PS_SAMPLED;
}

}  // namespace mk

// mk_geodesic.cu -- camera initialisation, geodesic integration and the
// shadow-bisection pass (geodesics.py), one thread per ray: cameras in
// binary64, geodesics in float triples (mk_tri.cuh) with binary64 where those
// do not hold.
#include <algorithm>

#include "mk_common.cuh"
#include "mk_kerr.cuh"
#include "mk_tri.cuh"

namespace mk {

constexpr int GEO_THREADS = 128;

__global__ void camera_kernel(mk_camera cam, int64_t npx, double *__restrict__ s0) {
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= npx) return;
    double s[8];
    camera_ray(cam, p, s);
#pragma unroll
    for (int i = 0; i < 8; i++) s0[8 * p + i] = s[i];
}

__global__ void camera_points_kernel(const double *__restrict__ xs, const double *__restrict__ ys, int64_t n,
                                     double a, double ci, double si, double d, double *__restrict__ s0) {
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= n) return;
    double s[8];
    camera_pixel(xs[p], ys[p], ci, si, d, a, s);
#pragma unroll
    for (int i = 0; i < 8; i++) s0[8 * p + i] = s[i];
}

// Distance to the horizon below which a step's accelerations are binary64 (see
// mk_tri.cuh): a ray stopped farther out has fewer binary64 steps behind it.
// End states of captured rays, times as far from a 64-bit-significand
// integration as binary64's (geometric mean of 40 to 80 rays) with 0.1 and 0.3
// M: tol 1e-2 at spins 0 to 0.94 1.6-3.1 and 0.8-1.0; tol <= 1e-4 0.06-0.7 up to
// spin 0.5 and 0.7-1.4 at 0.94 with 0.1 M.
constexpr float TRI_NEAR = 0.1f;
static float near_distance(double tol) { return tol > 2e-4 ? 0.3f : TRI_NEAR; }
// Above this spin the reference rule's rays linger near the horizon: at 0.998
// their last wavevectors are 3.5-4.6, 1.6-1.8 and 0.8-1.3 times as far off with
// 0.1, 0.3 and 1 M, and 128^2 rays take 65, 70 and 80 ms.  In binary64 from the
// start they take 55.  Below it (spins 0.9, 0.92, 0.95) 0.1 M gives 0.2-1.2.
constexpr double TRI_MAX_SPIN = 0.95;

__device__ __forceinline__ bool tri_range(const double s[8]) {
    const double k = fmax(fmax(fabs(s[4]), fabs(s[5])), fmax(fabs(s[6]), fabs(s[7])));
    const double x = fmax(fmax(fabs(s[1]), fabs(s[2])), fabs(s[3]));
    return fabs(s[0]) <= TRI_MAX_R && x <= TRI_MAX_R && k <= TRI_MAX_K && k >= TRI_MIN_K;
}
// Whether binary64 rounds a ray under the fixed rule more than pairs do: by
// 2^-54 of each coordinate, of which the part across the ray counts, t^2 = sum
// x_i^2 (1 - k_i^2 / k^2).  Ratios as above, hfrac 0.05 and 0.1, escaped rays:
// at 1000 M and 10 deg (t = 240 M) 0.4, 85 deg (120 M) 0.7-0.9, 3 deg (70 M)
// 0.9-1.4, 88 and 1 deg 1.1-2; from 200 and 100 M at 60 deg (120, 60 M) 1.1-1.7
// and 1.5-2.9.  hfrac 0.02: 0.3-1.0 everywhere.
__device__ __forceinline__ bool fixed_range(const double s[8], double hfrac) {
    if (hfrac <= 0.02) return true;
    const double kk = s[5] * s[5] + s[6] * s[6] + s[7] * s[7], xx = s[1] * s[1] + s[2] * s[2] + s[3] * s[3];
    const double a = s[1] * s[5], b = s[2] * s[6], c = s[3] * s[7];
    return xx >= 9e4 && xx * kk - (a * a + b * b + c * c) >= 6.4e3 * kk;
}

// one RK4 step of the triple state by its binary64 increment (s: the state)
__device__ __noinline__ void rk4_step_near(TriState &st, const double s[8], double dt, double a) {
    double d1[4], sum[8];
    kerr_accel(s[1], s[2], s[3], s[4], s[5], s[6], s[7], a, d1[0], d1[1], d1[2], d1[3]);
    rk4_sum_k1(s, d1, dt, a, sum);
    const double c = dt * SIXTH;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        st.X[i] = t_add(st.X[i], t_from(c * sum[i]));
        st.K[i] = t_add(st.K[i], t_from(c * sum[4 + i]));
    }
}

// 16-byte stores where the caller's array allows them
__device__ __forceinline__ void store_row(double *__restrict__ rows, int64_t at, const double s[8]) {
    if (((uintptr_t)rows & 15) == 0) {
        double2 *o = reinterpret_cast<double2 *>(rows + at * 8);
#pragma unroll
        for (int i = 0; i < 4; i++) o[i] = make_double2(s[2 * i], s[2 * i + 1]);
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) rows[at * 8 + i] = s[i];
    }
}

// Rows j >= K[p] of stopped rays: the frozen state, dt = 0.  A pass of its
// own over (row, ray), 16 bytes a thread: written by the thread of the ray
// that stopped, a row at a time, they were two thirds of the time of 1600
// trajectories with 10000 rows.  V: double2, or double where the arrays are
// not 16-byte aligned.
template <typename V>
__global__ void freeze_rows_kernel(const double *__restrict__ state, const int32_t *__restrict__ K, int64_t npx,
                                   int nrows, double *__restrict__ rows, double *__restrict__ dts) {
    constexpr int PARTS = 8 * sizeof(double) / sizeof(V);
    const int64_t row = npx * PARTS;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < row; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p = e / PARTS;
        const V v = reinterpret_cast<const V *>(state)[e];
        for (int j = max(0, K[p]) + blockIdx.y; j < nrows; j += gridDim.y) {
            if (rows) reinterpret_cast<V *>(rows)[j * row + e] = v;
            if (dts && e % PARTS == 0) dts[j * npx + p] = 0.0;
        }
    }
}

// geodesic_integrator (geodesics.py:246-272) for one ray, in binary64, from
// its state s before step j0.  rows (N, npx, 8) / dts (N, npx) optional.
__device__ __noinline__ void integrate_reference_f64(double s[8], int j0, int64_t p, int64_t npx, double a, int N,
                                                     double div, double tol, double *rows, double *dts,
                                                     int32_t *Kout, int32_t *why_out, double *state_out) {
    double nw[8];
    const double reh = radius_eh(a);
    int K = N, why = MK_RAY_MAXSTEPS;
    // a step's dt is the previous step's dtn (the same radius_cal of the same
    // state), carried instead of recomputed
    int w0;
    double dt = reference_dt(radius_cal(s[1], s[2], s[3], a), reh, div, tol, w0);
    for (int j = j0; j < N; j++) {
        int w1;
        rk4_step(s, dt, a, nw);
        const double dtn = reference_dt(radius_cal(nw[1], nw[2], nw[3], a), reh, div, tol, w1);
        if (dtn == 0.0) {
            K = j;
            why = (w0 != MK_RAY_ACTIVE) ? w0 : w1;
            break;
        }
        if (rows) store_row(rows, (int64_t)j * npx + p, s);
        if (dts) dts[(int64_t)j * npx + p] = dt;
#pragma unroll
        for (int i = 0; i < 8; i++) s[i] = nw[i];
        dt = dtn;
        w0 = w1;
    }
    Kout[p] = K;
    why_out[p] = why;
    store_row(state_out, p, s);
}

// The same on triples (mk_tri.cuh).  rpw rays a warp: a ray's chain of steps
// sets the time of a small launch, so its rays are spread over every SM
// sub-partition before they share warps.  A warp's lanes near the horizon
// wait until none of the others moves: a binary64 step holds the warp ~31 k
// cycles whatever number of lanes takes it, so the lanes take them together,
// after as many steps on triples as the longest ray has (40^2 rays, spin 0.1:
// 12.3 -> 9.9 ms).
// ROWS: rows or dts wanted; the state is then converted to binary64 at every
// step, and the state before a rejected step is that row.
template <bool ROWS>
__global__ void __launch_bounds__(GEO_THREADS)
integrate_reference_kernel(const double *__restrict__ s0, int64_t npx, double a, SpinTri sp, RuleTri R, float near_d,
                           int N, double div, double tol, double *__restrict__ rows, double *__restrict__ dts,
                           int32_t *__restrict__ Kout, int32_t *__restrict__ why_out, double *__restrict__ state_out,
                           int rpw, int all_f64) {
    const int lane = threadIdx.x & 31;
    const int64_t p = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * rpw + lane;
    const unsigned team = __ballot_sync(0xffffffffu, lane < rpw && p < npx);
    if (lane >= rpw || p >= npx) return;
    double s64[8];
#pragma unroll
    for (int i = 0; i < 8; i++) s64[i] = s0[8 * p + i];
    bool out = all_f64 || !tri_range(s64);
    int K = N, why = MK_RAY_MAXSTEPS, j = 0;
    TriState s, last;
    tri_state(s64, s);
    last = s;
    {
        TriPoint q;
        tri dt = {0.0f, 0.0f, 0.0f};
        float d = 0.0f;
        int w;
        bool go = false, moving = !out && N > 0;
        if (moving) {
            tri_step<true>(s, q, dt, sp.a, sp.aa, sp.aa3, true);
            go = rule_dt(q.r, R, dt, d, w);
            if (tri_left_range(s, q.r.h)) {
                out = true;
                moving = false;
            }
        }
        while (__any_sync(team, moving)) {
            const bool near = go && d < near_d;
            if (__any_sync(team, moving && !near) && near) continue;
            if (!moving) continue;
            tri dtn = dt;
            if (!ROWS) last = s;
            else if (j) tri_doubles(s, s64);  // the first state is the caller's, bit for bit
            if (go) {
                if (near) {  // through a copy: s itself stays in registers
                    TriState n = s;
                    double sc[8];
                    if (!ROWS) tri_doubles(s, s64);
#pragma unroll
                    for (int i = 0; i < 8; i++) sc[i] = s64[i];
                    rk4_step_near(n, sc, t_to(dt), a);
                    s = n;
                }
                tri_step<true>(s, q, dt, sp.a, sp.aa, sp.aa3, near);
                if (tri_left_range(s, q.r.h)) {
                    out = true;
                    moving = false;
                    continue;
                }
                go = rule_dt(q.r, R, dtn, d, w);
            }
            if (!go) {
                K = j;
                why = w;
                moving = false;
                continue;
            }
            if (ROWS && rows) store_row(rows, (int64_t)j * npx + p, s64);
            if (ROWS && dts) dts[(int64_t)j * npx + p] = t_to(dt);
            dt = dtn;
            moving = ++j < N;
        }
    }
    if (out) {
        if (!ROWS && j) tri_doubles(last, s64);
        double sc[8];
#pragma unroll
        for (int i = 0; i < 8; i++) sc[i] = s64[i];
        integrate_reference_f64(sc, j, p, npx, a, N, div, tol, rows, dts, Kout, why_out, state_out);
        return;
    }
    Kout[p] = K;
    why_out[p] = why;
    if (K == N && N) tri_doubles(s, s64);
    else if (!ROWS && K) tri_doubles(last, s64);  // a rejected step leaves the state before it
    store_row(state_out, p, s64);
}

// fixed-fraction vacuum policy: h = clamp(hfrac r, hmin, hmax), backwards, in
// binary64 from the state before step j0
__device__ __noinline__ void integrate_fixed_f64(double s[8], int j0, int64_t p, double a, int N, double hfrac,
                                                 double hmin, double hmax, double capture, double r_escape,
                                                 int32_t *Kout, int32_t *why_out, double *state_out) {
    double nw[8];
    const double rcap = capture * radius_eh(a);
    double r = radius_cal(s[1], s[2], s[3], a);
    int st = MK_RAY_MAXSTEPS, j;
    for (j = j0; j < N; j++) {
        double h = hfrac * r;
        h = h < hmin ? hmin : (h > hmax ? hmax : h);
        rk4_step(s, -h, a, nw);
        const double rn = radius_cal(nw[1], nw[2], nw[3], a);
#pragma unroll
        for (int i = 0; i < 8; i++) s[i] = nw[i];
        if (isnan(rn) || isnan(s[4])) { st = MK_RAY_NAN; j++; break; }
        if (rn < rcap) { st = MK_RAY_CAPTURED; j++; break; }
        if (rn > r_escape && rn > r) { st = MK_RAY_ESCAPED; j++; break; }
        r = rn;
    }
    Kout[p] = j;
    why_out[p] = st;
    store_row(state_out, p, s);
}

// Lanes near the horizon do not wait here: the fixed-fraction rule takes few
// steps there (128^2 rays 1.80 ms, 1.82 with the wait).
__global__ void __launch_bounds__(GEO_THREADS)
integrate_fixed_kernel(const double *__restrict__ s0, int64_t npx, double a, int N, double hfrac, double hmin,
                       double hmax, double capture, double r_escape, int32_t *__restrict__ Kout,
                       int32_t *__restrict__ why_out, double *__restrict__ state_out, int rpw, int all_f64) {
    const int lane = threadIdx.x & 31;
    const int64_t p = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * rpw + lane;
    if (lane >= rpw || p >= npx) return;
    double s64[8];
#pragma unroll
    for (int i = 0; i < 8; i++) s64[i] = s0[8 * p + i];
    bool out = all_f64 || !tri_range(s64) || !fixed_range(s64, hfrac);
    const double reh = radius_eh(a);
    const tri rcap = t_near(capture * reh), resc = t_near(r_escape), hf = t_from(hfrac), h0 = t_near(hmin),
              h1 = t_near(hmax);
    const float near_r = (float)reh + TRI_NEAR;
    TriState s, last;
    tri_state(s64, s);
    last = s;
    const SpinTri sp = spin_tri(a);
    int st = MK_RAY_MAXSTEPS, j = 0;
    if (!out) {
        TriPoint q;
        tri_step<true>(s, q, {0.0f, 0.0f, 0.0f}, sp.a, sp.aa, sp.aa3, true);
        out = tri_left_range(s, q.r.h);
        for (j = 0; j < N && !out; j++) {
            tri h = t_add(t_mul(hf, q.r), {0.0f, 0.0f, 0.0f});
            h = t_less(h, h0) ? h0 : (t_less(h1, h) ? h1 : h);
            h = t_neg(h);
            const tri r = q.r;
            const bool near = r.h < near_r;
            last = s;
            if (near) {  // through a copy: s itself stays in registers
                TriState n = s;
                double sc[8];
                tri_doubles(s, sc);
                rk4_step_near(n, sc, t_to(h), a);
                s = n;
            }
            tri_step<true>(s, q, h, sp.a, sp.aa, sp.aa3, near);
            if (tri_left_range(s, q.r.h)) { out = true; break; }
            if (t_less(q.r, rcap)) { st = MK_RAY_CAPTURED; j++; break; }
            if (t_less(resc, q.r) && t_less(r, q.r)) { st = MK_RAY_ESCAPED; j++; break; }
        }
    }
    if (out) {
        double sc[8];
        tri_doubles(last, sc);
        if (!j)
#pragma unroll
            for (int i = 0; i < 8; i++) sc[i] = s64[i];
        integrate_fixed_f64(sc, j, p, a, N, hfrac, hmin, hmax, capture, r_escape, Kout, why_out, state_out);
        return;
    }
    Kout[p] = j;
    why_out[p] = st;
    if (j) tri_doubles(s, s64);
    store_row(state_out, p, s64);
}

__global__ void radius_kernel(const double *__restrict__ x, int64_t n, int64_t stride, double a,
                              double *__restrict__ r) {
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= n) return;
    const double *q = x + p * stride;
    r[p] = radius_cal(q[1], q[2], q[3], a);
}

// One bisection pass (select_photons_integrator, geodesics.py:354-378):
// integrate each polar ray with div 40, tol 1e-2 and record what the host
// needs to evaluate r[argmax(dt) - 1] on the trimmed trajectory.
__device__ __noinline__ void shadow_ray_f64(const double start[8], int64_t p, double a, int N, int32_t *Kout,
                                            int32_t *best_out, double *best_dt_out, double *r_km1, double *r_best,
                                            double *r_last) {
    double s[8], nw[8];
#pragma unroll
    for (int i = 0; i < 8; i++) s[i] = start[i];
    const double reh = radius_eh(a);
    int K = N, best = -1;
    double best_dt = -INFINITY, r_prev = nan(""), rb = nan(""), rk = nan(""), rl = nan("");
    int w0;
    double r_here = radius_cal(s[1], s[2], s[3], a);
    double dt = reference_dt(r_here, reh, 40.0, 1e-2, w0);  // carried from step to step, as above
    for (int j = 0; j < N; j++) {
        int w1;
        rk4_step(s, dt, a, nw);
        const double r_next = radius_cal(nw[1], nw[2], nw[3], a);
        const double dtn = reference_dt(r_next, reh, 40.0, 1e-2, w1);
        if (dtn == 0.0) {
            K = j;
            rk = r_prev;   // row K-1
            rl = r_here;   // frozen state = every later row
            break;
        }
        if (dt > best_dt) { best_dt = dt; best = j; rb = r_prev; }
        r_prev = r_here;
        if (j == N - 1) rl = r_here;  // row N-1 = state before step N-1
#pragma unroll
        for (int i = 0; i < 8; i++) s[i] = nw[i];
        r_here = r_next;
        dt = dtn;
    }
    Kout[p] = K;
    best_out[p] = best;
    best_dt_out[p] = best_dt;
    r_km1[p] = rk;
    r_best[p] = rb;
    r_last[p] = rl;
}

// The pass on triples.  NEAR: within near_d of the horizon in binary64 steps, as
// integrate_reference_kernel, for its radii (an outline of 48 angles would take
// 18 ms with 0.3 M, 9.2 without); without, in pairs down to the 1e-2 M where it
// stops, for the sides of the shadow's edge they lie on.  Radii at the horizon, in pairs and with NEAR,
// against long double, median: spin 0.94 2.6e-15, 6e-16 (binary64 7e-16); spin
// 0.998 4.2e-14, 1.3e-15 with 1 M (4e-15; NEAR takes it there).
template <bool NEAR>
__global__ void __launch_bounds__(GEO_THREADS)
shadow_pass_kernel(const double *__restrict__ ca, const double *__restrict__ sa, const double *__restrict__ mid,
                   int64_t n, double a, SpinTri sp, RuleTri R, float near_d, double ci, double si, double dist, int N,
                   int32_t *__restrict__ Kout, int32_t *__restrict__ best_out, double *__restrict__ best_dt_out,
                   double *__restrict__ r_km1, double *__restrict__ r_best, double *__restrict__ r_last, int rpw) {
    const int lane = threadIdx.x & 31;
    const int64_t p = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * rpw + lane;
    const unsigned team = __ballot_sync(0xffffffffu, lane < rpw && p < n);
    if (lane >= rpw || p >= n) return;
    double s64[8];
    camera_pixel(ca[p] * mid[p], sa[p] * mid[p], ci, si, dist, a, s64);
    bool out = !tri_range(s64) || (NEAR && fabs(a) > TRI_MAX_SPIN);
    TriState s;
    tri_state(s64, s);
    const tri none = {NAN, NAN, NAN};
    int K = N, best = -1;
    tri best_dt = {-INFINITY, 0.0f, 0.0f}, r_prev = none, rb = none, rk = none, rl = none;
    TriPoint q;
    tri dt = {0.0f, 0.0f, 0.0f}, r_here = none;
    float d = 0.0f;
    int w;
    bool go = false;
    // step j: to the rule's next dt, false where the ray stops or leaves the range
    auto step = [&](int j, bool near) {
        tri dtn = dt;
        if (go) {
            if (NEAR && near) {  // through a copy: s itself stays in registers
                TriState n = s;
                double sc[8];
                tri_doubles(s, sc);
                rk4_step_near(n, sc, t_to(dt), a);
                s = n;
            }
            tri_step<false>(s, q, dt, sp.a, sp.aa, sp.aa3, NEAR && near);
            if (tri_left_range(s, q.r.h)) { out = true; return false; }
            go = rule_dt(q.r, R, dtn, d, w);
        }
        if (!go) {
            K = j;
            rk = r_prev;   // row K-1
            rl = r_here;   // frozen state = every later row
            return false;
        }
        if (t_less(best_dt, dt)) { best_dt = dt; best = j; rb = r_prev; }
        r_prev = r_here;
        if (j == N - 1) rl = r_here;  // row N-1 = state before step N-1
        r_here = q.r;
        dt = dtn;
        return true;
    };
    if (!out) {
        tri_step<false>(s, q, dt, sp.a, sp.aa, sp.aa3, true);
        r_here = q.r;
        go = rule_dt(q.r, R, dt, d, w);
        out = tri_left_range(s, q.r.h);
    }
    if (NEAR) {
        int j = 0;
        bool moving = !out;
        while (__any_sync(team, moving)) {  // a warp's lanes near the horizon step together
            const bool near = go && d < near_d;
            if (__any_sync(team, moving && !near) && near) continue;
            if (moving) moving = step(j, near) && ++j < N;
        }
    } else if (!out) {
        for (int j = 0; j < N; j++)
            if (!step(j, false)) break;
    }
    if (out) {
        shadow_ray_f64(s64, p, a, N, Kout, best_out, best_dt_out, r_km1, r_best, r_last);
        return;
    }
    Kout[p] = K;
    best_out[p] = best;
    best_dt_out[p] = t_to(best_dt);
    r_km1[p] = t_to(rk);
    r_best[p] = t_to(rb);
    r_last[p] = t_to(rl);
}

// rays a warp: the fewest (a power of two) with which the launch's warps
// still fit one to an SM sub-partition, 32 at most
static int rays_per_warp(int64_t n) {
    const int64_t slots = (int64_t)device_sm_count() * 4;
    int w = 1;
    while (w < 32 && n > slots * w) w *= 2;
    return w;
}
static unsigned ray_grid(int64_t n, int rpw) {
    const int64_t warps = (n + rpw - 1) / rpw;
    return (unsigned)((warps + GEO_THREADS / 32 - 1) / (GEO_THREADS / 32));
}
// Step rules that the triples' range covers and whose accelerations pairs hold
// exactly enough: a long step multiplies their error.  End states against a
// 64-bit-significand integration, times as far off as binary64's (geometric
// means, spins 0.5 and 0.94, escaped and captured): div 1 29-33, 2 2.2-2.5, 4
// 1.1-1.7, 7 0.6-0.9, 10 0.4-0.7, 40 0.1-0.7.  The fixed rule from 1000 M at 60
// deg: hfrac 0.5 1.0-5.4, 0.2 0.7-1.1, 0.05 0.2, 0.01 0.1.
static bool tri_policy(const mk_step_policy &p, double a) {
    if (p.kind == MK_POLICY_REFERENCE) return fabs(a) <= TRI_MAX_SPIN && p.div >= 7.0 && p.div <= 1e6 && p.tol >= 1e-12;
    return p.hfrac >= 1e-6 && p.hfrac <= 0.1 && p.hmin >= 1e-9 && p.hmax >= 1e-9 && p.hmin <= 0.2;
}

}  // namespace mk

using namespace mk;

extern "C" int mk_camera_init(const mk_camera *camera, double *s0_dev, void *stream) {
    MK_REQUIRE(camera && s0_dev, MK_ERR_ARG, "mk_camera_init: null pointer");
    MK_REQUIRE(camera->pixels > 0, MK_ERR_ARG, "mk_camera_init: pixels must be positive");
    MK_REQUIRE(camera->kind == MK_CAMERA_GRID || camera->kind == MK_CAMERA_EQUATOR, MK_ERR_ARG,
               "mk_camera_init: unknown camera kind %d", (int)camera->kind);
    const int64_t npx = camera->kind == MK_CAMERA_GRID ? (int64_t)camera->pixels * camera->pixels : camera->pixels;
    camera_kernel<<<grid_for(npx, 128), 128, 0, as_stream(stream)>>>(*camera, npx, s0_dev);
    MK_LAUNCHED("camera_kernel");
    return MK_OK;
}

extern "C" int mk_camera_points(const double *x_dev, const double *y_dev, int64_t n, double bhspin, double cos_inc,
                                double sin_inc, double distance, double *s0_dev, void *stream) {
    MK_REQUIRE(x_dev && y_dev && s0_dev, MK_ERR_ARG, "mk_camera_points: null pointer");
    MK_REQUIRE(n >= 0, MK_ERR_ARG, "mk_camera_points: negative size");
    if (n == 0) return MK_OK;
    camera_points_kernel<<<grid_for(n, 128), 128, 0, as_stream(stream)>>>(x_dev, y_dev, n, bhspin, cos_inc,
                                                                          sin_inc, distance, s0_dev);
    MK_LAUNCHED("camera_points_kernel");
    return MK_OK;
}

static int integrate(const double *s0_dev, int64_t npx, double bhspin, const mk_step_policy *policy, double *rows_dev,
                     double *dt_dev, int32_t *K_dev, int32_t *why_dev, double *state_dev, void *stream) {
    MK_REQUIRE(s0_dev && policy && K_dev && why_dev && state_dev, MK_ERR_ARG, "mk_integrate: null pointer");
    MK_REQUIRE(npx >= 0 && policy->nmax >= 0, MK_ERR_ARG, "mk_integrate: negative size");
    if (npx == 0) return MK_OK;
    cudaStream_t st = as_stream(stream);
    const int rpw = rays_per_warp(npx);
    if (policy->kind == MK_POLICY_REFERENCE) {
        const auto kernel = rows_dev || dt_dev ? integrate_reference_kernel<true> : integrate_reference_kernel<false>;
        kernel<<<ray_grid(npx, rpw), GEO_THREADS, 0, st>>>(
            s0_dev, npx, bhspin, spin_tri(bhspin), rule_tri(bhspin, policy->div, policy->tol),
            near_distance(policy->tol), policy->nmax, policy->div, policy->tol, rows_dev, dt_dev, K_dev, why_dev,
            state_dev, rpw, !tri_policy(*policy, bhspin));
        MK_LAUNCHED("integrate_reference_kernel");
    } else if (policy->kind == MK_POLICY_FIXED) {
        MK_REQUIRE(!rows_dev && !dt_dev, MK_ERR_UNSUPPORTED, "mk_integrate: rows only for the reference policy");
        integrate_fixed_kernel<<<ray_grid(npx, rpw), GEO_THREADS, 0, st>>>(
            s0_dev, npx, bhspin, policy->nmax, policy->hfrac, policy->hmin, policy->hmax, policy->capture,
            policy->r_escape, K_dev, why_dev, state_dev, rpw, !tri_policy(*policy, bhspin));
        MK_LAUNCHED("integrate_fixed_kernel");
    } else {
        MK_REQUIRE(false, MK_ERR_ARG, "mk_integrate: unknown policy %d", (int)policy->kind);
    }
    return MK_OK;
}

extern "C" int mk_freeze_rows(const double *state_dev, const int32_t *K_dev, int64_t npx, int32_t nrows,
                              double *rows_dev, double *dt_dev, void *stream) {
    MK_REQUIRE(state_dev && K_dev, MK_ERR_ARG, "mk_freeze_rows: null pointer");
    MK_REQUIRE(npx >= 0 && nrows >= 0, MK_ERR_ARG, "mk_freeze_rows: negative size");
    if (npx == 0 || nrows == 0 || (!rows_dev && !dt_dev)) return MK_OK;
    // about 16 blocks an SM over (ray, row)
    const bool wide = (((uintptr_t)state_dev | (uintptr_t)rows_dev) & 15) == 0;
    const int64_t bx = std::min<int64_t>((npx * (wide ? 4 : 8) + 255) / 256, 65535);
    const int64_t by = std::max<int64_t>(1, std::min<int64_t>(nrows, (int64_t)device_sm_count() * 16 / bx));
    const dim3 grid((unsigned)bx, (unsigned)by);
    if (wide)
        freeze_rows_kernel<double2><<<grid, 256, 0, as_stream(stream)>>>(state_dev, K_dev, npx, nrows, rows_dev, dt_dev);
    else
        freeze_rows_kernel<double><<<grid, 256, 0, as_stream(stream)>>>(state_dev, K_dev, npx, nrows, rows_dev, dt_dev);
    MK_LAUNCHED("freeze_rows_kernel");
    return MK_OK;
}

extern "C" int mk_integrate_moving(const double *s0_dev, int64_t npx, double bhspin, const mk_step_policy *policy,
                                   double *rows_dev, double *dt_dev, int32_t *K_dev, int32_t *why_dev,
                                   double *state_dev, void *stream) {
    return integrate(s0_dev, npx, bhspin, policy, rows_dev, dt_dev, K_dev, why_dev, state_dev, stream);
}

extern "C" int mk_integrate(const double *s0_dev, int64_t npx, double bhspin, const mk_step_policy *policy,
                            double *rows_dev, double *dt_dev, int32_t *K_dev, int32_t *why_dev, double *state_dev,
                            void *stream) {
    const int rc = integrate(s0_dev, npx, bhspin, policy, rows_dev, dt_dev, K_dev, why_dev, state_dev, stream);
    if (rc != MK_OK || (!rows_dev && !dt_dev)) return rc;
    return mk_freeze_rows(state_dev, K_dev, npx, policy->nmax, rows_dev, dt_dev, stream);
}

extern "C" int mk_radius_cal(const double *x_dev, int64_t npts, int64_t stride, double bhspin, double *r_dev,
                             void *stream) {
    MK_REQUIRE(x_dev && r_dev, MK_ERR_ARG, "mk_radius_cal: null pointer");
    MK_REQUIRE(npts >= 0 && stride >= 4, MK_ERR_ARG, "mk_radius_cal: bad size/stride");
    if (npts == 0) return MK_OK;
    radius_kernel<<<grid_for(npts, 256), 256, 0, as_stream(stream)>>>(x_dev, npts, stride, bhspin, r_dev);
    MK_LAUNCHED("radius_kernel");
    return MK_OK;
}

template <bool NEAR>
static int shadow(const char *name, const double *cos_dev, const double *sin_dev, const double *mid_dev, int64_t n,
                  double bhspin, double cos_inc, double sin_inc, double distance, int32_t max_steps, int32_t *K_dev,
                  int32_t *best_dev, double *best_dt_dev, double *r_km1_dev, double *r_best_dev, double *r_last_dev,
                  void *stream) {
    MK_REQUIRE(cos_dev && sin_dev && mid_dev && K_dev && best_dev && best_dt_dev && r_km1_dev && r_best_dev &&
                   r_last_dev,
               MK_ERR_ARG, "%s: null pointer", name);
    MK_REQUIRE(n >= 0 && max_steps >= 1, MK_ERR_ARG, "%s: bad sizes", name);
    if (n == 0) return MK_OK;
    const int rpw = rays_per_warp(n);
    shadow_pass_kernel<NEAR><<<ray_grid(n, rpw), GEO_THREADS, 0, as_stream(stream)>>>(
        cos_dev, sin_dev, mid_dev, n, bhspin, spin_tri(bhspin), rule_tri(bhspin, 40.0, 1e-2),
        near_distance(1e-2), cos_inc, sin_inc, distance, max_steps, K_dev, best_dev, best_dt_dev, r_km1_dev,
        r_best_dev, r_last_dev, rpw);
    MK_LAUNCHED("shadow_pass_kernel");
    return MK_OK;
}

extern "C" int mk_shadow_pass(const double *cos_dev, const double *sin_dev, const double *mid_dev, int64_t n,
                              double bhspin, double cos_inc, double sin_inc, double distance, int32_t max_steps,
                              int32_t *K_dev, int32_t *best_dev, double *best_dt_dev, double *r_km1_dev,
                              double *r_best_dev, double *r_last_dev, void *stream) {
    return shadow<true>("mk_shadow_pass", cos_dev, sin_dev, mid_dev, n, bhspin, cos_inc, sin_inc, distance, max_steps,
                        K_dev, best_dev, best_dt_dev, r_km1_dev, r_best_dev, r_last_dev, stream);
}

extern "C" int mk_shadow_sides(const double *cos_dev, const double *sin_dev, const double *mid_dev, int64_t n,
                               double bhspin, double cos_inc, double sin_inc, double distance, int32_t max_steps,
                               int32_t *K_dev, int32_t *best_dev, double *best_dt_dev, double *r_km1_dev,
                               double *r_best_dev, double *r_last_dev, void *stream) {
    return shadow<false>("mk_shadow_sides", cos_dev, sin_dev, mid_dev, n, bhspin, cos_inc, sin_inc, distance,
                         max_steps, K_dev, best_dev, best_dt_dev, r_km1_dev, r_best_dev, r_last_dev, stream);
}

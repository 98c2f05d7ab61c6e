// Host check of the FP32-pipe geodesic pieces (mk_tri.cuh) against long
// double: accel_pair's geodesic acceleration against one from sixth-order
// differences of the Kerr-Schild metric, relative to 2 f/r (|k^0| + |k|)^2,
// the size of its terms; t_radius against the closed form; the triple's sum,
// product and conversions.  Prints the largest of each.
#include <math.h>
#include <stdio.h>

#include <random>

#include "mk_tri.cuh"

typedef long double LD;
using mk::pr;
using mk::tri;

static LD L(pr v) { return (LD)v.h + v.l; }
static LD L(tri v) { return (LD)v.h + v.m + v.l; }

static LD radius(const LD x[4], LD a) {
    const LD kk = 0.5L * (x[1] * x[1] + x[2] * x[2] + x[3] * x[3] - a * a);
    return sqrtl(kk + sqrtl(kk * kk + a * a * x[3] * x[3]));
}
static void kerr(const LD x[4], LD a, LD &f, LD l[4]) {
    const LD r = radius(x, a), rr = r * r;
    f = 2 * rr * r / (rr * rr + a * a * x[3] * x[3]);
    l[0] = 1;
    l[1] = (r * x[1] + a * x[2]) / (rr + a * a);
    l[2] = (r * x[2] - a * x[1]) / (rr + a * a);
    l[3] = x[3] / r;
}
// -Gamma^mu_ab k^a k^b; g = eta + f l l, its inverse eta - f l l (raised l)
static void accel(const LD x[4], const LD k[4], LD a, LD out[4]) {
    LD D[4][4][4] = {};  // d_c g_ab
    const LD h = 1e-3L * radius(x, a);
    for (int c = 1; c < 4; c++)
        for (int s = 1; s <= 3; s++) {
            const LD w[4] = {0, 0.75L, -0.15L, 1.0L / 60};
            for (int sign = -1; sign <= 1; sign += 2) {
                LD y[4] = {x[0], x[1], x[2], x[3]}, f, l[4];
                y[c] += sign * s * h;
                kerr(y, a, f, l);
                for (int i = 0; i < 4; i++)
                    for (int j = 0; j < 4; j++) D[c][i][j] += sign * w[s] / h * f * l[i] * l[j];
            }
        }
    LD low[4], f, l[4];
    for (int m = 0; m < 4; m++) {
        low[m] = 0;
        for (int i = 0; i < 4; i++)
            for (int j = 0; j < 4; j++) low[m] -= (D[i][m][j] - 0.5L * D[m][i][j]) * k[i] * k[j];
    }
    kerr(x, a, f, l);
    const LD dot = -l[0] * low[0] + l[1] * low[1] + l[2] * low[2] + l[3] * low[3];
    for (int m = 0; m < 4; m++) out[m] = (m ? 1 : -1) * (low[m] - f * l[m] * dot);
}

int main() {
    std::mt19937_64 g(7);
    std::uniform_real_distribution<double> U(-1, 1);
    LD worst_a = 0, worst_r = 0, worst_add = 0, worst_mul = 0;
    int round_trip = 1, n = 0;
    const double spins[4] = {0.0, 0.5, 0.94, -0.998};
    for (int t = 0; t < 40000; t++) {
        const double a = spins[t & 3], scale = pow(10.0, 0.1 + 2.95 * fabs(U(g)));
        double v[4] = {0, scale * U(g), scale * U(g), scale * U(g)}, kv[4];
        if (t % 16 == 0) v[3] = 0.0;  // the equator
        for (int i = 0; i < 4; i++) kv[i] = U(g) * (t % 3 ? 1.0 : 100.0);
        tri X[4], K[4];
        LD x[4], k[4], kn = 0;
        for (int i = 0; i < 4; i++) {
            X[i] = mk::t_from(v[i]);
            K[i] = mk::t_from(kv[i]);
            if (mk::t_to(X[i]) != v[i]) round_trip = 0;
            x[i] = L(mk::t_pair(X[i]));  // what the pairs are given
            k[i] = L(mk::t_pair(K[i]));
            if (i) kn += k[i] * k[i];
        }
        const mk::SpinTri s = mk::spin_tri(a);
        const LD as = L(s.a), r = radius(x, as);
        if (r < 1.0L + sqrtl(1 - as * as)) continue;
        ++n;
        pr A[4];
        mk::PairPoint o;
        mk::accel_pair(mk::t_pair(X[1]), mk::t_pair(X[2]), mk::t_pair(X[3]), mk::t_pair(K[0]), mk::t_pair(K[1]),
                       mk::t_pair(K[2]), mk::t_pair(K[3]), s.a, s.aa, A, o);
        LD ref[4], f, l[4];
        accel(x, k, as, ref);
        kerr(x, as, f, l);
        const LD size = 2 * f / r * (fabsl(k[0]) + sqrtl(kn)) * (fabsl(k[0]) + sqrtl(kn));
        for (int i = 0; i < 4; i++) worst_a = fmaxl(worst_a, fabsl(L(A[i]) - ref[i]) / size);
        const LD xf[4] = {0, v[1], v[2], v[3]}, rf = radius(xf, sqrtl((LD)(a * a)));
        worst_r = fmaxl(worst_r, fabsl(L(mk::t_radius(X[1], X[2], X[3], s.aa3, o.r, o.iq, o.ir)) - rf) / rf);
        worst_add = fmaxl(worst_add, fabsl(L(mk::t_add(X[1], K[1])) - (L(X[1]) + L(K[1]))) / (fabsl(L(X[1])) + fabsl(L(K[1]))));
        worst_mul = fmaxl(worst_mul, fabsl(L(mk::t_mulr(X[1], K[1])) - L(X[1]) * L(K[1])) / fabsl(L(X[1]) * L(K[1])));
    }
    printf("%d %Lg %Lg %Lg %Lg %d\n", n, worst_a, worst_r, worst_add, worst_mul, round_trip);
    return 0;
}

"""Writes wide.npz: end states of captured rays, and the radii at which those of
a polar camera are captured, in more than binary64, for the tests that ask how
far from the exact trajectory a binary64 result is.

The integrator is the oracle's C source (oracle/mk_oracle.c) with `double`
compiled as `long double` (64 bits of significand on x86-64, 113 on aarch64)
and its literals and library calls to match.  Each state is stored as the sum
of two doubles.  Run from the repository's root: python tests/golden/make_wide.py
"""

import ctypes
import os
import re
import subprocess
import sys
import tempfile

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
CASES = ((0.0, 1e-4), (0.5, 1e-2), (0.94, 1e-2), (0.94, 1e-4), (0.998, 1e-4))  # spin, tol
# spin, inclination, distance, then the step rule: div, or hfrac of the fixed-fraction rule
RULES = ((0.5, 60.0, 1000.0, "div", 2.0), (0.94, 60.0, 1000.0, "div", 10.0), (0.5, 60.0, 1000.0, "hfrac", 0.05),
         (0.94, 85.0, 1000.0, "hfrac", 0.05), (0.5, 60.0, 100.0, "hfrac", 0.1), (0.94, 90.0, 1000.0, "hfrac", 0.1),
         (0.5, 60.0, 100.0, "hfrac", 0.5), (0.94, 60.0, 100.0, "hfrac", 0.02))
CALLS = "sqrt cbrt exp pow sin cos acos fabs fmin fmax fmod floor copysign".split()


def wide_library(directory):
    src = open(os.path.join(ROOT, "oracle", "mk_oracle.c")).read()
    head, body = src.split("#include <string.h>", 1)
    for name in "dadd dsub dmul ddiv dsqrt dsq dscale".split():   # names the C library takes for itself
        body = re.sub(r"\b%s\b" % name, "dual_" + name, body)
    body = re.sub(r"(?<![\w.])(\d+\.\d*(?:e[+-]?\d+)?|\d+e[+-]?\d+)(?![\w.])", r"\1L", body)
    defs = "#define double long double\n" + "".join("#define %s %sl\n" % (c, c) for c in CALLS)
    c = os.path.join(directory, "wide.c")
    with open(c, "w") as f:
        f.write(head + "#include <string.h>\n" + defs + body)
    lib = os.path.join(directory, "libwide.so")
    subprocess.run(["gcc", "-O2", "-std=c11", "-D_GNU_SOURCE", "-fopenmp", "-ffp-contract=off", "-shared", "-fPIC", c,
                    "-o", lib, "-lm"], check=True)
    return ctypes.CDLL(lib)


def end_states(lib, s0, N, div, tol, spin):
    """K and the state after K steps of the reference's rule, in long double."""
    s = np.ascontiguousarray(s0, dtype=np.longdouble)
    n, state = len(s), np.empty(s.shape, np.longdouble)
    K, why = np.empty(n, np.int32), np.empty(n, np.int32)
    lib.orc_integrate(s.ctypes.data_as(ctypes.c_void_p), n, N, ctypes.c_longdouble(div), ctypes.c_longdouble(tol),
                      ctypes.c_longdouble(spin), None, None, K.ctypes.data_as(ctypes.c_void_p),
                      why.ctypes.data_as(ctypes.c_void_p), state.ctypes.data_as(ctypes.c_void_p))
    return K, why, state


def fixed_end_states(lib, s0, N, hfrac, spin):
    """Steps and last state of the fixed-fraction rule, in long double."""
    s = np.ascontiguousarray(s0, dtype=np.longdouble)
    n, state = len(s), np.empty(s.shape, np.longdouble)
    K, why = np.empty(n, np.int32), np.empty(n, np.int32)
    numbers = [ctypes.c_longdouble(v) for v in (spin, hfrac, 0.01, 10.0, 1.01, 1000.0)]
    lib.orc_trace_fixed(s.ctypes.data_as(ctypes.c_void_p), n, N, *numbers, state.ctypes.data_as(ctypes.c_void_p),
                        K.ctypes.data_as(ctypes.c_void_p), why.ctypes.data_as(ctypes.c_void_p))
    return K, why, state


def polar_camera(oracle, ang, rad, spin):
    s0 = np.empty((len(ang), 8))
    ci, si = oracle.inclination_cos_sin(60.0)
    c, s, r = (np.ascontiguousarray(v) for v in (np.cos(ang), np.sin(ang), rad))
    p = lambda v: v.ctypes.data_as(ctypes.c_void_p)
    d = ctypes.c_double
    oracle.lib().orc_camera_polar(p(c), p(s), p(r), len(r), d(ci), d(si), d(1000.0), d(spin), p(s0))
    return s0


def radius(x, a):
    R2 = x[1] ** 2 + x[2] ** 2 + x[3] ** 2 - a ** 2
    return np.sqrt((R2 + np.sqrt(R2 ** 2 + 4 * a ** 2 * x[3] ** 2)) / 2)


def main():
    sys.path.insert(0, ROOT)
    import oracle
    out = {}
    with tempfile.TemporaryDirectory() as d:
        lib = wide_library(d)
        for i, (spin, tol) in enumerate(CASES):
            s0 = oracle.initialize_geodesics_at_camera(spin, 60.0, 1000, -10, 10, 20)
            K, why, state = end_states(lib, s0, 4000, 40.0, tol, spin)
            keep = np.flatnonzero((why == oracle.ST_CAPTURED) & (K == oracle.integrate(s0, 4000, 40.0, tol, spin)["K"]))[:40]
            hi = state[keep].astype(np.float64)
            out.update({f"s0_{i}": s0[keep], f"K_{i}": K[keep], f"hi_{i}": hi,
                        f"lo_{i}": (state[keep] - hi).astype(np.float64), f"spin_{i}": spin, f"tol_{i}": tol})
            if spin < 0.9 or tol != 1e-4:
                continue
            # radii of select_photons_integrator: row argmax(dt) - 1 = K - 1 of captured rays
            rng = np.random.default_rng(i)
            ang, rad = rng.uniform(0, 2 * np.pi, 300), rng.uniform(0.5, 4.5, 300)
            s0 = polar_camera(oracle, ang, rad, spin)
            K, why, _ = end_states(lib, s0, 2000, 40.0, 1e-2, spin)
            keep = np.flatnonzero(why == oracle.ST_CAPTURED)
            r = np.empty(len(keep), np.longdouble)
            for j, p in enumerate(keep):
                x = end_states(lib, s0[p:p + 1], int(K[p]) - 1, 40.0, 1e-2, spin)[2][0]
                r[j] = radius(x, np.longdouble(spin))
            hi = r.astype(np.float64)
            out.update({f"angle_{i}": ang[keep], f"radius_{i}": rad[keep], f"r_hi_{i}": hi,
                        f"r_lo_{i}": (r - hi).astype(np.float64)})
        for i, (spin, inc, distance, rule, value) in enumerate(RULES):
            s0 = oracle.initialize_geodesics_at_camera(spin, inc, distance, -10, 10, 14)
            if rule == "div":
                K, why, state = end_states(lib, s0, 4000, value, 1e-4, spin)
                same = K == oracle.integrate(s0, 4000, value, 1e-4, spin)["K"]
            else:
                K, why, state = fixed_end_states(lib, s0, 4000, value, spin)
                same = K == oracle.trace_fixed(s0, 4000, spin, hfrac=value)["nsteps"]
            keep = np.flatnonzero((why == oracle.ST_ESCAPED) & same)[:100]
            hi = state[keep].astype(np.float64)
            out.update({f"rule_s0_{i}": s0[keep], f"rule_K_{i}": K[keep], f"rule_hi_{i}": hi,
                        f"rule_lo_{i}": (state[keep] - hi).astype(np.float64), f"rule_spin_{i}": spin,
                        f"rule_{i}": rule, f"rule_value_{i}": value})
    np.savez_compressed(os.path.join(os.path.dirname(os.path.abspath(__file__)), "wide.npz"), **out)


if __name__ == "__main__":
    main()

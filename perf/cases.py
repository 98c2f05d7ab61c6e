"""Performance cases of the imaging path: what a user's program has it do.

Each case is one call sequence through the public Python entry points, at
the sizes of this package's workloads (``mahakala_gb300/configs.py``), its
tests and its benchmark, and at generic sizes between them:

* ``image``      one ``make_image`` call, the image back in host memory;
* ``batch``      several requests in one ``render_requests`` launch;
* ``geodesics``  the trajectories of a camera's rays
  (``geodesic_integrator``), the head of the step-by-step sequence a
  notebook runs;
* ``vacuum``     end states under the fixed-fraction step rule (``trace``);
* ``shadow``     the shadow outline by bisection (``find_shadow_bisection``);
* ``fluid``      ``get_fluid_scalars_from_geodesics`` over trajectories;
* ``radiation``  electron temperature, synchrotron coefficients and the
  transfer solve over (steps, pixels) arrays, the tail of that sequence;
* ``load``       a snapshot's host arrays made resident on the GPU.

``exact`` evaluates the same quantities in plain torch, in 64 bits and
without this package's compute code (the package's generator of synthetic
snapshots supplies the input arrays of both).
"""

import functools
import math

import numpy as np
import torch

import mahakala_gb300 as mk
from mahakala_gb300 import configs, electrons, geodesics
from mahakala_gb300.grmhd.athenak import AthenakFluidModel
from mahakala_gb300.grmhd.synthetic import make_multilevel_snapshot, make_synthetic_snapshot
from mahakala_gb300.images import RenderRequest, make_image, render_requests

MSUN = 1.989e33
M_BH = 6.5e9 * MSUN
GAMMA = 13.0 / 9.0
EXTENT = 50.0
SPINS = (0.0, 0.5, 0.94)


# ------------------------------------------------------------------ cases
def listed():
    return [
        # a preview of a view in the plain form: few rays, so one ray's chain
        # of steps and the call's own overhead are what the user waits for
        dict(name="image_fp64_24", kind="image", precision="fp64", resolution=24, nfreq=1, fov=20.0, blocks=8),
        # the plain form's render of the standard 256^3-cell workload
        dict(name="image_fp64_256", kind="image", precision="fp64", resolution=256, nfreq=1, fov=50.0, blocks=16),
        # an odd-sized thumbnail in the fast form
        dict(name="image_mixed_63", kind="image", precision="mixed", resolution=63, nfreq=1, fov=30.0, blocks=8),
        # the standard workload in the fast form
        dict(name="image_mixed_256", kind="image", precision="mixed", resolution=256, nfreq=1, fov=50.0, blocks=16),
        # a publication-size image at three frequencies in one pass
        dict(name="image_mixed_1024", kind="image", precision="mixed", resolution=1024, nfreq=3, fov=80.0, blocks=16),
        # a server's batch: requests of several sizes, spins, views and
        # frequencies over two resident snapshots in one launch
        dict(name="batch_mixed_12", kind="batch", precision="mixed", requests=12, mix=5, largest=256, blocks=8),
        # trajectories of a small camera for the step-by-step sequence, with
        # the notebooks' limit of 10000 steps
        dict(name="geodesics_40", kind="geodesics", pixels=40, steps=10000, fov=20.0, bhspin=0.0, inclination=60.0),
        # the vacuum shadow test: end states, stop reasons and step counts (these
        # two cases take little or no spin: around a fast-spinning hole a captured
        # ray winds about the horizon, and its last states are not determined to
        # six digits by 64-bit arithmetic)
        dict(name="vacuum_128", kind="vacuum", pixels=128, steps=4096, fov=20.0, bhspin=0.0),
        # the outline of a shadow at 48 angles
        dict(name="shadow_48", kind="shadow", angles=48, steps=2000),
        # sampling a camera's trajectories (most points lie outside the
        # snapshot, as along any camera ray)
        dict(name="fluid_400x96", kind="fluid", rows=400, pixels=96, blocks=8, levels=1),
        # coefficients and transfer along a default-size camera's trajectories
        dict(name="radiation_500x160", kind="radiation", rows=500, pixels=160),
        # loading a 128^3-cell snapshot
        dict(name="load_128", kind="load", blocks=8, cells=16, levels=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("image", "image", "image", "batch", "geodesics", "vacuum", "shadow", "fluid", "radiation",
                       "load"))
    if kind == "image":
        precision = rng.choice(("fp64", "mixed"))
        res = _log_int(rng, 8, 256) if precision == "fp64" else _log_int(rng, 16, 1024)
        return dict(kind=kind, precision=precision, resolution=res, nfreq=rng.choice((1, 1, 2, 3)),
                    fov=round(rng.uniform(16.0, 80.0), 1), blocks=rng.choice((4, 8)))
    if kind == "batch":
        precision = rng.choice(("fp64", "mixed"))
        return dict(kind=kind, precision=precision, requests=rng.randint(2, 20), mix=rng.randrange(1000),
                    largest=_log_int(rng, 16, 64) if precision == "fp64" else _log_int(rng, 32, 256), blocks=8)
    if kind == "geodesics":
        return dict(kind=kind, pixels=rng.randint(5, 48), steps=_log_int(rng, 300, 10000),
                    fov=round(rng.uniform(12.0, 50.0), 1), bhspin=rng.choice((0.0, 0.1, 0.2)),
                    inclination=round(rng.uniform(10.0, 85.0), 1))
    if kind == "vacuum":
        return dict(kind=kind, pixels=_log_int(rng, 8, 128), steps=4096, fov=round(rng.uniform(12.0, 50.0), 1),
                    bhspin=0.0)
    if kind == "shadow":
        return dict(kind=kind, angles=rng.randint(7, 48), steps=2000)
    if kind == "fluid":
        return dict(kind=kind, rows=_log_int(rng, 1, 500), pixels=_log_int(rng, 5, 128), blocks=rng.choice((4, 8)),
                    levels=rng.choice((1, 1, 2)))
    if kind == "radiation":
        return dict(kind=kind, rows=_log_int(rng, 2, 800), pixels=_log_int(rng, 5, 200))
    return dict(kind=kind, blocks=rng.choice((2, 4, 6, 8)), cells=rng.choice((4, 8, 12, 16)),
                levels=rng.choice((1, 1, 2)))


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=8)
def _snapshot(blocks, cells, levels, seed):
    """Host arrays of a synthetic snapshot; two levels: the central blocks refined once."""
    if levels == 1:
        return make_synthetic_snapshot(nblocks=blocks, cells_per_block=cells, extent=EXTENT, seed=seed)
    c = (blocks // 2 - 1, blocks // 2)
    return make_multilevel_snapshot(nblocks=blocks, cells_per_block=cells, extent=EXTENT, seed=seed,
                                    refine=[(0, i, j, k) for i in c for j in c for k in c])


def _device():
    return torch.device("cuda") if torch.cuda.is_available() else torch.device("cpu")


def _view(rng, nfreq):
    """A view of the torus: spin, inclination, electron model, frequencies and a
    density scale that keeps the explicit transfer stable."""
    inc, r_high = float(rng.uniform(10.0, 85.0)), float(np.exp(rng.uniform(0.0, np.log(80.0))))
    freqs = [230e9] if nfreq == 1 else [86e9, 230e9, 345e9][:nfreq]
    return dict(bhspin=float(rng.choice(SPINS)), inclination=inc, r_high=r_high, freqs=freqs,
                mass_scale=configs.stable_mass_scale(r_high, inc, min(freqs)))


def _batch(case, rng):
    """The requests of a batch: sizes from the case, views from the generator."""
    sizes = np.random.default_rng(case["mix"])
    out = []
    for _ in range(case["requests"]):
        res = int(round(np.exp(sizes.uniform(np.log(8.0), np.log(case["largest"])))))
        v = _view(rng, int(sizes.integers(1, 4)))
        out.append(dict(v, resolution=res, fov=float(sizes.uniform(16.0, 80.0)), snapshot=int(sizes.integers(0, 2))))
    return out


def _turned_camera(case, rng, dev):
    """(pixels^2, 8) camera rays of the case's view from an azimuth of the
    generator's: other positions and directions, and (the hole being
    axisymmetric) trajectories of the same lengths."""
    x, k = _camera(case["bhspin"], case["inclination"], 1000.0, *_grid(case["pixels"], case["fov"] / 2.0, dev))
    t = float(rng.uniform(0.0, 2.0 * math.pi))
    turn = torch.tensor([[math.cos(t), -math.sin(t), 0.0], [math.sin(t), math.cos(t), 0.0], [0.0, 0.0, 1.0]],
                        dtype=torch.float64, device=dev)
    one = torch.ones_like(x[:1])
    return torch.cat([0.0 * one, turn @ x, one, turn @ k]).T.contiguous()


def _trajectory_points(case, rng, dev):
    """(rows, pixels^2, 8) points along straight camera lines with null
    wavevectors, spaced by the step rule (r - r_EH) / 40 from 1000 M on: the
    positions a trajectory visits, without an integrator."""
    n, a = case["pixels"], 0.94
    reh = 1.0 + math.sqrt(1.0 - a * a)
    inc = float(rng.uniform(10.0, 85.0)) * math.pi / 180
    grid = torch.linspace(-1.0, 1.0, 2 * n + 1, dtype=torch.float64, device=dev)[1::2] * float(rng.uniform(10.0, 40.0))
    X, Y = (g.reshape(-1) for g in torch.meshgrid(grid, grid, indexing="ij"))
    si, ci = math.sin(inc), math.cos(inc)
    s = torch.full_like(X, 1000.0)
    rows = []
    start = 200 if case["rows"] < 200 else 0  # a short run of rows lies near the hole
    for j in range(start + case["rows"]):
        x = torch.stack([s * si - Y * ci, X, Y * si + s * ci])
        r = _radius(x, a)
        if j >= start:
            rows.append(x)
        dt = (r - reh) / 40.0
        s = torch.where(dt * 40.0 < 1e-4, s, s - dt)
    x = torch.stack(rows, 1)
    k = _null(x, torch.tensor([si, 0.0, ci], dtype=torch.float64, device=dev)[:, None, None].expand_as(x), a)
    zero = torch.zeros_like(x[:1])
    return torch.cat([zero, x, zero + 1.0, k]).permute(1, 2, 0).contiguous()


def _radiation_inputs(case, seed, dev):
    """Fluid quantities along trajectories: log-normal about a torus' values,
    zero in the part outside the snapshot (where the electron model gives NaN
    and the coefficients are zero)."""
    rows, npx = case["rows"], case["pixels"] ** 2
    g = torch.Generator(device=dev)
    g.manual_seed(seed)

    def normal():
        return torch.randn((rows, npx), generator=g, dtype=torch.float64, device=dev)

    def uniform(lo, hi):
        return lo + (hi - lo) * torch.rand((rows, npx), generator=g, dtype=torch.float64, device=dev)

    inside = (torch.arange(rows, device=dev)[:, None] >= rows // 2).to(torch.float64)
    dens = inside * torch.exp(0.8 * normal())
    u = dens * uniform(0.01, 0.1)
    beta = 10.0 * torch.exp(0.5 * normal())
    Ne = 2.0e5 * dens
    B = inside * 8.0 * torch.exp(0.4 * normal())
    pitch = uniform(0.01, math.pi - 0.01)
    nu = 230e9 * uniform(0.4, 2.0)
    dt = -uniform(0.02, 1.0)
    dt[-2:] = 0.0
    return dict(dens=dens, u=u, beta=beta, Ne=Ne, B=B, pitch=pitch, nu=nu, dt=dt)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    dev = _device()
    if kind == "image":
        v = _view(rng, case["nfreq"])
        model = AthenakFluidModel(_snapshot(case["blocks"], 16, 1, 0), v["bhspin"], fluid_gamma=GAMMA)
        return dict(kind=kind, case=case, view=v, model=model)
    if kind == "batch":
        models = [AthenakFluidModel(_snapshot(case["blocks"], 16, 1, s), 0.94, fluid_gamma=GAMMA) for s in (0, 1)]
        reqs = [RenderRequest(models[q["snapshot"]], camera_inclination=q["inclination"], mass_scale=q["mass_scale"],
                              M_bh=M_BH, r_high=q["r_high"], observing_frequency=q["freqs"], fov=q["fov"],
                              resolution=q["resolution"], max_nsteps=8192, bhspin=q["bhspin"])
                for q in _batch(case, rng)]
        return dict(kind=kind, case=case, requests=reqs)
    if kind == "geodesics":
        return dict(kind=kind, case=case, s0=_turned_camera(case, rng, dev))
    if kind == "vacuum":  # the camera's rays are in hand; the call integrates them
        v = dict(_view(rng, 1), bhspin=case["bhspin"])
        s0 = mk.initialize_geodesics_at_camera(v["bhspin"], v["inclination"], 1000.0, -case["fov"] / 2,
                                               case["fov"] / 2, case["pixels"])
        return dict(kind=kind, case=case, view=v, s0=s0, policy=geodesics.step_policy(case["steps"], kind="fixed"))
    if kind == "shadow":
        return dict(kind=kind, case=case, view=_view(rng, 1))
    if kind == "fluid":
        model = AthenakFluidModel(_snapshot(case["blocks"], 16, case["levels"], 0), 0.94, fluid_gamma=GAMMA)
        return dict(kind=kind, case=case, model=model, S=_trajectory_points(case, rng, dev))
    if kind == "radiation":
        return dict(kind=kind, case=case, arrays=_radiation_inputs(case, seed, dev))
    arrs = make_multilevel_snapshot(nblocks=case["blocks"], cells_per_block=case["cells"], extent=EXTENT, seed=seed,
                                    refine=[(0, i, j, k) for i in (case["blocks"] // 2 - 1, case["blocks"] // 2)
                                            for j in (0, 1) for k in (0, 1)] if case["levels"] == 2 else ())
    return dict(kind=kind, case=case, arrays=arrs)


# -------------------------------------------------------------------- run
def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "image":
        v = state["view"]
        return make_image(state["model"], camera_inclination=v["inclination"], mass_scale=v["mass_scale"], M_bh=M_BH,
                          r_high=v["r_high"],
                          observing_frequency=v["freqs"] if len(v["freqs"]) > 1 else v["freqs"][0], fov=case["fov"],
                          resolution=case["resolution"], max_nsteps=8192, precision=case["precision"])
    if kind == "batch":
        return render_requests(state["requests"], precision=case["precision"])
    if kind == "geodesics":
        S, dt = mk.geodesic_integrator(case["steps"], state["s0"], 40, 1e-4, case["bhspin"])
        return dict(S=S, dt=dt)
    if kind == "vacuum":
        return geodesics.trace(state["s0"], state["view"]["bhspin"], state["policy"])
    if kind == "shadow":
        v = state["view"]
        angles, radii = mk.find_shadow_bisection(v["bhspin"], v["inclination"], case["angles"],
                                                 max_steps=case["steps"])
        return dict(angles=angles, radii=radii)
    if kind == "fluid":
        return state["model"].get_fluid_scalars_from_geodesics(state["S"])
    if kind == "radiation":
        q = state["arrays"]
        theta = electrons.rlow_rhigh_model(q["dens"], q["u"], q["beta"], r_low=1, r_high=40)
        em, ab = mk.synchrotron_coefficients(q["Ne"], theta, q["B"], q["pitch"], q["nu"], invariant=True,
                                             rescale_nu=1.0 / 230e9)
        return dict(theta=theta, em=em, ab=ab, I=mk.solve_specific_intensity(em, ab, q["dt"], L_UNIT))
    model = AthenakFluidModel(state["arrays"], 0.94, fluid_gamma=GAMMA)
    return dict(blocks=model.snapshot.blocks(), table=model.snapshot.table, faces=model.snapshot.faces)


def _image_work(rays, nfreq):
    # about 230 accepted steps a ray, 893 operations each, and 90 samples at
    # 379 operations and 41 for each further frequency; one stencil of cells a
    # sample stays cached, so the traffic is the touched cells (64 B a ray and
    # crossed cell column) and the image
    return dict(flops=rays * (230 * 893 + 90 * (379 + 41 * (nfreq - 1))), bytes=rays * (8 * nfreq + 128 * 32))


def work(case):
    kind = case["kind"]
    if kind == "image":
        return _image_work(case["resolution"] ** 2, case["nfreq"])
    if kind == "batch":
        parts = [_image_work(q["resolution"] ** 2, len(q["freqs"]))
                 for q in _batch(case, np.random.default_rng(0))]
        return dict(flops=sum(p["flops"] for p in parts), bytes=sum(p["bytes"] for p in parts))
    if kind == "geodesics":
        # every kept row is written; the longest ray keeps about 700
        n = case["pixels"] ** 2
        return dict(flops=n * 430 * 893, bytes=n * min(case["steps"], 700) * 72)
    if kind == "vacuum":
        n = case["pixels"] ** 2
        return dict(flops=n * 250 * 893, bytes=n * (64 + 64 + 8))
    if kind == "shadow":
        return dict(flops=case["angles"] * 14 * 450 * 893, bytes=case["angles"] * 14 * 64)
    if kind == "fluid":
        n = case["rows"] * case["pixels"] ** 2
        return dict(flops=n * 300, bytes=n * (64 + 40))
    if kind == "radiation":
        n = case["rows"] * case["pixels"] ** 2
        return dict(flops=n * 120, bytes=n * 8 * (4 + 6 + 3))
    nmb = case["blocks"] ** 3 + (56 if case["levels"] == 2 else 0)
    return dict(flops=0, bytes=nmb * 32 * (case["cells"] ** 3 + (case["cells"] + 2) ** 3))


# -------------------------------------------------- the same in plain torch
EE, CL, ME, MP, HPL, GNEWT = 4.8032e-10, 2.99792458e10, 9.1094e-28, 1.6726e-24, 6.6261e-27, 6.6743e-8
L_UNIT = GNEWT * M_BH / CL ** 2


def _radius(x, a):
    """Kerr-Schild radius of x (3, ...)."""
    q = (x * x).sum(0) - a * a
    return torch.sqrt((q + torch.sqrt(q * q + 4.0 * a * a * x[2] * x[2])) / 2.0)


def _metric(x, a):
    """(f, l_i) of g = eta + f l l at x (3, ...)."""
    r = _radius(x, a)
    rr, aa, z = r * r, a * a, x[2]
    f = 2.0 * rr * r / (rr * rr + aa * z * z)
    return f, torch.stack([(r * x[0] + a * x[1]) / (rr + aa), (r * x[1] - a * x[0]) / (rr + aa), z / r])


def _null(x, v, a):
    """v (3, ...) rescaled so that (1, v) is null."""
    f, l = _metric(x, a)
    lv = (l * v).sum(0)
    A, b, C = f - 1.0, f * lv, (v * v).sum(0) + f * lv * lv
    return v * ((-b + torch.sqrt(b * b - A * C)) / C)


def _accel(x, k0, k, a):
    """-Gamma^mu_ab k^a k^b from the derivatives of f and l, as (a^0, a^i)."""
    aa, z = a * a, x[2]
    e = torch.eye(3, dtype=x.dtype, device=x.device)[:, :, None]
    kk = 0.5 * ((x * x).sum(0) - aa)
    q = torch.sqrt(kk * kk + aa * z * z)
    rr = kk + q
    r = torch.sqrt(rr)
    dr = (rr * x + aa * z * e[2]) / (2.0 * r * q)
    den, s = rr * rr + aa * z * z, rr + aa
    f = 2.0 * rr * r / den
    df = f * (3.0 * dr / r - (4.0 * rr * r * dr + 2.0 * aa * z * e[2]) / den)
    l = torch.stack([(r * x[0] + a * x[1]) / s, (r * x[1] - a * x[0]) / s, z / r])
    dl = torch.stack([(dr * x[0] + r * e[0] + a * e[1] - 2.0 * r * dr * l[0]) / s,
                      (dr * x[1] + r * e[1] - a * e[0] - 2.0 * r * dr * l[1]) / s,
                      (e[2] - dr * l[2]) / r])            # (component j, derivative c, n)
    lv = k0 + (l * k).sum(0)
    Dl = (dl * k[None]).sum(1)
    dlk = (dl * k[:, None]).sum(0)
    Dlk = (Dl * k).sum(0)
    F0 = -((k * df).sum(0) * lv + f * Dlk)
    F = l * F0 + f * lv * (dlk - Dl) + 0.5 * df * lv * lv
    lF = (l * F).sum(0) - F0
    return f * lF - F0, F - f * l * lF


class _Rays:
    """RK4 rays (x^mu, k^mu) in 64 bits; the state's rounding errors are carried along."""

    def __init__(self, x, k, a):
        self.a = a
        one = torch.ones_like(x[:1])
        self.y = torch.cat([0.0 * one, x, one, k])
        self.lo = torch.zeros_like(self.y)

    def _f(self, y):
        a0, ai = _accel(y[1:4], y[4], y[5:], self.a)
        return torch.cat([y[4:], a0[None], ai])

    def step(self, dt):
        y = self.y
        f1 = self._f(y)
        f2 = self._f(y + 0.5 * dt * f1)
        f3 = self._f(y + 0.5 * dt * f2)
        f4 = self._f(y + dt * f3)
        d = dt * (f1 + 2.0 * (f2 + f3) + f4) / 6.0 + self.lo
        new = y + d
        v = new - y
        return new, (y - (new - v)) + (d - v)

    def take(self, new, ok):
        self.y = torch.where(ok, new[0], self.y)
        self.lo = torch.where(ok, new[1], self.lo)

    def keep(self, idx):
        self.y, self.lo = self.y[:, idx], self.lo[:, idx]


def _rule(r, a, div, tol):
    """Step size of the reference rule, 0 where the ray stops."""
    d = r - (1.0 + math.sqrt(1.0 - a * a))
    dt = -d / div
    return torch.where((d.abs() >= tol) & (d.abs() <= 1500.0), dt, torch.zeros_like(dt))


def _camera(a, inc, d, X, Y):
    """Camera rays at image-plane points (X, Y): positions and null directions."""
    ci, si = float(np.cos(inc * np.pi / 180)), float(np.sin(inc * np.pi / 180))

    def place(x, y):
        return torch.stack([-y * ci + 0.0 * si + d * si, x, y * si + 0.0 * ci + d * ci])

    org, ini = place(torch.zeros_like(X), torch.zeros_like(Y)), place(X, Y)
    p, q = org - ini, place(X + Y, Y - X) - ini
    # products and differences rounded one by one, as the reference rounds them:
    # the direction's rounding moves a ray by 1e-10 over the 1000 M to the hole
    v = torch.stack([p[1] * q[2] - p[2] * q[1], p[2] * q[0] - p[0] * q[2], p[0] * q[1] - p[1] * q[0]])
    return ini, _null(ini, v, a)


def _grid(n, half, dev):
    c = torch.as_tensor(np.linspace(-half, half, 2 * n + 1)[1::2], device=dev)
    return (g.reshape(-1) for g in torch.meshgrid(c, c, indexing="ij"))


@functools.lru_cache(maxsize=2)
def _global_cells(blocks, seed):
    """The snapshot's cells as one zero-padded (8, n+2, n+2, n+2) float32 array."""
    arrs = _snapshot(blocks, 16, 1, seed)
    n = 16 * blocks
    g = np.concatenate([arrs.uov, arrs.B]).reshape(8, blocks, blocks, blocks, 16, 16, 16)
    g = g.transpose(0, 1, 4, 2, 5, 3, 6).reshape(8, n, n, n)
    return torch.nn.functional.pad(torch.as_tensor(np.ascontiguousarray(g)), (1, 1) * 3)


def _primitives(cells, x):
    """Trilinear primitives (8, n) at x (3, n), zero outside the grid."""
    n = cells.shape[1] - 2
    w = 2.0 * EXTENT / n
    inside = ((x > -EXTENT) & (x <= EXTENT)).all(0)
    t = torch.where(inside, (x + EXTENT) / w + 0.5, torch.ones_like(x))
    i = torch.floor(t).clamp(0, n)
    d = t - i
    i = i.long()
    flat = cells.reshape(8, -1)
    at = (i[2] * (n + 2) + i[1]) * (n + 2) + i[0]
    v = [flat[:, at + c * (n + 2) ** 2 + b * (n + 2) + a].double() for c in (0, 1) for b in (0, 1) for a in (0, 1)]
    v = [p + (q - p) * d[0] for p, q in zip(v[::2], v[1::2])]
    v = [p + (q - p) * d[1] for p, q in zip(v[::2], v[1::2])]
    return torch.where(inside, v[0] + (v[1] - v[0]) * d[2], torch.zeros_like(v[0])), inside


def _frame(p, x, k0, k, a):
    """dens, u, pitch angle, k.u and |b| from primitives p (8, n)."""
    f, l = _metric(x, a)
    U, Bi = p[1:4], p[5:8]
    alpha = 1.0 / torch.sqrt(1.0 + f)
    gamma = torch.sqrt(1.0 + (U * U).sum(0) + f * (l * U).sum(0) ** 2)
    u0, ui = gamma / alpha, U - gamma * alpha * f * l

    def lower(v0, vi):
        s = f * (v0 + (l * vi).sum(0))
        return s - v0, vi + l * s

    ud0, ud = lower(u0, ui)
    b0 = (Bi * ud).sum(0)
    bi = (Bi + ui * b0) / u0
    bd0, bd = lower(b0, bi)
    kdotu = k0 * ud0 + (k * ud).sum(0)
    b = torch.sqrt(b0 * bd0 + (bi * bd).sum(0))
    c = (k0 * bd0 + (k * bd).sum(0)) / (kdotu.abs() * b)
    c = torch.where(c.isnan(), torch.full_like(c, math.cos(math.pi / 3.0)), c).clamp(-1.0, 1.0)
    return p[0], p[4], torch.acos(c), kdotu, b


def _theta(dens, u, beta, r_low, r_high):
    g, i = 4.0 / 3 - 1.0, 5.0 / 3 - 1.0
    T = (r_high * beta ** 2 + r_low) / (1.0 + beta ** 2)
    return MP * u * g * i / (dens * (i + g * T)) / ME


def _synchrotron(Ne, th, B, pitch, nu, rescale):
    nus = 2.0 / 9.0 * (EE * B / (2.0 * math.pi * ME * CL)) * th ** 2 * torch.sin(pitch)
    X = nu / nus
    f = (X ** 0.5 + 2.0 ** (11.0 / 12) * X ** (1.0 / 6)) ** 2
    em = math.sqrt(2.0) * math.pi * EE ** 2 * Ne * nus / (3.0 * CL) * f * torch.exp(-X ** (1.0 / 3)) / (2.0 * th ** 2)
    em = torch.where((X > 1e12) | (th < 0.3), torch.zeros_like(em), em)
    ab = em / (2.0 * HPL * nu ** 3 / CL ** 2) * torch.expm1(HPL * nu / (ME * CL ** 2 * th))
    return torch.nan_to_num(em / (nu * rescale) ** 2, nan=0.0), torch.nan_to_num(ab * nu * rescale, nan=0.0)


def _exact_image(v, res, fov, blocks, seed, nmax=8192):
    dev = _device()
    cells = _global_cells(blocks, seed).to(dev)
    a = v["bhspin"]
    dens_unit = v["mass_scale"] / L_UNIT ** 3
    Ne_unit, B_unit = dens_unit / (MP + ME), CL * math.sqrt(4.0 * math.pi * dens_unit)
    X, Y = _grid(res, fov / 2.0, dev)
    rays = _Rays(*_camera(a, v["inclination"], 1000.0, X, Y), a)
    npx, nnu = res * res, len(v["freqs"])
    I = torch.zeros((nnu, npx), dtype=torch.float64, device=dev)
    Ia, Pa = torch.zeros_like(I), torch.ones_like(I)      # of the rays still moving
    idx = torch.arange(npx, device=dev)
    dt = _rule(_radius(rays.y[1:4], a), a, 40.0, 1e-4)
    for j in range(1, nmax):
        if j % 32 == 1:
            I[:, idx] = Ia
            on = torch.nonzero(dt != 0)[:, 0]
            if not len(on):
                break
            idx, dt, Ia, Pa = idx[on], dt[on], Ia[:, on], Pa[:, on]
            rays.keep(on)
        new = rays.step(dt)
        dtn = _rule(_radius(new[0][1:4], a), a, 40.0, 1e-4)
        ok = (dtn != 0) & (dt != 0)
        x, k0, k = new[0][1:4], new[0][4], new[0][5:]
        p, inside = _primitives(cells, x)
        dens, u, pitch, kdotu, b = _frame(p, x, k0, k, a)
        th = _theta(dens, u, u * (GAMMA - 1.0) * 2.0 / (b * b), 1.0, v["r_high"])
        lit = ok & inside & ~(b * b / dens > 100.0)
        w = -dt * L_UNIT
        for c, nu in enumerate(v["freqs"]):
            em, ab = _synchrotron(Ne_unit * dens, th, B_unit * b, pitch, -kdotu * nu, 1.0 / nu)
            em, ab = torch.where(lit, em, 0.0), torch.where(lit, ab, 0.0)
            Ia[c] += w * em * Pa[c]
            Pa[c] *= 1.0 - w * ab
        rays.take(new, ok)
        dt = torch.where(ok, dtn, torch.zeros_like(dtn))
    I[:, idx] = Ia
    I = I.reshape(nnu, res, res).cpu().numpy()
    return I


def _exact_rows(x, k, a, N, div, tol):
    """Trajectory rows (N_t, n, 8) and steps (N_t, n), kept to two rows past
    the last moving one as the integrator keeps them."""
    rays = _Rays(x, k, a)
    dt = _rule(_radius(x, a), a, div, tol)
    S, D = [], []
    while len(S) < N:
        new = rays.step(dt)
        dtn = _rule(_radius(new[0][1:4], a), a, div, tol)
        ok = (dtn != 0) & (dt != 0)
        S.append(rays.y)
        D.append(torch.where(ok, dt, torch.zeros_like(dt)))
        rays.take(new, ok)
        dt = torch.where(ok, dtn, torch.zeros_like(dtn))
        if len(S) % 16 == 0 and not bool(dt.any()):
            break
    moving = torch.stack([d.any() for d in D]).nonzero()
    nt = min(int(moving[-1]) + 3, N)
    while len(S) < nt:
        S.append(rays.y)
        D.append(torch.zeros_like(dt))
    return torch.stack(S[:nt]).permute(0, 2, 1), torch.stack(D[:nt])


def _exact_vacuum(v, case, dev):
    a, p = v["bhspin"], geodesics.step_policy(case["steps"], kind="fixed")
    reh = 1.0 + math.sqrt(1.0 - a * a)
    rays = _Rays(*_camera(a, v["inclination"], 1000.0, *_grid(case["pixels"], case["fov"] / 2.0, dev)), a)
    n = case["pixels"] ** 2
    state = torch.zeros((8, n), dtype=torch.float64, device=dev)
    idx = torch.arange(n, device=dev)
    r = _radius(rays.y[1:4], a)
    on = torch.ones(n, dtype=torch.bool, device=dev)
    for j in range(p.nmax):
        if j % 32 == 0:
            state[:, idx] = rays.y
            left = on.nonzero()[:, 0]
            if not len(left):
                break
            idx, r, on = idx[left], r[left], on[left]
            rays.keep(left)
        new = rays.step(-(p.hfrac * r).clamp(p.hmin, p.hmax))
        rn = _radius(new[0][1:4], a)
        rays.take(new, on)
        on = on & ~(rn.isnan() | (rn < p.capture * reh) | ((rn > p.r_escape) & (rn > r)))
        r = torch.where(on, rn, r)
    state[:, idx] = rays.y
    return dict(K=None, why=None, state=state.T)


def _exact_shadow(v, case, dev):
    a = v["bhspin"]
    angles = np.arange(case["angles"]) / case["angles"] * 2.0 * np.pi
    c, s = (torch.as_tensor(f(angles), device=dev) for f in (np.cos, np.sin))
    inner, outer = torch.full_like(c, 0.5), torch.full_like(c, 10.0)
    for _ in range(40):
        if float((outer - inner).max()) <= 1e-3:
            break
        mid = (outer - inner) / 2 + inner
        S, dt = _exact_rows(*_camera(a, v["inclination"], 1000.0, c * mid, s * mid), a, case["steps"], 40.0, 1e-2)
        row = dt.argmax(0) - 1
        row = torch.where(row < 0, row + len(dt), row)
        r = _radius(S.permute(2, 0, 1)[1:4], a).gather(0, row[None])[0]
        inner, outer = torch.where(r < 100, mid, inner), torch.where(r >= 100, mid, outer)
    close = lambda x: np.append(x, x[0])  # noqa: E731
    return dict(angles=close(angles), radii=close(inner.cpu().numpy()))


def exact(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    dev = _device()
    if kind == "image":
        I = _exact_image(_view(rng, case["nfreq"]), case["resolution"], case["fov"], case["blocks"], 0)
        return I[0] if case["nfreq"] == 1 else I
    if kind == "batch":
        if case["requests"] > 12:
            return None     # each image costs about a second
        return [_exact_image(q, q["resolution"], q["fov"], case["blocks"], q["snapshot"]) for q in _batch(case, rng)]
    if kind == "geodesics":
        s0 = _turned_camera(case, rng, dev).T
        S, dt = _exact_rows(s0[1:4], s0[5:], case["bhspin"], case["steps"], 40.0, 1e-4)
        return dict(S=S, dt=dt)
    if kind == "vacuum":
        return _exact_vacuum(dict(_view(rng, 1), bhspin=case["bhspin"]), case, dev)
    if kind == "shadow":
        return _exact_shadow(_view(rng, 1), case, dev)
    if kind == "fluid":
        if case["levels"] == 2:
            return None     # the refined mesh's ghost rules are the framework's own
        S = _trajectory_points(case, rng, dev)
        cells = _global_cells(case["blocks"], 0).to(dev)
        out = []
        for s in S.split(max(1, (1 << 20) // S.shape[1])):
            y = s.reshape(-1, 8).T
            p, _ = _primitives(cells, y[1:4])
            out.append([q.reshape(s.shape[:2]) for q in _frame(p, y[1:4], y[4], y[5:], 0.94)])
        dens, u, pitch, kdotu, b = (torch.cat(q) for q in zip(*out))
        return dict(dens=dens, u=u, pitch_angle=pitch, kdotu=kdotu, b=b)
    if kind == "radiation":
        q = _radiation_inputs(case, seed, dev)
        th = _theta(q["dens"], q["u"], q["beta"], 1.0, 40.0)
        em, ab = _synchrotron(q["Ne"], th, q["B"], q["pitch"], q["nu"], 1.0 / 230e9)
        I = torch.zeros_like(em[0])
        for j in range(len(em) - 1, 0, -1):
            I = I - q["dt"][j - 1] * L_UNIT * (em[j] - ab[j] * I)
        return dict(theta=th, em=em, ab=ab, I=I)
    return None

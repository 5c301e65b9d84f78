"""The work a user of this framework has it do, as cases to measure.

A case is one call sequence of a user's program on one grain (or one batch of
grains): self-consistency iterations, an LDOS postprocess, a free energy with
its gradients, or a batch of grains.  ``prepare`` makes what the program holds
before the call (the context and its seeded state), ``run`` makes one pass
through the public entry points, and ``exact`` computes the same outputs in
64 bits with plain torch (no code of this package), for discs and squares with
the accelerator's first step, which is what one pass on a new state takes.
"""
from __future__ import annotations

import ctypes
import json
import math

import numpy as np
import torch

import superconga_b200 as sb
from superconga_b200 import autograd, workloads

DEV = "cuda"
# Iterations of one pass of self-consistency work: the state a pass returns
# then holds one whole iteration's result, its residual and free energy another.
ITERATIONS = 2
CUTOFF = 8.0  # energy cutoff in units of 2 pi k_B T_c, as in the benchmark workloads
TIGHT_BINDING = {"type": "tight_binding", "hopping_nnn": -0.25, "hopping_nnnn": 0.0, "chemical_potential": 0.0}


def listed():
    return [
        # The smallest grain of a parameter study: launch latency and the
        # host path count, and the GPU is nearly empty.
        dict(name="small_disc_mixed", kind="solve", shape="disc", size=4.0, ppxi=10.0, angles=32, t=0.7, sym="s",
             field=0.05, kappa=2.0, mode="mixed"),
        # An ordinary s-wave disc in a field in plain double precision, the
        # form that users of the reference compare against.
        dict(name="disc_fp64", kind="solve", shape="disc", size=10.0, ppxi=10.0, angles=64, t=0.5, sym="s",
             field=0.02, kappa=2.0, mode="fp64"),
        # A square at a very low temperature: 81 Ozaki energies, in energy passes.
        dict(name="cold_square_mixed", kind="solve", shape="square", size=12.0, ppxi=8.0, angles=64, t=0.003,
             sym="dx2-y2", field=0.0, kappa=2.0, mode="mixed"),
        # Production size in both precisions: the benchmark's d-wave square of
        # side 30 xi0 with pair-breaking edges (14 energies, 256 angles).
        dict(name="square_fp64", kind="solve", shape="square", size=30.0, ppxi=20.0, angles=256, t=0.1,
             sym="dx2-y2", field=0.0, kappa=2.0, mode="fp64"),
        dict(name="square_mixed", kind="solve", shape="square", size=30.0, ppxi=20.0, angles=256, t=0.1,
             sym="dx2-y2", field=0.0, kappa=2.0, mode="mixed"),
        # A non-circular Fermi surface (per-angle Riccati step), ragged sizes.
        dict(name="tight_binding_mixed", kind="solve", shape="square", size=17.3, ppxi=11.0, angles=90, t=0.25,
             sym="dx2-y2", field=0.0, kappa=2.0, mode="mixed", surface="tight_binding"),
        # Density of states of a solved grain: blocks of 32 real energies, and
        # a small odd number of them in double precision.
        dict(name="ldos_square_mixed", kind="ldos", shape="square", size=40.0, ppxi=16.0, angles=128, t=0.5, sym="s",
             field=0.3, kappa=5.0, mode="mixed", energies=32, block=32),
        dict(name="ldos_disc_fp64", kind="ldos", shape="disc", size=10.0, ppxi=12.0, angles=64, t=0.3, sym="dx2-y2",
             field=0.05, kappa=2.0, mode="fp64", energies=33, block=20),
        # Free energy and edge current with their gradients (forward and
        # backward through torch.autograd): one small grain, and the chiral
        # two-component disc of the benchmark.
        dict(name="gradient_disc", kind="gradient", shape="disc", size=6.0, ppxi=10.0, angles=32, t=0.5, sym="s",
             field=0.02, kappa=2.0, mode="fp64"),
        dict(name="gradient_chiral", kind="gradient", shape="disc", size=15.0, ppxi=15.0, angles=128, t=0.3,
             sym="dx2-y2+dxy", field=0.05, kappa=2.0, mode="fp64"),
        # A parameter study: many grains of mixed shape, size, temperature and
        # field advanced together.
        dict(name="batch_mixed", kind="batch", grains=24, smallest=4.0, largest=14.0, ppxi=10.0, study=3,
             mode="mixed"),
        dict(name="batch_fp64", kind="batch", grains=8, smallest=4.0, largest=10.0, ppxi=10.0, study=5, mode="fp64"),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case: any kind, grains of 4 to 20 xi0 radius (8 to 40 xi0
    side) at 8 to 20 points/xi0, odd and even angle counts, T from 0.02 to
    0.9, with and without field, both precisions."""
    kind = rng.choice(["solve", "solve", "solve", "ldos", "gradient", "batch"])
    mode = "fp64" if kind == "gradient" else rng.choice(["mixed", "fp64"])
    if kind == "batch":
        return dict(kind=kind, grains=rng.randint(3, 20), smallest=4.0, largest=round(rng.uniform(6.0, 14.0), 2),
                    ppxi=round(rng.uniform(8.0, 12.0), 1), study=rng.randrange(1 << 20), mode=mode)
    shape = rng.choice(["disc", "square"])
    most = {"solve": 20.0, "ldos": 12.0, "gradient": 10.0}[kind]
    size = round(_log_uniform(rng, 4.0, most) * (1 if shape == "disc" else 2), 2)
    case = dict(kind=kind, shape=shape, size=size, ppxi=round(rng.uniform(8.0, 14.0), 1),
                angles=rng.choice([32, 45, 48, 62, 64, 81, 96, 128]), t=round(rng.uniform(0.1, 0.9), 3),
                sym=rng.choice(["s", "dx2-y2", "dx2-y2+dxy"]), field=rng.choice([0.0, round(rng.uniform(0.01, 0.1), 3)]),
                kappa=2.0, mode=mode)
    if kind == "solve" and rng.random() < 0.2:  # low temperatures: many Ozaki energies
        case.update(size=round(_log_uniform(rng, 4.0, 8.0) * (1 if shape == "disc" else 2), 2), t=round(_log_uniform(rng, 0.01, 0.1), 4))
    if kind == "solve" and rng.random() < 0.2:
        case.update(surface="tight_binding", sym=rng.choice(["s", "dx2-y2"]))
    if kind == "ldos":
        case.update(energies=rng.randint(9, 64), block=rng.choice([8, 16, 20, 32]))
    return case


# ------------------------------------------------------------ configurations --
def _symmetries(case):
    return [s for s in ("dx2-y2", "dxy", "g", "s") if s in case["sym"].split("+")]


def _config(case):
    """The case in the JSON schema of the framework."""
    radius = case["size"]
    if case["shape"] == "disc":
        geometry = [{"disc": {"add": True, "radius": radius, "center_x": 0.0, "center_y": 0.0}}]
        area = math.pi * radius ** 2
    else:
        geometry = [{"regular_polygon": {"add": True, "num_edges": 4, "side_length": radius, "rotation": 0.0,
                                         "center_x": 0.0, "center_y": 0.0}}]
        area = radius ** 2
    order = {s: {"critical_temperature": 1.0} for s in _symmetries(case)}
    if len(order) > 1:
        order["dxy"]["initial_phase_shift"] = 0.25
    physics = {"temperature": case["t"], "external_flux_quanta": case["field"] * area / math.pi,
               "penetration_depth": case["kappa"], "charge_sign": -1, "gauge": "symmetric",
               "crystal_axes_rotation": 0.125 if case["shape"] == "square" and case["sym"] == "dx2-y2" else 0.0,
               "order_parameter": order}
    if case.get("surface") == "tight_binding":
        physics["fermi_surface"] = TIGHT_BINDING
        physics["crystal_axes_rotation"] = 0.0
    return {
        "physics": physics, "geometry": geometry,
        "numerics": {"points_per_coherence_length": case["ppxi"], "num_fermi_momenta": case["angles"],
                     "energy_cutoff": CUTOFF, "convergence_criterion": 1e-30, "norm": "l2",
                     "vector_potential_error": 1e-6, "num_iterations_burnin": 0, "num_iterations_min": 0,
                     "num_iterations_max": -1},
        "accelerator": {"name": "congacc"},
        "misc": {"verbose": False, "save_path": "", "load_path": ""},
    }


def _spectroscopy(case):
    d0 = workloads.S_WAVE_BULK
    return {"spectroscopy": {"energy_min": -2.0 * d0, "energy_max": 2.0 * d0, "num_energies": case["energies"],
                             "energy_broadening": 0.05 * d0},
            "numerics": {"convergence_criterion": 1e-30, "norm": "l2", "num_energies_per_block": case["block"],
                         "num_fermi_momenta": case["angles"]}}


def _study(case):
    """The grains of a parameter study, spread as the benchmark's batch is."""
    rng = np.random.default_rng(case["study"])
    out = []
    for i in range(case["grains"]):
        disc = i % 2 == 0
        r = rng.uniform(case["smallest"], case["largest"])
        out.append(dict(kind="solve", shape="disc" if disc else "square", size=float(r if disc else 2 * r),
                        ppxi=case["ppxi"], angles=int(min(128, max(32, 32 * round(2 * r / 10.0)))),
                        t=float(rng.uniform(0.1, 0.9)), sym="s" if rng.uniform() < 0.5 else "dx2-y2",
                        field=float(rng.uniform(0.0, 0.1)), kappa=2.0, mode=case["mode"]))
    return out


def _inputs(case, n0, seed):
    """Seeded state: the bulk order parameter with a slowly varying phase and
    2% of noise, and a smooth induced vector potential.  delta [Nc][2][N0][N0]
    and a [2][N0][N0], float64 on the GPU."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    rnd = lambda *s: torch.rand(*s, generator=gen, device=DEV, dtype=torch.float64)  # noqa: E731
    nrm = lambda *s: torch.randn(*s, generator=gen, device=DEV, dtype=torch.float64)  # noqa: E731
    syms = _symmetries(case)
    u = torch.linspace(-0.5, 0.5, n0, device=DEV, dtype=torch.float64)
    yy, xx = torch.meshgrid(u, u, indexing="ij")

    def wave():
        p = rnd(6)
        return torch.cos(2 * math.pi * (2 * p[0] * xx + 2 * p[1] * yy + p[2])) + torch.cos(
            2 * math.pi * (3 * p[3] * xx + 3 * p[4] * yy + p[5]))

    phase = 0.5 * wave()
    delta = torch.empty(len(syms), 2, n0, n0, device=DEV, dtype=torch.float64)
    for c, s in enumerate(syms):
        z = workloads.delta_bulk(case["t"], s) * torch.complex(1 + 0.02 * nrm(n0, n0), 0.02 * nrm(n0, n0))
        z = z * torch.polar(torch.ones_like(phase), phase + (0.5 * math.pi * c))
        delta[c, 0], delta[c, 1] = z.real, z.imag
    a = torch.stack([0.02 * wave(), 0.02 * wave()])
    return delta.contiguous(), a.contiguous()


# ------------------------------------------------------------- prepare, run --
def prepare(case, seed):
    if case["kind"] == "batch":
        cases = _study(case)
        batch = sb.Batch([json.dumps(_config(c)) for c in cases], mode=case["mode"])
        outs = []
        for k, (c, g) in enumerate(zip(cases, batch.grains)):
            delta, a = _inputs(c, g.dims.n0, 1000 * seed + k)
            torch.cuda.synchronize()
            g.set_state_device(delta.data_ptr(), a.data_ptr())
            outs.append((torch.empty_like(delta), torch.empty_like(a)))
        torch.cuda.synchronize()
        return dict(case=case, batch=batch, outs=outs)
    cfg = _config(case)
    if case["kind"] == "ldos":
        ctx = sb.LdosContext(cfg, _spectroscopy(case), mode=case["mode"])
    else:
        ctx = sb.Context(cfg, mode=case["mode"])
    delta, a = _inputs(case, ctx.dims.n0, seed)
    torch.cuda.synchronize()
    ctx.set_state_device(delta.data_ptr(), a.data_ptr())
    state = dict(case=case, ctx=ctx)
    if case["kind"] == "solve":
        state["delta"], state["a"] = torch.empty_like(delta), torch.empty_like(a)
    elif case["kind"] == "ldos":
        state["ldos"] = torch.empty(case["energies"], ctx.dims.n0, ctx.dims.n0, device=DEV, dtype=torch.float64)
    else:
        ctx.boundary_initial()
        ctx.burn_in(1)
        state["delta"] = torch.complex(delta[:, 0], delta[:, 1]).requires_grad_()
        state["a"] = a.requires_grad_()
        state["b"] = torch.tensor(ctx.external_field(), dtype=torch.float64, device=DEV, requires_grad=True)
        state["beta"] = autograd.edge_current_weights(ctx.domain(), 1.0 / case["ppxi"], 2.0)
    torch.cuda.synchronize()
    return state


def run(state):
    kind = state["case"]["kind"]
    if kind == "solve":  # what runSimulation's loop asks for: iterate, look at the residual and the free energy
        ctx = state["ctx"]
        residual, _ = ctx.compute(ITERATIONS)
        ctx.get_state_device(state["delta"].data_ptr(), state["a"].data_ptr())
        return {"delta": state["delta"], "a": state["a"], "residual": residual,
                "free_energy": ctx.scalars()["free_energy"]}
    if kind == "ldos":  # every block: burn-in, two LDOS iterations
        ctx = state["ctx"]
        for b in range(ctx.n_blocks):
            ctx.begin_block(b)
            ctx.burn_in(1)
            ctx.iterate(2)
        sb._lib.check(sb.load().sc_ldos_get_device(ctx._h, ctypes.c_void_p(state["ldos"].data_ptr())), ctx._h)
        return {"ldos": state["ldos"]}
    if kind == "gradient":
        inputs = [state["delta"], state["a"], state["b"]]
        loss = autograd.FreeEnergy.apply(*inputs, state["ctx"], 1.0, state["beta"])
        grads = torch.autograd.grad(loss, inputs)
        return {"loss": loss.detach(), "g_delta": grads[0], "g_a": grads[1], "g_b": grads[2]}
    batch = state["batch"]
    batch.compute(ITERATIONS)
    for g, (delta, a) in zip(batch.grains, state["outs"]):
        g.get_state_device(delta.data_ptr(), a.data_ptr())
    _, _, residual = batch.status()
    return {"residual": residual, "delta": torch.cat([d.reshape(-1) for d, _ in state["outs"]]),
            "a": torch.cat([a.reshape(-1) for _, a in state["outs"]])}


# --------------------------------------------------------- work, tolerance --
# Arithmetic the path cannot do without: one Riccati midpoint step is about 80
# floating-point operations (three complex products, a complex square root, a
# complex division, counting a root or a quotient as one), the Green functions
# of one site and energy with their four sums about 50, shared by two steps;
# the reverse of a step about twice the step.
STEP_FLOPS, GREEN_FLOPS = 80.0, 50.0


def _updates(case, n_energies):
    """Site-updates of one iteration: two functions, every angle, energy and grain site."""
    area = math.pi * case["size"] ** 2 if case["shape"] == "disc" else case["size"] ** 2
    return 2.0 * n_energies * case["angles"] * area * case["ppxi"] ** 2


def _lattice_side(case):
    width = 2 * case["size"] if case["shape"] == "disc" else case["size"]
    return int(math.ceil(width * case["ppxi"])) + 6


def work(case):
    if case["kind"] == "batch":
        parts = [work(c) for c in _study(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n0, nc = _lattice_side(case), len(_symmetries(case))
    state = 8.0 * (2 * nc + 2) * n0 * n0
    per_update = STEP_FLOPS + 0.5 * GREEN_FLOPS
    if case["kind"] == "ldos":
        blocks = -(-case["energies"] // case["block"])
        su = _updates(case, case["block"]) * blocks
        return {"bytes": state + 8.0 * case["energies"] * n0 * n0, "flops": su * (STEP_FLOPS + 2 * (STEP_FLOPS + 10.0))}
    su = _updates(case, _pole_count(case["t"], CUTOFF))
    if case["kind"] == "gradient":
        return {"bytes": 2 * state, "flops": su * (per_update + STEP_FLOPS + 2 * STEP_FLOPS + GREEN_FLOPS)}
    return {"bytes": 2 * state, "flops": ITERATIONS * su * per_update}


def tolerance(case):
    """About four times what was measured on B200 between the framework and
    exact(), and between its packed and its scalar single-precision sweep over
    two passes (four iterations)."""
    if case["mode"] == "fp64":
        # 2e-14 for the vector potential of the largest square; the accelerator's
        # adaptive steps let rounding differences grow from pass to pass.
        return {"rel": 1e-12}
    if case["kind"] == "ldos":
        return {"rel": 4e-6}  # 8e-7 against exact()
    # Single-precision Riccati steps: 8e-5 in a batch's residuals and 2e-5 in
    # free energies, which are a cancellation of two terms (state: 1e-7 in the
    # order parameter, 5e-6 in A); 8e-4 in single values of A in a batch.
    return {"rel": 3e-4, "max": 4e-3}


# ------------------------------------------------------------------- exact --
# A plain restatement in 64 bits: every angle's grain rasterised in its
# trajectory frame, the midpoint Riccati recursion row by row over all columns
# and energies at once, Green sums, specular walls by interpolation over two
# angles and two columns, the separable-filter vector potential by matrix
# products, and the accelerator's first step (half of g(x) - x).  Rotations
# use single-precision sines and cosines, as the method defines them.
_LIBM = ctypes.CDLL("libm.so.6")
for _f in ("cosf", "sinf"):
    getattr(_LIBM, _f).restype = ctypes.c_float
    getattr(_LIBM, _f).argtypes = [ctypes.c_float]
F8, C16 = torch.float64, torch.complex128


def _trig32(angle):
    f = -np.float32(angle)
    return float(_LIBM.cosf(float(f))), float(_LIBM.sinf(float(f)))


def _wrap(v, lo, hi):
    if lo <= v < hi:
        return v
    s = (v - lo) / (hi - lo)
    return (s - math.floor(s)) * (hi - lo) + lo


def _poles(n):
    e = np.array([-0.5 / math.sqrt((2.0 * (i - 1) + 1.0) * (2.0 * i + 1.0)) for i in range(1, 2 * n)])
    w, z = np.linalg.eigh(np.diag(e, 1) + np.diag(e, -1))
    pole = -1.0 / w[:n]
    return pole, (0.5 * z[0, :n] * pole) ** 2


def _pole_count(t, cutoff):
    """The fewest Ozaki poles whose largest exceeds 2 pi cutoff / T; above 60
    poles a quadratic fit of that largest pole decides."""
    val = 2.0 * math.pi * (cutoff / t)
    if val < 9244.2425:
        n = 1
        while _poles(n)[0].max() <= val:
            n += 1
        return n
    i = 60
    while i * (2.5465 * i + 1.2744) + 0.4651 < val:
        i += 1
    return i


def _tight_binding(na, wts):
    t1, t2, mu = TIGHT_BINDING["hopping_nnn"], TIGHT_BINDING["hopping_nnnn"], TIGHT_BINDING["chemical_potential"]
    cos, sin = math.cos, math.sin

    def energy(x, y):
        return -2 * (cos(x) + cos(y)) - 4 * t1 * cos(x) * cos(y) - 2 * t2 * (cos(2 * x) + cos(2 * y)) - mu

    def grad(x, y):
        return (2 * sin(x) + 4 * t1 * sin(x) * cos(y) + 4 * t2 * sin(2 * x),
                2 * sin(y) + 4 * t1 * cos(x) * sin(y) + 4 * t2 * sin(2 * y))

    o = 0.0 if energy(0.0, math.pi) * energy(math.pi, math.pi) > 0 else math.pi
    out = []
    for k in range(na):
        ph = _wrap(math.pi * 2 * k / na + 0.5 * math.pi, 0.0, 2 * math.pi)
        ux, uy = cos(ph), sin(ph)
        lo, hi = 0.0, math.pi / max(abs(ux), abs(uy))
        e_lo = energy(o, o)
        for _ in range(60):
            mid = 0.5 * (lo + hi)
            if (energy(mid * ux + o, mid * uy + o) > 0) == (e_lo > 0):
                lo = mid
            else:
                hi = mid
        r = 0.5 * (lo + hi)
        px, py = _wrap(r * ux + o, -math.pi, math.pi), _wrap(r * uy + o, -math.pi, math.pi)
        vx, vy = grad(px, py)
        kx, ky = r * ux, r * uy
        out.append((px, py, vx, vy, abs((kx * kx + ky * ky) / (kx * vx + ky * vy)) * wts[k]))
    px, py, vx, vy, w = np.array(out).T
    theta = np.arctan2(vy, vx) - 0.5 * math.pi
    speed = np.sum(np.hypot(vx, vy) * w) / np.sum(w)
    return o, theta, px, py, vx / speed, vy / speed, w / np.sum(w)


def _filters(n0, h, max_error):
    i = np.arange(n0, dtype=np.float64)
    ii, jj = np.meshgrid(i, i, indexing="ij")
    q = np.zeros((n0, n0))
    for sj in (-1.0, 1.0):
        for si in (-1.0, 1.0):
            a, b = 1.0 + 2.0 * si * ii, 1.0 + 2.0 * sj * jj
            fac = 0.5 * ((2.0 - a + b) * (a + b) - 2.0)
            caf = 0.5 * ((2.0 - b + a) * (a + b) - 2.0)
            q += a * b * (2.0 * np.log(np.hypot(a, b)) - math.log(2.0)) + fac * np.arctan(a / b) + caf * np.arctan(b / a)
    scale = 1.0 / (4.0 * math.pi)
    q = 0.25 * 0.5 * (q + q.T) * scale
    const = (2.0 * math.log(h) - math.log(2.0) - 3.0) * scale + q.mean()
    q -= q.mean()
    w, v = torch.linalg.eigh(torch.as_tensor(q, device=DEV))
    w, v = w.cpu().numpy(), v.cpu().numpy()
    terms = [(np.ones(n0), const)]
    left = 1.0
    for k in np.argsort(-np.abs(w), kind="stable"):
        terms.append((v[:, k], w[k]))
        left -= w[k] ** 2 / np.sum(w ** 2)
        if math.sqrt(max(left, 0.0)) < max_error:
            break
    return terms


def _shift(v, dy, dx):
    """v[..., y + dy, x + dx], zero beyond the edge."""
    n, m = v.shape[-2:]
    out = torch.zeros_like(v)
    out[..., max(0, -dy):n - max(0, dy), max(0, -dx):m - max(0, dx)] = \
        v[..., max(0, dy):n - max(0, -dy), max(0, dx):m - max(0, -dx)]
    return out


def _extend(inside, fields):
    """Sites outside within two sites of the grain take the mean of their nearest grain sites."""
    rings = {}
    for dy in range(-2, 3):
        for dx in range(-2, 3):
            rings.setdefault(dx * dx + dy * dy, []).append((dy, dx))
    left = ~inside
    ins = inside.to(F8)
    out = list(fields)
    masked = [f * ins for f in fields]
    for d2 in sorted(rings)[1:]:
        count = sum(_shift(ins, *o) for o in rings[d2])
        take = left & (count > 0)
        if bool(take.any()):
            for k, f in enumerate(masked):
                out[k] = torch.where(take, sum(_shift(f, *o) for o in rings[d2]) / count.clamp(min=1.0), out[k])
            left = left & ~take
    return out


def _lookup(n_out, n_in, c, s):
    """Bilinear lookups of an n_out lattice in an n_in lattice rotated by angles (c, s) [A]."""
    sh = (n_in - 1) / 2.0
    u = torch.arange(n_out, device=DEV, dtype=F8) + (n_in - n_out) / 2.0 - sh
    xs, ys = u[None, None, :], u[None, :, None]
    c, s = c[:, None, None], s[:, None, None]
    xr, yr = xs * c - ys * s + sh, xs * s + ys * c + sh
    xi, yi = xr.trunc(), yr.trunc()
    ok = (xi >= 0) & (xi + 1 < n_in) & (yi >= 0) & (yi + 1 < n_in)
    i00 = torch.where(ok, yi * n_in + xi, torch.zeros_like(xi)).long()
    return i00, xr - xi, yr - yi, ok, n_in


def _sample(lk, flat):
    """flat [n_in^2] or [A][n_in^2] at the lookups [A][n_out][n_out]."""
    i00, xf, yf, ok, n = lk

    def at(off):
        if flat.dim() == 1:
            return flat[i00 + off]
        return torch.gather(flat, 1, (i00 + off).reshape(flat.shape[0], -1)).reshape(i00.shape)

    v = (1 - yf) * ((1 - xf) * at(0) + xf * at(1)) + yf * ((1 - xf) * at(n) + xf * at(n + 1))
    return torch.where(ok, v, torch.zeros_like(v))


def _step(d, e, g, h):
    """Midpoint Riccati step over the distance h (order parameter d, energy e)."""
    a = 0.25j * h * d.conj()
    ihe = 1j * h * e
    ag = a * g
    b = 2 * ag + ihe - 1
    c = (ag + ihe + 1) * g + 1j * h * d
    return 2 * c / (torch.sqrt(b * b - 4 * a * c) - b)


class _Grain:
    """One grain's tables: lattice, energies, Fermi surface, geometry of every frame."""

    def __init__(self, case, e=None):
        cfg = _config(case)
        ph, num = cfg["physics"], cfg["numerics"]
        self.case, self.t, self.h = case, case["t"], 1.0 / case["ppxi"]
        self.lam, self.na = case["kappa"], case["angles"]
        if case["shape"] == "disc":
            verts, width = None, case["size"] - -case["size"]
        else:
            radius = case["size"] / math.hypot(math.cos(0.5 * math.pi) - 1.0, math.sin(0.5 * math.pi))
            corner = [0.25 * math.pi + 0.5 * math.pi * k for k in range(4)]
            vx, vy = [radius * math.cos(p) for p in corner], [radius * math.sin(p) for p in corner]
            ex, ey = max(vx) - min(vx), max(vy) - min(vy)
            width, verts = max(ex, ey), corner
            off = (min(vx) + 0.5 * ex, min(vy) + 0.5 * ey)
        frac = width * case["ppxi"]
        self.n0 = n0 = int(math.ceil(frac)) + 6
        self.n1 = n1 = n0 + 2 * int(math.ceil(0.5 * (math.sqrt(2.0) - 1.0) * n0))
        gf = frac / n0
        if verts is None:
            self.disc, self.verts = case["size"] / width * gf, None
        else:
            side = case["size"] / width
            rp = side / math.hypot(math.cos(0.5 * math.pi) - 1.0, math.sin(0.5 * math.pi)) * gf
            self.disc = None
            self.verts = [(rp * math.cos(p) - off[0] / width * gf, rp * math.sin(p) - off[1] / width * gf) for p in verts]
        if e is None:
            n = _pole_count(self.t, CUTOFF)
            pole, res = _poles(n)
            e_im = pole * self.t / (2 * math.pi)
            self.e, self.res = torch.as_tensor(1j * e_im, device=DEV), torch.as_tensor(res, device=DEV)
            self.sum_inv = float(np.sum(res / e_im)) * self.t
        else:
            self.e, self.sum_inv = torch.as_tensor(e, device=DEV), 0.0
        # Fermi surface
        na = self.na
        if na % 4 == 0:
            wts = [28 / 45 if k % 4 == 0 else 24 / 45 if k % 2 == 0 else 64 / 45 for k in range(na)]
        elif na % 3 == 0:
            wts = [6 / 8 if k % 3 == 0 else 9 / 8 for k in range(na)]
        elif na % 2 == 0:
            wts = [2 / 3 if k % 2 == 0 else 4 / 3 for k in range(na)]
        else:
            wts = [1.0] * na
        self.tb = "fermi_surface" in ph
        if self.tb:
            self.p_off, self.theta, self.px, self.py, self.vx, self.vy, self.w = _tight_binding(na, wts)
            step = self.h / np.hypot(self.vx, self.vy)
        else:
            phi = [_wrap(math.pi * 2 * k / na + 0.5 * math.pi, 0.0, 2 * math.pi) for k in range(na)]
            self.theta = np.array([p - 0.5 * math.pi for p in phi])
            self.vx, self.vy = np.array([math.cos(p) for p in phi]), np.array([math.sin(p) for p in phi])
            self.px, self.py, self.p_off = self.vx, self.vy, 0.0
            self.w = np.array(wts) / na
            step = np.full(na, self.h)
        self.step = torch.as_tensor(step, device=DEV)

        def basis(s, x, y):
            if self.tb:
                cx, cy, sn = np.cos(x), np.cos(y), np.sin(x) * np.sin(y)
                return {"s": cx + cy, "dx2-y2": cx - cy, "dxy": sn, "g": sn * (cx - cy)}[s]
            return {"s": np.ones_like(x), "dx2-y2": x * x - y * y, "dxy": x * y, "g": x * y * (x * x - y * y)}[s]

        rot = 2 * math.pi * ph["crystal_axes_rotation"]
        rx = self.px * math.cos(rot) - self.py * math.sin(rot)
        ry = self.px * math.sin(rot) + self.py * math.cos(rot)
        self.syms = _symmetries(case)
        self.eta = torch.as_tensor(np.array([basis(s, rx, ry) / math.sqrt(np.sum(basis(s, self.px, self.py) ** 2 * self.w))
                                             for s in self.syms]), device=DEV)
        self.log_t = math.log(self.t)
        trig = lambda sign, idx: torch.tensor([_trig32(sign * self.theta[i]) for i in idx], device=DEV, dtype=F8).T  # noqa: E731
        self.rot_d = trig(1.0, [(-k) % na for k in range(na)])
        self.rot_a, self.rot_b = trig(-1.0, range(na)), trig(1.0, range(na))
        self.fields_b = math.pi * ph["external_flux_quanta"]
        self.charge = -1.0
        # reference domain
        ix = np.arange(n0)
        if self.disc is not None:
            lab = self._disc_labels(n0, n0)[0]
            dom = lab > 0
        else:
            cx, cy = ix / (n0 - 1) - 0.5, ix / (n0 - 1) - 0.5
            dom = np.ones((n0, n0), bool)
            for i in range(4):
                (ax, ay), (bx, by) = self.verts[i], self.verts[(i + 1) % 4]
                dom &= (bx - ax) * (cy[:, None] - ay) - (by - ay) * (cx[None, :] - ax) >= 0.0
        self.dom = torch.as_tensor(dom, device=DEV)
        self.n_grain = int(dom.sum())
        self.area = self.h * self.h * self.n_grain
        self.flux_b = self.fields_b / self.area
        self._frames()
        self._walls()

    def _disc_labels(self, n0, n):
        o = (n0 - 1) * 0.5 + 0.5 * (n - n0)
        r = self.disc * (n0 - 1)
        u = np.arange(-1, n + 1) - o
        raw = (u[None, :] ** 2 + u[:, None] ** 2 <= r * r).astype(np.int64)
        row = (raw[:, :-2] + raw[:, 1:-1] + raw[:, 2:]) > 1
        lo, mid, hi = row[:-2], row[1:-1], row[2:]
        lab = np.zeros((n, n), np.int64)
        lab[lo & mid & hi] = 1
        lab[~lo & mid & hi] = 2
        lab[lo & mid & ~hi] = 3
        x, y = np.broadcast_to(u[None, 1:-1], (n, n)), np.broadcast_to(u[1:-1, None], (n, n))
        wall = lab > 1
        d = np.where(wall, np.sqrt(np.maximum(r * r - x * x, 0.0)) - np.abs(y), 0.0)
        nx = np.where(wall, -x / r, 0.0)
        ny = np.where(wall, np.where(y <= 0, -(y - d) / r, -(y + d) / r), 0.0)
        return lab, d, nx, ny

    def _polygon_labels(self, angle):
        n0, n = self.n0, self.n1
        c, s = math.cos(angle), math.sin(angle)
        p = [((c * x - s * y) * (n0 - 1.0), (s * x + c * y) * (n0 - 1.0)) for x, y in self.verts]
        u = np.arange(n) - (n - 1) * 0.5
        cx, cy = u[None, :], u[:, None]
        raw = np.ones((n, n), bool)
        dist, nx, ny = np.full((n, n), 1e5), np.zeros((n, n)), np.zeros((n, n))
        for i in range(4):
            (ax, ay), (bx, by) = p[i], p[(i + 1) % 4]
            lx, ly = bx - ax, by - ay
            raw &= lx * (cy - ay) - ly * (cx - ax) >= 0.0
            inv = 1.0 / math.sqrt(lx * lx + ly * ly)
            td = np.full((n, n), 1e4)
            if abs(lx) > 1e-5:
                k = ly / lx
                td = np.abs(k * cx + (ay - k * ax) - cy)
            near = td < dist
            dist, nx, ny = np.where(near, td, dist), np.where(near, -ly * inv, nx), np.where(near, lx * inv, ny)
        below, above = np.zeros_like(raw), np.zeros_like(raw)
        below[1:], above[:-1] = raw[:-1], raw[1:]
        lab = np.where(raw, 1, 0)
        lab[raw & ~below] = 2
        lab[raw & below & ~above] = 3
        lab[raw & ~below & ~above] = 0
        lab[0], lab[-1] = 0, 0
        return lab, dist, nx, ny

    def _frames(self):
        """Labels [A][y][x]; per column the lowest (entry) and highest (exit) site with distance and normal."""
        n1, na = self.n1, self.na
        shape = (na, n1)
        self.lab = np.zeros((na, n1, n1), np.uint8)
        self.node = {}
        for lbl in (2, 3):
            self.node[lbl] = {k: np.zeros(shape) for k in ("y", "d", "nx", "ny")}
            self.node[lbl]["on"] = np.zeros(shape, bool)
        same = self._disc_labels(self.n0, n1) if self.disc is not None else None
        for a in range(na):
            lab, d, nx, ny = same or self._polygon_labels(-self.theta[a])
            self.lab[a] = lab
            for lbl in (2, 3):
                y, x = np.nonzero(lab == lbl)
                nd = self.node[lbl]
                assert len(x) == len(set(x.tolist())), "one crossing per column"
                r = 1.0 / np.hypot(nx[y, x], ny[y, x])
                nd["on"][a, x], nd["y"][a, x], nd["d"][a, x] = True, y, np.maximum(d[y, x], 0.0)
                nd["nx"][a, x], nd["ny"][a, x] = nx[y, x] * r, ny[y, x] * r
        self.dist = {lbl: torch.as_tensor(self.node[lbl]["d"], device=DEV) for lbl in (2, 3)}
        self.on = {lbl: torch.as_tensor(self.node[lbl]["on"], device=DEV) for lbl in (2, 3)}
        self.lab = torch.as_tensor(self.lab, device=DEV)

    def _walls(self):
        """Specular gather tables: entries at label 2 read exits at label 3, and the other way round."""
        na, n1 = self.na, self.n1
        off = (n1 - 1) * 0.5
        self.wall = {}
        for into, out, sign in ((2, 3, 1.0), (3, 2, -1.0)):
            nd, present = self.node[into], self.node[out]["on"]
            a, x = np.nonzero(nd["on"])
            th = self.theta[a]
            c, s = np.cos(-th), np.sin(-th)
            px, py = self.px[a] * c - self.py[a] * s, self.px[a] * s + self.py[a] * c
            nx, ny = nd["nx"][a, x], nd["ny"][a, x]
            td = 2 * (px * nx + py * ny)
            src, wgt = np.zeros((len(a), 4), np.int64), np.zeros((len(a), 4))
            todo = np.ones(len(a), bool)
            for qx, qy in ((px - td * nx, py - td * ny), (-px, -py)):
                mx, my = qx * np.cos(th) - qy * np.sin(th), qx * np.sin(th) + qy * np.cos(th)
                wrap = np.vectorize(_wrap)
                kx = wrap(mx, self.p_off - math.pi, self.p_off + math.pi) - self.p_off
                ky = wrap(my, self.p_off - math.pi, self.p_off + math.pi) - self.p_off
                fai = na * wrap(np.arctan2(ky, kx) - 0.5 * math.pi, 0.0, 2 * math.pi) / (2 * math.pi)
                bx, by = x - off, nd["y"][a, x] - sign * nd["d"][a, x] - off
                s4, w4 = np.zeros_like(src), np.zeros_like(wgt)
                for r in range(2):
                    ia = (fai.astype(int) + r) % na
                    aw = fai - np.floor(fai) if r else 1 - (fai - np.floor(fai))
                    ra = th - self.theta[ia]
                    rx = bx * np.cos(ra) - by * np.sin(ra) + off
                    for pt in range(2):
                        col = rx.astype(int) + pt
                        pw = rx - np.floor(rx) if pt else 1 - (rx - np.floor(rx))
                        ok = (col >= 0) & (col < n1)
                        col = np.clip(col, 0, n1 - 1)
                        ok &= present[ia, col]
                        s4[:, 2 * r + pt] = np.where(ok, ia * n1 + col, 0)
                        w4[:, 2 * r + pt] = np.where(ok, pw * aw, 0.0)
                src[todo], wgt[todo] = s4[todo], w4[todo]
                todo &= w4.sum(1) < 1e-7
            tot = wgt.sum(1, keepdims=True)
            wgt = np.where(tot > 0, wgt / np.where(tot > 0, tot, 1.0), 0.0)
            self.wall[into] = tuple(torch.as_tensor(v, device=DEV) for v in (a * n1 + x, src, wgt))

    # -- physics of one state: x = (delta complex [Nc][n0][n0], a [2][n0][n0]) --
    def fields(self, delta, a, sl):
        """Order parameter and Doppler shift in the frames of the angles sl: [A][n1][n1] each."""
        n0, n1 = self.n0, self.n1
        ext = _extend(self.dom, [c.real for c in delta] + [c.imag for c in delta])
        nc = len(self.syms)
        lk = _lookup(n1, n0, self.rot_d[0][sl], self.rot_d[1][sl])
        d = 0
        for c in range(nc):
            z = torch.complex(_sample(lk, ext[c].reshape(-1)), _sample(lk, ext[nc + c].reshape(-1)))
            d = d + z * self.eta[c][sl][:, None, None]
        la = _lookup(n1, n0, self.rot_a[0][sl], self.rot_a[1][sl])
        th = torch.as_tensor(self.theta, device=DEV)[sl][:, None, None]
        u = (torch.arange(n1, device=DEV, dtype=F8) - 0.5 * (n1 - 1)) * self.h
        xs, ys = u[None, None, :], u[None, :, None]
        xr, yr = xs * torch.cos(th) - ys * torch.sin(th), xs * torch.sin(th) + ys * torch.cos(th)
        v = [torch.as_tensor(q, device=DEV)[sl][:, None, None] for q in (self.vx, self.vy)]
        sx = _sample(la, a[0].reshape(-1)) / self.lam ** 2 - 0.5 * self.flux_b * yr
        sy = _sample(la, a[1].reshape(-1)) / self.lam ** 2 + 0.5 * self.flux_b * xr
        return d, self.charge * (v[0] * sx + v[1] * sy)

    def initial_walls(self, delta, a):
        out = {lbl: torch.zeros(self.na, self.n1, len(self.e), device=DEV, dtype=C16) for lbl in (2, 3)}
        for sl in self.chunks(64):
            d, es = self.fields(delta, a, sl)
            for lbl in (2, 3):
                y = torch.as_tensor(self.node[lbl]["y"], device=DEV)[sl].long()
                dn = torch.gather(d, 1, y[:, None, :])[:, 0, :, None]
                en = self.e + torch.gather(es, 1, y[:, None, :])[:, 0, :, None]
                om = torch.sqrt((dn * dn.conj()).real - en * en)
                g = (-dn if lbl == 3 else dn.conj()) / (en + 1j * om)
                out[lbl][sl] = torch.where(self.on[lbl][sl][..., None], g, torch.zeros_like(g))
        return self.reflect(out)

    def reflect(self, out):
        """Incoming values from outgoing ones."""
        into = {}
        for lbl, other in ((2, 3), (3, 2)):
            dst, src, wgt = self.wall[lbl]
            v = out[other].reshape(-1, out[other].shape[-1])
            t = torch.zeros(self.na * self.n1, v.shape[1], device=DEV, dtype=C16)
            t[dst] = sum(v[src[:, k]] * wgt[:, k, None] for k in range(4))
            into[lbl] = t.reshape(self.na, self.n1, -1)
        return into

    def chunks(self, per=None):
        row = self.n1 * self.n1 * len(self.e) * 16.0
        per = per or max(1, min(self.na, int(12e9 / row)))
        return [slice(k, min(self.na, k + per)) for k in range(0, self.na, per)]

    def sweep_one(self, d, es, into, sl, downward):
        """One coherence function through every row; yields (row, value) and finally the exit values."""
        lbl_in, lbl_out = (3, 2) if downward else (2, 3)
        if downward:
            d = -d.conj()
        h = self.step[sl][:, None, None]
        g = torch.zeros_like(into[lbl_in][sl])
        exits = torch.zeros_like(g)
        n1 = self.n1
        rows = range(n1 - 1, -1, -1) if downward else range(n1)
        lab_any = (self.lab[sl] > 0).any(2).any(0).tolist()
        rows = [y for y in rows if lab_any[y]]
        for y in rows:
            lab = self.lab[sl, y, :, None]
            dy, ey = d[:, y, :, None], es[:, y, :, None]
            p = y + 1 if downward else y - 1
            dp, ep = d[:, p, :, None], es[:, p, :, None]
            entry, leave = lab == lbl_in, lab == lbl_out
            dm, em = torch.where(entry, dy, 0.5 * (dy + dp)), torch.where(entry, ey, 0.5 * (ey + ep))
            hm = torch.where(entry, self.dist[lbl_in][sl][..., None] * h, h)
            g0 = torch.where(entry, into[lbl_in][sl], g)
            g = torch.where(lab > 0, _step(dm, self.e + em, g0, hm), torch.zeros_like(g))
            if bool(leave.any()):
                last = _step(dy, self.e + ey, g, self.dist[lbl_out][sl][..., None] * h)
                exits = torch.where(leave, last, exits)
            yield y, g
        yield None, exits

    def sums(self, delta, a, into, sl, want_ldos=False, want_out=True):
        """Frame sums of the angles sl (F, Re g, Re I), or Im g of every energy, and the exit values."""
        d, es = self.fields(delta, a, sl)
        down, out2, out3 = {}, None, None
        for y, g in self.sweep_one(d, es, into, sl, True):
            if y is None:
                out2 = g
            else:
                down[y] = g
        zero = torch.zeros(d.shape[0], self.n1, device=DEV, dtype=F8)
        f, gr, ir, im = {}, {}, {}, {}
        for y, g in self.sweep_one(d, es, into, sl, False):
            if y is None:
                out3 = g
                continue
            gt = down.pop(y)
            live = (self.lab[sl, y] > 0)
            q = -1j * (1 - g * gt) / (1 + g * gt)
            if want_ldos:
                im[y] = torch.where(live[..., None], q.imag, torch.zeros_like(q.imag))
                continue
            fac = 2j / (1 + g * gt)
            dy = d[:, y, :, None]
            fs = ((-fac * g + (fac * gt).conj()) * self.res).sum(-1)
            f[y] = torch.where(live, fs, torch.zeros_like(fs))
            gr[y] = torch.where(live, (q.real * self.res).sum(-1), zero)
            ir[y] = torch.where(live, -((dy.conj() * g - dy * gt).imag * self.res).sum(-1), zero)
        outs = {2: out2, 3: out3}
        if want_ldos:
            return im, outs
        pack = lambda m, z: torch.stack([m.get(y, z) for y in range(self.n1)], 1)  # noqa: E731
        return (pack(f, zero.to(C16)), pack(gr, zero), pack(ir, zero)), outs

    def back(self, planes, sl):
        """Extended frame planes [A][n1][n1] at the reference sites, per angle."""
        inside = self.lab[sl] > 0
        lk = _lookup(self.n0, self.n1, self.rot_b[0][sl], self.rot_b[1][sl])
        return [_sample(lk, p.reshape(p.shape[0], -1)) for p in _extend(inside, planes)]

    def evaluate(self, delta, a, into):
        """g(x): new order parameter, current, sum of the free-energy kernel; and the outgoing values."""
        n0 = self.n0
        acc_d = torch.zeros(len(self.syms), n0, n0, device=DEV, dtype=C16)
        acc_j, acc_f = torch.zeros(2, n0, n0, device=DEV, dtype=F8), torch.zeros(n0, n0, device=DEV, dtype=F8)
        outs = {2: [], 3: []}
        for sl in self.chunks():
            (f, gr, ir), o = self.sums(delta, a, into, sl)
            fr, fi, g, i = self.back([f.real, f.imag, gr, ir], sl)
            w, vx, vy = (torch.as_tensor(q, device=DEV)[sl][:, None, None] for q in (self.w, self.vx, self.vy))
            fz = torch.complex(fr, fi) * w
            acc_d = acc_d + torch.stack([(fz * e[sl][:, None, None]).sum(0) for e in self.eta])
            acc_j = acc_j + torch.stack([(g * vx * w).sum(0), (g * vy * w).sum(0)])
            acc_f = acc_f + (i * w).sum(0)
            for lbl in (2, 3):
                outs[lbl].append(o[lbl].detach())
        m = self.dom.to(F8)
        new = acc_d * m * (0.5 * self.t / (self.log_t + self.sum_inv))
        return new, acc_j * m * (2.0 * self.charge * self.t), (acc_f * m).sum(), {l: torch.cat(v) for l, v in outs.items()}

    def free_energy(self, delta, a, kernel):
        n = self.n0
        idx = torch.arange(n, device=DEV)
        up, dn = (idx + 1).clamp(max=n - 1), (idx - 1).clamp(min=0)
        width = (up - dn).to(F8)
        bz = ((a[1][:, up] - a[1][:, dn]) / width[None, :] - (a[0][up] - a[0][dn]) / width[:, None]) / self.h
        m = self.dom.to(F8)
        cond = sum(((c.real ** 2 + c.imag ** 2) * m).sum() for c in delta) * (self.log_t + self.sum_inv)
        return (self.t * kernel + cond + 0.5 / self.lam ** 2 * (bz * bz).sum()) * self.h ** 2

    def vector_potential(self, j):
        s = j - j.sum((1, 2), keepdim=True) / self.n_grain
        idx = (torch.arange(self.n0, device=DEV)[:, None] - torch.arange(self.n0, device=DEV)[None, :]).abs()
        out = torch.zeros_like(s)
        for vec, val in _filters(self.n0, self.h, 1e-6):
            t = torch.as_tensor(np.ascontiguousarray(vec), device=DEV)[idx]
            out -= self.h ** 2 * float(val) * (t @ s @ t)
        return out


def _ratio(old, new, count):
    """The L2 residual of real values old -> new."""
    return float(torch.linalg.vector_norm(new - old)) / max(float(torch.linalg.vector_norm(old)), 1e-4 * count)


def _planes(z):
    return torch.stack([z.real, z.imag])


def _exact_solve(case, delta, a):
    gr = _Grain(case)
    delta = torch.complex(delta[:, 0], delta[:, 1]) * gr.dom
    nn, ne = 2 * gr.n0 ** 2, len(gr.e)
    into = gr.initial_walls(delta, a)
    j_old, fe_old = torch.zeros(2, gr.n0, gr.n0, device=DEV, dtype=F8), None
    for it in range(ITERATIONS):
        if it:
            delta, a = delta + 0.5 * (new - delta), a + 0.5 * (a_new - a)
        new, j, kernel, outs = gr.evaluate(delta, a, into)
        fe = float(gr.free_energy(delta, a, kernel))
        nxt = gr.reflect(outs)
        a_new = gr.vector_potential(j)
        res = [_ratio(_planes(o), _planes(n), nn) for o, n in zip(delta, new)]
        res += [_ratio(a, a_new, nn)] + ([_ratio(j_old, j, nn)] if it else [])
        res += [_ratio(_planes(into[l]), _planes(nxt[l]), 2 * ne * int(gr.on[l].sum())) for l in (2, 3)]
        if it:
            per = gr.h ** 2 * gr.n_grain
            res.append(abs(fe - fe_old) / per / max(abs(fe_old) / per, 1e-4))
        into, j_old, fe_old = nxt, j, fe
    return {"delta": torch.stack([delta.real, delta.imag], 1), "a": a, "residual": max(res), "free_energy": fe}


def exact(case, seed):
    if case["kind"] == "batch":
        res, deltas, pots = [], [], []
        for k, c in enumerate(_study(case)):
            r = _exact_solve(c, *_inputs(c, _side(c), 1000 * seed + k))
            res.append(r["residual"])
            deltas.append(r["delta"].reshape(-1))
            pots.append(r["a"].reshape(-1))
        return {"residual": np.array(res), "delta": torch.cat(deltas), "a": torch.cat(pots)}
    delta, a = _inputs(case, _side(case), seed)
    if case["kind"] == "solve":
        return _exact_solve(case, delta, a)
    if case["kind"] == "ldos":
        return {"ldos": _exact_ldos(case, delta, a)}
    return _exact_gradient(case, delta, a)


def _side(case):
    """The lattice side, from the grain's width as the lattice is laid out."""
    if case["shape"] == "disc":
        width = case["size"] - -case["size"]
    else:
        r = case["size"] / math.hypot(math.cos(0.5 * math.pi) - 1.0, math.sin(0.5 * math.pi))
        c = [0.25 * math.pi + 0.5 * math.pi * k for k in range(4)]
        xs, ys = [r * math.cos(p) for p in c], [r * math.sin(p) for p in c]
        width = max(max(xs) - min(xs), max(ys) - min(ys))
    return int(math.ceil(width * case["ppxi"])) + 6


def _exact_ldos(case, delta, a):
    sp = _spectroscopy(case)["spectroscopy"]
    n, block = case["energies"], min(case["block"], case["energies"])
    lo, hi = sp["energy_min"], sp["energy_max"]
    energies = [lo + (hi - lo) / (n - 1) * i for i in range(n)]
    gr = _Grain(case, e=np.zeros(1, complex))
    delta = torch.complex(delta[:, 0], delta[:, 1]) * gr.dom
    out = torch.zeros(n, gr.n0, gr.n0, device=DEV, dtype=F8)
    for b in range(0, n, block):
        real = [energies[min(b + i, n - 1)] for i in range(block)]
        gr.e = torch.as_tensor(np.array(real) + 1j * sp["energy_broadening"], device=DEV)
        count = min(block, n - b)
        into = gr.initial_walls(delta, a)
        for it in range(3):  # a burn-in and two iterations; the last one's values are kept
            outs = {2: [], 3: []}
            for sl in gr.chunks():
                im, o = gr.sums(delta, a, into, sl, want_ldos=True)
                for lbl in (2, 3):
                    outs[lbl].append(o[lbl])
                if it == 2:
                    w = torch.as_tensor(gr.w, device=DEV)[sl][:, None, None]
                    zero = torch.zeros(o[2].shape[0], gr.n1, block, device=DEV, dtype=F8)
                    plane = torch.stack([im.get(y, zero) for y in range(gr.n1)], 1)
                    for k in range(count):
                        out[b + k] -= (gr.back([plane[..., k]], sl)[0] * w).sum(0) * gr.dom
            into = gr.reflect({l: torch.cat(v) for l, v in outs.items()})
    return out


def _exact_gradient(case, delta, a):
    """Loss and gradients at frozen incoming values, by reverse mode over a few angles at a time."""
    gr = _Grain(case)
    z = torch.complex(delta[:, 0], delta[:, 1])
    flux_b = gr.flux_b
    masked = z * gr.dom
    into = gr.initial_walls(masked, a)
    _, _, _, outs = gr.evaluate(masked, a, into)
    into = gr.reflect(outs)
    beta = torch.as_tensor(_edge_weights(gr, 2.0), device=DEV)
    z, a = z.requires_grad_(), a.clone().requires_grad_()
    b = torch.tensor(flux_b, dtype=F8, device=DEV, requires_grad=True)
    grads, loss = [torch.zeros_like(z), torch.zeros_like(a), torch.zeros_like(b)], 0.0
    m = gr.dom.to(F8)
    per = max(1, int(60e9 / (gr.n1 * gr.n1 * len(gr.e) * 16.0 * 110)))
    for sl in [slice(0, 0)] + gr.chunks(per):
        gr.flux_b = b
        if sl.stop == 0:  # the explicit terms, without the angles
            part = gr.free_energy(z * m, a, torch.zeros((), device=DEV, dtype=F8))
        else:
            (_, g_re, i_re), _ = gr.sums(z * m, a, into, sl)
            g, i = gr.back([g_re, i_re], sl)
            w, vx, vy = (torch.as_tensor(q, device=DEV)[sl][:, None, None] for q in (gr.w, gr.vx, gr.vy))
            j = torch.stack([(g * vx * w).sum(0), (g * vy * w).sum(0)]) * m * (2.0 * gr.charge * gr.t)
            part = gr.t * gr.h ** 2 * ((i * w).sum(0) * m).sum() + (j * beta).sum()
        got = torch.autograd.grad(part, [z, a, b], allow_unused=True)
        grads = [x if y is None else x + y for x, y in zip(grads, got)]
        loss += float(part.detach())
        del part, got
    return {"loss": torch.tensor(loss, dtype=F8), "g_delta": grads[0], "g_a": grads[1], "g_b": grads[2]}


def _edge_weights(gr, width):
    """Weights of the azimuthal current in the outermost ring of the given width."""
    n = gr.n0
    u = (np.arange(n) - 0.5 * (n - 1)) * gr.h
    x, y = np.meshgrid(u, u)
    r = np.hypot(x, y)
    inside = gr.dom.cpu().numpy()
    ring = inside & (r > r[inside].max() - width)
    safe = np.where(r > 0, r, 1.0)
    return np.stack([np.where(ring, -y / safe, 0.0), np.where(ring, x / safe, 0.0)])

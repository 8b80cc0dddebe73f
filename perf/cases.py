"""The work that users of this library have it do, as cases that can be timed and compared.

Every case is one pass through the public entry points on a state that a program keeps (Solver, State):
the program writes this time step's concentrations into the state's device buffer, calls
update_state_parameters (temperature, pressure and photolysis change every step of a host model) and solves.
The concentrations are restored in every pass, so each pass does the same work.

Mechanisms are the repository's own: micm_bench's Chapman and TS1, and the synthetic mechanisms of
micm_b200.synthetic.CONFIGS (60, 210 and 600 species).  Inputs are drawn on the GPU from the seed, with the
distributions of synthetic.cell_inputs and micm_bench.inputs.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from micm_b200 import Solver, micm_bench, synthetic
from micm_b200._native import check, lib

# name: mechanism, tableau, time step [s]; what the arithmetic of one pass takes: step attempts per cell
# (measured; a property of the inputs, the same for every implementation of the method)
MECHANISMS = {
    "chapman": dict(make=lambda: micm_bench.mechanism("chapman"), stages=3, dt=30.0, attempts=13),
    "ts1": dict(make=lambda: micm_bench.mechanism("ts1"), stages=3, dt=30.0, attempts=57),
    "c60": dict(make=synthetic.CONFIGS["c60_adjoint"]["mech"], stages=4, dt=3600.0, attempts=58),
    "c210": dict(make=synthetic.CONFIGS["c210_uneven"]["mech"], stages=4, dt=600.0, attempts=58),
    "c600": dict(make=synthetic.CONFIGS["c600"]["mech"], stages=4, dt=600.0, attempts=69),
}
GAS_CONSTANT = 8.31446261815324
MAX_CHECKPOINTS = 160


def listed():
    return [
        # a box model: one cell of a small mechanism, micm's default solve; launches and latency
        dict(name="chapman_1_plain", op="plain", control="global", mech="chapman", cells=1, L=1),
        # one block of grid columns per call, as a CPU-parallel host model hands them over
        dict(name="ts1_128_plain", op="plain", control="global", mech="ts1", cells=128, L=128),
        # micm_bench's default case on its two GPU backends ("gpu" and "gpu-fused")
        dict(name="ts1_10000_plain", op="plain", control="global", mech="ts1", cells=10000, L=128),
        dict(name="ts1_10000_fused", op="fused", control="per_cell", mech="ts1", cells=10000, L=128, variant=0),
        # a small regional domain of a condensed mechanism, a count that fills neither groups nor warps
        dict(name="c60_1013_fused", op="fused", control="per_cell", mech="c60", cells=1013, L=32, variant=0),
        # a regional domain of a full mechanism in the default configuration
        dict(name="c210_4096_fused", op="fused", control="per_cell", mech="c210", cells=4096, L=128, variant=0),
        # a global model's share of one GPU, the configuration that the tuner picks for large states
        dict(name="c210_65536_fused", op="fused", control="per_cell", mech="c210", cells=65536, L=128, variant=2),
        dict(name="ts1_200000_fused", op="fused", control="per_cell", mech="ts1", cells=200000, L=128, variant=2),
        # a mechanism whose factor is larger than a block's share of on-chip memory
        dict(name="c600_700_fused", op="fused", control="per_cell", mech="c600", cells=700, L=128, variant=0),
        # an integrator of the user's own on the single-stage entry points: f, alpha I - J, LU, solve
        dict(name="c210_16384_stages", op="stages", control="global", mech="c210", cells=16384, L=128),
        # gradients of a loss with respect to the initial state and the rates (data assimilation)
        dict(name="c60_8192_adjoint", op="adjoint", control="per_cell", mech="c60", cells=8192, L=32, variant=2),
        # micm's second integrator
        dict(name="c60_3001_euler", op="euler", control="per_cell", mech="c60", cells=3001, L=32),
    ]


def draw(rng):
    op = rng.choice(["plain", "plain", "fused", "fused", "fused", "stages", "adjoint", "euler"])
    # mechanisms and counts that keep every pass at most as long as the longest listed one
    mech = rng.choice({"adjoint": ["chapman", "c60"], "euler": ["chapman", "c60"],
                       "plain": ["chapman", "ts1", "c60", "c210"]}.get(
        op, ["chapman", "ts1", "c60", "c210", "c600"]))
    most = {"chapman": 262144, "ts1": 65536, "c60": 65536, "c210": 32768, "c600": 1024}[mech]
    if op in ("adjoint", "euler"):
        most = min(most, 8192)
    if op == "stages":
        most = {"chapman": 262144, "ts1": 32768, "c60": 65536, "c210": 32768, "c600": 4096}[mech]
    case = dict(op=op, mech=mech, cells=max(1, int(round(math.exp(rng.uniform(0.0, math.log(most)))))),
                L=rng.choice([1, 8, 32, 100, 128]),
                control=rng.choice(["global", "per_cell"]) if op in ("plain", "euler") else
                ("global" if op == "stages" else "per_cell"))
    if op == "fused":
        # the tuner picks one cell per thread for large states only
        case["variant"] = 2 if mech != "c600" and case["cells"] >= 16384 and rng.random() < 0.5 else 0
    elif op == "adjoint":
        case["variant"] = rng.choice([0, 2])
    return case


# ---------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def mechanism(name):
    m = MECHANISMS[name]["make"]()
    if name == "ts1":
        # with micm's builder default (1e-3 mol m-3) some of the varied cells do not converge, in micm either
        m.absolute_tolerance = np.full(m.n_species, 1e-5)
    return m


@functools.lru_cache(maxsize=None)
def solver_of(name, L, variant):
    s = Solver(mechanism(name), MECHANISMS[name]["stages"], vector_length=L)
    if variant is not None:
        s.set_fused_config(variant=variant, lu_in_shared=0 if variant == 2 else 1)
    return s


def draw_inputs(case, seed):
    """Temperature, pressure, air density [n], concentrations [n, S] in system order, parameters [n, P], on the GPU."""
    m, n = mechanism(case["mech"]), case["cells"]
    g = torch.Generator(device="cuda").manual_seed(int(seed))

    def uniform(lo, hi, *shape):
        return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo

    labels = m.custom_param_labels()
    if case["mech"] in ("chapman", "ts1"):
        # micm_bench's state, every cell varied as micm_bench.inputs does with a seed
        base = micm_bench.inputs(case["mech"], 1)
        put = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
        T = float(base["temperature"][0]) + uniform(-30.0, 10.0, n)
        P = torch.full((n,), float(base["pressure"][0]), device="cuda", dtype=torch.float64)
        y = put(base["concentrations"]) * 10.0 ** uniform(-0.5, 0.5, n, m.n_species)
        params = put(base["custom_params"]).repeat(n, 1)
        photolysis = torch.tensor([l.startswith("j") for l in labels], device="cuda", dtype=torch.bool)
        params[:, photolysis] *= uniform(0.0, 1.0, n, int(photolysis.sum()))
    else:
        # half the cells at night: their step counts differ from the day cells'
        T, P = uniform(200.0, 310.0, n), uniform(9.0e4, 1.02e5, n)
        y = 10.0 ** uniform(-14.0, -6.0, n, m.n_species)
        day = uniform(0.5, 1.0, n) * (uniform(0.0, 1.0, n) >= 0.5)
        params = torch.zeros(n, len(labels), device="cuda", dtype=torch.float64)
        k = torch.as_tensor(m.photolysis_base, device="cuda")
        params[:, : len(k)] = day[:, None] * k[None, :]
    return dict(T=T, P=P, rho=P / (GAS_CONSTANT * T), y=y, params=params)


def to_layout(a, L):
    """[cell, column] to the state's vector layout: groups of L cells, column by column."""
    n, c = a.shape
    pad = torch.zeros(-(-n // L) * L, c, device=a.device, dtype=a.dtype)
    pad[:n] = a
    return pad.reshape(-1, L, c).transpose(1, 2).reshape(-1).contiguous()


class DeviceArray:
    """A state's device buffer; holds the state, so that a tensor over it keeps the buffer alive."""

    def __init__(self, state, ptr, count):
        self.state = state
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f8", "data": (ptr, False), "version": 3,
                                         "strides": None}


VARIABLES, PARAMS, JACOBIAN, CONDITIONS, TOLERANCES, FORCING = 0, 1, 3, 4, 5, 6


def view(state, buffer):
    ptr, count = state.device_buffer(buffer)
    return torch.as_tensor(DeviceArray(state, ptr, count), device="cuda") if count else None


def prepare(case, seed):
    solver = solver_of(case["mech"], case["L"], case.get("variant"))
    x = draw_inputs(case, seed)
    L, S = case["L"], solver.mech.n_species
    state = solver.get_state(case["cells"])
    stream = torch.cuda.Stream()
    check(lib().micmb_state_set_stream(state.handle, ctypes.c_void_p(stream.cuda_stream)))
    state.upload(TOLERANCES, state.absolute_tolerance)
    check(lib().micmb_state_set_relative_tolerance(state.handle, float(state.relative_tolerance)))
    columns = torch.as_tensor(solver.compiled.species_columns.astype(np.int64), device="cuda")
    by_column = torch.empty_like(x["y"])
    by_column[:, columns] = x["y"]
    y0 = to_layout(by_column, L)
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        view(state, CONDITIONS).copy_(to_layout(torch.stack([x["T"], x["P"], x["rho"]], 1), L))
        if x["params"].shape[1]:
            view(state, PARAMS).copy_(to_layout(x["params"], L))
        view(state, VARIABLES).copy_(y0)
    stream.synchronize()
    s = dict(case=case, solver=solver, state=state, stream=stream, y0=y0, y=view(state, VARIABLES),
             dt=MECHANISMS[case["mech"]]["dt"])
    if case["op"] == "stages":
        s["f"], s["jac"] = view(state, FORCING), view(state, JACOBIAN)
    if case["op"] == "adjoint":
        s["grad"] = loss_gradient(case["cells"], S, seed)
    return s


def loss_gradient(n, S, seed):
    return np.random.default_rng(int(seed)).standard_normal((n, S))


COUNTS = ("function_calls", "jacobian_updates", "number_of_steps", "accepted", "rejected", "decompositions",
          "solves", "cells_not_converged")


def counts(result):
    return {k: int(result.stats[k]) for k in COUNTS}


def run(s):
    case, solver, state, dt = s["case"], s["solver"], s["state"], s["dt"]
    with torch.cuda.stream(s["stream"]):
        s["y"].copy_(s["y0"])
        if case["op"] == "stages":
            s["f"].zero_()
            s["jac"].zero_()
    solver.update_state_parameters(state)
    op = case["op"]
    if op in ("plain", "fused"):
        r = solver.solve(dt, state, method=op, step_control=case["control"])
        return {"y": s["y"], "counts": counts(r)}
    if op == "euler":
        r = solver.solve_backward_euler(dt, state, step_control=case["control"])
        return {"y": s["y"], "counts": counts(r)}
    if op == "adjoint":
        dy0, dlogk, r = solver.solve_adjoint(dt, state, s["grad"], MAX_CHECKPOINTS)
        return {"y": s["y"], "dy0": dy0, "dlogk": dlogk, "counts": counts(r)}
    check(lib().micmb_add_forcing_terms(solver.handle, state.handle))
    check(lib().micmb_subtract_jacobian_terms(solver.handle, state.handle))
    check(lib().micmb_alpha_minus_jacobian(solver.handle, state.handle, ALPHA))
    check(lib().micmb_lu_decompose(solver.handle, state.handle))
    check(lib().micmb_linear_solve(solver.handle, state.handle))
    return {"x": s["f"], "lu": s["jac"]}


ALPHA = 0.25  # 1 / (H gamma) of a step of a few seconds


def work(case):
    m = mechanism(case["mech"])
    info = solver_of(case["mech"], case["L"], case.get("variant")).compiled.info
    n, S, R, P = case["cells"], m.n_species, m.n_reactions, info["n_custom_params"]
    stages, attempts = MECHANISMS[case["mech"]]["stages"], MECHANISMS[case["mech"]]["attempts"]
    nnz = info["jacobian_nnz"]
    forcing = 3 * R + 2 * info["n_forcing_terms"]
    jacobian = 3 * info["n_jacobian_infos"] + 2 * info["n_jacobian_terms"] + S
    lu = 2 * info["lu_updates"] + info["lu_lower"] + S
    solve = 2 * (nnz - S) + S
    # conditions, parameters and concentrations in; rate constants and concentrations out
    words, rates = 3 + P + 2 * S + R, 20 * R
    if case["op"] == "stages":
        return dict(bytes=8.0 * n * (words + nnz), flops=float(n) * (rates + forcing + jacobian + lu + solve))
    if case["op"] == "euler":
        return dict(bytes=8.0 * n * words, flops=float(n) * (rates + 20 * (forcing + jacobian + lu + solve)))
    attempt = 3 * forcing + jacobian + lu + stages * solve + S * (2 * stages * stages + 4 * stages + 8)
    flops = float(n) * (rates + attempts * attempt)
    if case["op"] == "adjoint":
        return dict(bytes=8.0 * n * (words + 2 * S), flops=3.0 * flops)
    return dict(bytes=8.0 * n * words, flops=flops)


# ---------------------------------------------------------------------------------------------------------
# the same values from dense 64-bit linear algebra
# ---------------------------------------------------------------------------------------------------------
class Dense:
    """Rate constants, f and J of a mechanism on [n, S] states in system order, written out in torch."""

    def __init__(self, m, x):
        self.m, self.n, self.S = m, x["y"].shape[0], m.n_species
        T, P, rho = x["T"], x["P"], x["rho"]
        labels = {l: i for i, l in enumerate(m.custom_param_labels())}
        k = []

        def falloff(p, numerator):
            k0 = p[0] * torch.exp(p[2] / T) * (T / 300.0) ** p[1]
            kinf = p[3] * torch.exp(p[5] / T) * (T / 300.0) ** p[4]
            ratio = k0 * rho / kinf
            return k0 * numerator / (1.0 + ratio) * p[6] ** (p[7] / (p[7] + torch.log10(ratio) ** 2))

        for rx in m.reactions:
            p = list(rx.params)
            if rx.kind == 0:
                v = p[0] * torch.exp(p[2] / T) * (T / p[3]) ** p[1] * (1.0 + p[4] * P)
            elif rx.kind == 1:
                v = falloff(p, rho)
            elif rx.kind == 2:
                v = falloff(p, 1.0)
            elif rx.kind == 7:
                v = x["params"][:, labels[rx.label]] * p[0]
            elif rx.kind == 8:
                r = x["params"][:, labels[rx.label + ".effective radius [m]"]]
                c = x["params"][:, labels[rx.label + ".particle number concentration [# m-3]"]]
                speed = torch.sqrt(8.0 * GAS_CONSTANT / (math.pi * p[1]) * T)
                v = 4.0 * c * math.pi * r * r / (r / p[0] + 4.0 / (speed * p[2]))
            else:
                raise NotImplementedError
            for i in rx.reactants:
                if i < 0:
                    c = m.parameterized[-i - 1]
                    v = v * (c[0] + c[1] * T + c[2] * P + c[3] * rho)
            k.append(v)
        self.k = torch.stack(k, 1)
        self.reactants = [[i for i in rx.reactants if i >= 0] for rx in m.reactions]
        R = len(m.reactions)
        self.nu = torch.zeros(R, self.S, device="cuda", dtype=torch.float64)
        for r, rx in enumerate(m.reactions):
            for i in self.reactants[r]:
                self.nu[r, i] -= 1.0
            for i, c in rx.products:
                self.nu[r, i] += c
        width = max(1, max(len(a) for a in self.reactants))
        ids = torch.full((R, width), self.S, dtype=torch.int64)
        for r, a in enumerate(self.reactants):
            ids[r, : len(a)] = torch.tensor(a, dtype=torch.int64)
        self.ids = ids.cuda()

    def padded(self, y, cells):
        y1 = torch.cat([y, torch.ones(y.shape[0], 1, device="cuda", dtype=torch.float64)], 1)
        return y1[:, self.ids]  # [n, R, width], ones where a reaction has fewer reactants

    def f(self, y, cells):
        return (self.k[cells] * self.padded(y, cells).prod(2)) @ self.nu

    def jacobian(self, y, cells):
        v, k = self.padded(y, cells), self.k[cells]
        J = torch.zeros(y.shape[0], self.S + 1, self.S, device="cuda", dtype=torch.float64)
        for q in range(v.shape[2]):
            others = k.clone()
            for o in range(v.shape[2]):
                if o != q:
                    others *= v[:, :, o]
            # d f / d y_i += nu * (rate without its q-th reactant), i that reactant
            for r in range(k.shape[1]):
                i = int(self.where[r][q])
                if i < self.S:
                    J[:, i, :] += others[:, r, None] * self.nu[r]
        return J[:, : self.S].transpose(1, 2)

    @functools.cached_property
    def where(self):
        return self.ids.cpu().tolist()


def dense_rosenbrock(d, params, y, dt, atol, rtol, per_cell):
    """micm's adaptive Rosenbrock method on dense matrices; one step size for all cells or one per cell."""
    n, S = y.shape
    s, a, c = params.stages, list(params.a), list(params.c)
    one = torch.ones(n, device="cuda", dtype=torch.float64)
    t, H = 0.0 * one, (1e-6 * dt) * one
    h_min = 1e-15 * dt
    rejected, again = torch.zeros(n, dtype=torch.bool, device="cuda"), torch.zeros(n, dtype=torch.bool, device="cuda")
    y = y.clone()
    eye = torch.eye(S, device="cuda", dtype=torch.float64)
    while True:
        cells = torch.nonzero(t - dt + params.round_off <= 0).flatten()
        if not len(cells):
            break
        h = torch.minimum(H[cells], (dt - t[cells]).abs())
        yc = y[cells]
        lu, piv = torch.linalg.lu_factor(eye / (h * params.gamma[0])[:, None, None] - d.jacobian(yc, cells))
        K, F = [], d.f(yc, cells)
        for i in range(s):
            at = i * (i - 1) // 2
            if i > 0 and params.new_function_evaluation[i]:
                F = d.f(yc + sum(a[at + j] * K[j] for j in range(i)), cells)
            rhs = F + sum((c[at + j] / h)[:, None] * K[j] for j in range(i)) if i else F
            K.append(torch.linalg.lu_solve(lu, piv, rhs[:, :, None])[:, :, 0])
        yn = yc + sum(params.m[j] * K[j] for j in range(s))
        e = sum(params.e[j] * K[j] for j in range(s)) / (atol + rtol * torch.maximum(yc.abs(), yn.abs()))
        total = (e * e).sum(1)
        err = torch.sqrt(total / S if per_cell else total.sum().expand_as(total) / (S * len(cells)))
        err = err.clamp(min=1e-10)
        fac = (params.safety_factor / err ** (1.0 / params.estimator_of_local_order)).clamp(params.factor_min,
                                                                                            params.factor_max)
        good = (err < 1) | (h < h_min)
        new = h * fac
        up = new.clamp(h_min, dt)
        up = torch.where(rejected[cells], torch.minimum(up, h), up)
        down = torch.where(again[cells], h * params.rejection_factor_decrease, new)
        H[cells] = torch.where(good, up, down)
        t[cells] = torch.where(good, t[cells] + h, t[cells])
        y[cells] = torch.where(good[:, None], yn, yc)
        again[cells] = ~good & rejected[cells]
        rejected[cells] = ~good
    return y.clamp(min=0.0)


def exact(case, seed):
    m, n, L = mechanism(case["mech"]), case["cells"], case["L"]
    S = m.n_species
    if case["op"] not in ("plain", "fused", "stages") or case["mech"] == "c600" or 8 * n * S * S > 1 << 30:
        return None
    solver = solver_of(case["mech"], L, case.get("variant"))
    x = draw_inputs(case, seed)
    d = Dense(m, x)
    columns = torch.as_tensor(solver.compiled.species_columns.astype(np.int64), device="cuda")
    atol = torch.as_tensor(m.atol(), device="cuda")
    if case["op"] != "stages":
        y = dense_rosenbrock(d, solver.params, x["y"], MECHANISMS[case["mech"]]["dt"], atol, m.relative_tolerance,
                             case["control"] == "per_cell")
        out = torch.empty_like(y)
        out[:, columns] = y
        return {"y": to_layout(out, L), "counts": {k: None for k in COUNTS}}
    cells = torch.arange(n, device="cuda")
    A = ALPHA * torch.eye(S, device="cuda", dtype=torch.float64) - d.jacobian(x["y"], cells)
    f = d.f(x["y"], cells)
    order = torch.argsort(columns)  # species of each column
    A, f = A[:, order][:, :, order].contiguous(), f[:, order]
    sol = torch.linalg.solve(A, f[:, :, None])[:, :, 0]
    for k in range(S - 1):  # LU without pivoting, in place
        A[:, k + 1:, k] /= A[:, k, k, None]
        A[:, k + 1:, k + 1:] -= A[:, k + 1:, k, None] * A[:, k, None, k + 1:]
    rows = torch.as_tensor(solver.compiled.rows.astype(np.int64), device="cuda")
    cols = torch.as_tensor(solver.compiled.cols.astype(np.int64), device="cuda")
    return {"x": to_layout(sol, L), "lu": to_layout(A[:, rows, cols], L)}

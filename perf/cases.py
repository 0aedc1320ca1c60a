"""The measured cases: what a program built on this library has it do.

Every case goes through the public entry points (multigrid_meshless_b200.api
and the C ABI of include/mgm.h behind it).  The families:

  weights  create_derivative_matrices on one level: host arrays in, the
           operator rows [n][k] out (api.derivative_weights)
  setup    a hierarchy built from its clouds (api.Multigrid: kNN clouds,
           reorder, derivative and transfer rows, solver data) and the first
           time step on it -- what a program pays before its loop starts
  steps    a short episode of fractional steps from rest (boundary conditions,
           then mgm_run_steps and mgm_step_host into page-locked buffers)
  timple   the same for the implicit TIMPLE loop
  batch    many Poisson right-hand sides through one batched V-cycle
  train    loss and gradient of the learned warm start on one sample

A pass of `steps` and `timple` starts from rest, so it does the same work each
time it is called; the fields it returns are those after its last step.
"""
import ctypes as C
import math
import random
import weakref

import numpy as np

from multigrid_meshless_b200 import (BC_LID, BC_TAYLOR_COUETTE, GUESS_EXTRAPOLATE, GUESS_LEARNED, MODE_FP32_IR,
                                     MODE_FP64, MODE_REFERENCE, api, clouds, load)
from multigrid_meshless_b200._lib import check

MODES = {"fp32": MODE_FP32_IR, "fp64": MODE_FP64, "reference": MODE_REFERENCE}


def listed():
    return [
        # the CPU-runnable configuration of the reference (128^2 cavity, k = 20, poly 3): its operator rows alone
        {"name": "weights-c1", "family": "weights", "shape": "cavity", "m": 128, "k": 20, "poly": 3},
        # set-up and first step of a 2D production cloud at the benchmark's stencils
        {"name": "setup-cavity", "family": "setup", "shape": "cavity", "m": 500, "levels": 5, "k": 30, "poly": 4,
         "mode": "fp32"},
        # the same in 3D
        {"name": "setup-cube", "family": "setup", "shape": "cube", "m": 40, "levels": 3, "k": 35, "poly": 2,
         "mode": "fp32"},
        # small interactive run: the reference's own size, bound by latency and launches
        {"name": "step-c1", "family": "steps", "shape": "cavity", "m": 128, "levels": 3, "k": 20, "poly": 3,
         "mode": "fp32", "guess": 0, "steps": 10, "courant": 0.3},
        # the benchmark's size: 1M-node cavity, extrapolated initial guess
        {"name": "step-cavity-1m", "family": "steps", "shape": "cavity", "m": 1000, "levels": 6, "k": 30, "poly": 4,
         "mode": "fp32", "guess": 1, "steps": 4, "courant": 0.3},
        # the plain FP64 arm, at a size between the two and not a power of two
        {"name": "step-cavity-fp64", "family": "steps", "shape": "cavity", "m": 411, "levels": 5, "k": 30, "poly": 4,
         "mode": "fp64", "guess": 0, "steps": 4, "courant": 0.3},
        # 3D lid-driven cube at the benchmark's stencil
        {"name": "step-cube", "family": "steps", "shape": "cube", "m": 64, "levels": 4, "k": 35, "poly": 2,
         "mode": "fp32", "guess": 0, "steps": 3, "courant": 0.1},
        # the benchmark's headline arm: extrapolation and the network's direction together
        {"name": "step-learned", "family": "steps", "shape": "cavity", "m": 500, "levels": 5, "k": 30, "poly": 4,
         "mode": "fp32", "guess": 3, "steps": 4, "courant": 0.3},
        # the reference's own multigrid (10 V-cycles of 3 sweeps), the drop-in program's mode
        {"name": "step-reference", "family": "steps", "shape": "cavity", "m": 256, "levels": 4, "k": 30, "poly": 4,
         "mode": "reference", "guess": 0, "steps": 2, "courant": 0.3},
        # the reference main's default loop, on the Taylor-Couette annulus it is shipped with
        {"name": "timple-annulus", "family": "timple", "nodes": 250000, "levels": 5, "k": 30, "poly": 4,
         "mode": "fp32", "compat": False, "steps": 2},
        # 64 right-hand sides on the sphere-in-sphere shell with per-node stencils
        {"name": "batch-shell", "family": "batch", "nodes": 100000, "levels": 3, "nrhs": 64, "mode": "fp32"},
        # one training sample of the warm-start network, forward and backward
        {"name": "train-sample", "family": "train", "m": 300, "levels": 4, "k": 30, "poly": 4},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cavity_levels(m):
    # the coarsest level is solved densely: 16 to 60 nodes across
    levels = 1
    while m > 40:
        m //= 2
        levels += 1
    return max(2, levels)


def draw(rng):
    fam = rng.choice(["weights", "setup", "setup", "steps", "steps", "steps", "steps", "steps", "timple", "batch",
                      "train"])
    k, poly = rng.choice([(20, 3), (25, 3), (30, 4), (33, 4)])
    if fam == "weights":
        if rng.random() < 0.3:
            return {"family": fam, "shape": "cube", "m": _logint(rng, 10, 36), "k": rng.choice([25, 35]), "poly": 2}
        return {"family": fam, "shape": "cavity", "m": _logint(rng, 40, 220), "k": k, "poly": poly}
    if fam == "setup":
        if rng.random() < 0.3:
            m = _logint(rng, 20, 44)
            return {"family": fam, "shape": "cube", "m": m, "levels": 3 if m >= 28 else 2, "k": rng.choice([30, 35]),
                    "poly": 2, "mode": "fp32"}
        m = _logint(rng, 64, 500)
        return {"family": fam, "shape": "cavity", "m": m, "levels": _cavity_levels(m), "k": k, "poly": poly,
                "mode": rng.choice(["fp32", "fp64"])}
    if fam == "steps":
        mode = rng.choice(["fp32", "fp32", "fp32", "fp64", "reference"])
        guess = rng.choice([0, 1, 1, 3]) if mode != "reference" else 0
        if rng.random() < 0.25:
            m = _logint(rng, 20, 56)
            return {"family": fam, "shape": "cube", "m": m, "levels": 3 if m >= 28 else 2, "k": rng.choice([30, 35]),
                    "poly": 2, "mode": mode, "guess": min(guess, 1), "steps": 3, "courant": 0.1}
        m = _logint(rng, 64, 600)
        return {"family": fam, "shape": "cavity", "m": m, "levels": _cavity_levels(m), "k": k, "poly": poly,
                "mode": mode, "guess": guess, "steps": rng.randint(2, 5), "courant": 0.3}
    if fam == "timple":
        nodes = _logint(rng, 8000, 250000)
        return {"family": fam, "nodes": nodes, "levels": 3 if nodes < 60000 else 4, "k": 30, "poly": 4,
                "mode": rng.choice(["fp32", "fp64"]), "compat": rng.random() < 0.5, "steps": 2}
    if fam == "batch":
        nodes = _logint(rng, 8000, 100000)
        return {"family": fam, "nodes": nodes, "levels": 3 if nodes >= 25000 else 2,
                "nrhs": rng.choice([5, 16, 32, 40, 64]), "mode": rng.choice(["fp32", "fp32", "fp64"])}
    m = _logint(rng, 64, 300)
    return {"family": fam, "m": m, "levels": _cavity_levels(m), "k": k, "poly": poly}


# ---------------------------------------------------------------------------
def _clouds(case, seed):
    if case["shape"] == "cube":
        return clouds.cube_hierarchy(case["m"], case.get("levels", 1), seed=seed)
    return clouds.cavity_hierarchy(case["m"], case.get("levels", 1), seed=seed)


def _reynolds(case, seed):
    # the benchmarks' ranges: U[100, 1000] in the cavity, 400 in the cube
    return 400.0 if case["shape"] == "cube" else random.Random(seed).uniform(100.0, 1000.0)


def _pinned(n):
    """Page-locked doubles as (array, address), given back when the last view of them goes."""
    p = api.PinnedArray(n)
    owner = p.array
    while isinstance(owner, np.ndarray):
        owner = owner.base
    weakref.finalize(owner, load().mgm_host_free, p.ptr).atexit = False
    return p.array, p.ptr


class _Steps:
    """A hierarchy, the flow's settings and page-locked buffers for the fields."""

    def __init__(self, case, cl, bc):
        nl = len(cl)
        self.mg = api.Multigrid(cl, [case["k"]] * nl, [case["poly"]] * nl, reference_transfer=case["mode"] == "reference")
        self.bc, self.mode = bc, MODES[case["mode"]]
        self.steps = case.get("steps", 1)
        n = self.mg.n()
        self.buf = {f: _pinned(n) for f in ("u", "v", "p")}

    def settings(self, Re, courant, deg, ratio):
        # omega: data-parallel sweeps of the reference's cycle need under-relaxation on Neumann rows
        self.mg.set_flow(Re=Re, courant=courant, omega=0.25, num_relax=3, num_vcycles=10)
        self.mg.set_solver(rel_tol=1e-8, max_iters=100, cheb_degree=deg, cheb_ratio=ratio)

    def episode(self):
        mg = self.mg
        mg.apply_bc(self.bc)
        if self.steps > 1:
            mg.run_steps(self.mode, self.steps - 1)
        err = mg.step_host(self.mode, u_out=self.buf["u"][1], v_out=self.buf["v"][1], p_out=self.buf["p"][1])
        out = {f: b[0] for f, b in self.buf.items()}
        out["steady"] = err
        if mg.dim == 3:
            out["w"] = mg.get_field("w")
        return out


def _solver(case):
    # the benchmark's smoother settings: degree 3 / ratio 20 on the cavity, 4 / 10 elsewhere
    return (3, 20.0) if case.get("shape") == "cavity" else (4, 10.0)


def prepare(case, seed):
    fam = case["family"]
    if fam == "weights":
        c = _clouds(dict(case, levels=1), seed)[0]
        cloud = api.knn_cloud(c.x, c.y, c.z, c.btag, c.nb, case["k"], c.dim)
        nx, ny, nz = api.correct_normals(c.x, c.y, c.z, c.btag, cloud, c.nx, c.ny, c.nz)
        return {"fam": fam, "args": (c.x, c.y, c.z, nx, ny, nz, c.btag, cloud, c.dim, 3, case["poly"])}
    if fam == "setup":
        return {"fam": fam, "case": case, "clouds": _clouds(case, seed), "Re": _reynolds(case, seed)}
    if fam == "steps":
        st = _Steps(case, _clouds(case, seed), BC_LID)
        st.settings(_reynolds(case, seed), case["courant"], *_solver(case))
        if case["guess"] & GUESS_LEARNED:
            check(load().mgm_mpnn_init(st.mg.h, seed, 0))
        st.mg.set_initial_guess(case["guess"])
        return {"fam": fam, "steps": st}
    if fam == "timple":
        cl = clouds.annulus_hierarchy(clouds.annulus_h_for_nodes(case["nodes"]), case["levels"], seed=seed)
        nl = len(cl)
        mg = api.Multigrid(cl, [case["k"]] * nl, [case["poly"]] * nl)
        mg.set_flow(Re=100.0, courant=0.5)
        mg.set_solver(rel_tol=1e-8, max_iters=100, cheb_degree=4, cheb_ratio=10.0)
        mg.set_timple(1, 5, 1.0, 1.0)
        if case["compat"]:
            mg.set_compatible_rhs(True)
        return {"fam": fam, "mg": mg, "mode": MODES[case["mode"]], "steps": case["steps"]}
    if fam == "batch":
        # one mesh, other right-hand sides with each seed
        cl = clouds.shell_hierarchy(clouds.shell_h_for_nodes(case["nodes"]), case["levels"], seed=1)
        ks = [clouds.shell_stencil_sizes(cl[0], 40, 60)] + [clouds.shell_stencil_sizes(c, 25, 35) for c in cl[1:]]
        b = api.Batch(cl, ks, [3] + [2] * (len(cl) - 1), autotune=True)
        b.set_solver(1e-8, 24, 4, 10.0)
        lev = b.level(0)
        c0 = clouds.Cloud(lev["x"], lev["y"], lev["z"], lev["nx"], lev["ny"], lev["nz"], lev["btag"], 0, 3, 0.0,
                          "shell3d", {"r_in": 0.5, "r_out": 1.0})
        f = clouds.gaussian_fields(c0, case["nrhs"], seed=seed, bumps=4)
        inner = lev["btag"] == 0
        f[:, ~inner] = 0.0
        f[:, inner] -= f[:, inner].mean(1, keepdims=True)
        f[:, 0] = 0.0
        rhs, sol = (_pinned(f.size)[0].reshape(f.shape) for _ in range(2))
        rhs[:] = f
        return {"fam": fam, "b": b, "rhs": rhs, "sol": sol, "mode": MODES[case["mode"]]}
    # train: normalised smooth fields, as the recorded samples are
    cl = clouds.cavity_hierarchy(case["m"], case["levels"], seed=seed)
    mg = api.Multigrid(cl, [case["k"]] * len(cl), [case["poly"]] * len(cl))
    check(load().mgm_mpnn_init(mg.h, seed, 0))
    g = mg.geometry(0)
    rng = np.random.default_rng(seed)
    fields = []
    for _ in range(4):
        f = np.zeros(mg.n())
        for _ in range(6):
            a, b, ph = rng.uniform(0.5, 6.0), rng.uniform(0.5, 6.0), rng.uniform(0, 2 * math.pi)
            f += rng.standard_normal() * np.cos(a * math.pi * g["x"] + ph) * np.cos(b * math.pi * g["y"])
        fields.append((f / math.sqrt(float(np.mean(f * f)))).astype(np.float32))
    return {"fam": fam, "mg": mg, "fields": fields, "np": load().mgm_mpnn_num_params()}


def run(state):
    fam = state["fam"]
    if fam == "weights":
        return api.derivative_weights(*state["args"])
    if fam == "setup":
        case = state["case"]
        st = _Steps(case, state["clouds"], BC_LID)
        st.settings(state["Re"], 0.1 if case["shape"] == "cube" else 0.3, *_solver(case))
        out = st.episode()
        out["dt"] = st.mg.dt
        return out
    if fam == "steps":
        return state["steps"].episode()
    if fam == "timple":
        mg = state["mg"]
        mg.apply_bc(BC_TAYLOR_COUETTE)
        mg.timple_run(state["mode"], state["steps"])
        return {f: mg.get_field(f) for f in ("u_new", "v_new", "p_old")}
    if fam == "batch":
        sol, _, rr, _ = state["b"].solve(state["rhs"], state["mode"], out=state["sol"])
        return sol
    L, mg = load(), state["mg"]
    loss = C.c_double()
    grads, pred = np.zeros(state["np"], np.float32), np.zeros(mg.n(), np.float32)
    b, p, dp, t = (f.ctypes.data for f in state["fields"])
    check(L.mgm_mpnn_loss_grad(mg.h, b, p, dp, t, C.byref(loss), grads.ctypes.data, pred.ctypes.data))
    return {"loss": loss.value, "grads": grads, "prediction": pred}


# ---------------------------------------------------------------------------
def _exact_weights(x, y, z, nx, ny, nz, btag, cloud, dim, phs, poly):
    """The RBF-FD rows (PHS r^3 plus monomials) from batched 64-bit solves in
    coordinates scaled by each stencil's radius."""
    n, k = cloud.shape
    P = np.stack([x, y, z][:dim], 1)
    if dim == 2:
        ex = [(i, j) for i in range(poly + 1) for j in range(poly + 1 - i)]
    else:
        ex = [(i, j, l) for i in range(poly + 1) for j in range(poly + 1 - i) for l in range(poly + 1 - i - j)]
    npoly = len(ex)
    N = k + npoly
    names = ["Dx", "Dy"] + (["Dz"] if dim == 3 else []) + ["lap"]
    out = {nm: np.zeros((n, k)) for nm in names}
    for a in range(0, n, 4096):
        cl = cloud[a:a + 4096]
        X = P[cl] - P[cl[:, :1]]
        h = np.sqrt((X ** 2).sum(2)).max(1)
        X = X / h[:, None, None]
        r = np.sqrt(((X[:, :, None] - X[:, None]) ** 2).sum(3))
        M = np.zeros((len(cl), N, N))
        M[:, :k, :k] = r ** 3
        for t, e in enumerate(ex):
            v = np.ones(X.shape[:2])
            for d in range(dim):
                v = v * X[:, :, d] ** e[d]
            M[:, :k, k + t] = v
            M[:, k + t, :k] = v
        rhs = np.zeros((len(cl), N, len(names)))
        r0 = np.sqrt((X ** 2).sum(2))
        for d in range(dim):
            rhs[:, :k, d] = -phs * X[:, :, d] * r0
            e1 = tuple(1 if q == d else 0 for q in range(dim))
            if e1 in ex:
                rhs[:, k + ex.index(e1), d] = 1.0
        rhs[:, :k, dim] = phs * phs * r0
        for d in range(dim):
            e2 = tuple(2 if q == d else 0 for q in range(dim))
            if e2 in ex:
                rhs[:, k + ex.index(e2), dim] = 2.0
        w = np.linalg.solve(M, rhs)[:, :k]
        for q, nm in enumerate(names):
            out[nm][a:a + 4096] = w[:, :, q] / (h[:, None] ** 2 if nm == "lap" else h[:, None])
    bnd = (np.asarray(btag) != 0)[:, None]
    dn = out["Dx"] * nx[:, None] + out["Dy"] * ny[:, None]
    if dim == 3:
        dn = dn + out["Dz"] * nz[:, None]
    out["lapP"] = np.where(bnd, dn, out["lap"])
    return out


def exact(case, seed):
    """64-bit values where plain numpy gives them in seconds: the operator
    rows.  The other families end in sparse solves on up to a million
    unknowns, or a network of 16-bit weights on their operators."""
    if case["family"] != "weights":
        return None
    return _exact_weights(*prepare(case, seed)["args"])


# ---------------------------------------------------------------------------
def _sizes(case):
    if case.get("shape") == "cube":
        return [max(3, case["m"] >> l) ** 3 for l in range(case.get("levels", 1))]
    if case["family"] in ("timple", "batch"):
        f = 8 if case["family"] == "batch" else 4
        return [max(64, case["nodes"] // f ** l) for l in range(case["levels"])]
    return [max(3, case["m"] >> l) ** 2 for l in range(case.get("levels", 1))]


def _weights_work(n, k, poly, dim, ops):
    npoly = (poly + 1) * (poly + 2) // 2 if dim == 2 else (poly + 1) * (poly + 2) * (poly + 3) // 6
    N = k + npoly
    # one symmetric system of order N solved for `ops` right-hand sides
    return {"bytes": n * (k * (4 + 8 * (ops + 1)) + 60), "flops": n * (N ** 3 / 3.0 + 4.0 * N * N * ops)}


def _vcycle_bytes(sizes, k, wb, deg):
    # each smoothing step and the residual read the operator (weight + 2-byte
    # offset) and the step's vectors once; the transfers theirs
    tot = 0
    for l, n in enumerate(sizes[:-1]):
        tot += (2 * deg + 1) * n * (k * (wb + 2) + 6 * wb)
        tot += (sizes[l + 1] + n) * (k * (wb + 2) + 3 * wb)
    return tot + sizes[-1] ** 2 * wb


def _solve_bytes(sizes, k, wb, deg, vcycles):
    n = sizes[0]
    return vcycles * (_vcycle_bytes(sizes, k, wb, deg) + n * (12 * k + 8 * (vcycles + 4))) + n * (12 * k + 40)


def _step_work(case, steps):
    sizes, k = _sizes(case), case["k"]
    dim = 3 if case.get("shape") == "cube" else 2
    wb = 4 if case["mode"] == "fp32" else 8
    step = sizes[0] * (k * (8 * (3 * dim + 1) + 12) + 8 * 8 * dim)
    if case["mode"] == "reference":
        # 10 V-cycles: per level 2 x 3 sweeps, a residual and the transfers
        step += sum(10 * 7 * n * (12 * k + 24) for n in sizes)
    else:
        vc = 6 if case.get("guess", 0) else 12  # V-cycles a step takes from rest, about
        step += _solve_bytes(sizes, k, wb, _solver(case)[0], vc)
    flops = 0.0
    if case.get("guess", 0) & GUESS_LEARNED:
        step += sizes[0] * 4 * (k * 8 + 256)
        flops = sizes[0] * 4 * 2.0 * 192 * 64
    return {"bytes": steps * step, "flops": steps * (flops + step / 4.0)}


def work(case):
    fam = case["family"]
    dim = 3 if case.get("shape") == "cube" else 2
    if fam == "weights":
        return _weights_work(_sizes(case)[0], case["k"], case["poly"], dim, dim + 1)
    if fam == "setup":
        sizes = _sizes(case)
        w = [_weights_work(n, case["k"], case["poly"], dim, dim + 1) for n in sizes]
        # prolongation rows on every level but the coarsest, restriction rows on every level but the finest
        w += [_weights_work(n, case["k"], case["poly"], dim, 1) for n in sizes[:-1] + sizes[1:]]
        s = _step_work(case, 1)
        return {"bytes": sum(v["bytes"] for v in w) + s["bytes"], "flops": sum(v["flops"] for v in w) + s["flops"]}
    if fam == "steps":
        return _step_work(case, case["steps"])
    if fam == "timple":
        sizes, k = _sizes(case), case["k"]
        per = 5 * sizes[0] * (28 * k + 80) + 2 * sizes[0] * (20 * k + 64)
        per += _solve_bytes(sizes, k, 4 if case["mode"] == "fp32" else 8, 4, 14)
        return {"bytes": case["steps"] * per, "flops": case["steps"] * per / 4.0}
    if fam == "batch":
        sizes, k, B, wb = _sizes(case), 45, case["nrhs"], 4 if case["mode"] == "fp32" else 8
        vc = 14
        per = sum((2 * 4 + 1) * n * (k * (wb + 4) + 4 * wb * B) for n in sizes[:-1]) + sizes[-1] ** 2 * wb
        per += sizes[0] * (12 * k + 8 * B * (vc + 4))
        flops = vc * B * sum(2.0 * 10 * n * k for n in sizes)
        return {"bytes": vc * per + 2 * 8 * B * sizes[0], "flops": flops}
    n, k = case["m"] ** 2, case["k"]
    # forward and backward of four 192 -> 64 layers: three GEMMs each, the gathers' rows read once
    return {"bytes": n * 4.0 * (2 * k * 8 + 64 * (2 + 4 + 4 + 2) + 192 * 4), "flops": n * 4 * 3 * 2.0 * 192 * 64}

"""The solves whose speed is measured: what a user's program has the library do, through its public binding.

Every case is one whole call as a program makes it: new right-hand sides go to the resident hierarchy from device
memory, the solve runs to its tolerance (1e-10 of the initial residual, as the benchmark and the fixtures ask), and
phi of every level comes back to device memory.  The hierarchy (box layouts, plans, operator coefficients) is made
beforehand, as a program keeps it over many right-hand sides; CUDA graphs are on, as in the benchmark.
"""
import ctypes
import functools
import importlib.util
import math
import os

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GRID_SEED = 20261203  # the seed of the benchmark's hierarchies


@functools.lru_cache(maxsize=None)
def _cmg():
    spec = importlib.util.spec_from_file_location("cmg", os.path.join(ROOT, "chombo_3.2_b200", "cmg.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def _solve(name, n0, **kw):
    case = dict(name=name, kind="solve", n0=n0, levels=1, max_box=32, block=8, grid_seed=GRID_SEED, op=0, alpha=0.0,
                beta=1.0, bc="DDDDDD", mixed=False, steps=0, members=1)
    case.update(kw)
    return case


VC = dict(op=1, alpha=1.0, beta=-1.0)  # variable-coefficient Helmholtz
HELM = dict(op=0, alpha=1.0, beta=-0.1)  # constant-coefficient Helmholtz


def listed():
    return [
        # A small constant-coefficient solve (the fixtures' smallest one-level size): launches and latency.
        _solve("poisson_32", 32, max_box=16),
        # The benchmark's configuration 0: one level of 64^3 in eight boxes.
        _solve("poisson_64", 64),
        # A channel as the projection's pressure solves set it up: periodic, wall and outflow faces, boxes of 24^3
        # that coarsen only twice, so the bottom level is large.
        _solve("helmholtz_96_ppnndd", 96, max_box=24, bc="PPNNDD", **HELM),
        # A small refined hierarchy.
        _solve("vc_2lev_64", 64, levels=2, **VC),
        # The benchmark's configuration 1, in FP64 and with FP32 V-cycles inside FP64 refinement.
        _solve("vc_3lev_128", 128, levels=3, **VC),
        _solve("vc_3lev_128_mixed", 128, levels=3, mixed=True, **VC),
        # The benchmark's configuration 2 (149M cells): the largest hierarchy.
        _solve("vc_3lev_256_mixed", 256, levels=3, mixed=True, **VC),
        # The configuration of the reference's published timing: one periodic level of 512^3 in 4096 boxes.
        _solve("helmholtz_512_periodic", 512, bc="PPPPPP", **HELM),
        # Batching: twelve independent two-level hierarchies solved as one forest (a group of configuration 3).
        _solve("forest_12x64_mixed", 64, kind="forest", levels=2, max_box=16, members=12, mixed=True, **VC),
        # A regrid's coarse-to-fine interpolation of a new finest level.
        _solve("fineinterp_128_l2", 128, kind="fineinterp", levels=3),
        # Time stepping: backward-Euler heat steps, each a solve with new coefficients.
        _solve("heat_3lev_32", 32, kind="heat", levels=3, steps=3, alpha=1.0),
        # The variable-coefficient example's solver: BiCGStab preconditioned by AMR V-cycles.
        _solve("bicgstab_3lev_64", 64, kind="bicgstab", levels=3, **VC),
    ]


def _size(rng, lo, hi, step):
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(step, int(round(n / step)) * step)


def draw(rng):
    kind = rng.choice(["level", "level", "amr", "amr", "amr", "forest", "fineinterp", "heat", "bicgstab"])
    seed = rng.randrange(1, 1 << 30)
    operator = rng.choice([VC, VC, HELM, {}])
    if kind == "level":
        # Boxes of 12, 20 and 24 cells stop coarsening early and leave a large bottom level.
        block, max_box = rng.choice([(8, 16), (8, 32), (8, 32), (8, 24), (4, 12), (4, 20)])
        top = 320 if max_box in (16, 32) else 96
        bc = rng.choice(["DDDDDD", "DDDDDD", "NNNNND", "PPNNDD", "PPPPPP"])
        constant = HELM if bc == "PPPPPP" else rng.choice([HELM, {}])
        return _solve("", _size(rng, 24, top, block), max_box=max_box, block=block, bc=bc, grid_seed=seed,
                      mixed=rng.random() < 0.3, **constant)
    levels = rng.choice([2, 3])
    max_box = rng.choice([16, 24, 32, 32])
    if kind == "amr":
        return _solve("", _size(rng, 16, 128, 8), levels=levels, max_box=max_box, grid_seed=seed,
                      bc=rng.choice(["DDDDDD", "DDDDDD", "NNNNND"]), mixed=rng.random() < 0.5, **operator)
    if kind == "forest":
        n0 = _size(rng, 32, 96, 16)
        return _solve("", n0, kind="forest", levels=2, max_box=rng.choice([16, 32]), grid_seed=seed,
                      members=rng.randrange(2, 17), mixed=rng.random() < 0.7, **operator)
    if kind == "fineinterp":
        return _solve("", _size(rng, 16, 128, 8), kind="fineinterp", levels=levels, max_box=max_box, grid_seed=seed)
    if kind == "heat":
        return _solve("", _size(rng, 16, 64, 8), kind="heat", levels=rng.choice([1, 2, 3]), max_box=max_box,
                      grid_seed=seed, steps=rng.randrange(1, 4), alpha=1.0)
    return _solve("", _size(rng, 16, 64, 8), kind="bicgstab", levels=rng.choice([1, 2, 3]), max_box=max_box,
                  grid_seed=seed, **operator)


# ------------------------------------------------------------------ layouts
@functools.lru_cache(maxsize=64)
def _boxes(n0, levels, max_box, block, seed):
    cmg = _cmg()
    if levels == 1:
        return [cmg.domain_split((0, 0, 0), (n0 - 1,) * 3, max_box, block)]
    return cmg.synthetic_hierarchy(n0, levels, max_box=max_box, block_factor=block, seed=seed)


def _members(case):
    """The box lists of every hierarchy of a case (one, or a forest's)."""
    return [_boxes(case["n0"], case["levels"], case["max_box"], case["block"], case["grid_seed"] + m)
            for m in range(case["members"])]


def _cells(boxes):
    return sum((b[3] - b[0] + 1) * (b[4] - b[1] + 1) * (b[5] - b[2] + 1) for b in boxes)


def _gather(dense, boxes):
    """A level's cells in the binding's order (box by box, x fastest) from a dense [z, y, x] array."""
    return torch.cat([dense[b[2]:b[5] + 1, b[1]:b[4] + 1, b[0]:b[3] + 1].reshape(-1) for b in boxes])


def _bumps(n, seed):
    """The benchmark's kind of right-hand side on an n^3 grid, dense [z, y, x]: 16 Gaussian bumps with centres in
    [0.2, 0.8]^3, widths in [0.02, 0.1] and amplitudes +-[0.5, 2]."""
    r = np.random.RandomState(seed % (1 << 31))
    centre, width = r.uniform(0.2, 0.8, (16, 3)), r.uniform(0.02, 0.1, 16)
    amp = r.uniform(0.5, 2.0, 16) * r.choice([-1.0, 1.0], 16)
    x = (np.arange(n) + 0.5) / n
    e = [torch.from_numpy(np.exp(-(x[None, :] - centre[:, d:d + 1]) ** 2 / (2 * width[:, None] ** 2))).cuda()
         for d in range(3)]
    plane = (e[1][:, :, None] * e[0][:, None, :]).reshape(16, n * n)
    return ((e[2] * torch.from_numpy(amp).cuda()[:, None]).T @ plane).reshape(n, n, n)


# -------------------------------------------------------------------- state
def _coarse_field(case, seed):
    """A solution-like field on the level below the interpolated one: smooth bumps, a jump and a little noise, so
    that the limiter takes all its branches."""
    n = case["n0"] << (case["levels"] - 2)
    g = torch.Generator(device="cuda").manual_seed(seed)
    f = _bumps(n, seed)
    f[:, :, n // 2:] += 0.25
    return f + 1e-3 * torch.randn(f.shape, dtype=torch.float64, device="cuda", generator=g)


def prepare(case, seed):
    cmg = _cmg()
    kind = case["kind"]
    members = _members(case)
    st = {"kind": kind, "cmg": cmg, "steps": case["steps"], "mixed": case["mixed"], "params": cmg.solve_params(eps=1e-10)}
    if kind == "fineinterp":
        coarse, fine = members[0][-2], members[0][-1]
        n = case["n0"] << (len(members[0]) - 1)
        st["op"] = cmg.FineInterp((0, 0, 0, n - 1, n - 1, n - 1), fine, coarse)
        st["coarse"] = _gather(_coarse_field(dict(case, levels=len(members[0])), seed), coarse)
        st["out"] = torch.empty(_cells(fine), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        return st
    if kind == "forest":
        h = cmg.Forest(case["n0"], members, op=case["op"], alpha=case["alpha"], beta=case["beta"], bc=case["bc"])
        h.fill_synthetic([seed * 1000 + m for m in range(case["members"])])
    else:
        h = cmg.Hierarchy(case["n0"], members[0], op=case["op"], alpha=case["alpha"], beta=case["beta"],
                          bc=case["bc"])
        h.fill_synthetic(seed, device=True)
    h.use_graphs(True)
    st["h"] = h
    levels = range(h.nlev)
    # fill_synthetic has made the coefficients and the right-hand sides on the device
    st["rhs"] = [torch.empty(h.num_cells(l), dtype=torch.float64, device="cuda") for l in levels]
    st["out"] = [torch.empty_like(r) for r in st["rhs"]]
    if kind == "solve" and h.nlev == 1:
        st["rhs"] = [_gather(_bumps(case["n0"], seed), members[0][0])]
    else:
        torch.cuda.synchronize()
        for l in levels:
            h.get_rhs_ptr(l, st["rhs"][l].data_ptr(), True)
    if kind == "heat":
        # the state before the steps starts as the source, as in the fixtures
        st["phi0"] = [r.clone() for r in st["rhs"]]
    st["ml"] = cmg.mlsolve_params(mg_iters=2, mg_smooth=4, imax=100, eps=1e-10)
    torch.cuda.synchronize()
    return st


def run(state):
    if state["kind"] == "fineinterp":
        state["op"].interp_to_fine_device(state["coarse"].data_ptr(), state["out"].data_ptr())
        return state["out"]
    cmg, h = state["cmg"], state["h"]
    for l, r in enumerate(state["rhs"]):
        h.set_rhs_ptr(l, r.data_ptr(), True)
    if state["kind"] == "heat":
        for l, p in enumerate(state["phi0"]):
            cmg._check(cmg.lib().cmg_set_phi(h.h, l, ctypes.c_void_p(p.data_ptr()), 1))
        h.backward_euler(state["params"], 1e-3, state["steps"])
    elif state["kind"] == "bicgstab":
        h.solve_bicgstab(state["ml"])
    else:
        h.solve(state["params"], mixed=state["mixed"])
    for l, p in enumerate(state["out"]):
        h.get_phi_ptr(l, p.data_ptr(), True)
    return state["out"]


# --------------------------------------------------------------------- cost
def work(case):
    """Bytes and operations of one pass.  A solve: ten V-cycles (what 1e-10 takes, give or take two; six for the
    periodic Helmholtz operator), each with eight red-black sweeps and two residuals per level, every operand of a
    sweep read once and its result written once (the correction in and out, the right-hand side and, for variable
    coefficients, a, lambda and three face arrays)."""
    members = _members(case)
    vc = case["op"] == 1
    if case["kind"] == "fineinterp":
        fine = _cells(members[0][-1])
        return {"bytes": fine * 9.0, "flops": fine * 6.0}
    cells = sum(_cells(b) for m in members for b in m)
    cells += sum(_cells(m[0]) for m in members) / 7.0  # the multigrid depths below level 0
    cycles = 6 if case["bc"] == "PPPPPP" else 10
    if case["kind"] == "heat":
        cycles = 7 * case["steps"]
    elif case["kind"] == "bicgstab":
        cycles = 32  # eight iterations of two preconditioner calls of two V-cycles
    sweep, resid = (8, 7) if vc else (3, 3)
    word = 4 if case["mixed"] else 8
    return {"bytes": float(cells * cycles * word * (8 * sweep + 2 * resid)),
            "flops": float(cells * cycles * 10 * (26 if vc else 11))}


def tolerance(case):
    if case["kind"] == "fineinterp":
        return {"rel": 1e-14, "max": 1e-12}
    if case["mixed"] and case["levels"] > 1:
        # Coarse cells under a finer level take no part in the composite residual and keep the rounding of the FP32
        # cycles: up to 5e-8 (3e-7 in one cell) between the mixed and the FP64 solve.
        return {"rel": 2e-7, "max": 1.5e-6}
    # Two solves to 1e-10 may stop one V-cycle apart: up to 1.2e-10 from the exact solution, 8e-10 (2e-9) after
    # three heat steps.
    return {"rel": 3e-9, "max": 1e-8} if case["kind"] == "heat" else {"rel": 5e-10, "max": 2e-9}


# -------------------------------------------------------------------- exact
def _second_difference(n, lo, hi):
    a = np.diag(-2.0 * np.ones(n)) + np.diag(np.ones(n - 1), 1) + np.diag(np.ones(n - 1), -1)
    if lo == "P":
        a[0, -1] += 1.0
        a[-1, 0] += 1.0
    else:
        a[0, 0] += 1.0 if lo == "N" else -1.0
        a[-1, -1] += 1.0 if hi == "N" else -1.0
    return a * (float(n) * n)


def exact(case, seed):
    """One level with constant coefficients: the discrete operator is a sum of three one-dimensional ones, solved by
    their eigenvectors.  FineInterp: the limited linear interpolation on dense arrays.  A composite solve over
    several refined levels has no such direct form (an iteration to 64 bits in plain torch takes minutes)."""
    if case["kind"] == "fineinterp":
        return _exact_interp(case, seed)
    if case["kind"] != "solve" or case["levels"] != 1 or case["op"] != 0:
        return None
    n, bc = case["n0"], case["bc"]
    val, vec = [], []
    for d in range(3):
        w, v = torch.linalg.eigh(torch.from_numpy(_second_difference(n, bc[2 * d], bc[2 * d + 1])).cuda())
        val.append(w)
        vec.append(v)
    f = _bumps(n, seed)
    turn = lambda t, m: torch.einsum("zyx,zc,yb,xa->cba", t, m[2], m[1], m[0])  # noqa: E731
    lap = val[2][:, None, None] + val[1][None, :, None] + val[0][None, None, :]
    u = turn(turn(f, vec) / (case["alpha"] + case["beta"] * lap), [v.T for v in vec])
    return [_gather(u, _members(case)[0][0])]


def _exact_interp(case, seed):
    boxes = _members(case)[0]
    c = _coarse_field(dict(case, levels=len(boxes)), seed)
    m = c[1:-1, 1:-1, 1:-1]
    n = c.shape[0]
    shifted = lambda k, j, i: c[1 + k:n - 1 + k, 1 + j:n - 1 + j, 1 + i:n - 1 + i]  # noqa: E731
    s = [0.5 * (shifted(0, 0, 1) - shifted(0, 0, -1)), 0.5 * (shifted(0, 1, 0) - shifted(0, -1, 0)),
         0.5 * (shifted(1, 0, 0) - shifted(-1, 0, 0))]
    hi, lo = m.clone(), m.clone()
    for k in (-1, 0, 1):
        for j in (-1, 0, 1):
            for i in (-1, 0, 1):
                hi, lo = torch.maximum(hi, shifted(k, j, i)), torch.minimum(lo, shifted(k, j, i))
    total = 0.5 * (s[0].abs() + s[1].abs() + s[2].abs())
    eta = torch.minimum(hi - m, m - lo)
    eta = torch.where(eta <= 1e-9 * hi.abs(), torch.zeros_like(eta),
                      torch.where(total > eta, eta / total, torch.ones_like(eta)))
    out = torch.empty((2 * n,) * 3, dtype=torch.float64, device=c.device)
    for k in (0, 1):
        for j in (0, 1):
            for i in (0, 1):
                v = c.clone()  # cells next to the domain boundary stay piecewise constant
                v[1:-1, 1:-1, 1:-1] += eta * ((i - 0.5) * 0.5 * s[0] + (j - 0.5) * 0.5 * s[1] + (k - 0.5) * 0.5 * s[2])
                out[k::2, j::2, i::2] = v
    return _gather(out, boxes[-1])

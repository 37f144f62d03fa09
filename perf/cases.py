"""Performance cases of the operator path: what a program built on dage_b200
has it do, through the public entry points, over the range of sizes,
precisions and options in use.

A case is a dict of plain values; ``prepare`` makes the inputs from a seed on
the GPU and the operator that such a program keeps, ``run`` is one pass,
``work`` the bytes and operations a pass cannot do without, ``exact`` the same
outputs in 64 bits from plain torch, without the library's code.

Families:

* ``cube``: the tensor-product operator on one cube, V and the energy.
* ``cube_host``: a batch of host (pinned) cubes through one operator.
* ``gbfmm``: the multipole operator on one cube, V and the energy.
* ``gbfmm_batch``: many densities of uneven grids through the batched one.
* ``inject``: bubbles into a cube.
* ``product``: the product of two functions held as cube plus bubbles.
"""
import math

import numpy as np
import torch

import dage_b200 as dage

NLIP = 7
TLIN, TLOG = 2.0, 1.0e3
DEV = "cuda"


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def _cube(name, precision, cells, step, nlin, nlog, gaussians, energy=0.0):
    return {"name": name, "family": "cube", "precision": precision, "cx": cells[0], "cy": cells[1],
            "cz": cells[2], "step": step, "nlin": nlin, "nlog": nlog, "gaussians": gaussians,
            "energy": energy}


def listed():
    return [
        # the smallest cubes of the test suite: launches and host calls count
        _cube("cube_fp64_25", "fp64", (4, 4, 4), 0.4, 10, 8, 1),
        # a molecule's bounding box: three different axes, the Helmholtz
        # kernel of an orbital update, the reference's default quadrature
        _cube("cube_fp64_helmholtz_97x121x73", "fp64", (16, 20, 12), 0.2, 10, 8, 4, energy=-0.5),
        # the FP64 drop-in at an ordinary production size
        _cube("cube_fp64_241", "fp64", (40, 40, 40), 0.2, 20, 20, 8),
        # the split-precision operator at the size of the single-box
        # validation configuration
        _cube("cube_fp16x3_121", "fp16x3", (20, 20, 20), 0.2, 20, 20, 2),
        # the headline benchmark: 481^3, 64 t-points, 32 Gaussians
        _cube("cube_fp16x3_481", "fp16x3", (80, 80, 80), 0.1, 32, 32, 32),
        # the split precision with the smallest error, mid size
        _cube("cube_bf16x6_253", "bf16x6", (42, 42, 42), 0.1, 32, 32, 16),
        # a host program (the Fortran caller) with its cubes in host memory
        {"name": "cube_host_fp16x3_181", "family": "cube_host", "precision": "fp16x3", "cx": 30,
         "cy": 30, "cz": 30, "step": 0.2, "nlin": 20, "nlog": 20, "gaussians": 4, "energy": 0.0,
         "count": 3},
        # the FP64 multipole operator, box edges of 30 points
        {"name": "gbfmm_fp64_121", "family": "gbfmm", "precision": "fp64", "cx": 20, "cy": 20,
         "cz": 20, "step": 0.2, "nlin": 20, "nlog": 20, "gaussians": 16, "energy": 0.0, "lmax": 12},
        # the GBFMM benchmark: 241^3, lmax 12, 4x4x4 boxes, 16 Gaussians
        {"name": "gbfmm_fp16x3_241", "family": "gbfmm", "precision": "fp16x3", "cx": 40, "cy": 40,
         "cz": 40, "step": 0.2, "nlin": 20, "nlog": 20, "gaussians": 16, "energy": 0.0, "lmax": 12},
        # one SCF step's densities of uneven sizes, Coulomb and Helmholtz
        {"name": "gbfmm_batch_mixed_sizes", "family": "gbfmm_batch", "precision": "fp16x3",
         "cells": "10 20 15 10 30 25", "step": 0.2, "nlin": 20, "nlog": 20, "lmax": 10,
         "gaussians": 4, "emin": 0.125, "emax": 2.0},
        # a 20-atom molecule's bubbles onto a 301^3 cube
        {"name": "inject_301", "family": "inject", "cx": 50, "cy": 50, "cz": 50, "step": 0.1,
         "atoms": 20, "lmax": 2, "radial_cells": 33},
        # a density from two orbitals with cusps
        {"name": "product_181", "family": "product", "cx": 30, "cy": 30, "cz": 30, "step": 0.15,
         "atoms": 12, "lmax": 2, "radial_cells": 33},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["cube", "cube", "cube", "cube_host", "gbfmm", "gbfmm", "gbfmm_batch",
                         "inject", "product"])
    nlin, nlog = rng.randint(6, 32), rng.randint(6, 32)
    if family in ("cube", "cube_host"):
        precision = rng.choice(["fp64", "fp16x3", "fp16x3", "bf16x3", "bf16x6"])
        most = {"fp64": 44, "fp16x3": 72, "bf16x3": 60, "bf16x6": 56}[precision]
        base = _log_int(rng, 3, most if family == "cube" else 32)
        cells = [max(3, int(round(base * rng.uniform(0.7, 1.15)))) for _ in range(3)]
        if rng.random() < 0.4:
            cells = [base] * 3
        case = {"family": family, "precision": precision, "cx": cells[0], "cy": cells[1],
                "cz": cells[2], "step": rng.choice([0.1, 0.15, 0.2, 0.3]), "nlin": nlin,
                "nlog": nlog, "gaussians": rng.randint(1, 16),
                "energy": rng.choice([0.0, 0.0, -0.5, -1.7]) if family == "cube" else 0.0}
        if family == "cube_host":
            case["count"] = rng.randint(2, 5)
        return case
    if family == "gbfmm":
        base = _log_int(rng, 8, 40)
        cells = [max(8, int(round(base * rng.uniform(0.8, 1.1)))) for _ in range(3)]
        if rng.random() < 0.5:
            cells = [base] * 3
        return {"family": family, "precision": rng.choice(["fp64", "fp16x3"]), "cx": cells[0],
                "cy": cells[1], "cz": cells[2], "step": 0.2, "nlin": rng.randint(10, 25),
                "nlog": rng.randint(10, 25), "gaussians": rng.randint(1, 16),
                "energy": rng.choice([0.0, 0.0, -0.5]), "lmax": rng.randint(6, 14)}
    if family == "gbfmm_batch":
        cells = [str(rng.choice([10, 13, 15, 20, 25, 30])) for _ in range(rng.randint(2, 8))]
        return {"family": family, "precision": rng.choice(["fp64", "fp16x3"]),
                "cells": " ".join(cells), "step": 0.2, "nlin": rng.randint(10, 25),
                "nlog": rng.randint(10, 25), "lmax": rng.randint(6, 12),
                "gaussians": rng.randint(1, 8), "emin": 0.125, "emax": 2.0}
    base = _log_int(rng, 6, 50 if family == "inject" else 32)
    cells = [max(5, int(round(base * rng.uniform(0.75, 1.0)))) for _ in range(3)]
    return {"family": family, "cx": cells[0], "cy": cells[1], "cz": cells[2],
            "step": rng.choice([0.1, 0.15, 0.2]), "atoms": rng.randint(1, 24),
            "lmax": rng.choice([0, 1, 2, 2, 3] if family == "inject" else [0, 1, 2]),
            "radial_cells": rng.choice([33, 33, 20, 48])}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _cells(case):
    return (case["cx"], case["cy"], case["cz"])


def _axis(ncell, step):
    """Points of an equidistant axis centred at 0."""
    return -0.5 * ncell * (NLIP - 1) * step + step * np.arange(ncell * (NLIP - 1) + 1)


def _grid(cells, step):
    return dage.Grid3D(tuple(dage.Grid1D.equidistant(-0.5 * c * (NLIP - 1) * step, c, step)
                             for c in cells))


def _density(rng, cells, step, count, device=DEV):
    """Sum of normalised Gaussians, widths the grid resolves, charges of both
    signs but mostly positive, inside the cube; [z, y, x]."""
    pts = [torch.tensor(_axis(c, step), dtype=torch.float64, device=device) for c in cells]
    alpha = np.exp(rng.uniform(np.log(0.1), np.log(0.2 / step ** 2), count))
    charge = rng.uniform(-0.5, 2.0, count)
    half = np.array([0.5 * c * (NLIP - 1) * step for c in cells])
    centre = rng.uniform(-0.6, 0.6, (count, 3)) * half
    e = [torch.stack([torch.exp(-a * (p - c[d]) ** 2) for a, c in zip(alpha, centre)])
         for d, p in enumerate(pts)]
    norm = torch.tensor(charge * (alpha / np.pi) ** 1.5, dtype=torch.float64, device=device)
    ez = e[2] * norm[:, None]
    rho = torch.empty((len(pts[2]), len(pts[1]), len(pts[0])), dtype=torch.float64, device=device)
    for z0 in range(0, rho.shape[0], 64):
        rho[z0:z0 + 64] = torch.matmul(ez[:, z0:z0 + 64].T[:, None, :] * e[1].T[None, :, :], e[0])
    return rho


def _densities(case, seed):
    """[(cells, density)] of a case."""
    rng = np.random.default_rng([seed, 17])
    if case["family"] == "gbfmm_batch":
        cells = [(int(c),) * 3 for c in case["cells"].split()]
    else:
        cells = [_cells(case)] * case.get("count", 1)
    return [(c, _density(rng, c, case["step"], case["gaussians"])) for c in cells]


def _energies(case, seed):
    """Batch: every other density has the Helmholtz kernel."""
    rng = np.random.default_rng([seed, 23])
    n = len(case["cells"].split())
    e = -rng.uniform(case["emin"], case["emax"], n)
    e[1::2] = 0.0
    return e


def _radial(case):
    """Radial cell steps: cell ends at 0 and log-spaced on [1e-5, 15] bohr."""
    nc = case["radial_cells"]
    edges = np.concatenate([[0.0], 1e-5 * (15.0 / 1e-5) ** (np.arange(nc) / (nc - 1))])
    return np.diff(edges) / (NLIP - 1)


def _radial_points(h):
    starts = np.concatenate([[0.0], np.cumsum(h * (NLIP - 1))])
    return np.concatenate([[0.0]] + [s + hh * np.arange(1, NLIP) for s, hh in zip(starts, h)])


def _bubble_sets(case, seed, lmaxs):
    """Centres and, per set (one lmax each), per atom ((lmax+1)^2, points)
    radial values c r^l e^(-zeta r)."""
    rng = np.random.default_rng([seed, 31])
    half = np.array([0.5 * c * (NLIP - 1) * case["step"] for c in _cells(case)])
    centres = rng.uniform(-1.0, 1.0, (case["atoms"], 3)) * half
    r = _radial_points(_radial(case))
    sets = []
    for lmax in lmaxs:
        fs = []
        for _ in range(case["atoms"]):
            fs.append(np.stack([rng.uniform(-1, 1) * r ** l * np.exp(-rng.uniform(0.5, 3) * r)
                                for l in range(lmax + 1) for _ in range(2 * l + 1)]))
        sets.append(fs)
    return centres, sets


def _lmaxs(case):
    """inject: one set; product: the two factors and the result's bubbles."""
    return (case["lmax"],) if case["family"] == "inject" else (case["lmax"], case["lmax"], 2 * case["lmax"])


def _smooth_cubes(case, seed, count):
    rng = np.random.default_rng([seed, 41])
    return [_density(rng, _cells(case), case["step"], 3) for _ in range(count)]


def prepare(case, seed):
    family = case["family"]
    if family in ("inject", "product"):
        grid = _grid(_cells(case), case["step"])
        radial = dage.Grid1D(0.0, case["radial_cells"], NLIP, 1, _radial(case))
        centres, sets = _bubble_sets(case, seed, _lmaxs(case))
        b = [dage.Bubbles(centres, [radial] * case["atoms"], f, lmax) for f, lmax in zip(sets, _lmaxs(case))]
        if family == "inject":
            (base,) = _smooth_cubes(case, seed, 1)
            return {"case": case, "grid": grid, "b": b[0], "base": base, "cube": torch.empty_like(base)}
        c1, c2 = _smooth_cubes(case, seed, 2)
        return {"case": case, "grid": grid, "b1": b[0], "b2": b[1], "b12": b[2], "c1": c1,
                "c2": c2, "out": torch.empty_like(c1)}
    quad = dage.GaussQuad(case["nlin"], case["nlog"], 0.0, TLIN, TLOG)
    dens = _densities(case, seed)
    rhos = [r for _, r in dens]
    if family == "gbfmm_batch":
        op = dage.GBFMMBatch([_grid(c, case["step"]) for c, _ in dens], lmax=case["lmax"], quad=quad,
                             precision=case["precision"])
        op.set_energies(_energies(case, seed))
        return {"case": case, "op": op, "rho": rhos, "V": [torch.empty_like(r) for r in rhos]}
    grid = _grid(_cells(case), case["step"])
    if family == "gbfmm":
        if case["energy"] < 0.0:
            op = dage.GBFMMHelmholtz3D(grid, case["energy"], lmax=case["lmax"], quad=quad,
                                       precision=case["precision"])
        else:
            op = dage.GBFMMCoulomb3D(grid, lmax=case["lmax"], quad=quad, precision=case["precision"])
        return {"case": case, "op": op, "rho": rhos[0], "V": torch.empty_like(rhos[0])}
    op = dage.Coulomb3D(grid, quad=quad, precision=case["precision"])
    if family == "cube_host":
        host = [torch.empty(r.shape, dtype=torch.float64, pin_memory=True) for r in rhos]
        for h, r in zip(host, rhos):
            h.copy_(r)
        return {"case": case, "op": op, "rho": host,
                "V": [torch.empty(r.shape, dtype=torch.float64, pin_memory=True) for r in rhos]}
    if case["energy"] < 0.0:
        op = dage.Helmholtz3D(op, case["energy"])
    return {"case": case, "op": op, "rho": rhos[0], "V": torch.empty_like(rhos[0])}


def run(state):
    family = state["case"]["family"]
    if family == "inject":
        state["cube"].copy_(state["base"])
        return state["b"].inject(state["grid"], state["cube"])
    if family == "product":
        return dage.multiply(state["grid"], state["c1"], state["c2"], state["b1"], state["b2"],
                             state["b12"], out=state["out"])
    if family == "cube_host":
        n = len(state["rho"])
        e = dage.apply_batched([state["op"]] * n, state["rho"], state["V"], energy=True)
        return {"V": state["V"], "E": e}
    if family == "gbfmm_batch":
        e = state["op"].apply(state["rho"], state["V"], energy=True)
        return {"V": state["V"], "E": e}
    v, e = state["op"].apply(state["rho"], out=state["V"], energy=True)
    return {"V": v, "E": np.float64(e)}


# ---------------------------------------------------------------------------
# Work and tolerance
# ---------------------------------------------------------------------------
def _tpoints(nlin, nlog):
    """t-points and weights: Gauss-Legendre on [0, TLIN] and on log t over
    [TLIN, TLOG]."""
    x, w = np.polynomial.legendre.leggauss(nlin)
    t, tw = 0.5 * TLIN * (1 + x), 0.5 * TLIN * w
    x, w = np.polynomial.legendre.leggauss(nlog)
    tl = TLIN * (TLOG / TLIN) ** (0.5 * (x + 1))
    return np.concatenate([t, tl]), np.concatenate([tw, 0.5 * math.log(TLOG / TLIN) * w * tl])


def _band_entries(n, step, t):
    """Entries of an n x n operator matrix above 2^-64 of their row's scale:
    |i - j| within the Gaussian's reach and one cell of basis function."""
    w = int(min(n, math.sqrt(64 * math.log(2)) / (t * step) + NLIP - 1))
    return n * (2 * w + 1) - w * (w + 1) if w < n else n * n


def _cube_flops(points, step, tps):
    """Three mode products per t-point on the entries of the matrices that matter."""
    total = 0.0
    for t in tps:
        k = [_band_entries(n, step, t) / n for n in points]
        total += 2.0 * float(np.prod(points, dtype=np.float64)) * sum(k)
    return total


def _gbfmm_work(cells, case):
    n = [6 * c + 1 for c in cells]
    pts = float(np.prod(n, dtype=np.float64))
    tps, _ = _tpoints(case["nlin"], case["nlog"])
    nlm = (case["lmax"] + 1) ** 2
    flops = 0.0
    # near field: per axis the box's own points against 2 or 3 boxes' points
    for t in tps:
        reach = math.sqrt(64 * math.log(2)) / (t * case["step"]) + NLIP - 1
        near = [sum(min(nn * f / 4, 2 * reach + 1) for f in (2, 3, 3, 2)) / 4 for nn in n]
        # rows of a stage relative to its output points: near y z, near z, own
        flops += 2.0 * pts * (near[0] * 6.25 + near[1] * 2.5 + near[2])
    # moments and local expansions: separable polynomials of degree lmax per axis
    flops += 2 * 2.0 * pts * (case["lmax"] + 1)
    flops += 2.0 * 3096 * nlm ** 2  # far-field pairs of 4x4x4 boxes
    return {"bytes": 16.0 * pts, "flops": flops}


def work(case):
    family = case["family"]
    if family == "gbfmm_batch":
        ws = [_gbfmm_work((int(c),) * 3, case) for c in case["cells"].split()]
        return {"bytes": sum(w["bytes"] for w in ws), "flops": sum(w["flops"] for w in ws)}
    n = [6 * c + 1 for c in _cells(case)]
    pts = float(np.prod(n, dtype=np.float64))
    if family == "gbfmm":
        return _gbfmm_work(_cells(case), case)
    if family == "inject":
        nlm = (case["lmax"] + 1) ** 2
        return {"bytes": 16.0 * pts, "flops": pts * case["atoms"] * (14.0 * nlm + 40)}
    if family == "product":
        nlm = 2 * (case["lmax"] + 1) ** 2 + (2 * case["lmax"] + 1) ** 2
        return {"bytes": 24.0 * pts, "flops": pts * case["atoms"] * (14.0 * nlm + 40)}
    tps, _ = _tpoints(case["nlin"], case["nlog"])
    count = case.get("count", 1)
    return {"bytes": 16.0 * pts * count, "flops": _cube_flops(n, case["step"], tps) * count}


def tolerance(case):
    precision = case.get("precision", "fp64")
    if case["family"] in ("inject", "product"):
        return {"rel": 1e-13, "max": 1e-11}  # 64-bit polynomials and sums
    return {
        # 64 bits; the closed-form matrix entries cancel to ~1e-9 of V
        "fp64": {"rel": 1e-9, "max": 4e-8},
        # two FP16 parts (22 bits), FP32 partial sums
        "fp16x3": {"rel": 1e-6, "max": 2e-5},
        # three BF16 parts, FP32 sums
        "bf16x6": {"rel": 1e-6, "max": 2e-5},
        # two BF16 parts (16 bits)
        "bf16x3": {"rel": 8e-6, "max": 1e-4},
    }[precision]


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------
def _lagrange():
    """Coefficients c[j][k] of x^k of the NLIP Lagrange polynomials on the
    nodes -3 .. 3."""
    nodes = np.arange(NLIP) - (NLIP - 1) // 2
    return np.linalg.inv(np.vander(nodes.astype(np.float64), increasing=True)).T.copy()


def _lip_weights(ncell, step):
    """Integration weights of the points of `ncell` cells."""
    half = (NLIP - 1) // 2
    c = _lagrange()
    k = np.arange(NLIP)
    per = step * (c * ((half ** (k + 1.0) - (-half) ** (k + 1.0)) / (k + 1))).sum(1)
    w = np.zeros(ncell * (NLIP - 1) + 1)
    for i in range(ncell):
        w[i * (NLIP - 1):i * (NLIP - 1) + NLIP] += per
    return w


def _operator_matrices(ncell, step, first, out, tps):
    """T[p, i, j] = integral of basis function j of the `ncell` cells that
    start at `first` times exp(-t_p^2 (x_i - x)^2), by Gauss-Legendre
    quadrature on both sides of x_i (out to exp(-44))."""
    gx, gw = np.polynomial.legendre.leggauss(40)
    gx = torch.tensor(gx, dtype=torch.float64, device=DEV)
    gw = torch.tensor(gw, dtype=torch.float64, device=DEV)
    lag = torch.tensor(_lagrange(), dtype=torch.float64, device=DEV)
    xi = torch.tensor(out, dtype=torch.float64, device=DEV)[:, None]
    lo = torch.tensor(first + step * (NLIP - 1) * np.arange(ncell), dtype=torch.float64, device=DEV)[None, :]
    hi, mid = lo + step * (NLIP - 1), lo + 0.5 * step * (NLIP - 1)
    n_in = ncell * (NLIP - 1) + 1
    T = torch.zeros((len(tps), len(out), n_in), dtype=torch.float64, device=DEV)
    for p, t in enumerate(tps):
        reach = math.sqrt(44.0) / t
        for a, b in ((torch.maximum(lo, xi - reach), torch.minimum(hi, xi.expand(-1, ncell))),
                     (torch.maximum(lo, xi.expand(-1, ncell)), torch.minimum(hi, xi + reach))):
            half = 0.5 * (b - a).clamp_min(0.0)
            x = (0.5 * (a + b))[..., None] + half[..., None] * gx
            e = torch.exp(-(t * (xi[..., None] - x)) ** 2) * (half[..., None] * gw)
            s = (x - mid[..., None]) / step
            mom, cur = [], e
            for _ in range(NLIP):
                mom.append(cur.sum(-1))
                cur = cur * s
            mom = torch.stack(mom, -1) @ lag.T  # [i, cell, j]
            for j in range(NLIP):
                T[p, :, j:j + ncell * (NLIP - 1):NLIP - 1] += mom[..., j]
    return T


def _weights(case_energy, tps, tw):
    w = 2.0 / math.sqrt(math.pi) * tw
    return w * np.exp(2.0 * case_energy / (4.0 * tps ** 2)) if case_energy < -0.005 else w


def _contract(Tx, Ty, Tz, w, rho):
    """sum_p w_p Tx Ty Tz rho for rho [z, y, x]."""
    V = torch.zeros((Tz.shape[1], Ty.shape[1], Tx.shape[1]), dtype=torch.float64, device=DEV)
    for p in range(len(w)):
        a = torch.matmul(rho, Tx[p].T)          # z y i
        a = torch.matmul(Ty[p], a)              # z j i
        s = a.shape
        V += w[p] * (Tz[p] @ a.reshape(s[0], -1)).reshape(V.shape)
    return V


def _integral(cells, step, a, b):
    wx, wy, wz = (torch.tensor(_lip_weights(c, step), dtype=torch.float64, device=DEV) for c in cells)
    return float(((a * b) @ wx @ wy @ wz).item())


def _exact_cube(cells, case, rho, energy):
    tps, tw = _tpoints(case["nlin"], case["nlog"])
    T = {}
    for c in set(cells):
        T[c] = _operator_matrices(c, case["step"], _axis(c, case["step"])[0], _axis(c, case["step"]), tps)
    V = _contract(T[cells[0]], T[cells[1]], T[cells[2]], _weights(energy, tps, tw), rho)
    V += math.pi / TLOG ** 2 * rho
    return V, _integral(cells, case["step"], rho, V)


def _harmonics(lmax, x, y, z):
    """Racah-normalised real regular solid harmonics [(lmax+1)^2, ...], lm at l(l+1)+m."""
    S = [None] * (lmax + 1) ** 2
    S[0] = torch.ones_like(x)
    r2 = x * x + y * y + z * z
    for l in range(1, lmax + 1):
        top, bot = S[l * l - 1], S[(l - 1) ** 2] if l > 1 else torch.zeros_like(x)
        f = 1.0 if l == 1 else math.sqrt((2 * l - 1.0) / (2 * l))
        S[l * l + 2 * l] = f * (x * top - y * bot)
        S[l * l] = f * (y * top + x * bot)
        for m in range(-l + 1, l):
            v = (2 * l - 1) / math.sqrt((l + m) * (l - m)) * z * S[(l - 1) * l + m]
            if l - abs(m) > 1:
                v = v - math.sqrt((l + m - 1.0) * (l - m - 1.0) / ((l + m) * (l - m))) * r2 * S[(l - 2) * (l - 1) + m]
            S[l * (l + 1) + m] = v
    return torch.stack(S)


def _bessel_ratio(lmax, x):
    """i_l(x) / x^l of the modified spherical Bessel functions, [lmax+1, ...]."""
    out = [None] * (lmax + 2)
    for l in (lmax, lmax + 1):
        term = torch.full_like(x, 1.0 / float(np.prod(np.arange(1, 2 * l + 2, 2, dtype=np.float64))))
        out[l] = term.clone()
        for k in range(1, 30 + int(1.5 * float(x.max()))):
            term = term * (x * x / 2) / (k * (2 * l + 2 * k + 1))
            out[l] += term
    for l in range(lmax, 0, -1):
        out[l - 1] = x * x * out[l + 1] + (2 * l + 1) * out[l]
    return torch.stack(out[:lmax + 1])


def _regular(lmax, kappa, x, y, z):
    """Solid harmonics, or i_l(kappa r) Y_lm for kappa > 0."""
    S = _harmonics(lmax, x, y, z)
    if kappa > 0:
        f = _bessel_ratio(lmax, kappa * torch.sqrt(x * x + y * y + z * z))
        for l in range(lmax + 1):
            S[l * l:(l + 1) ** 2] *= f[l] * kappa ** l
    return S


def _coulomb_m2l(lmax, d, scale):
    """Local expansions about 0 of the multipoles at d (rows [displacement]):
    the potentials S_lm(r - d) / |r - d|^(2l+1) on a sphere of radius `scale`,
    projected on its harmonics."""
    nt, npz = 40, 80
    u, wu = np.polynomial.legendre.leggauss(nt)
    ph = 2 * np.pi * np.arange(npz) / npz
    s = np.sqrt(1 - u * u)
    n = np.stack([(s[:, None] * np.cos(ph)).ravel(), (s[:, None] * np.sin(ph)).ravel(), np.repeat(u, npz)])
    n = torch.tensor(n, dtype=torch.float64, device=DEV)
    wq = torch.tensor(np.repeat(wu, npz) / (2.0 * npz), dtype=torch.float64, device=DEV)  # sums to 1
    Y = _harmonics(lmax, n[0], n[1], n[2])
    ls = torch.tensor(np.repeat(np.arange(lmax + 1.0), 2 * np.arange(lmax + 1) + 1), device=DEV)
    proj = Y * wq * ((2 * ls + 1) / scale ** ls)[:, None]
    d = torch.tensor(np.asarray(d), device=DEV)
    out = []
    for dv in d.split(32):
        x, y, z = (scale * n[i] - dv[:, i, None] for i in range(3))
        r = torch.sqrt(x * x + y * y + z * z)
        phi = _harmonics(lmax, x / r, y / r, z / r) / r ** (ls[:, None, None] + 1)
        out.append(torch.einsum("ln,mdn->dlm", proj, phi))
    return torch.cat(out)


def _helmholtz_m2l(lmax, kappa, d):
    """The multipole-to-local conversion for e^(-kappa r)/r as the operator
    defines it: coaxial coefficients by recurrence from k_0 .. k_(lmax+1)
    (entries the recurrence never reaches are zero), rotated to each
    displacement.  d [displacement]: source - target."""
    L = lmax
    d = np.asarray(d)
    dist = np.linalg.norm(d, axis=1)
    x = (kappa * dist).astype(np.longdouble)
    k = [np.exp(-x) / x * np.pi / 2, np.exp(-x) * (x + 1) / (x * x) * np.pi / 2]
    for l in range(2, L + 2):
        k.append((2 * l - 1) * k[l - 1] / x + k[l - 2])
    k = [v.astype(np.float64) for v in k]
    C = np.zeros((L + 3, L + 3, L + 3, len(d)))  # index -1 .. L+1 at 0 .. L+2

    def at(l, n, m):
        return C[l + 1, n + 1, m + 1]

    def a(n, m):
        return 0.0 if n < 0 else math.sqrt((n + 1 + abs(m)) * (n + 1 - abs(m)) / ((2 * n + 1) * (2 * n + 3)))

    def b(n, m):
        if n < 0 or abs(m) > n:
            return 0.0
        v = math.sqrt((n - m - 1) * (n - m) / ((2 * n - 1) * (2 * n + 1)))
        return -v if m < 0 else v

    at(0, 0, 0)[:] = k[0]
    for n in range(1, L + 2):
        at(n, 0, 0)[:] = (-1) ** n * math.sqrt(2 * n + 1) * k[n]
        at(0, n, 0)[:] = math.sqrt(2 * n + 1) * k[n]
    for n in range(1, L + 1):
        at(1, n, 0)[:] = (-a(n, 0) * at(0, n + 1, 0) - a(n - 1, 0) * at(0, n - 1, 0)) / a(0, 0)
        at(n, 1, 0)[:] = (-1) ** (1 + n) * at(1, n, 0)
    for m in range(L + 1):
        for n in range(m, L + 1):
            for l in range(m, L + 1):
                at(l, n + 1, m)[:] = (-a(l, m) * at(l + 1, n, m) - a(l - 1, m) * at(l - 1, n, m)
                                      - a(n - 1, m) * at(l, n - 1, m)) / a(n, m)
        for l in range(m, L + 1):
            at(l, m + 1, m + 1)[:] = (-b(l, -m - 1) * at(l - 1, m, m) - b(l + 1, m) * at(l + 1, m, m)) \
                / b(m + 1, -m - 1)
    N = (L + 1) ** 2
    dirs = np.random.default_rng(7).normal(size=(3, 4 * (2 * L + 1)))
    dirs /= np.linalg.norm(dirs, axis=0)
    ls = np.repeat(np.arange(L + 1), 2 * np.arange(L + 1) + 1)
    ms = np.concatenate([np.arange(-l, l + 1) for l in range(L + 1)])
    zz = -d / dist[:, None]
    t = np.where(np.abs(zz[:, :1]) > 0.9, [[0.0, 1.0, 0.0]], [[1.0, 0.0, 0.0]])
    xx = np.cross(t, zz)
    xx /= np.linalg.norm(xx, axis=1, keepdims=True)
    Q = np.stack([xx, np.cross(zz, xx), zz], 2)
    turned = torch.tensor(np.einsum("dij,jn->idn", Q, dirs), device=DEV)
    here = _harmonics(L, *torch.tensor(dirs, device=DEV))
    there = _harmonics(L, *turned)
    R = torch.zeros((len(d), N, N), dtype=torch.float64, device=DEV)
    for l in range(L + 1):  # S_lm(Q n) = sum_m' R[m', m] S_lm'(n)
        s = slice(l * l, (l + 1) ** 2)
        R[:, s, s] = torch.einsum("mdn,nk->dkm", there[s], torch.linalg.pinv(here[s]))
    axial = np.where(ms[:, None] == ms[None, :], 1.0, 0.0)[..., None] * \
        C[ls[:, None] + 1, ls[None, :] + 1, np.abs(ms)[None, :] + 1]
    axial = torch.tensor(np.moveaxis(axial, 2, 0), device=DEV)
    f = torch.tensor(np.sqrt(4 * np.pi / (2 * ls + 1)), device=DEV)
    return f[:, None] * (R.transpose(1, 2) @ axial @ R) / f


def _exact_gbfmm(cells, case, rho, energy):
    step, lmax, nb = case["step"], case["lmax"], 4
    kappa = math.sqrt(-2 * energy) if energy < 0 else 0.0
    tps, tw = _tpoints(case["nlin"], case["nlog"])
    w = _weights(energy, tps, tw)
    pts = [_axis(c, step) for c in cells]

    def split(c, v):  # first and one-past-last cell of box position v
        base, rem = divmod(c, nb)
        c0 = v * base + min(v, rem)
        return c0, c0 + base + (1 if v < rem else 0)

    mats, own = {}, {}
    for d, c in enumerate(cells):
        for v in range(nb):
            c0, c1 = split(c, v)
            n0, n1 = split(c, max(v - 1, 0))[0], split(c, min(v + 1, nb - 1))[1]
            own[d, v] = (c0 * 6, c1 * 6 + (1 if c1 == c else 0))
            if (c, v) not in mats:
                mats[c, v] = (n0 * 6, n1 * 6 + 1, _operator_matrices(
                    n1 - n0, step, pts[d][n0 * 6], pts[d][own[d, v][0]:own[d, v][1]], tps))
    boxes = [(x, y, z) for z in range(nb) for y in range(nb) for x in range(nb)]
    centre, q = {}, {}
    for bx in boxes:
        cc, sub = [], []
        for d in range(3):
            c0, c1 = split(cells[d], bx[d])
            cc.append(0.5 * (pts[d][c0 * 6] + pts[d][c1 * 6]))
            sub.append((c0 * 6, c1 * 6 + 1, torch.tensor(_lip_weights(c1 - c0, step), device=DEV)))
        centre[bx] = np.array(cc)
        (x0, x1, wx), (y0, y1, wy), (z0, z1, wz) = sub
        X, Y, Z = (torch.tensor(pts[d][s[0]:s[1]] - cc[d], device=DEV) for d, s in enumerate(sub))
        q[bx] = torch.zeros((lmax + 1) ** 2, dtype=torch.float64, device=DEV)
        for k in range(z0, z1, 64):  # slabs of planes
            e = min(k + 64, z1)
            g = rho[k:e, y0:y1, x0:x1] * wx * wy[:, None] * wz[k - z0:e - z0, None, None]
            ZZ, YY, XX = (v.reshape(-1) for v in torch.meshgrid(Z[k - z0:e - z0], Y, X, indexing="ij"))
            q[bx] += _regular(lmax, kappa, XX, YY, ZZ) @ g.reshape(-1)
    disp, index = [], {}
    width = max(step * 6 * split(c, 0)[1] for c in cells)
    pairs = {}
    for t in boxes:
        pairs[t] = []
        for s in boxes:
            if max(abs(s[d] - t[d]) for d in range(3)) > 1 and max(abs(s[d] // 2 - t[d] // 2) for d in range(3)) <= 1:
                dv = centre[s] - centre[t]
                key = tuple(np.round(dv, 9))
                if key not in index:
                    index[key] = len(disp)
                    disp.append(dv)
                pairs[t].append((s, index[key]))
    T = _helmholtz_m2l(lmax, kappa, disp) if kappa > 0 else _coulomb_m2l(lmax, disp, 0.8 * width)
    V = torch.empty_like(rho)
    ls = torch.tensor(np.repeat(np.arange(lmax + 1.0), 2 * np.arange(lmax + 1) + 1), device=DEV)
    for bx in boxes:
        L = sum(T[i] @ q[s] for s, i in pairs[bx])
        if kappa > 0:
            L = L * 8 * kappa * (2 * ls + 1) / (4 * math.pi)
        (ax0, ax1, Tx), (ay0, ay1, Ty), (az0, az1, Tz) = (mats[cells[d], bx[d]] for d in range(3))
        near = _contract(Tx, Ty, Tz, w, rho[az0:az1, ay0:ay1, ax0:ax1])
        o = [own[d, bx[d]] for d in range(3)]
        X, Y, Z = (torch.tensor(pts[d][o[d][0]:o[d][1]] - centre[bx][d], device=DEV) for d in range(3))
        for k in range(0, len(Z), 64):
            ZZ, YY, XX = (v.reshape(-1) for v in torch.meshgrid(Z[k:k + 64], Y, X, indexing="ij"))
            near[k:k + 64] += (L @ _regular(lmax, kappa, XX, YY, ZZ)).reshape(-1, len(Y), len(X))
        V[o[2][0]:o[2][1], o[1][0]:o[1][1], o[0][0]:o[0][1]] = near
    return V, _integral(cells, step, rho, V)


def _exact_bubbles(case, centres, fs, lmax):
    """Sum over atoms of f_lm(|r - R|) Y_lm at the cube's points, [z, y, x]."""
    h = _radial(case)
    starts = torch.tensor(np.concatenate([[0.0], np.cumsum(h * (NLIP - 1))]), device=DEV)
    hh = torch.tensor(h, device=DEV)
    nc = len(h)
    lag = _lagrange()
    pts = [torch.tensor(_axis(c, case["step"]), device=DEV) for c in _cells(case)]
    out = torch.zeros(tuple(len(p) for p in pts[::-1]), dtype=torch.float64, device=DEV)
    coef = []
    for f in fs:  # [cell, lm, power]
        cells = np.stack([f[:, 6 * c:6 * c + NLIP] @ lag for c in range(nc)])
        coef.append(torch.tensor(cells, device=DEV))
    for z0 in range(0, out.shape[0], 8):
        Z, Y, X = torch.meshgrid(pts[2][z0:z0 + 8], pts[1], pts[0], indexing="ij")
        acc = torch.zeros_like(X)
        for c, k in zip(centres, coef):
            dx, dy, dz = X - c[0], Y - c[1], Z - c[2]
            r = torch.sqrt(dx * dx + dy * dy + dz * dz)
            inside = (r <= starts[-1]) & (r > 0)
            dx, dy, dz, r = dx[inside], dy[inside], dz[inside], r[inside]
            cell = (torch.searchsorted(starts, r, right=True) - 1).clamp(0, nc - 1)
            t = (r - starts[cell]) / hh[cell] - (NLIP - 1) // 2
            S = _harmonics(lmax, dx / r, dy / r, dz / r)
            v = torch.zeros_like(r)
            for lm in range((lmax + 1) ** 2):
                p = k[cell, lm, NLIP - 1]
                for e in range(NLIP - 2, -1, -1):
                    p = p * t + k[cell, lm, e]
                v += p * S[lm]
            acc[inside] += v
        out[z0:z0 + 8] = acc
    return out


def exact(case, seed):
    family = case["family"]
    if family == "inject":
        centres, sets = _bubble_sets(case, seed, _lmaxs(case))
        (base,) = _smooth_cubes(case, seed, 1)
        return base + _exact_bubbles(case, centres, sets[0], case["lmax"])
    if family == "product":
        centres, sets = _bubble_sets(case, seed, _lmaxs(case))
        f1, f2 = (c + _exact_bubbles(case, centres, f, case["lmax"])
                  for c, f in zip(_smooth_cubes(case, seed, 2), sets))
        return f1 * f2 - _exact_bubbles(case, centres, sets[2], 2 * case["lmax"])
    got = []
    energies = _energies(case, seed) if family == "gbfmm_batch" else None
    for i, (cells, rho) in enumerate(_densities(case, seed)):
        energy = float(energies[i]) if energies is not None else case["energy"]
        if family in ("gbfmm", "gbfmm_batch"):
            got.append(_exact_gbfmm(cells, case, rho, energy))
        else:
            got.append(_exact_cube(cells, case, rho, energy))
    if family in ("gbfmm_batch", "cube_host"):
        return {"V": [v.cpu() if family == "cube_host" else v for v, _ in got],
                "E": np.array([e for _, e in got])}
    return {"V": got[0][0], "E": np.float64(got[0][1])}

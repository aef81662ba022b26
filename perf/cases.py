"""The work that programs have this framework do, as cases that can be timed.

Every case goes through the public Python layer (`aphi_b200`): assembly of a
frequency sweep, one request of a solver service, a frequency sweep in FP64
and in mixed precision, solves with a resident factor, the host-array
pipeline, the residual check of given solutions and the fields of a solution.

`listed()` gives the fixed cases, `draw(rng)` more of the same ranges;
`prepare(case, seed)` builds what a program has in hand (mesh, ordering,
analysis, assembly, systems, right-hand sides), `run(state)` makes one pass
and returns its outputs, `work(case)` says what the pass cannot do without
and `exact(case, seed)` what the outputs are in plain torch FP64.

Materials, port voltages, frequencies and right-hand sides come from the seed.
Frequencies of the solved systems lie between 50 Hz and 1 kHz: further up the
systems' own conditioning (their smallest pivot falls like 1 / omega) leaves
fewer than nine digits of a solution to compare on the larger meshes, while
the work of a factorization does not depend on the frequency.
"""
from __future__ import annotations

import functools
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "hybrid-aphi-solver_b200"))

import aphi_b200 as ab  # noqa: E402

F_LO, F_HI = 50.0, 1.0e3          # Hz, solved systems
F_LO_FILL, F_HI_FILL = 50.0, 1.0e6  # Hz, assembly and fields alone
DENSE_FLOPS = 2.5e14              # exact(): the dense factorizations stay within seconds


def listed():
    return [
        # One small system filled at one frequency: what a tuning loop or a
        # service with small meshes calls between solves; launches and latency.
        {"name": "refill_8", "do": "refill", "mesh": "cylinder", "cells": 8, "freqs": 1, "form": "row_scaled"},
        # The benchmark's sweep: 16 frequencies of the 32^3 cylinder filled in
        # one call; the largest fill.
        {"name": "refill_32", "do": "refill", "mesh": "cylinder", "cells": 32, "freqs": 16, "form": "row_scaled"},
        # Relative residual and backward error of given solutions, as a
        # program checks what it serves or hands on.
        {"name": "check_24", "do": "check", "mesh": "cylinder", "cells": 24, "freqs": 4, "rhs": 2},
        # Fields of one solution of the torus with its cut port.
        {"name": "fields_16", "do": "fields", "mesh": "torus", "cells": 16, "freqs": 1, "form": "row_scaled"},
        # The smallest configuration (6^3 at 50 Hz) through the pipeline on
        # host arrays that replaces the reference's solve_symmetric.
        {"name": "host_6", "do": "host", "mesh": "cylinder", "cells": 6, "freqs": 1, "rhs": 1},
        # One request of the service on its smallest mesh: four excitations of
        # one frequency, factorized in FP64 and solved.
        {"name": "request_8", "do": "request", "mesh": "cylinder", "cells": 8, "freqs": 1, "rhs": 4},
        # A batch of requests on a medium mesh.
        {"name": "request_16", "do": "request", "mesh": "cylinder", "cells": 16, "freqs": 4, "rhs": 2},
        # Eight excitations solved with a factor that is kept.
        {"name": "solve_24", "do": "solve", "mesh": "cylinder", "cells": 24, "freqs": 1, "rhs": 8},
        # Plain FP64 sweeps: eight frequencies of a medium mesh, two of the
        # benchmark's mesh (nearly all of it the trailing updates).
        {"name": "sweep64_24", "do": "sweep", "mesh": "cylinder", "cells": 24, "freqs": 8, "precision": "fp64"},
        {"name": "sweep64_32", "do": "sweep", "mesh": "cylinder", "cells": 32, "freqs": 2, "precision": "fp64"},
        # Mixed sweeps: FP32 factors refined in FP64; the band in which the
        # benchmark's sweep stays in FP32.
        {"name": "sweep_mixed_24", "do": "sweep", "mesh": "cylinder", "cells": 24, "freqs": 8, "precision": "mixed"},
        {"name": "sweep_mixed_32", "do": "sweep", "mesh": "cylinder", "cells": 32, "freqs": 6, "precision": "mixed"},
    ]


def draw(rng: random.Random):
    def size(lo, hi):  # over the logarithm, odd sizes among them
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    do = rng.choice(["refill", "check", "fields", "host", "request", "request", "solve", "sweep64", "sweep64", "mixed"])
    form = rng.choice(["row_scaled", "scaled_phi"])
    if do == "refill":
        cells = size(6, 32)
        return {"do": do, "mesh": "cylinder", "cells": cells, "freqs": size(1, 16), "form": form}
    if do == "check":
        return {"do": do, "mesh": "cylinder", "cells": size(6, 24), "freqs": size(1, 4), "rhs": rng.randint(1, 4)}
    if do == "fields":
        if rng.random() < 0.5:
            return {"do": do, "mesh": "torus", "cells": 2 * size(7, 14), "freqs": 1, "form": form}   # even ones only
        return {"do": do, "mesh": "cylinder", "cells": size(6, 24), "freqs": 1, "form": form}
    if do == "host":
        return {"do": do, "mesh": "cylinder", "cells": size(4, 14), "freqs": 1, "rhs": 1}
    if do == "request":
        return {"do": do, "mesh": "cylinder", "cells": size(6, 20), "freqs": rng.randint(1, 4), "rhs": rng.randint(1, 8)}
    if do == "solve":
        return {"do": do, "mesh": "cylinder", "cells": size(8, 26), "freqs": rng.randint(1, 3), "rhs": rng.randint(1, 8)}
    if do == "mixed":
        cells = size(12, 30)
        return {"do": "sweep", "mesh": "cylinder", "cells": cells, "freqs": rng.randint(2, 6), "precision": "mixed"}
    cells = size(10, 30)
    return {"do": "sweep", "mesh": "cylinder", "cells": cells, "freqs": rng.randint(2, 2 if cells > 26 else 6),
            "precision": "fp64"}


# ---------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=6)
def _mesh(mesh: str, cells: int):
    """The mesh's host tables and ordering, which a program makes once."""
    w = ab.Workload.torus(cells) if mesh == "torus" else ab.Workload.cylinder(cells)
    return w, ab.workload_arrays(w), ab.amd_ordering(w.row_ptr, w.col_idx)


def _form(case) -> int:
    return ab.COND_SCALED_PHI if case.get("form") == "scaled_phi" else ab.COND_ROW_SCALED


def _inputs(case, seed: int):
    """(mesh tables with the seed's materials and excitation, angular frequencies, numpy generator)."""
    _, arrays, _ = _mesh(case["mesh"], case["cells"])
    rng = np.random.default_rng([seed, case["cells"], case["freqs"]])
    a = dict(arrays)
    material = a["material"].reshape(-1, 3).copy()
    material[:, 0] *= rng.uniform(0.8, 1.25, len(material))   # conductivities
    a["material"] = material.reshape(-1)
    a["port_value"] = a["port_value"] * rng.uniform(0.5, 2.0)
    a["port_amplitude"] = a["port_amplitude"] * rng.uniform(0.5, 2.0)
    a["tet_fixed"] = a["tet_fixed"] * rng.uniform(0.5, 2.0)
    solved = case["do"] not in ("refill", "fields")
    lo, hi = (F_LO, F_HI) if solved else (F_LO_FILL, F_HI_FILL)
    hz = np.geomspace(lo, hi, case["freqs"] + 1)
    hz = hz[:-1] * (hz[1:] / hz[:-1]) ** rng.uniform(0.0, 1.0, case["freqs"])   # one in each part of the band
    return a, 2.0 * np.pi * hz, rng


def _vectors(case, rng, n: int) -> np.ndarray:
    shape = (case["freqs"], case["rhs"], n)
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def prepare(case, seed: int):
    w, _, perm = _mesh(case["mesh"], case["cells"])
    arrays, omegas, rng = _inputs(case, seed)
    s = {"case": case, "omegas": omegas, "form": _form(case), "assembly": ab.Assembly(arrays)}
    do = case["do"]
    if do == "refill":
        return s
    n = s["assembly"].num_unknowns
    if do == "fields":
        x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        return s | {"fields": ab.Fields.of_workload(s["assembly"], w), "x": torch.from_numpy(x).cuda()}
    s["analysis"] = ab.Analysis(w.row_ptr, w.col_idx, perm)
    if do == "sweep":
        s["solver"] = ab.SweepSolver(s["analysis"], s["assembly"], case["freqs"], case["precision"])
        return s
    if do == "host":
        s["values"], s["rhs"] = s["assembly"].refill_host(float(omegas[0]))
        return s
    if do in ("check", "solve"):
        s["values"], _ = s["assembly"].refill(omegas)
        s["b"] = torch.from_numpy(_vectors(case, rng, n)).cuda()
    if do == "check":
        s["x"] = torch.from_numpy(_vectors(case, rng, n)).cuda()
    if do in ("request", "solve"):
        s["factor"] = ab.Factor(s["analysis"], ab.PREC_FP64, case["freqs"])
    if do == "solve":
        s["factor"].factorize(s["values"])
    if do == "request":  # a request's excitations scale the port's right-hand side
        v = rng.standard_normal((case["freqs"], case["rhs"], 1)) + 1j * rng.standard_normal((case["freqs"], case["rhs"], 1))
        s["voltages"] = torch.from_numpy(v).cuda()
    return s


def run(s):
    do = s["case"]["do"]
    if do == "refill":
        return s["assembly"].refill(s["omegas"], s["form"])
    if do == "fields":
        return s["fields"].compute(s["x"], float(s["omegas"][0]), s["form"])
    if do == "check":
        return ab.residuals(s["analysis"], s["values"], s["x"], s["b"])
    if do == "host":
        ok, x, report = ab.solve_symmetric(s["analysis"], s["values"], s["rhs"])
        return {"ok": ok, "x": x, "columns_done": int(report["columns_done"])}
    if do == "solve":
        return s["factor"].solve(s["b"])
    if do == "request":
        values, rhs = s["assembly"].refill(s["omegas"])
        ok = s["factor"].factorize(values)
        return {"ok": ok, "x": s["factor"].solve(s["voltages"] * rhs[:, None, :])}
    x, values, rhs, _ = s["solver"].solve(s["omegas"])
    return {"x": x, "values": values, "rhs": rhs}


# ---------------------------------------------------------------- work
def work(case):
    """Bytes and operations of one pass: each input read and each output
    written once; a factorization's flops are the unpadded count of the
    elimination tree, and its factor is written once and read twice (forward
    and backward); an element fill is counted by its outputs and tables."""
    w, _, perm = _mesh(case["mesh"], case["cells"])
    nf, n, nnz, t = case["freqs"], w.num_unknowns, w.nnz, w.num_tets
    do = case["do"]
    fill = {"bytes": 16.0 * nf * (nnz + n) + 4.0 * nnz + 350.0 * t, "flops": 60.0 * 100 * t + 500.0 * nf * t}
    if do == "refill":
        return fill
    if do == "fields":
        p2 = w.num_nodes + w.num_edges
        return {"bytes": 16.0 * n + 350.0 * t + t * (12 * 16 + 8) + p2 * (16 * 16 + 9.0), "flops": 1.0e3 * t}
    if do == "check":
        return {"bytes": 16.0 * nf * nnz + 4.0 * nnz + 32.0 * nf * case["rhs"] * n, "flops": 16.0 * nf * case["rhs"] * nnz}
    info = ab.Analysis(w.row_ptr, w.col_idx, perm).info
    nnz_l, flops, rhs = info["nnz_l"], info["flops"], case.get("rhs", 1)
    size = 8.0 if case.get("precision") == "mixed" else 16.0
    solve = {"bytes": nf * (2 * size * nnz_l + 32.0 * rhs * n), "flops": 16.0 * nf * rhs * nnz_l}
    if do == "solve":
        return solve
    out = {"bytes": solve["bytes"] + nf * (size * nnz_l + 16.0 * nnz), "flops": solve["flops"] + nf * flops}
    if do in ("request", "sweep"):
        out = {k: out[k] + fill[k] for k in out}
    return out


# ---------------------------------------------------------------- exact
_EDGES = ((0, 1), (0, 2), (0, 3), (1, 2), (2, 3), (1, 3))


def _elements(a):
    """Per tet, over the degree-2 rule: curl.curl and Whitney mass (6 x 6),
    Whitney . P2 gradient (6 x 10) and gradient . gradient (10 x 10)
    integrals, on the GPU."""
    dev = dict(dtype=torch.float64, device="cuda")
    p = torch.from_numpy(a["xyz"].reshape(-1, 3)[a["tets"].reshape(-1, 4)]).to(**dev)
    one = torch.cat([torch.ones(p.shape[:2] + (1,), **dev), p], 2)
    grad = torch.linalg.inv(one)[:, 1:, :].transpose(1, 2)               # T, vertex, xyz
    vol = torch.linalg.det(one).abs() / 6.0
    i, j = torch.tensor(_EDGES).T
    curl = 2.0 * torch.linalg.cross(grad[:, i], grad[:, j], dim=2)
    s5 = math.sqrt(5.0)
    hi, lo = (5.0 + 3.0 * s5) / 20.0, (5.0 - s5) / 20.0
    cc = torch.einsum("t,tik,tjk->tij", vol, curl, curl)
    ww = torch.zeros_like(cc)
    wg = torch.zeros(cc.shape[0], 6, 10, **dev)
    gg = torch.zeros(cc.shape[0], 10, 10, **dev)
    for q in range(4):
        b = torch.full((4,), lo, **dev)
        b[q] = hi
        wh = grad[:, j] * b[i][None, :, None] - grad[:, i] * b[j][None, :, None]
        g = torch.cat([grad * (4.0 * b - 1.0)[None, :, None],
                       4.0 * (grad[:, i] * b[j][None, :, None] + grad[:, j] * b[i][None, :, None])], 1)
        ww += torch.einsum("t,tik,tjk->tij", vol / 4, wh, wh)
        wg += torch.einsum("t,tik,tjk->tij", vol / 4, wh, g)
        gg += torch.einsum("t,tik,tjk->tij", vol / 4, g, g)
    return cc, ww, wg, gg


def _systems(case, seed):
    """(values [freqs, nnz], rhs [freqs, n]) of the case's systems, plain torch."""
    a, omegas, _ = _inputs(case, seed)
    n, nnz, t = a["row_ptr"].size - 1, a["col_idx"].size, a["tets"].size // 4
    cc, ww, wg, gg = _elements(a)
    idx = torch.from_numpy(a["tet_idx"].reshape(t, 16).astype(np.int64)).cuda()
    co = torch.from_numpy(a["tet_coeff"].reshape(t, 16)).cuda()
    fixed = torch.view_as_complex(torch.from_numpy(a["tet_fixed"].reshape(t, 10, 2).copy()).cuda())
    body = np.zeros(t, np.int64)
    for b in range(a["body_ptr"].size - 1):
        body[a["body_tets"][a["body_ptr"][b]:a["body_ptr"][b + 1]]] = b
    sigma, eps, mu = (torch.from_numpy(c).cuda() for c in a["material"].reshape(-1, 3)[body].T.copy())
    mu, eps = mu * 4.0e-7 * math.pi, eps * 8.8541878128e-12
    rows = np.repeat(np.arange(n, dtype=np.int64), np.diff(a["row_ptr"]))
    key = torch.from_numpy(rows * n + a["col_idx"]).cuda()
    row, col = idx[:, :, None].expand(t, 16, 16), idx[:, None, :].expand(t, 16, 16)
    keep = (row >= 0) & (col >= row)
    slot = torch.searchsorted(key, (row * n + col)[keep])
    values = torch.zeros(len(omegas), nnz, dtype=torch.complex128, device="cuda")
    rhs = torch.zeros(len(omegas), n, dtype=torch.complex128, device="cuda")
    for f, om in enumerate(omegas):
        jw = 1j * om
        r, c = (1.0, jw) if _form(case) == ab.COND_SCALED_PHI else (1.0 / jw, 1.0)
        alpha, beta = torch.complex(-om * om * eps, om * sigma), torch.complex(sigma, om * eps)
        e = torch.zeros(t, 16, 16, dtype=torch.complex128, device="cuda")
        e[:, :6, :6] = cc / mu[:, None, None] + alpha[:, None, None] * ww
        e[:, :6, 6:] = c * beta[:, None, None] * wg
        e[:, 6:, :6] = r * jw * (beta[:, None, None] * wg).transpose(1, 2)
        e[:, 6:, 6:] = r * c * beta[:, None, None] * gg
        given = torch.where(idx[:, 6:] < 0, fixed / c, torch.zeros_like(fixed))   # prescribed potentials
        b = -(co * torch.einsum("tij,tj->ti", e[:, :, 6:], given))
        rhs[f].index_add_(0, idx[idx >= 0], b[idx >= 0])
        values[f].index_add_(0, slot, (e * (co[:, :, None] * co[:, None, :]))[keep])
        diag = a["row_ptr"][a["port_row"]]                                        # upper rows begin on the diagonal
        for p in range(a["port_row"].size):
            if a["port_current"][p]:
                rhs[f, int(a["port_row"][p])] += r * complex(*a["port_amplitude"].reshape(-1, 2)[p])
            else:
                values[f, int(diag[p])] += 1.0
                rhs[f, int(a["port_row"][p])] += complex(*a["port_value"].reshape(-1, 2)[p]) / c
    return values, rhs, torch.from_numpy(rows).cuda(), torch.from_numpy(a["col_idx"].astype(np.int64)).cuda()


def _full(values, rows, cols, n):
    off = rows != cols
    return torch.sparse_coo_tensor(torch.stack([torch.cat([rows, cols[off]]), torch.cat([cols, rows[off]])]),
                                   torch.cat([values, values[off]]), (n, n)).coalesce()


def _solve(values, rows, cols, b):
    """A^-1 b by a dense LU of the scaled system, refined in FP64 (b: [rhs, n])."""
    n = b.shape[1]
    a = _full(values, rows, cols, n)
    d = torch.zeros(n, dtype=torch.float64, device="cuda").index_reduce_(0, a.indices()[0], a.values().abs(), "amax")
    d = d.rsqrt()
    dense = torch.sparse_coo_tensor(a.indices(), a.values() * d[a.indices()[0]] * d[a.indices()[1]], (n, n)).to_dense()
    lu, piv = torch.linalg.lu_factor(dense)
    del dense
    x = torch.zeros_like(b.T)
    for _ in range(3):
        r = b.T - torch.sparse.mm(a, x)
        x = x + d[:, None] * torch.linalg.lu_solve(lu, piv, d[:, None] * r)
    return x.T


def exact(case, seed: int):
    do = case["do"]
    if do == "fields":
        return None
    n = _mesh(case["mesh"], case["cells"])[0].num_unknowns
    if do not in ("refill", "check") and 8.0 / 3.0 * n ** 3 * case["freqs"] > DENSE_FLOPS:
        return None
    values, rhs, rows, cols = _systems(case, seed)
    if do == "refill":
        return values, rhs
    _, _, rng = _inputs(case, seed)
    if do == "check":
        b = torch.from_numpy(_vectors(case, rng, n)).cuda()
        x = torch.from_numpy(_vectors(case, rng, n)).cuda()
        out = np.zeros(b.shape[:2] + (2,))
        for f in range(b.shape[0]):
            a = _full(values[f], rows, cols, n)
            for k in range(b.shape[1]):
                r = float(torch.linalg.vector_norm(b[f, k] - torch.mv(a, x[f, k])))
                bn = float(torch.linalg.vector_norm(b[f, k]))
                size = float(values[f].abs().max() * torch.linalg.vector_norm(x[f, k]))
                out[f, k] = r / bn, r / (size + bn)
        return out
    if do == "solve":
        b = torch.from_numpy(_vectors(case, rng, n)).cuda()
    elif do == "request":
        v = rng.standard_normal((case["freqs"], case["rhs"], 1)) + 1j * rng.standard_normal((case["freqs"], case["rhs"], 1))
        b = torch.from_numpy(v).cuda() * rhs[:, None, :]
    else:
        b = rhs[:, None, :]
    x = torch.stack([_solve(values[f], rows, cols, b[f]) for f in range(case["freqs"])])
    if do == "host":
        return {"ok": True, "x": x[0, 0].cpu().numpy(), "columns_done": None}
    if do == "solve":
        return x
    if do == "request":
        return {"ok": True, "x": x}
    return {"x": x[:, 0], "values": values, "rhs": rhs}

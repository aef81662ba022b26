"""Post-solve fields against their definition in NumPy, on meshes whose tets
fill a block of k_field_tets (16) not at all, exactly, by one more, and many
times, with nodes of no tet and an interface of both sigma and mu.

The bound: an entry sums at most about 40 contributions of some 100 rounded
operations on gradients whose own error is a few units times the tets' shape
factor (below 20): (40 + 100) * 20 * 1.1e-16 < 1e-12 of an array's largest."""
import numpy as np
import pytest
import torch

import aphi_b200 as ab

pytestmark = pytest.mark.gpu

EDGES = [(0, 1), (0, 2), (0, 3), (1, 2), (2, 3), (1, 3)]


def fields_numpy(a, tet_edges, num_edges, x, omega, scale):
    xyz, tets = a["xyz"].reshape(-1, 3), a["tets"].reshape(-1, 4)
    idx, coeff = a["tet_idx"].reshape(-1, 16), a["tet_coeff"].reshape(-1, 16)
    fixed = a["tet_fixed"].reshape(-1, 10, 2) @ [1.0, 1.0j]
    mat, T, nv = a["material"].reshape(-1, 3), len(tets), len(xyz)
    body = np.zeros(T, int)
    for i in range(len(mat)):
        body[a["body_tets"][a["body_ptr"][i]:a["body_ptr"][i + 1]]] = i
    sigma, mu = mat[body, 0], 4e-7 * np.pi * mat[body, 2]
    M = np.concatenate([np.ones((T, 4, 1)), xyz[tets]], axis=2)
    grad, vol = np.linalg.inv(M)[:, 1:, :].transpose(0, 2, 1), np.abs(np.linalg.det(M)) / 6
    u = np.where(idx >= 0, x[idx], 0)
    av, ph = u[:, :6] * coeff[:, :6], np.where(idx[:, 6:] >= 0, scale * coeff[:, 6:] * u[:, 6:], fixed)
    b = sum(2 * av[:, k, None] * np.cross(grad[:, i], grad[:, j]) for k, (i, j) in enumerate(EDGES))

    def at(L):
        A = sum(av[:, k, None] * (grad[:, j] * L[i] - grad[:, i] * L[j]) for k, (i, j) in enumerate(EDGES))
        g = sum(ph[:, n, None] * grad[:, n] * (4 * L[n] - 1) for n in range(4))
        g = g + sum(ph[:, 4 + k, None] * 4 * (grad[:, i] * L[j] + grad[:, j] * L[i]) for k, (i, j) in enumerate(EDGES))
        return A, -1j * omega * A - g

    out = {"a_tet": at([0.25] * 4)[0], "e_tet": at([0.25] * 4)[1], "b_tet": b, "sigma_tet": sigma}
    out["j_tet"] = sigma[:, None] * out["e_tet"]
    points = list(np.eye(4)) + [(np.eye(4)[i] + np.eye(4)[j]) / 2 for i, j in EDGES]
    nodes = np.concatenate([tets, nv + tet_edges.reshape(-1, 6)], axis=1)
    Pn = nv + num_edges
    smax, mmax, smin, mmin = np.full(Pn, -1.0), np.full(Pn, -1.0), np.full(Pn, 1e300), np.full(Pn, 1e300)
    for k in range(10):
        np.maximum.at(smax, nodes[:, k], sigma), np.minimum.at(smin, nodes[:, k], sigma)
        np.maximum.at(mmax, nodes[:, k], mu), np.minimum.at(mmin, nodes[:, k], mu)
    vw, ew, bw = np.zeros(Pn), np.zeros(Pn), np.zeros(Pn)
    an, en, bn, phi = (np.zeros((Pn, 3), complex) for _ in range(4))
    for k in range(10):
        A, E = at(points[k])
        n, on_e, on_b = nodes[:, k], sigma == smax[nodes[:, k]], mu == mmax[nodes[:, k]]
        np.add.at(vw, n, vol), np.add.at(ew, n, vol * on_e), np.add.at(bw, n, vol * on_b)
        np.add.at(an, n, vol[:, None] * A)
        np.add.at(en, n, (vol * on_e)[:, None] * E), np.add.at(bn, n, (vol * on_b)[:, None] * b)
        live = idx[:, 6 + k] >= 0
        phi[n, 0] = np.where(live, scale * u[:, 6 + k], fixed[:, k])
    has = vw > 0
    out["a_node"] = an / np.where(has, vw, 1)[:, None]
    out["e_node"] = en / np.where(has, ew, 1)[:, None]
    out["b_node"] = bn / np.where(has, bw, 1)[:, None]
    out["j_node"] = out["e_node"] * np.where(has, smax, 0)[:, None]
    out["h_node"] = out["b_node"] / np.where(has, mmax, 1)[:, None]
    out |= {"phi_node": phi[:, 0], "vertex_weight": vw,
            "on_interface": (has & ((smax != smin) | (mmax != mmin))).astype(np.uint8)}
    return out


@pytest.mark.parametrize("num_tets", [1, 15, 16, 17, 162])
@pytest.mark.parametrize("form", [ab.COND_ROW_SCALED, ab.COND_SCALED_PHI])
def test_fields_match_their_definition(num_tets, form, cuda):
    w = ab.Workload.cylinder(3)
    a = dict(ab.workload_arrays(w))
    a["material"] = np.array(a["material"])
    a["material"].reshape(-1, 3)[0, 2] = 50.0
    # Some tets of each body, in their order, renumbered.
    order = np.random.default_rng(5).permutation(162)[:num_tets] if num_tets < 162 else np.arange(162)
    new = np.full(162, -1)
    new[order] = np.arange(num_tets)
    per_body = [new[a["body_tets"][a["body_ptr"][i]:a["body_ptr"][i + 1]]] for i in range(2)]
    per_body = [p[p >= 0] for p in per_body]
    a["body_tets"] = np.concatenate(per_body).astype(np.int32)
    a["body_ptr"] = np.cumsum([0] + [len(p) for p in per_body]).astype(np.int32)
    for key, width in (("tets", 4), ("tet_idx", 16), ("tet_coeff", 16), ("tet_fixed", 20)):
        a[key] = np.ascontiguousarray(a[key].reshape(-1, width)[order]).ravel()
    te = np.ascontiguousarray(w.tet_edges.reshape(-1, 6)[order]).ravel()
    asm = ab.Assembly(a)
    fields = ab.Fields(asm, w.num_nodes, w.num_edges, te)
    rng = np.random.default_rng(7)
    x = rng.standard_normal(w.num_unknowns) + 1j * rng.standard_normal(w.num_unknowns)
    omega = 2 * np.pi * 50.0
    want = fields_numpy(a, te, w.num_edges, x, omega, 1j * omega if form == ab.COND_SCALED_PHI else 1.0)
    got = fields.compute(torch.from_numpy(x).cuda(), omega, form)
    for key, ref in want.items():
        g = got[key].cpu().numpy()
        if key == "on_interface":
            np.testing.assert_array_equal(g, ref)
        else:
            assert np.abs(g - ref).max() <= 1e-12 * max(np.abs(ref).max(), 1e-300), key

"""The kernels that give a matrix row to eight lanes (residuals, products,
equilibration, the scatter into the panels) at the edges of their blocks, on
rows from one entry to several hundred, against numpy. Sums of at most a few
hundred FP64 terms in another order: 1e-12 relative to the terms' magnitudes."""
import numpy as np
import pytest
import torch

import aphi_b200 as ab

pytestmark = pytest.mark.gpu


def system(n, seed):
    """Upper CSR: a diagonal, a few random neighbours, one full row and column."""
    rng = np.random.default_rng([n, seed])
    hub = n // 2
    rows = [{i} | {int(c) for c in rng.integers(i, n, rng.integers(0, 9))} for i in range(n)]
    rows[hub] |= set(range(hub, n))
    for i in range(hub):
        rows[i].add(hub)
    ci = [sorted(r) for r in rows]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in ci])]).astype(np.int32)
    ci = np.concatenate(ci).astype(np.int32)
    r = np.repeat(np.arange(n), np.diff(rp))
    v = (rng.standard_normal(ci.size) + 1j * rng.standard_normal(ci.size)) * 10.0 ** rng.uniform(-6, 6, ci.size)
    v[r == ci] += 1e8
    a = np.zeros((n, n), np.complex128)
    a[r, ci] = v
    a[ci, r] = v
    return rp, ci, v, a, rng


@pytest.mark.parametrize("n", [1, 7, 31, 33, 255, 256, 257, 700])
@pytest.mark.parametrize("nrhs", [1, 2, 3, 4, 5])
def test_residuals_and_products(n, nrhs, cuda):
    rp, ci, v, a, rng = system(n, nrhs)
    an = ab.Analysis(rp, ci)
    f = ab.Factor(an)
    vals = torch.from_numpy(np.stack([v, 2.0 * v])).cuda()
    x, b = (rng.standard_normal((2, nrhs, n)) + 1j * rng.standard_normal((2, nrhs, n)) for _ in range(2))
    y = ab.spmv(an, vals, torch.from_numpy(x).cuda()).cpu().numpy()
    res = ab.residuals(an, vals, torch.from_numpy(x).cuda(), torch.from_numpy(b).cuda())
    for e in range(2):
        m = a * (1.0 + e)
        mag = np.abs(x[e]) @ np.abs(m)
        assert (np.abs(y[e] - x[e] @ m) <= 1e-12 * mag).all()
        for k in range(nrhs):
            r = np.linalg.norm(b[e, k] - m @ x[e, k])
            bn, xn = np.linalg.norm(b[e, k]), np.linalg.norm(x[e, k])
            np.testing.assert_allclose(res[e, k], [r / bn, r / (np.abs(m).max() * xn + bn)], rtol=1e-11)
    f.close()


@pytest.mark.parametrize("n", [1, 33, 257, 700])
@pytest.mark.parametrize("steps", [0, 1, 2, 9, 10])
def test_equilibration_and_scatter(n, steps, cuda):
    """D equals the Ruiz steps in numpy, and L D L^T the scaled matrix."""
    rp, ci, v, a, _ = system(n, 100 + steps)
    d = np.ones(n)
    for _ in range(steps):
        m = (np.abs(a) * np.outer(d, d)).max(1)
        d = np.where(m > 0, d / np.sqrt(np.where(m > 0, m, 1.0)), d)
    an = ab.Analysis(rp, ci)
    f = ab.Factor(an)
    assert f.factorize(torch.from_numpy(v).cuda().unsqueeze(0), steps)
    e = f.export()
    np.testing.assert_allclose(e["d"], d, rtol=1e-13)
    low = np.eye(n, dtype=np.complex128)
    for j in range(n):
        t = slice(e["col_ptr"][j], e["col_ptr"][j + 1])
        low[e["row_index"][t], j] = e["value"][t]
    want = a * np.outer(d, d)
    got = (low * e["diagonal"]) @ low.T
    assert np.abs(got - want).max() <= 1e-13 * n * np.abs(want).max()

"""The solves at the edges of their 64-column blocks, 64-row chunks and
512-row gathers, for one to nine right-hand sides and both precisions,
against numpy on diagonally dominant systems (condition below 10: n eps, with
n <= 1200, is under 3e-13 in FP64 and 2e-4 in FP32)."""
import numpy as np
import pytest
import torch

import aphi_b200 as ab

pytestmark = pytest.mark.gpu


def dense_and_tails(n, tail, rng):
    """A dense block of n unknowns, ordered last, and `tail` unknowns before it
    that each touch three of the block's: one front of n rows with children."""
    tot = n + tail
    a = np.zeros((tot, tot), np.complex128)
    blk = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    a[tail:, tail:] = np.triu(blk, 1)
    for i in range(tail):
        at = tail + rng.choice(n, min(3, n), replace=False)
        a[i, at] = rng.standard_normal(at.size) + 1j * rng.standard_normal(at.size)
    a = a + a.T
    a[np.arange(tot), np.arange(tot)] = 2.0 * np.abs(a).sum(1) + 1.0
    return a


@pytest.mark.parametrize("precision,tol", [(ab.PREC_FP64, 3e-13), (ab.PREC_FP32, 2e-4)])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 128, 129, 511, 513, 600, 1030])
def test_solves_match_numpy(precision, tol, n, cuda):
    rng = np.random.default_rng(n)
    a = dense_and_tails(n, 150, rng)
    r, c = np.nonzero(np.triu(a))
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=len(a)))]).astype(np.int32)
    an = ab.Analysis(rp, c.astype(np.int32), np.arange(len(a), dtype=np.int32))
    f = ab.Factor(an, precision, 2)
    vals = torch.from_numpy(np.stack([a[r, c], 3.0 * a[r, c]])).cuda()
    assert f.factorize(vals)
    b = rng.standard_normal((2, 9, len(a))) + 1j * rng.standard_normal((2, 9, len(a)))
    want = np.stack([np.linalg.solve(a, b[0].T).T, np.linalg.solve(3.0 * a, b[1].T).T])
    got = f.solve(torch.from_numpy(b).cuda()).cpu().numpy()
    for e in range(2):
        for k in range(9):
            assert np.linalg.norm(got[e, k] - want[e, k]) <= tol * np.linalg.norm(want[e, k])
    for k in (1, 5, 8):   # fewer right-hand sides give the same bits
        part = f.solve(torch.from_numpy(np.ascontiguousarray(b[:, :k])).cuda()).cpu().numpy()
        np.testing.assert_array_equal(part, got[:, :k])
    f.close()


@pytest.mark.parametrize("small_front", [96, 8])
@pytest.mark.parametrize("n", [2, 8, 9, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 191, 193])
def test_dense_factors_reconstruct(n, small_front, cuda):
    """One dense front of n rows through the one-CTA and the blocked kernels:
    L D L^T is the matrix to n eps of its largest entry (its growth is below
    2: diagonally dominant), multipliers and pivots match a host LDL^T."""
    rng = np.random.default_rng([n, small_front])
    a = dense_and_tails(n, 0, rng)
    r, c = np.nonzero(np.triu(a))
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
    o = ab.default_analysis_options()
    o.small_front = small_front
    an = ab.Analysis(rp, c.astype(np.int32), np.arange(n, dtype=np.int32), options=o)
    f = ab.Factor(an)
    assert f.factorize(torch.from_numpy(a[r, c]).cuda().unsqueeze(0), 0)
    e = f.export()
    low, host = np.eye(n, dtype=np.complex128), a.copy()
    for j in range(n):
        t = slice(e["col_ptr"][j], e["col_ptr"][j + 1])
        low[e["row_index"][t], j] = e["value"][t]
        host[j + 1:, j] /= host[j, j]
        host[j + 1:, j + 1:] -= np.outer(host[j + 1:, j] * host[j, j], host[j + 1:, j])
    assert np.abs((low * e["diagonal"]) @ low.T - a).max() <= 2.3e-16 * 4 * n * np.abs(a).max()
    np.testing.assert_allclose(e["diagonal"], np.diag(host), rtol=1e-12)
    assert np.abs(np.tril(low, -1) - np.tril(host, -1)).max() <= 1e-12
    f.close()

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

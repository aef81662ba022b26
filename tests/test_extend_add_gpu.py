"""Extend-add at the edges of its tables: one to five children (taken two at a
time), fronts just above and below its 32-column items, and one with more rows
than a row map holds (4096).

The check is the backward error of a solve, |b - A x| / (|A| |x|) in the
maximum norm, on diagonally dominant systems: with an element growth below 2 it
is at most 2 n eps. The children carry most of the weight of the entries that
they reach: one contribution that is lost or added twice shows as 1e-4 or more
(the FP32 bound is 2e-5 for the smallest case, 5e-4 for the largest)."""
import numpy as np
import pytest
import torch

import aphi_b200 as ab

pytestmark = pytest.mark.gpu


def cliques_on_a_block(n, kids, rng):
    """A dense block of n unknowns, ordered last; before it `kids` cliques of 40
    unknowns, each coupled strongly to 60 (at most n) of the block's, the last
    two rows among them."""
    tot = n + 40 * kids
    r, c, v = [], [], []

    def dense(rows, cols, scale):
        i, j = np.meshgrid(rows, cols, indexing="ij")
        keep = i < j
        r.append(i[keep]), c.append(j[keep])
        v.append(scale * (rng.standard_normal(keep.sum()) + 1j * rng.standard_normal(keep.sum())))

    block = np.arange(40 * kids, tot)
    dense(block, block, 1e-3)
    for k in range(kids):
        own = np.arange(40 * k, 40 * k + 40)
        dense(own, own, 1.0)
        at = rng.choice(n - 2, min(58, n - 2), replace=False)
        dense(own, 40 * kids + np.sort(np.concatenate([at, [n - 2, n - 1]])), 1.0)
    r, c, v = np.concatenate(r), np.concatenate(c), np.concatenate(v)
    diag = np.bincount(r, np.abs(v), tot) + np.bincount(c, np.abs(v), tot) + 1.0
    r, c, v = np.concatenate([r, np.arange(tot)]), np.concatenate([c, np.arange(tot)]), np.concatenate([v, diag])
    order = np.lexsort((c, r))
    return tot, r[order], c[order], v[order]


@pytest.mark.parametrize("precision,eps", [(ab.PREC_FP64, 1.1e-16), (ab.PREC_FP32, 6e-8)])
@pytest.mark.parametrize("n,kids", [(97, 1), (127, 2), (129, 3), (160, 4), (191, 5), (1030, 3), (4300, 3)])
def test_children_reach_their_front(precision, eps, n, kids, cuda):
    rng = np.random.default_rng([n, kids])
    tot, r, c, v = cliques_on_a_block(n, kids, rng)
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=tot))]).astype(np.int32)
    an = ab.Analysis(rp, c.astype(np.int32), np.arange(tot, dtype=np.int32))
    f = ab.Factor(an, precision, 1)
    assert f.factorize(torch.from_numpy(v[None]).cuda())
    b = rng.standard_normal(tot) + 1j * rng.standard_normal(tot)
    x = f.solve(torch.from_numpy(b[None, None]).cuda()).cpu().numpy().reshape(-1)
    off = r != c
    ax = np.zeros(tot, complex)
    np.add.at(ax, r, v * x[c])
    np.add.at(ax, c[off], v[off] * x[r[off]])
    rows = np.bincount(r, np.abs(v), tot) + np.bincount(c[off], np.abs(v[off]), tot)
    assert np.abs(b - ax).max() <= 2 * tot * eps * rows.max() * np.abs(x).max()
    f.close()

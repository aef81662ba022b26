"""The trailing updates on INT8 digits (csrc/i8_update.cuh) at the edges of
its tiles: rows and columns around multiples of 128, 64 and 32, K around
multiples of 32, one panel and groups of two and four.

Each front's contribution block must be -L21 D L21^T of the panel that the same
call returns, formed here in extended precision. Tolerance, per entry: with
the pivots' magnitudes shared out as the kernel does (|a|, |b| <= A_i, B_j,
the rows' largest components), an operand is off by at most 2^-62 A_i, so a
sum of w complex products is off by at most 4 w 2^-62 A_i B_j, plus the
dropped digit levels (below 2^-56 w A_i B_j) and at most three roundings of a
sum below 2 w A_i B_j per group: together under 8 w 2^-53 A_i B_j. In FP32
the operands' own products are rounded to 24 bits (8 w 2^-24 A_i B_j over a
sum), a group's sum twice (4 w) and the destination once for each of up to
five groups (10 w); digits and dropped levels add less than 2 w: 32 w 2^-24."""
import numpy as np
import pytest
import torch

import aphi_b200 as ab

pytestmark = pytest.mark.gpu

SHAPES = [(97, 1), (98, 96), (128, 31), (129, 32), (130, 33), (160, 64), (161, 97), (225, 100), (256, 127),
          (257, 128), (300, 129), (392, 130), (393, 256), (450, 255), (520, 257), (641, 511), (700, 513)]


def panels_of(rng, shapes, spread):
    out = []
    for m, w in shapes:
        p = rng.standard_normal((m, w)) + 1j * rng.standard_normal((m, w))
        top = np.tril(p[:w])
        p[:w] = top + np.tril(top, -1).T
        # pivots of very different sizes, the columns scaled with them
        c = 2.0 ** rng.integers(-spread, spread + 1, w)
        p[:w] *= c[:, None]
        p *= c[None, :]
        p[np.arange(w), np.arange(w)] += 4.0 * m * c * c
        p[w:] *= (2.0 ** rng.integers(-8 * spread, 8 * spread + 1, m - w))[:, None]
        out.append(p)
    return out


def factorize(shapes, panels, precision=ab.PREC_FP64):
    fr = ab.Fronts([m for m, _ in shapes], [w for _, w in shapes])
    flat = np.zeros(fr.stored, np.complex128)
    for o, p in zip(fr.panel_offset, panels):
        flat[o:o + p.size] = p.reshape(-1, order="F")
    f = ab.Factor(fr, precision, 1)
    if precision == ab.PREC_FP32:
        f.set_tc_split(2)
    ok = f.factorize_fronts(torch.from_numpy(flat).cuda().unsqueeze(0))
    P, C = (t.cpu().numpy() for t in f.read_fronts(0))
    got = []
    for s, (m, w) in enumerate(shapes):
        o, q, c = fr.panel_offset[s], fr.cb_offset[s], m - w
        got.append((P[o:o + m * w].reshape(m, w, order="F"), C[q:q + c * c].reshape(c, c, order="F")))
    return ok, got


@pytest.mark.parametrize("precision,spread", [(ab.PREC_FP64, 0), (ab.PREC_FP64, 12), (ab.PREC_FP32, 0), (ab.PREC_FP32, 2)])
def test_trailing_update_at_the_tile_edges(precision, spread, cuda):
    rng = np.random.default_rng(11 + spread)
    panels = panels_of(rng, SHAPES, spread)
    ok, got = factorize(SHAPES, panels, precision)
    assert ok
    unit = 8.0 * 2.0 ** -53 if precision == ab.PREC_FP64 else 32.0 * 2.0 ** -24
    for (m, w), (L, C) in zip(SHAPES, got):
        d = np.diag(L[:w, :w])
        h = 2.0 ** np.floor(np.floor(np.log2(np.maximum(abs(d.real), abs(d.imag)))) / 2)
        A, B = (L[w:] * d) / h, L[w:] * h
        big = lambda x: np.maximum(abs(x.real), abs(x.imag)).max(1)  # noqa: E731
        Lx = L[w:].astype(np.clongdouble)
        want = -(Lx * d.astype(np.clongdouble)) @ Lx.T
        low = np.tril(np.ones(C.shape, bool))
        err = np.abs((C.astype(np.clongdouble) - want)[low]).astype(np.float64)
        tol = (unit * w * np.outer(big(A), big(B)))[low]
        assert (err <= tol).all(), (m, w, (err / tol).max())


@pytest.mark.parametrize("precision", [ab.PREC_FP64, ab.PREC_FP32])
def test_a_row_that_is_not_finite_reaches_its_entries_only(precision, cuda):
    """A NaN below the pivots makes its row and column of the contribution
    block NaN, as a floating-point update does, and changes nothing else."""
    shapes = [(300, 130)]
    rng = np.random.default_rng(3)
    panels = panels_of(rng, shapes, 0)
    _, clean = factorize(shapes, panels, precision)
    bad = panels[0].copy()
    bad[200, 5] = np.nan
    _, got = factorize(shapes, [bad], precision)
    C, D = got[0][1], clean[0][1]
    low = np.tril(np.ones(C.shape, bool))
    hit = np.zeros_like(low)
    hit[70, :] = hit[:, 70] = True
    assert np.isnan(C[low & hit]).all()
    np.testing.assert_array_equal(C[low & ~hit], D[low & ~hit])

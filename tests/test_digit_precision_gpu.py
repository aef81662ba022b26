"""What the trailing updates' byte digits keep, and the form that keeps more.

Rows graded within themselves: each row's components fall by many binades away
from a column of its own, so that two rows' products are far below the product of
their largest components. With A, B the powers of two next above those (pivots
shared out as the kernel does) and S the sum of the products' magnitudes, an
entry formed on digits may be off by the bounds that include/aphi_b200.h states,
  FP64: sqrt(2) w (2^-61 + 2^-58) A B < w 2^-57 A B,
  FP32: sqrt(2) w (2^-29 + 2^-27.4) A B < w 2^-26 A B,
beside the arithmetic's own roundings: W = L D (4 units of S) and, for each of at
most 2 + w / 128 groups, the sum (once in FP64, three times in FP32) and the
result (sqrt(2) units of S each): (7 + 1.5 w / 128) and (10 + 1.5 w / 128) units
of S, 2^-53 or 2^-24. In FP64 arithmetic there is no A B at all: a chain of 2 w
multiply-adds on W, 4 w units of S, and the groups' results.

Scaling: a symmetric scaling by powers of two moves every row's A and B with it,
so the digits of D M D are those of M: the same solution, scaled, bit for bit,
without equilibration."""
import numpy as np
import pytest
import torch

import aphi_b200 as ab

pytestmark = pytest.mark.gpu

SHAPES = [(97, 1), (225, 100), (300, 128), (393, 256), (450, 255), (641, 511), (700, 513)]


def graded_panels(rng, span):
    out = []
    for m, w in SHAPES:
        p = np.zeros((m, w), np.complex128)
        p[np.arange(w), np.arange(w)] = rng.uniform(1, 2, w) * np.exp(1j * rng.uniform(-1, 1, w))
        k = np.arange(w)
        # every third row falls from the left, from the right, and from a column of its own
        top = np.where(np.arange(m - w) % 3 == 0, 0, np.where(np.arange(m - w) % 3 == 1, w - 1, rng.integers(0, w, m - w)))
        p[w:] = rng.uniform(0.5, 1, (m - w, w)) * np.exp(2j * np.pi * rng.uniform(0, 1, (m - w, w)))
        p[w:] *= 2.0 ** (-span * np.abs(k[None, :] - top[:, None]) / w)
        out.append(p)
    return out


def factorize(panels, precision, digits):
    fr = ab.Fronts([m for m, _ in SHAPES], [w for _, w in SHAPES])
    flat = np.zeros(fr.stored, np.complex128)
    for o, p in zip(fr.panel_offset, panels):
        flat[o:o + p.size] = p.reshape(-1, order="F")
    f = ab.Factor(fr, precision, 1)
    if precision == ab.PREC_FP32:
        f.set_tc_split(2)
    else:
        f.set_fp64_digits(digits)
    assert f.factorize_fronts(torch.from_numpy(flat).cuda().unsqueeze(0))
    P, C = (t.cpu().numpy() for t in f.read_fronts(0))
    for s, (m, w) in enumerate(SHAPES):
        o, q, c = fr.panel_offset[s], fr.cb_offset[s], m - w
        yield m, w, P[o:o + m * w].reshape(m, w, order="F"), C[q:q + c * c].reshape(c, c, order="F")


@pytest.mark.parametrize("precision,digits,span", [(ab.PREC_FP64, True, 40), (ab.PREC_FP64, False, 40),
                                                   (ab.PREC_FP32, True, 16)])
def test_rows_graded_within_themselves(precision, digits, span, cuda):
    panels = graded_panels(np.random.default_rng(span), span)
    unit = 2.0 ** -53 if precision == ab.PREC_FP64 else 2.0 ** -24
    worst = 0.0   # the error in units of S: what the grading costs an entry
    for m, w, L, C in factorize(panels, precision, digits):
        d = np.diag(L[:w, :w])
        h = 2.0 ** np.floor(np.floor(np.log2(np.maximum(abs(d.real), abs(d.imag)))) / 2)
        a, b = (L[w:] * d) / h, L[w:] * h
        above = lambda x: 2.0 ** (np.floor(np.log2(np.maximum(abs(x.real), abs(x.imag)).max(1))) + 1)  # noqa: E731
        Lx = L[w:].astype(np.clongdouble)
        want = -(Lx * d.astype(np.clongdouble)) @ Lx.T
        low = np.tril(np.ones(C.shape, bool))
        err = np.abs((C.astype(np.clongdouble) - want)[low]).astype(np.float64)
        S = (np.abs(a) @ np.abs(b).T)[low]
        AB = np.outer(above(a), above(b))[low]
        if not digits:
            tol = unit * (4 * w + 7 + 1.5 * w / 128) * S
        elif precision == ab.PREC_FP64:
            tol = w * 2.0 ** -57 * AB + unit * (7 + 1.5 * w / 128) * S
        else:
            tol = w * 2.0 ** -26 * AB + unit * (10 + 1.5 * w / 128) * S
        assert (err <= tol).all(), (m, w, (err / tol).max())
        if w > 1:
            worst = max(worst, (err / (unit * S)).max())
    if digits:   # the rows are graded enough to show: some entry lost more than eight bits of itself
        assert worst > 256


@pytest.mark.parametrize("precision,digits,spread", [(ab.PREC_FP64, True, 40), (ab.PREC_FP64, False, 40),
                                                     (ab.PREC_FP32, True, 12)])
def test_scaling_by_powers_of_two_keeps_the_bits(precision, digits, spread, cuda):
    w = ab.Workload.cylinder(9)
    an = ab.Analysis(w.row_ptr, w.col_idx, ab.amd_ordering(w.row_ptr, w.col_idx))
    assert an.plan_stats(0)["update_wide"][0] > 0 and an.plan_stats(1)["update_tc"][0] > 0
    asm = ab.Assembly(ab.workload_arrays(w))
    values, rhs = asm.refill(2 * np.pi * 400.0)
    # rows of one size first, so that the FP32 factor's numbers stay in range
    rows = np.repeat(np.arange(an.n), np.diff(w.row_ptr))
    diag = values[0].abs().cpu().numpy()[w.row_ptr[:-1]]
    level = -np.round(np.log2(diag) / 2)
    rng = np.random.default_rng(7)
    xs = []
    for extra in (np.zeros(an.n), rng.integers(-spread, spread + 1, an.n)):
        s = torch.from_numpy(np.ldexp(1.0, (level + extra).astype(int))).cuda()
        f = ab.Factor(an, precision, 1)
        if precision == ab.PREC_FP32:
            f.set_tc_split(2)
        else:
            f.set_fp64_digits(digits)
        scaled = values * s[torch.from_numpy(rows).cuda()] * s[torch.from_numpy(w.col_idx.astype(np.int64)).cuda()]
        assert f.factorize(scaled, equilibration_iterations=0)
        xs.append(f.solve(rhs * s) * s)
        f.close()
    assert torch.isfinite(torch.view_as_real(xs[0])).all() and xs[0].abs().max() > 0
    assert torch.equal(torch.view_as_real(xs[0]), torch.view_as_real(xs[1]))


def test_the_form_is_a_factors_own_choice(cuda):
    """Two factors of one analysis, one of each form, in turn; refused for FP32."""
    w = ab.Workload.cylinder(10)
    an = ab.Analysis(w.row_ptr, w.col_idx, ab.amd_ordering(w.row_ptr, w.col_idx))
    asm = ab.Assembly(ab.workload_arrays(w))
    values, rhs = asm.refill(2 * np.pi * 400.0)
    a, b = ab.Factor(an), ab.Factor(an)
    b.set_fp64_digits(False)
    launches, xs = [], []
    for f in (a, b, a):
        f.profile(True)
        assert f.factorize(values)
        launches.append(f.profile_read().get("dmma_scale", (0, 0.0))[0])
        f.profile(False)
        xs.append(f.solve(rhs))
    assert launches[0] == launches[2] > 0 and launches[1] == 0
    assert torch.equal(torch.view_as_real(xs[0]), torch.view_as_real(xs[2]))
    assert not torch.equal(torch.view_as_real(xs[0]), torch.view_as_real(xs[1]))
    b.set_fp64_digits(True)
    assert b.factorize(values)
    assert torch.equal(torch.view_as_real(b.solve(rhs)), torch.view_as_real(xs[0]))
    with pytest.raises(ab.InvalidArgument):
        ab.Factor(an, ab.PREC_FP32).set_fp64_digits(False)

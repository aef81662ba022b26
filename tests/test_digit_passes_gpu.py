"""Trailing updates whose digits do not fit the workspace for the whole batch:
28 multiples (powers of four) of one dense matrix of 4300 rows, 1.4 GB of digits
in FP64, go through in two passes. Scaling by a power of four is exact in every
step, so each entry's solution is the single factorization's, bit for bit, over
its factor (8.5 GB on the device)."""
import numpy as np
import pytest
import torch

import aphi_b200 as ab

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [ab.PREC_FP64, ab.PREC_FP32])
def test_passes_give_the_bits_of_one_factorization(precision, cuda):
    n, batch = 4300, 28
    rng = np.random.default_rng(3)
    r, c = np.triu_indices(n)
    rp = np.concatenate([[0], np.cumsum(np.arange(n, 0, -1))]).astype(np.int32)
    v = rng.standard_normal(r.size) + 1j * rng.standard_normal(r.size)
    v[r == c] = 4.0 * n
    an = ab.Analysis(rp, c.astype(np.int32), np.arange(n, dtype=np.int32))
    base = torch.from_numpy(v).cuda()
    scale = torch.from_numpy(np.ldexp(1.0, 2 * np.arange(-14, 14))).cuda()
    b = torch.from_numpy(rng.standard_normal(n) + 1j * rng.standard_normal(n)).cuda()
    one, many = ab.Factor(an, precision, 1), ab.Factor(an, precision, batch)
    if precision == ab.PREC_FP32:
        one.set_tc_split(2), many.set_tc_split(2)
    assert one.factorize(base[None].contiguous())
    want = one.solve(b[None, None].contiguous())[0, 0]
    one.close()
    assert many.factorize(base[None] * scale[:, None])
    got = many.solve(b.expand(batch, 1, n).contiguous())[:, 0]
    many.close()
    assert torch.isfinite(torch.view_as_real(want)).all() and want.abs().max() > 0
    assert torch.equal(torch.view_as_real(got * scale[:, None]), torch.view_as_real(want.expand(batch, n)))

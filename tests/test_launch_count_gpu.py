"""aphi_launch_count and the per-kind profile count the kernels that ran, also
where a trailing update goes through the batch in several passes (28 dense
matrices of 4300 rows: more digits than the workspace holds at once): each pass
is a launch of its operands' kind and one of the update's."""
import numpy as np
import pytest
import torch

import aphi_b200 as ab

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,kinds", [(ab.PREC_FP64, ("dmma_scale", "update_wide")),
                                             (ab.PREC_FP32, ("tc_split", "update_tc"))])
def test_every_pass_is_counted_under_its_kind(precision, kinds, cuda):
    n = 4300
    rng = np.random.default_rng(4)
    r, c = np.triu_indices(n)
    rp = np.concatenate([[0], np.cumsum(np.arange(n, 0, -1))]).astype(np.int32)
    v = rng.standard_normal(r.size) + 1j * rng.standard_normal(r.size)
    v[r == c] = 4.0 * n
    an = ab.Analysis(rp, c.astype(np.int32), np.arange(n, dtype=np.int32))
    planned = an.plan_stats(0 if precision == ab.PREC_FP64 else 1)
    values = torch.from_numpy(v).cuda()
    seen = {}
    for batch in (1, 28):
        f = ab.Factor(an, precision, batch)
        if precision == ab.PREC_FP32:
            f.set_tc_split(2)
        f.profile(True)
        before = ab.launch_count()
        assert f.factorize(values.expand(batch, -1).contiguous())
        seen[batch] = ab.launch_count() - before, f.profile_read()
        f.close()
    (one, k1), (many, k28) = seen[1], seen[28]
    assert {k: x[0] for k, x in k1.items()} == {k: planned[k][0] for k in k1}
    split, update = kinds
    assert k28[split][0] == k28[update][0] > planned[update][0]
    assert {k: x[0] for k, x in k28.items() if k not in kinds} == {k: x[0] for k, x in k1.items() if k not in kinds}
    assert many - one == sum(x[0] for x in k28.values()) - sum(x[0] for x in k1.values())
    assert all(ms > 0 for _, ms in k28.values())

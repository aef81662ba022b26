"""Refill at any batch of frequencies gives the bits of one frequency at a time:
every count around the kernels' switches (4 frequencies), a warp's 32 lanes and
the 64 of a launch, on meshes on both sides of the one / four tets a warp
switch, both formulations, upper and full storage, and the cut port's mesh."""
import numpy as np
import pytest

import aphi_b200 as ab

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh,cells", [("cylinder", 4), ("cylinder", 11), ("cylinder", 12), ("torus", 16)])
@pytest.mark.parametrize("form", [ab.COND_ROW_SCALED, ab.COND_SCALED_PHI])
@pytest.mark.parametrize("upper", [True, False])
def test_batches_equal_single_frequencies(mesh, cells, form, upper, cuda):
    w = ab.Workload.torus(cells) if mesh == "torus" else ab.Workload.cylinder(cells)
    arrays = ab.workload_arrays(w)
    if not upper:
        rp, ci = ab.pattern_build(w.num_unknowns, w.tet_idx, w.port_row[w.port_current == 0], upper_only=False)
        arrays |= {"row_ptr": rp, "col_idx": ci}
    asm = ab.Assembly(arrays, upper_only=upper)
    om = 2 * np.pi * np.geomspace(50.0, 1.0e6, 70)
    single = [tuple(t[0].cpu().numpy() for t in asm.refill(o, form)) for o in om]
    for nf in (2, 3, 4, 5, 16, 31, 33, 64, 70):
        v, b = (t.cpu().numpy() for t in asm.refill(om[:nf], form))
        for f in range(nf):
            assert np.array_equal(v[f], single[f][0]) and np.array_equal(b[f], single[f][1]), (nf, f)

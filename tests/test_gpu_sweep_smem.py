"""Staging capacities at the end of a CTA's 227 KB: where the plain sweep fits
but not the sweeps that take rows ahead (two more row tables, 128 bytes of
static shared memory instead of 64), the plain one runs."""
import numpy as np
import pytest

from adventure_fullwave_b200 import hddm, meshgen
from helpers import rel_l2

pytestmark = pytest.mark.gpu

SMEM = 227 * 1024


def _cap_for(total, max_interior, blocks, es):
    """The largest staging capacity whose plain sweep takes at most `total`
    bytes: the vector, two staging buffers, two blocks' vectors, two row
    tables, the barriers and the block table."""
    rest = max_interior * es + 64 * es + 64 * 8 + 32 + ((blocks + 1) * 8 + 15) // 16 * 16
    return (total - rest) // 32 * 16 // es  # each buffer a multiple of 16 bytes


@pytest.mark.parametrize("kernel", ["warp", "blockinv"])
@pytest.mark.parametrize("precision,es", [("fp64", 16), ("fp32_ir", 8)])
# the plain sweep's last byte; one buffer element from where both fit; both fit
@pytest.mark.parametrize("total", [SMEM - 64, SMEM - 128 - 512 + 64, SMEM - 128 - 512])
def test_plain_sweep_where_the_other_does_not_fit(kernel, precision, es, total):
    model = meshgen.make_model("w", n=6, size=1.0, npml=1, layers=2, nleaves=None, leaf_cap=110, jitter=(0.3, 0.7), seed=5)
    meshgen.round_trip_material(model)
    kw = dict(hddm_eps=1e-9, hddm_max_loop=2000, precision=precision, solve_kernel=kernel)
    with hddm.HddmSolver(model, **kw) as s:
        n = s.sizes()["max_interior"]
        assert 32 < n < 200  # a block of 32 rows is far below the capacities
        s.solve(0)
        want = s.edge_solution()
    cap = _cap_for(total, n, -(-n // 32), es)
    with hddm.HddmSolver(model, stage_cap=cap, **kw) as s:
        r = s.solve(0)
        assert r.converged and r.solve_kernel == kernel and r.stage_cap == cap
        # converged to 1e-9 in other row blocks
        assert rel_l2(s.edge_solution(), np.asarray(want)) <= 1e-6

"""The LDL^T factor of every subdomain against the oracle's restatement of the
reference (oracle.factor_sub), at sizes around the factor kernel's blocks of
16 columns: subdomains of a few DOFs, of one to three blocks, and one of
several hundred rows.  1e-12 relative per subdomain, as for the models of
test_gpu_parity.py (the sums are grouped differently)."""
import numpy as np
import pytest

from adventure_fullwave_b200 import hddm, meshgen
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,leaf", [(4, 7), (5, 30), (5, 60), (6, 110), (6, 1296)])
def test_factor_vs_oracle(n, leaf):
    model = meshgen.make_model("f", n=n, size=1.0, npml=1, layers=2, nleaves=None, leaf_cap=leaf, jitter=(0.3, 0.7), seed=3)
    meshgen.round_trip_material(model)
    part = oracle.partition(model)
    sizes = set()
    with hddm.HddmSolver(model, hddm_eps=1e-6, hddm_max_loop=1) as s:
        s.make_tmp_aij(0)
        s.solve_dom_1st()
        for k in range(model.nsub):
            want = oracle.factor_sub(model, part.subs[k])[3]
            got = s.factor(k)
            sizes.add(got.shape[0])
            assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max(), k
    assert leaf == 1296 or len(sizes) > 3


@pytest.mark.parametrize("n,leaf", [(6, 4), (8, 4)])
def test_factor_of_many_subdomains(n, leaf):
    """Models with more than two and more than four subdomains per SM, where the
    factor's CTAs are smaller: 1e-12 as above, on every tenth subdomain."""
    model = meshgen.make_model("f", n=n, size=1.0, npml=1, layers=2, nleaves=None, leaf_cap=leaf, jitter=(0.3, 0.7), seed=3)
    meshgen.round_trip_material(model)
    assert model.nsub > (296 if n == 6 else 592)
    part = oracle.partition(model)
    with hddm.HddmSolver(model, hddm_eps=1e-6, hddm_max_loop=1) as s:
        s.make_tmp_aij(0)
        s.solve_dom_1st()
        for k in range(0, model.nsub, 10):
            want = oracle.factor_sub(model, part.subs[k])[3]
            got = s.factor(k)
            if got.size:
                assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max(), k

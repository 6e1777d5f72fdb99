"""The staged sweeps with one, two and four warps per subdomain and with the
timed choice (which may take the rows ahead, with four or eight warps) give
the same bits: subdomains of one row block, of a few, and of one of many."""
import numpy as np
import pytest

from adventure_fullwave_b200 import hddm, meshgen
from helpers import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,leaf", [(4, 7), (5, 30), (6, 110), (8, 600), (8, 3072)])
@pytest.mark.parametrize("precision,kernel", [("fp64", "auto"), ("fp64", "blockinv"), ("fp32_ir", "auto")])
def test_same_bits_for_every_share(n, leaf, precision, kernel):
    model = meshgen.make_model("w", n=n, size=1.0, npml=1, layers=2, nleaves=None, leaf_cap=leaf, jitter=(0.3, 0.7),
                               seed=5)
    meshgen.round_trip_material(model)
    got = []
    for warps in (1, 2, 4, 0):
        x, r = hddm.hddm_solver_CS(model, 0, hddm_eps=1e-9, hddm_max_loop=40, precision=precision, solve_kernel=kernel,
                                   stage_warps=warps)
        got.append((np.asarray(x), r.iterations))
    for x, its in got[1:]:
        assert its == got[0][1] and np.array_equal(x, got[0][0], equal_nan=True)


@pytest.mark.parametrize("n,leaf", [(8, 1600), (9, 1500)])
def test_batched_sources_on_the_largest_subdomains(n, leaf):
    """FP64 batched sources where a subdomain of 1,451 interior DOFs leaves no
    shared memory for the pivots and a second row table, and where all of at
    most 1,094 leave it: each source against the one-source solve, 1e-8."""
    model = meshgen.make_model("w", n=n, size=1.0, npml=1, layers=2, nleaves=None, leaf_cap=leaf, jitter=(0.3, 0.7),
                               seed=5, nsources=3)
    meshgen.round_trip_material(model)
    with hddm.HddmSolver(model, hddm_eps=1e-10, hddm_max_loop=20000) as s:
        res = s.solve_multi([0, 1, 2])
        xs = [s.edge_solution_multi(k) for k in range(3)]
        for k in range(3):
            s.resolve(k)
            assert res[k].converged and rel_l2(xs[k], s.edge_solution()) <= 1e-8


@pytest.mark.parametrize("n,leaf", [(4, 7), (6, 110), (8, 4), (8, 600), (8, 1600)])
@pytest.mark.parametrize("precision", ["fp64", "fp32_ir"])
def test_auto_sweep_against_the_staged_one(n, leaf, precision):
    """The timed choice's block-inverse sweep, at the capacities it takes for
    one subdomain per SM, a few and many, against the staged sweep: both
    converged to 1e-10, 1e-8 (FP32 with refinement 1e-6, as against the oracle)."""
    model = meshgen.make_model("w", n=n, size=1.0, npml=1, layers=2, nleaves=None, leaf_cap=leaf, jitter=(0.3, 0.7),
                               seed=5)
    meshgen.round_trip_material(model)
    kw = dict(hddm_eps=1e-10, hddm_max_loop=20000, precision=precision, ir_max_steps=2)
    x, r = hddm.hddm_solver_CS(model, 0, **kw)
    want, rw = hddm.hddm_solver_CS(model, 0, solve_kernel="warp", **kw)
    assert r.solve_kernel == "blockinv" and r.converged and rw.converged
    assert rel_l2(np.asarray(x), np.asarray(want)) <= (1e-8 if precision == "fp64" else 1e-6)

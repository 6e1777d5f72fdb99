"""Calls without enough device memory, by a hook that fails the allocations
above a size: an error, never a solve in another order of sums, and the same
call with the memory there gives the bits of a context that always had it."""
import numpy as np
import pytest

from adventure_fullwave_b200 import _lib, hddm, meshgen

pytestmark = pytest.mark.gpu


def _model(n, leaf):
    model = meshgen.make_model("w", n=n, size=1.0, npml=1, layers=2, nleaves=None, leaf_cap=leaf, jitter=(0.3, 0.7),
                               seed=5)
    meshgen.round_trip_material(model)
    return model


def _limit(solver, nbytes):
    _lib.check(solver._lib.fwgpu_test_hook(solver._h, _lib.HOOK_ALLOC_MAX, int(nbytes)))


@pytest.mark.parametrize("precision", ["fp64", "fp32_ir"])
def test_no_room_for_the_block_inverse_copy(precision):
    model = _model(8, 1600)
    kw = dict(hddm_eps=1e-9, hddm_max_loop=2000, precision=precision)
    with hddm.HddmSolver(model, **kw) as s:
        r = s.solve(0)
        assert r.solve_kernel == "blockinv"
        want, n = s.edge_solution(), s.sizes()["nlen_interior"]
    # the copy holds each block's triangle in full, so it is larger than the
    # factor, which in FP64 is the largest allocation besides; in FP32 the
    # FP64 factor is larger than the copy, and takes its place here
    limit = 16 * (n + 64) if precision == "fp64" else 16 * (n + 64) - 1
    with hddm.HddmSolver(model, **kw) as s:
        _limit(s, limit)
        for _ in range(2):
            with pytest.raises(_lib.FwgpuError) as e:
                s.solve(0)
            assert e.value.code == _lib.ERR_NOMEM
        _limit(s, 0)
        got = s.solve(0)
        assert (got.solve_kernel, got.iterations) == ("blockinv", r.iterations)
        assert np.array_equal(s.edge_solution(), want)
    if precision == "fp64":  # the sweep that needs no copy
        with hddm.HddmSolver(model, solve_kernel="warp", **kw) as s:
            _limit(s, limit)
            assert s.solve(0).converged


def test_the_block_inverse_copy_takes_no_memory_of_its_own():
    """With FP64 factors of subdomains of a few hundred elements the first
    solve allocates nothing larger than the factor itself; the copy, which
    holds each block's triangle in full, is larger."""
    model = _model(10, 600)
    with hddm.HddmSolver(model, hddm_eps=1e-9, hddm_max_loop=2000) as s:
        r = s.solve(0)
        want, z = s.edge_solution(), s.sizes()
    limit = max(16 * (z["nlen_interior"] + 64), 8 * z["nnz_lower"])
    with hddm.HddmSolver(model, hddm_eps=1e-9, hddm_max_loop=2000) as s:
        s.make_tmp_aij(0)
        _limit(s, limit)
        got = s.solve(0)
        assert (got.solve_kernel, got.iterations) == ("blockinv", r.iterations)
        assert np.array_equal(s.edge_solution(), want)


@pytest.mark.parametrize("leaf", [110, 600])
@pytest.mark.parametrize("precision", ["fp64", "fp32_ir"])
def test_refused_source_leaves_the_factors_in_use(leaf, precision):
    model = _model(8, leaf)
    with hddm.HddmSolver(model, hddm_eps=1e-9, hddm_max_loop=2000, precision=precision) as s:
        s.solve(0)
        want = s.edge_solution()
        with pytest.raises(_lib.FwgpuError) as e:
            s.make_tmp_aij((np.array([model.n_edges]), np.array([1.0 + 0j])))
        assert e.value.code == _lib.ERR_ARG
        s.resolve(0)
        assert np.array_equal(s.edge_solution(), want)

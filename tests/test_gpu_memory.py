"""Calls without enough device memory, by a hook that fails the allocations
above a size: an error, never a solve in another order of sums, and the same
call with the memory there gives the bits of a context that always had it."""
import numpy as np
import pytest

from adventure_fullwave_b200 import _lib, hddm, meshgen
from helpers import golden, rel_l2

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


@pytest.mark.parametrize("precision,kernel", [("fp64", "auto"), ("fp64", "warp"), ("fp32_ir", "auto")])
def test_every_failed_allocation_can_be_repeated(precision, kernel):
    """Each device allocation of an element source, a solve and a batched
    solve fails once; the failed call is an error and its repetition gives what
    a context that always had the memory gives: AUTO the same bits, WARP, whose
    timed staging capacity sets the order of its sums, the solution that
    converged to 1e-10."""
    _, _, model = golden("gap")
    es, model.element_source = model.element_source, None
    src = (np.array([3, 17], np.int32), np.array([1.0 + 2j, -0.5j]))

    def run(fail):
        failed = 0
        with hddm.HddmSolver(model, hddm_eps=1e-10, hddm_max_loop=20000, precision=precision, solve_kernel=kernel) as s:
            _lib.check(s._lib.fwgpu_test_hook(s._h, _lib.HOOK_ALLOC_FAIL, fail))
            for call in (lambda: s.set_element_source(es), lambda: s.solve(src), lambda: s.solve_multi([src, src])):
                try:
                    call()
                except _lib.FwgpuError as e:
                    assert e.code == _lib.ERR_NOMEM
                    failed += 1
                    call()
            xs = [s.edge_solution_multi(0), s.edge_solution_multi(1)]
            s.resolve(src)
            return [s.edge_solution(), *xs], failed

    want, failed = run(0)
    assert failed == 0
    for k in range(1, 200):
        got, failed = run(k)
        for a, b in zip(got, want):
            assert np.array_equal(a, b) if kernel == "auto" else rel_l2(a, b) <= 1e-7
        if failed == 0:
            break
        assert failed == 1
    assert k > 30  # every allocation was met


@pytest.mark.parametrize("n,leaf,limit,kernel", [
    (10, 600, 1, "blockinv"),          # in the element matrices: at any size
    (8, 1600, 1, "warp"),              # memory of its own, over the limit
    (8, 1600, 1 << 30, "blockinv"),
])
def test_auto_weighs_the_memory_that_the_copy_costs(n, leaf, limit, kernel):
    model = _model(n, leaf)
    with hddm.HddmSolver(model, hddm_eps=1e-9, hddm_max_loop=2000) as s:
        _lib.check(s._lib.fwgpu_test_hook(s._h, _lib.HOOK_COPY_MAX, limit))
        r = s.solve(0)
        assert r.converged and r.solve_kernel == kernel
    if kernel == "warp":  # and FP32 factors, and a kernel asked for, are not limited
        for kw in (dict(precision="fp32_ir"), dict(solve_kernel="blockinv")):
            with hddm.HddmSolver(model, hddm_eps=1e-9, hddm_max_loop=2000, **kw) as s:
                _lib.check(s._lib.fwgpu_test_hook(s._h, _lib.HOOK_COPY_MAX, limit))
                assert s.solve(0).solve_kernel == "blockinv"

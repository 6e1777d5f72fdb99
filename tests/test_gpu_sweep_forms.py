"""Every form of the staged sweeps, one, two and four warps per subdomain and
four and eight that take the next block's rows ahead, on both layouts and in
both precisions, and the two kernels of the LDL^T factor: the same bits."""
import numpy as np
import pytest

from adventure_fullwave_b200 import _lib, hddm, meshgen

pytestmark = pytest.mark.gpu

FORMS = [(1, 0), (2, 0), (4, 0), (4, 1), (8, 1)]


def _model(n, leaf):
    model = meshgen.make_model("w", n=n, size=1.0, npml=1, layers=2, nleaves=None, leaf_cap=leaf, jitter=(0.3, 0.7),
                               seed=5)
    meshgen.round_trip_material(model)
    return model


def _hook(solver, hook, value):
    _lib.check(solver._lib.fwgpu_test_hook(solver._h, hook, value))


# subdomains of one row block, of a few, of many, and of blocks cut short by
# the staging buffer
@pytest.mark.parametrize("n,leaf,cap", [(4, 7, 512), (6, 110, 512), (6, 110, 1024), (8, 600, 768), (8, 3072, 1024)])
@pytest.mark.parametrize("precision", ["fp64", "fp32_ir"])
@pytest.mark.parametrize("kernel", ["warp", "blockinv"])
def test_same_bits_of_every_form(n, leaf, cap, precision, kernel):
    model = _model(n, leaf)
    got = []
    for warps, ahead in FORMS:
        with hddm.HddmSolver(model, hddm_eps=1e-9, hddm_max_loop=40, precision=precision, solve_kernel=kernel,
                             stage_cap=cap) as s:
            _hook(s, _lib.HOOK_SWEEP, warps + 16 * ahead)
            r = s.solve(0)
            assert (r.solve_kernel, r.stage_warps, r.stage_ahead) == (kernel, warps, ahead)
            got.append((s.edge_solution(), r.iterations, r.stage_cap))
    for x, its, c in got[1:]:
        assert (its, c) == got[0][1:] and np.array_equal(x, got[0][0], equal_nan=True)


# up to two, up to four and more subdomains per SM (1,024, 512 and 256 threads),
# of no row, one, a block of 16, its edges, and several hundred rows
@pytest.mark.parametrize("n,leaf", [(4, 7), (5, 30), (5, 60), (6, 110), (6, 1296), (6, 4), (8, 4), (12, 12)])
def test_same_bits_of_both_factor_kernels(n, leaf):
    model = _model(n, leaf)
    got = []
    for by_rows in (0, 1):
        with hddm.HddmSolver(model, hddm_eps=1e-9, hddm_max_loop=1) as s:
            _hook(s, _lib.HOOK_ROW_FACTOR, by_rows)
            s.make_tmp_aij(0)
            s.solve_dom_1st()
            got.append([s.factor(k) for k in range(model.nsub)])
    assert all(np.array_equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("warps", [0, 1])
def test_batched_result_names_its_own_sweep(warps):
    """Batched sources run eight warps, whatever the one-source sweep was
    given or timed to."""
    model = _model(5, 30)
    with hddm.HddmSolver(model, hddm_eps=1e-9, hddm_max_loop=2000, stage_warps=warps) as s:
        r, = s.solve_multi([0])
        assert (r.solve_kernel, r.stage_warps, r.stage_ahead) == ("warp", 8, 0)
        one = s.resolve(0)
        assert one.stage_warps == warps if warps else one.stage_warps > 1

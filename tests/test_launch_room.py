"""Shared memory of a sweep's CTA beside the kernel's static arrays: what compiled and ran with the
paths in device memory, or with less padding, still does."""
import types

import numpy as np
import pytest

from test_boundary import _cfg, _compile


def _quadratic(dof):
    return " + ".join(f"0.5 * x{i + 1} * x{i + 1}" for i in range(dof))


def test_learned_walkers_in_device_memory_compile():
    # a warp of walkers a CTA, 263168 bytes of paths and histogram: the paths stay in device memory
    kw = dict(dof=6, n_slices=512, bisection_level=8, n_walkers=64, hist_bins=16384, potential_cache=2)
    rc, log = _compile(_cfg(learned=1, global_path=1, **kw), _quadratic(6), "", ("x1 * x1",), (), ("x1",))
    assert rc == 0, log


@pytest.mark.parametrize("N,S,per_sm", [(1024, 3, 8), (2048, 4, 4), (1024, 3, 16)])
def test_lanes_leave_the_callers_register_budget(N, S, per_sm):
    # three walkers would take 4 or 8 lanes a segment thread: CTAs that no SM holds per_sm of, for
    # which ptxas drops the budget
    rc, log = _compile(_cfg(dof=6, n_slices=N, bisection_level=S, n_walkers=3, min_blocks_per_sm=per_sm), _quadratic(6),
                       "", ("x1 * x1",))
    assert rc == 0 and "will be ignored" not in log, log


@pytest.mark.parametrize("dof,kw", [
    (2, dict(n_slices=4, potential_cache=1)), (9, dict(n_slices=256)), (3, dict(n_slices=8, potential_cache=3, enable_ranlux=1)),
    (6, dict(n_slices=64, metro_steps_per_operator_run=0)), (1, dict(n_slices=8, potential_cache=1, enable_parallelize_path=0)),
])
def test_level_zero_compiles(dof, kw):
    # a move without nodes: no cached values to keep for a rejection
    rc, log = _compile(_cfg(dof=dof, bisection_level=0, n_walkers=64, **kw), _quadratic(dof), "", ("x1 * x1",))
    assert rc == 0, log


def test_measurements_without_moves_compile():
    # metroStepsPerOperatorRun = 0: RANLUX has no offsets to draw ahead
    rc, log = _compile(_cfg(enable_ranlux=1, metro_steps_per_operator_run=0), "0.5 * x1 * x1", "", ("x1 * x1",))
    assert rc == 0, log


def test_refused_size_is_named():
    rc, log = _compile(_cfg(dof=9, n_slices=512, bisection_level=9, walkers_per_block=16), _quadratic(9))
    assert rc == -1 and "does not fit in shared memory (" in log


@pytest.mark.gpu
def test_last_kilobytes_beside_static_arrays():
    # 320 walkers of 32 slices and 13632 histogram bins, 197888 bytes with the plain padding, and 34560
    # of RANLUX streams in static shared memory fill the 227 KB; the bank spread takes 219648
    from gpu_util import engine, require_gpu
    require_gpu()
    kernel, kernel_args = engine()

    def run(per_block):
        ka = kernel_args.KernelArgs(
            system=types.SimpleNamespace(DOF=3, potential=_quadratic(3), userCode=""), nbrOfWalkers=640, N=32, beta=1.0,
            S=5, enableOperator=True, enableCorrelator=False, enableBisection=True, enablePathShift=False,
            enableSingleNodeMove=False, enableBins=False, nbrOfWalkersPerWorkGroup=1, enableParallelizePath=True,
            enableGlobalPath=False, enableGlobalOldPath=False, enableRanlux=True, luxuaryFactor=2,
            ranluxIntMax=2 ** 32 - 1, operators=("x1 * x1",), operatorRuns=2, metroStepsPerOperatorRun=2,
            walkersPerBlock=per_block, potentialCache=False, seed=3, fastMath=False, histograms=("x1",),
            histRange=(-1.0, 1.0), histBins=13632)
        k = kernel.PIMCKernel(ka)
        k.initRanlux()
        k.groupInitRanlux()
        k.run()
        return k.getPaths(), k.getOperators(), k.getHistogram(density=False)[1]

    for a, b in zip(run(320), run(32)):
        assert np.array_equal(a, b)

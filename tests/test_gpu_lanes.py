"""Lanes that share a segment thread (FS_G) against one lane each (asked for by a number of walkers
per CTA): the same bits in paths, generator states, accepts, operator sums and histogram, for 2, 4
and 8 lanes, degrees of freedom they do and do not divide, walkers inside a warp and across
warps, every generator, FP32 and FP64, and in device memory.  IEEE builds, so that the compiler's
contraction of plugin expressions is the same at both."""
import types

import numpy as np
import pytest

from gpu_util import engine, require_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()


@pytest.mark.parametrize("dof,W,N,S,lux,double,cache,lanes", [
    (6, 20, 32, 4, None, False, None, 8), (6, 20, 32, 4, 2, False, False, 8), (3, 7, 16, 3, None, False, True, 4),
    (9, 33, 32, 3, None, False, None, 8), (27, 5, 64, 2, None, False, None, 4), (6, 3, 256, 3, None, False, "device", 4),
    (15, 2, 512, 3, None, False, None, 8), (6, 1200, 128, 4, 1, False, None, 4), (6, 40, 64, 5, 3, False, None, 8),
    (12, 9, 32, 3, 2, True, None, 8), (3, 11, 32, 2, None, True, False, 2), (8, 10, 16, 3, 2, False, None, 4)])
def test_lanes_bit_identical(dof, W, N, S, lux, double, cache, lanes):
    kernel, kernel_args = engine()
    squares = " + ".join(f"x{d + 1} * x{d + 1}" for d in range(dof))
    system = types.SimpleNamespace(DOF=dof, potential=f"0.3 * ({squares}) + 0.1 * x1 * x{dof}", userCode="")
    p0 = np.random.RandomState(3).randn(W, dof * N) * 0.4
    got = []
    for wpb in (0, 1):
        k = kernel.PIMCKernel(kernel_args.KernelArgs(
            system=system, nbrOfWalkers=W, N=N, beta=2.0, S=S, enableOperator=True, enableCorrelator=False,
            enableBisection=True, enablePathShift=False, enableSingleNodeMove=False, enableBins=False,
            nbrOfWalkersPerWorkGroup=1, enableParallelizePath=True, enableGlobalPath=False, enableGlobalOldPath=False,
            enableDouble=double, enableRanlux=lux is not None, luxuaryFactor=lux, ranluxIntMax=2 ** 32 - 1,
            operators=("x1 * x1", f"x{dof}"), operatorRuns=3, metroStepsPerOperatorRun=2, fastMath=False,
            histograms=("x1", f"x{dof} + 0.1"), histRange=(-3.0, 3.0), histBins=40, potentialCache=cache,
            walkersPerBlock=wpb, seed=S + W))
        if lux is not None:
            k.initRanlux()
            k.groupInitRanlux()
        k.setPaths(p0)
        k.run(2)
        rng = k.getRanluxTables() if lux is not None else (k.getSeeds(), k.getWalkerSeeds())
        got.append((k.getPaths(), k.getOperators(), k._raw_operators(), k.getAccepts(), *rng,
                    k.getHistogram(density=False)[1]))
        threads = k.getInfo().block_threads
        per_walker = threads // k.getInfo().walkers_per_block
        assert per_walker == (N >> S) * (lanes if wpb == 0 else 1)
        k.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    assert 0 < got[0][3].sum()

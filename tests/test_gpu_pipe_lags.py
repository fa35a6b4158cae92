"""Pipelined correlator helpers of two lags a lane against one walker per CTA (helpers after the
moves, or none), and of the library's own choice for a run of few walkers: the same bits, IEEE
builds."""
import types

import numpy as np
import pytest

from gpu_util import engine, require_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()


@pytest.mark.parametrize("N,S,W,accumulation", [(16, 1, 12, "fp64"), (16, 2, 16, "kahan"), (32, 2, 20, "fp64"),
                                                (64, 2, 6, "fp64"), (64, 1, 3, "fp64"), (128, 3, 40, "fp64"),
                                                (128, 3, 2, "kahan"), (64, 3, 8, "fp64")])
def test_two_lags_bit_identical(N, S, W, accumulation):
    kernel, kernel_args = engine()
    system = types.SimpleNamespace(DOF=1, potential="0.5 * x1 * x1", userCode="")
    p0 = (np.random.RandomState(N + S).randn(W, N) * 0.7).astype(np.float32)
    got = []
    for wpb in (0, 1):
        k = kernel.PIMCKernel(kernel_args.KernelArgs(
            system=system, nbrOfWalkers=W, N=N, beta=4.0, S=S, enableOperator=True, enableCorrelator=True,
            enableBisection=True, enablePathShift=False, enableSingleNodeMove=False, enableBins=False,
            nbrOfWalkersPerWorkGroup=1, enableParallelizePath=True, enableGlobalPath=False, enableGlobalOldPath=False,
            operators=("x1 * x1",), correlators=("x1", "x1 * x1"), operatorRuns=3, metroStepsPerOperatorRun=2,
            accumulation=accumulation, fastMath=False, walkersPerBlock=wpb, seed=S))
        k.setPaths(p0)
        k.run(2)
        got.append((k.getPaths(), k._raw_operators(), k.getAccepts(), k._raw_correlator()))
        k.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)

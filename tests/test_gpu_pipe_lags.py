"""Pipelined correlator helpers of two lags a lane, and with walkers that leave the last CTA
ragged, against one walker per CTA (helpers after the moves, or none): the same bits, IEEE
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
                                                (128, 3, 2, "kahan"), (64, 3, 8, "fp64"),
                                                (128, 3, 41, "fp64"), (32, 2, 5, "fp64"), (64, 4, 9, "kahan"),
                                                (16, 3, 1, "fp64"), (64, 2, 333, "fp64")])
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
            accumulation=accumulation, fastMath=False, walkersPerBlock=wpb, seed=S, histograms=("x1",),
            histRange=(-2.0, 2.0), histBins=16))
        k.setPaths(p0)
        k.run(2)
        got.append((k.getPaths(), k._raw_operators(), k.getAccepts(), k._raw_correlator(), k.getSeeds(), k.getWalkerSeeds(),
                    k.getHistogram(density=False)[1]))
        k.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("N,S,W", [(16, 1, 3), (64, 1, 5), (128, 1, 7), (128, 1, 64), (256, 2, 5), (512, 3, 3), (1024, 1, 2),
                                   (1024, 2, 3), (64, 3, 4), (8, 1, 6)])
def test_lag_sums_of_the_final_path(N, S, W):
    """One measurement after one step: its lag sums are those of the paths read back, to the
    documented bound of the FP32 partials, (gamma(N/4 + 2) + 2u) sum_s x_s^2."""
    kernel, kernel_args = engine()
    system = types.SimpleNamespace(DOF=1, potential="0.5 * x1 * x1", userCode="")
    k = kernel.PIMCKernel(kernel_args.KernelArgs(
        system=system, nbrOfWalkers=W, N=N, beta=4.0, S=S, enableOperator=True, enableCorrelator=True,
        enableBisection=True, enablePathShift=False, enableSingleNodeMove=False, enableBins=False,
        nbrOfWalkersPerWorkGroup=1, enableParallelizePath=True, enableGlobalPath=False, enableGlobalOldPath=False,
        operators=("x1 * x1",), correlators=("x1", "x1 + 0.5"), operatorRuns=1, metroStepsPerOperatorRun=1, seed=S))
    k.setPaths((np.random.RandomState(N).randn(W, N) * 0.7).astype(np.float32))
    k.run()
    x = k.getPaths().astype(np.float64)
    got = k._raw_correlator().reshape(W, 2, N // 2)
    u = 2.0 ** -24
    for c, f in enumerate((x, (x.astype(np.float32) + np.float32(0.5)).astype(np.float64))):
        want = np.stack([(f * np.roll(f, -t, axis=1)).sum(axis=1) for t in range(N // 2)], axis=1)
        n = N // 4 + 2
        bound = (n * u / (1 - n * u) + 2 * u) * (f * f).sum(axis=1, keepdims=True)
        assert np.all(np.abs(got[:, c] - want) <= bound), (np.abs(got[:, c] - want) / bound).max()
    k.close()

"""getCorrelatorMoments (two-stage reduction over the walkers, no atomics) against the raw
correlator sums reduced here, for fewer and more lags than a block's 256 threads, walker ranges
that leave blocks ragged or single, and every stored type.  Sums of W FP64 terms in another
order stay within 2 W u of the terms' magnitudes (u = 2^-53); W <= 700 and the standard error's
cancellation leaves 1e-9 with room."""
import types

import numpy as np
import pytest

from gpu_util import engine, require_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()


@pytest.mark.parametrize("accumulation", ["fp64", "fp32", "study"])
@pytest.mark.parametrize("W,N,cors", [(3, 4, 1), (700, 16, 3), (129, 128, 2), (37, 512, 1), (40, 1024, 2)])
def test_moments_match_raw(W, N, cors, accumulation):
    kernel, kernel_args = engine()
    system = types.SimpleNamespace(DOF=1, potential="0.5 * x1 * x1", userCode="")
    S = max(1, int(np.log2(N)) - 4)
    k = kernel.PIMCKernel(kernel_args.KernelArgs(
        system=system, nbrOfWalkers=W, N=N, beta=2.0, S=S, enableOperator=True, enableCorrelator=True,
        enableBisection=True, enablePathShift=False, enableSingleNodeMove=False, enableBins=False,
        nbrOfWalkersPerWorkGroup=1, enableParallelizePath=True, enableGlobalPath=False, enableGlobalOldPath=False,
        operators=("x1 * x1",), correlators=("x1", "x1 * x1", "1.0 + x1")[:cors], operatorRuns=2,
        metroStepsPerOperatorRun=1, accumulation=accumulation, seed=1))
    k.setPaths((np.random.RandomState(5).randn(W, N) * 0.5).astype(np.float32))
    k.run(2)
    ncol = 3 if accumulation == "study" else 1
    if ncol == 3:
        v = k.getCorrelatorStudy().reshape(3, W, cors, N // 2)
    else:
        v = k.getCorrelatorPerWalker().reshape(1, W, cors, N // 2)
    for lo, hi in ((0, W), (1, 2), (W // 3, W)):
        mean, se = k.getCorrelatorMoments((lo, hi))
        mean, se = np.reshape(mean, (ncol, cors, -1)), np.reshape(se, (ncol, cors, -1))
        part = v[:, lo:hi]
        scale = np.abs(part).max()
        np.testing.assert_allclose(mean, part.mean(axis=1), rtol=1e-12, atol=1e-13 * scale)
        # var = q / n - mean^2: the subtraction loses up to 1e-13 of the squares, 4e-7 of a root
        want = part.std(axis=1) / np.sqrt(hi - lo)
        np.testing.assert_allclose(se, want, rtol=1e-9, atol=1e-6 * scale)
    k.close()

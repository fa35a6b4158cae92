"""The precision study's per-walker operator means reduced on the device against the raw
per-work-item sums averaged here: T work-items a walker below, at and above a warp, two
operators, walkers shared out over work-groups.  Both average the same FP64 values; a sum of
T terms in another order is within 2 T u of the other, u = 2^-53, relative to the terms' sum of
magnitudes (positive here), far below the 1e-12 asked for."""
import types

import numpy as np
import pytest

from gpu_util import engine, require_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()


@pytest.mark.parametrize("W,N,S,per_group,parallel", [
    (5, 16, 4, 1, True), (33, 32, 2, 3, True), (12, 128, 2, 4, True), (9, 512, 1, 1, True), (7, 16, 2, 1, False)])
def test_device_means_match_raw(W, N, S, per_group, parallel):
    kernel, kernel_args = engine()
    system = types.SimpleNamespace(DOF=1, potential="0.5 * x1 * x1", userCode="")
    k = kernel.PIMCKernel(kernel_args.KernelArgs(
        system=system, nbrOfWalkers=W, N=N, beta=2.0, S=S, enableOperator=True, enableCorrelator=False,
        enableBisection=True, enablePathShift=False, enableSingleNodeMove=False, enableBins=False,
        nbrOfWalkersPerWorkGroup=per_group, enableParallelizePath=parallel, enableGlobalPath=False,
        enableGlobalOldPath=False, operators=("x1 * x1", "1.0 + x1 * x1 * x1 * x1"), operatorRuns=3,
        metroStepsPerOperatorRun=2, accumulation="study", seed=1))
    k.setPaths((np.random.RandomState(5).randn(W, N) * 0.5).astype(np.float32))
    k.run()
    raw = k._raw_operators().reshape(-1, 2, 3)
    want = np.stack([k._per_walker(raw[:, :, c]).T for c in range(3)])
    got = k.getOperatorsStudy()
    assert got.shape == (3, 2, W)
    np.testing.assert_allclose(got, want, rtol=1e-12, atol=0)
    k.close()

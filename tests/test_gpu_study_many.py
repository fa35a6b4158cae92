"""The precision study's operator means of more walkers than 2^32 threads in whole warps count."""
import types

import numpy as np
import pytest

from gpu_util import engine, require_gpu

pytestmark = pytest.mark.gpu


def test_walkers_beyond_32_bit_threads():
    require_gpu()
    kernel, kernel_args = engine()
    W = (1 << 27) + 37
    k = kernel.PIMCKernel(kernel_args.KernelArgs(
        system=types.SimpleNamespace(DOF=1, potential="0.5 * x1 * x1", userCode=""), nbrOfWalkers=W, N=2, beta=2.0, S=1,
        enableOperator=True, enableCorrelator=False, enableBisection=True, enablePathShift=False,
        enableSingleNodeMove=False, enableBins=False, nbrOfWalkersPerWorkGroup=1, enableParallelizePath=True,
        enableGlobalPath=False, enableGlobalOldPath=False, operators=("1.0 + x1 * x1",), operatorRuns=1,
        metroStepsPerOperatorRun=1, accumulation="study", seed=1))
    k.setPathsTiled(np.ones((4, 2), np.float32))
    k.run()
    got = k.getOperatorsStudy()
    # one work-item a walker: its means are its sums, to the bit
    assert np.array_equal(got[:, 0], k._raw_operators().reshape(W, 3).T)
    k.close()

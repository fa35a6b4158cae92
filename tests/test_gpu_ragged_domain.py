"""Spare threads of a ragged last CTA evaluate the plugin on a walker's coordinates only: a potential
that is defined about x = 100 and reports anything else."""
import types

import numpy as np
import pytest

from gpu_util import engine, require_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,S,W", [(128, 3, 777), (32, 2, 5), (16, 3, 1), (16, 1, 13)])
def test_spare_threads_stay_in_the_domain(N, S, W, capfd):
    require_gpu()
    kernel, kernel_args = engine()
    user = """FLOAT_TYPE well(FLOAT_TYPE x)
{
    if (x < 50.0f || x > 150.0f) printf("outside the domain: %f\\n", (double)x);
    return 0.5f * (x - 100.0f) * (x - 100.0f);
}"""
    system = types.SimpleNamespace(DOF=1, potential="well(x1)", userCode=user)
    p0 = (100.0 + 0.7 * np.random.RandomState(N).randn(W, N)).astype(np.float32)
    got = []
    for wpb in (0, 1):
        k = kernel.PIMCKernel(kernel_args.KernelArgs(
            system=system, nbrOfWalkers=W, N=N, beta=4.0, S=S, enableOperator=True, enableCorrelator=True,
            enableBisection=True, enablePathShift=False, enableSingleNodeMove=False, enableBins=False,
            nbrOfWalkersPerWorkGroup=1, enableParallelizePath=True, enableGlobalPath=False, enableGlobalOldPath=False,
            operators=("well(x1)",), correlators=("x1",), operatorRuns=3, metroStepsPerOperatorRun=2,
            accumulation="fp64", fastMath=False, walkersPerBlock=wpb, seed=S))
        k.setPaths(p0)
        k.run()
        got.append((k.getPaths(), k._raw_operators(), k.getAccepts()))
        k.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    assert abs(got[0][0] - 100.0).max() < 50.0
    assert "outside the domain" not in capfd.readouterr().out

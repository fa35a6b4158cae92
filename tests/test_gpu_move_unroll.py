"""The unrolled and the rolled bisection move (FS_MOVE_CODE in fs_pimc.cuh) against the oracle
on both sides of the line: one and six degrees of freedom, xorshift, shared and device-memory
paths.  IEEE arithmetic: generator rows bit-exact, at most one accept decision flipped by the
last place of log, sin and exp, paths to 1e-4."""
import types

import numpy as np
import pytest

from gpu_util import engine, require_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()


@pytest.mark.parametrize("global_path", [False, True], ids=["shared_path", "global_path"])
@pytest.mark.parametrize("dof,N,S", [(1, 64, 4), (1, 64, 5), (1, 128, 6), (2, 32, 4), (6, 16, 1), (6, 16, 2),
                                     (6, 32, 3), (6, 32, 5)])
def test_move_matches_oracle(dof, N, S, global_path):
    from oracle import oracle as orc
    kernel, kernel_args = engine()
    pot = "0.5 * (" + " + ".join(f"x{d + 1} * x{d + 1}" for d in range(dof)) + ")"
    system = types.SimpleNamespace(DOF=dof, potential=pot, userCode="")
    W = 10
    ka = kernel_args.KernelArgs(
        system=system, nbrOfWalkers=W, N=N, beta=2.0, S=S, enableOperator=True, enableCorrelator=False,
        enableBisection=True, enablePathShift=False, enableSingleNodeMove=False, enableBins=False,
        nbrOfWalkersPerWorkGroup=2, enableParallelizePath=True, enableGlobalPath=global_path,
        enableGlobalOldPath=False, operators=("x1 * x1",), operatorRuns=3, metroStepsPerOperatorRun=2, fastMath=False,
        seed=S)
    k = kernel.PIMCKernel(ka)
    o = orc.OracleSampler(orc.OracleConfig(
        DOF=dof, potential=pot, userCode="", nbrOfWalkers=W, N=N, beta=2.0, S=S, operatorRuns=3,
        metroStepsPerOperatorRun=2, nbrOfWalkersPerWorkGroup=2, enableParallelizePath=True, enableRanlux=False,
        operators=("x1 * x1",), compat=False, accum=1))
    p0 = (np.random.RandomState(3).randn(*o.paths.shape) * 0.4).astype(np.float32)
    o.paths[...] = p0
    k.setPaths(p0)
    o.seeds[...] = k.getSeeds()
    o.walker_seeds[...] = k.getWalkerSeeds()
    flips = 0
    for _ in range(2):
        k.run()
        o.run()
        assert np.array_equal(k.getSeeds(), o.seeds)
        assert np.array_equal(k.getWalkerSeeds(), o.walker_seeds)
        flips += int((k.getAccepts() != o.accepts).sum())
        assert flips <= 1
        if flips == 0:
            np.testing.assert_allclose(k.getPaths(), o.paths, rtol=1e-4, atol=1e-5)
    k.close()

"""Shared-memory layouts and the choice of where the paths live (fs_api.cu: the walker stride of
walkers that share a warp, walkers per CTA, path_in_shared) and the batched path shift: the same
bits from every placement, and the walker-mode moves against the oracle."""
import types

import numpy as np
import pytest

from gpu_util import engine, require_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()


def _system(dof):
    pot = "0.5 * (" + " + ".join(f"x{d + 1} * x{d + 1}" for d in range(dof)) + ")"
    return types.SimpleNamespace(DOF=dof, potential=pot, userCode="")


def _kernel(dof, W, N, S, **more):
    kernel, kernel_args = engine()
    d = dict(
        system=_system(dof), nbrOfWalkers=W, N=N, beta=2.0, S=S, enableOperator=True, enableCorrelator=False,
        enableBisection=True, enablePathShift=False, enableSingleNodeMove=False, enableBins=False,
        nbrOfWalkersPerWorkGroup=1, enableParallelizePath=True, enableGlobalPath=False, enableGlobalOldPath=False,
        operators=("x1 * x1",), operatorRuns=2, metroStepsPerOperatorRun=3, fastMath=False, seed=S + W)
    return kernel.PIMCKernel(kernel_args.KernelArgs(**dict(d, **more)))


@pytest.mark.parametrize("dof,W,N,S,stays", [
    (1, 5, 16, 4, False), (1, 333, 16, 3, False), (6, 33, 16, 2, False), (6, 700, 16, 1, False), (3, 40, 64, 1, False),
    (27, 3, 16, 2, False), (27, 200, 1024, 2, True), (27, 100, 1024, 2, False)])
def test_placements_bit_identical(dof, W, N, S, stays):
    """Shared memory (the same CTA shape asked for, or chosen), device memory kept by a register
    budget of more CTAs than shared memory admits, and the library's own choice."""
    p0 = (np.random.RandomState(3).randn(W, dof * N) * 0.4).astype(np.float32)
    got = []
    for more in ({}, {"enableGlobalPath": True}, {"enableGlobalPath": True, "minBlocksPerSM": 32}):
        k = _kernel(dof, W, N, S, **more)
        k.setPaths(p0)
        k.run()
        got.append((k.getPaths(), k.getOperators(), k.getAccepts(), k.getSeeds(), k.getInfo().smem_bytes))
        k.close()
    for other in got[1:]:
        for a, b in zip(got[0][:4], other[:4]):
            assert np.array_equal(a, b)
    assert (got[1][4] < dof * N * 4) == stays


@pytest.mark.parametrize("dof,N,W", [(1, 2, 3), (1, 4, 100), (1, 64, 33), (2, 16, 5), (3, 16, 40), (9, 8, 6)])
def test_walker_moves_match_oracle(dof, N, W):
    from oracle import oracle as orc
    k = _kernel(dof, W, N, 1, enableParallelizePath=False, enablePathShift=True, enableSingleNodeMove=True, alpha=0.4,
                PSAlpha=0.6)
    pot = _system(dof).potential
    o = orc.OracleSampler(orc.OracleConfig(
        DOF=dof, potential=pot, userCode="", nbrOfWalkers=W, N=N, beta=2.0, S=1, operatorRuns=2,
        metroStepsPerOperatorRun=3, nbrOfWalkersPerWorkGroup=1, enableParallelizePath=False, enableRanlux=False,
        enablePathShift=True, enableSingleNodeMove=True, alpha=0.4, PSAlpha=0.6, operators=("x1 * x1",), compat=False,
        accum=1))
    p0 = (np.random.RandomState(4).randn(*o.paths.shape) * 0.4).astype(np.float32)
    o.paths[...] = p0
    k.setPaths(p0)
    o.seeds[...] = k.getSeeds()
    o.walker_seeds[...] = k.getWalkerSeeds()
    flips = 0
    for _ in range(4):
        k.run()
        o.run()
        assert np.array_equal(k.getSeeds(), o.seeds)
        assert np.array_equal(k.getWalkerSeeds(), o.walker_seeds)
        flips += int((k.getAccepts() != o.accepts).sum())
        assert flips <= 1
        if flips == 0:
            np.testing.assert_allclose(k.getPaths(), o.paths, rtol=1e-4, atol=1e-5)
    k.close()

"""The automatic chunk count of fs_run_host: 1 to 6 chunks by the grid's size, the same bits as
one chunk, with a ragged last CTA and unequal chunks."""
import numpy as np
import pytest

from gpu_util import engine, require_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()
    engine()


@pytest.mark.parametrize("walkers,chunks", [(40, 1), (6075, 2), (42001, 6)])
@pytest.mark.parametrize("lux", [None, 0])
def test_automatic_chunks(walkers, chunks, lux):
    kernel, kernel_args = engine()
    from feynsimul_gb300.physical_systems.lm2m2 import Lm2m2Cluster
    sysm = Lm2m2Cluster(3, 1.0)
    p0 = sysm.initial_paths(walkers, 64, np.random.RandomState(5)).astype(np.float32)
    got = []
    for n in (0, 1):
        k = kernel.PIMCKernel(kernel_args.KernelArgs(
            system=sysm, nbrOfWalkers=walkers, N=64, beta=sysm.beta, S=3, enableOperator=True, enableCorrelator=False,
            enableBisection=True, enablePathShift=False, enableSingleNodeMove=False, enableBins=False,
            nbrOfWalkersPerWorkGroup=1, enableParallelizePath=True, enableGlobalPath=False, enableGlobalOldPath=False,
            enableRanlux=lux is not None, luxuaryFactor=lux or 0, ranluxIntMax=2 ** 32 - 1, operators=(sysm.energyOp,),
            operatorRuns=2, metroStepsPerOperatorRun=2, seed=9, walkersPerBlock=8, minBlocksPerSM=8))
        if lux is not None:
            k.initRanlux()
            k.groupInitRanlux()
        out = [k.runHost(p0, launches=2, chunks=n).copy(), k.getAccepts(), np.asarray(k.getOperators()), k.getPaths()]
        if n == 0:
            # 64-thread CTAs, 8 (registers) to 15 (shared memory) to an SM, so a wave is 1216 to 2280 CTAs:
            # 5 CTAs are less than a quarter of it, 760 less than 3/4, 5251 more than 2 1/4
            assert k.lastChunks == chunks
        got.append(out)
        k.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)

"""The walkers' bank spread does not cost a resident CTA of an SM."""
import pytest

from gpu_util import engine, require_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("atoms,N,S,W,ctas", [(5, 64, 4, 8000, 4)])
def test_spread_keeps_the_ctas(atoms, N, S, W, ctas):
    require_gpu()
    kernel, kernel_args = engine()
    from feynsimul_gb300.physical_systems.lm2m2 import Lm2m2Cluster
    s = Lm2m2Cluster(atoms, 1.0)
    k = kernel.PIMCKernel(kernel_args.KernelArgs(
        system=s, nbrOfWalkers=W, N=N, beta=2.0, S=S, enableOperator=True, enableCorrelator=False, enableBisection=True,
        enablePathShift=False, enableSingleNodeMove=False, enableBins=False, nbrOfWalkersPerWorkGroup=1,
        enableParallelizePath=True, enableGlobalPath=False, enableGlobalOldPath=False, operators=(s.energyOp,),
        operatorRuns=1, metroStepsPerOperatorRun=1, seed=1))
    assert ctas * (k._info.smem_bytes + 1024) <= 228 * 1024
    k.run()
    k.close()

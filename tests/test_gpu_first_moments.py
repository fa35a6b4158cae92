"""The first reading of correlator moments allocates no device memory."""
import numpy as np
import pytest

from gpu_util import engine, ho_system, require_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,N,S,accumulation", [(340, 512, 5, "fp64"), (222, 1024, 3, "fp32"), (900, 256, 4, "study")])
def test_first_moments_allocate_nothing(W, N, S, accumulation):
    require_gpu()
    import torch
    kernel, kernel_args = engine()
    torch.cuda.init()

    def make():
        k = kernel.PIMCKernel(kernel_args.KernelArgs(
            system=ho_system(), nbrOfWalkers=W, N=N, beta=4.0, S=S, enableOperator=False, enableCorrelator=True,
            enableBisection=True, enablePathShift=False, enableSingleNodeMove=False, enableBins=False,
            nbrOfWalkersPerWorkGroup=1, enableParallelizePath=True, enableGlobalPath=False, enableGlobalOldPath=False,
            correlators=("x1",), operatorRuns=2, metroStepsPerOperatorRun=1, accumulation=accumulation, seed=3))
        k.setPaths((np.random.RandomState(N).randn(W, N) * 0.5).astype(np.float32))
        k.run()
        return k

    # several handles: small allocations share mappings of 2 MB, so not every one shows in the free memory
    held, taken = [], []
    for _ in range(6):
        k = make()
        before = torch.cuda.mem_get_info()[0]
        mean, error = k.getCorrelatorMoments()
        taken.append(before - torch.cuda.mem_get_info()[0])
        assert np.isfinite(np.asarray(mean)).all() and np.isfinite(np.asarray(error)).all()
        held.append(k)
    assert max(taken) <= 0, taken
    for k in held:
        k.close()

"""A null result buffer is an error code at the C ABI, for results in page-locked host memory too."""
import numpy as np
import pytest

from gpu_util import engine, ho_system, require_gpu

pytestmark = pytest.mark.gpu


def test_null_buffers_are_refused():
    require_gpu()
    kernel, kernel_args = engine()
    from feynsimul_gb300 import _lib
    from feynsimul_gb300.batch import BatchSampler
    L = _lib.lib()
    k = kernel.PIMCKernel(kernel_args.KernelArgs(
        system=ho_system(), nbrOfWalkers=64, N=32, beta=4.0, S=2, enableOperator=False, enableCorrelator=False,
        enableBisection=True, enablePathShift=False, enableSingleNodeMove=False, enableBins=False,
        nbrOfWalkersPerWorkGroup=1, enableParallelizePath=True, enableGlobalPath=False, enableGlobalOldPath=False,
        operatorRuns=1, metroStepsPerOperatorRun=1, seed=3))
    k.run()
    assert L.fs_get_accepts(k._handle, None, 64 * 8) != _lib.FS_OK
    assert np.asarray(k.getAccepts()).size == 64 * 8
    b = BatchSampler([{"n": 3, "N": 32, "T": 1.0, "walkers": 8}], block_threads=64, tpw_target=8)
    b.run(1)
    assert L.fs_batch_get_accepts(b._h, 0, None, b.accepts(0).size) != _lib.FS_OK
    assert L.fs_batch_get_op_sums(b._h, 0, None, 8) != _lib.FS_OK
    assert np.isfinite(b.energy_sums(0)).all()

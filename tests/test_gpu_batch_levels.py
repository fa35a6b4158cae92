"""Batch tiles at every bisection level (constant up to 4, run-time above; the old segment in
registers or in scratch), T from 1 to 32 threads a walker and odd walker counts, against the
single-system sweep on the same paths and generator rows.  Both compute in fast math and differ
only where the compiler contracts a plugin expression differently, so at most a few accept
decisions flip; walkers without one keep the same paths and energies."""
import numpy as np
import pytest

from gpu_util import engine, require_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()


@pytest.mark.parametrize("target,ranlux,block", [
    (32, None, 512), (16, None, 64), (8, None, 512), (4, None, 64), (2, None, 512), (1, None, 64), (16, 2, 512),
    (8, 2, 64), (1, 2, 512)])
def test_levels_match_single_systems(target, ranlux, block):
    kernel, kernel_args = engine()
    from feynsimul_gb300.batch import BatchSampler
    workload = [{"n": n, "N": N, "T": 1.0, "walkers": W} for n, N, W in ((2, 64, 5), (3, 64, 37), (6, 64, 9), (10, 32, 3))]
    b = BatchSampler(workload, op_runs=2, msteps=2, block_threads=block, tpw_target=target, ranlux=ranlux)
    rng = np.random.RandomState(5)
    singles = []
    for i, w in enumerate(workload):
        c = b.clusters[w["n"]]
        S = b.systems[i].bisection_level
        T = w["N"] >> S
        paths = c.initial_paths(w["walkers"], w["N"], rng).astype(np.float32)
        ts = rng.randint(0, 2 ** 31 - 1, size=(w["walkers"] * T + 1, 4)).astype(np.uint32)
        ws = rng.randint(0, 2 ** 31 - 1, size=(w["walkers"], 4)).astype(np.uint32)
        b.set_state(i, paths, ts[:-1], ws)
        k = kernel.PIMCKernel(kernel_args.KernelArgs(
            system=c, nbrOfWalkers=w["walkers"], N=w["N"], beta=1.0, S=S, enableOperator=True, enableCorrelator=False,
            enableBisection=True, enablePathShift=False, enableSingleNodeMove=False, enableBins=False,
            nbrOfWalkersPerWorkGroup=1, enableParallelizePath=True, enableGlobalPath=False, enableGlobalOldPath=False,
            enableRanlux=ranlux is not None, luxuaryFactor=ranlux, ranluxIntMax=2 ** 32 - 1, operators=(c.energyOp,),
            operatorRuns=2, metroStepsPerOperatorRun=2))
        k.setPaths(paths)
        if ranlux is None:
            k.setSeeds(ts)
            k.setWalkerSeeds(ws)
        else:
            k.setRanluxTables(*b.ranlux_tables(i))
        singles.append(k)
    b.run(1)
    for i, (w, k) in enumerate(zip(workload, singles)):
        k.run()
        if ranlux is not None:
            for mine, other in zip(b.ranlux_tables(i), k.getRanluxTables()):
                assert np.array_equal(mine, other)
        flips = (b.accepts(i) != k.getAccepts()).reshape(w["walkers"], -1).any(axis=1)
        assert flips.sum() <= 1, i
        np.testing.assert_allclose(b.paths(i)[~flips], k.getPaths()[~flips], rtol=1e-3, atol=1e-4)
        np.testing.assert_allclose(b.energy_sums(i)[~flips] / (2 * w["N"]), k.getOperators()[0][~flips], rtol=1e-3,
                                   atol=1e-3)
        k.close()
    b.close()

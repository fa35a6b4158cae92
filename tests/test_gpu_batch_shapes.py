"""Launch shapes of small batches: tiles do not outnumber the CTAs where a launch of fewer tiles has
room for all walkers at once, and batches of small segments run with two 512-thread CTAs per SM."""
import pytest

from gpu_util import engine, require_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()
    engine()


def _sampler(n, N, S, walkers, block):
    from feynsimul_gb300.batch import BatchSampler
    b = BatchSampler([{"n": n, "N": N, "T": 1.0, "walkers": walkers}], 1, 2, block, N >> S)
    assert b.systems[0].bisection_level == S
    return b


@pytest.mark.parametrize("n,N,S,walkers,block", [(3, 64, 4, 6000, 64), (5, 64, 2, 2000, 64), (6, 256, 3, 1500, 512),
                                                 (10, 128, 2, 1500, 512), (3, 128, 2, 300, 512)])
def test_every_tile_has_a_cta(n, N, S, walkers, block):
    b = _sampler(n, N, S, walkers, block)
    assert b.n_items == -(-walkers // b.walkers_per_tile[0]) <= b.grid
    b.run(1)
    b.close()


@pytest.mark.parametrize("n,N,S,block", [(3, 256, 2, 256), (3, 256, 2, 512), (4, 128, 1, 512), (5, 128, 1, 256)])
def test_small_segments_keep_their_ctas(n, N, S, block):
    # 1024 threads on an SM, as before old segments moved to registers
    import torch
    b = _sampler(n, N, S, 6000, block)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert b.registers <= 64 and b.grid * block >= 1024 * sms
    b.run(1)
    b.close()

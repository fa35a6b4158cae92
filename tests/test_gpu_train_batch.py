"""fs_mlp_train_batch (rows gathered in place, the CTAs' gradients added in order) against the
pass over copied rows with atomics, and against itself: row counts of a part of a tile, one tile,
one row more, and more tiles than SMs."""
import ctypes

import numpy as np
import pytest

from gpu_util import engine, require_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()
    engine()


@pytest.mark.parametrize("rows,dof", [(1, 6), (100, 1), (128, 8), (129, 3), (4096, 6), (152 * 128 + 300, 6)])
def test_batch_matches_pass_and_repeats(rows, dof):
    import torch
    from feynsimul_gb300 import _lib, learned
    L = _lib.lib()
    rng = np.random.RandomState(rows)
    n = 5000
    p = learned.init_params(3, zero_output=False)
    x = rng.randn(n, 16).astype(np.float32)
    z = rng.randn(n, 8).astype(np.float32)
    idx = torch.from_numpy(rng.randint(0, n, rows)).cuda()
    tx, tz = torch.from_numpy(x).cuda(), torch.from_numpy(z).cuda()
    sizes = [ctypes.c_int64() for _ in range(4)]
    L.fs_mlp_sizes(*[ctypes.byref(v) for v in sizes])
    need = ctypes.c_int64()
    _lib.check(L.fs_mlp_workspace(rows, ctypes.byref(need)))
    n_parts = min(-(-rows // 128), 152)
    stride = need.value // n_parts
    stream = torch.cuda.current_stream().cuda_stream

    def fresh():
        tp = torch.from_numpy(p.copy()).cuda()
        tq = torch.zeros(sizes[1].value, dtype=torch.int16, device="cuda")
        tf = torch.zeros(sizes[2].value * 2, dtype=torch.int32, device="cuda")
        tb = torch.zeros(sizes[3].value, dtype=torch.float32, device="cuda")
        _lib.check(L.fs_mlp_pack(tp.data_ptr(), tq.data_ptr(), tf.data_ptr(), tb.data_ptr(), stream))
        return tp, torch.zeros_like(tp), torch.zeros_like(tp), tq

    def batch():
        tp, tm, tv, tq = fresh()
        work = torch.zeros(need.value, dtype=torch.float32, device="cuda")
        loss = torch.full((1,), 7.0, dtype=torch.float32, device="cuda")
        _lib.check(L.fs_mlp_train_batch(tp.data_ptr(), tm.data_ptr(), tv.data_ptr(), tq.data_ptr(), tx.data_ptr(),
                                        tz.data_ptr(), idx.data_ptr(), rows, dof, loss.data_ptr(), 1, 1e-3,
                                        work.data_ptr(), need.value, stream))
        torch.cuda.synchronize()
        return tp, tm, tq, loss, work

    tp, tm, tq, loss, work = batch()
    for a, b in zip((tp, tm, tq, loss, work), batch()):
        assert torch.equal(a, b)
    parts = work.cpu().numpy().astype(np.float64).reshape(n_parts, stride)[:, :p.size + 1]
    magnitude = np.abs(parts).sum(axis=0)
    u = 2.0 ** -24
    # the ordered sum of the CTAs' losses
    assert abs(float(loss[0]) - parts[:, -1].sum()) <= n_parts * u * magnitude[-1]
    # the pass over copied rows: the same partial gradients, added by atomics in FP32
    tg = torch.zeros_like(tp)
    l2 = torch.zeros(1, dtype=torch.float32, device="cuda")
    xb, zb = tx[idx].contiguous(), tz[idx].contiguous()
    qp, qm, qv, qq = fresh()
    _lib.check(L.fs_mlp_train_step(qp.data_ptr(), qq.data_ptr(), tg.data_ptr(), xb.data_ptr(), zb.data_ptr(), rows, dof,
                                   1.0 / rows, l2.data_ptr(), stream))
    torch.cuda.synchronize()
    g = tm.cpu().numpy().astype(np.float64) / 0.1          # m = 0.1 g after one step from zero
    want = tg.cpu().numpy().astype(np.float64)
    # magnitudes in the parameters' order: rows of W1..W3 are stored by quads of inputs
    mag = magnitude[:-1].copy()
    for at, k in ((0, 16), (2048 + 128, 128), (2048 + 128 + 16384 + 128, 128)):
        block = mag[at:at + 128 * k].reshape(k // 4, 128, 4)
        mag[at:at + 128 * k] = block.transpose(1, 0, 2).reshape(-1)
    assert np.all(np.abs(g - want) <= (2 * n_parts + 8) * u * mag)
    assert abs(float(loss[0]) - float(l2[0])) <= (2 * n_parts + 8) * u * magnitude[-1]
    assert np.abs(want).max() > 0

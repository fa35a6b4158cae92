"""LearnedProposal.train over several steps: the default adds the tiles' gradients as
fs_mlp_train_step and fs_mlp_adam do, in arrival order; reproducible=True adds them in order,
with equal bits from equal calls.  Both orders against 64 bits."""
import ctypes
import math

import numpy as np
import pytest

from gpu_util import engine, require_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()
    engine()


def _network(dof, seed):
    rng = np.random.RandomState(seed)
    parts = []
    for out, inp, scale in ((128, 16, 1.0), (128, 128, 1.0), (128, 128, 1.0), (16, 128, 0.2)):
        parts += [scale * math.sqrt(2.0 / inp) * rng.randn(out * inp), 0.05 * scale * rng.randn(out)]
    return np.concatenate(parts).astype(np.float32)


def _data(n, dof, seed):
    rng = np.random.RandomState(seed)
    x = np.zeros((n, 16), np.float32)
    x[:, :dof] = rng.randn(n, dof)
    x[:, dof:2 * dof] = 0.2 * rng.randn(n, dof)
    z = np.zeros((n, 8), np.float32)
    z[:, :dof] = 0.5 * np.tanh(x[:, :dof]) + (0.6 + 0.2 * np.cos(x[:, :dof])) * rng.randn(n, dof)
    return x, z


class _State:
    """Parameters, moments and the BF16 copy on the device."""

    def __init__(self, params):
        import torch
        from feynsimul_gb300 import _lib
        self.L, self.check = _lib.lib(), _lib.check
        sizes = [ctypes.c_int64() for _ in range(4)]
        self.check(self.L.fs_mlp_sizes(*[ctypes.byref(v) for v in sizes]))
        self.p = torch.from_numpy(params.copy()).cuda()
        self.m, self.v, self.g = (torch.zeros_like(self.p) for _ in range(3))
        self.q = torch.zeros(sizes[1].value, dtype=torch.int16, device="cuda")
        f = torch.zeros(sizes[2].value * 2, dtype=torch.int32, device="cuda")
        b = torch.zeros(sizes[3].value, dtype=torch.float32, device="cuda")
        self.stream = torch.cuda.current_stream().cuda_stream
        self.check(self.L.fs_mlp_pack(self.p.data_ptr(), self.q.data_ptr(), f.data_ptr(), b.data_ptr(), self.stream))
        self.loss = torch.zeros(1, dtype=torch.float32, device="cuda")

    def copy_from(self, o):
        for a in ("p", "m", "v", "q"):
            getattr(self, a).copy_(getattr(o, a))

    def step(self, xb, zb, dof, it, lr=1e-3):
        self.loss.zero_()
        n = xb.shape[0]
        self.check(self.L.fs_mlp_train_step(self.p.data_ptr(), self.q.data_ptr(), self.g.data_ptr(), xb.data_ptr(),
                                            zb.data_ptr(), n, dof, 1.0 / n, self.loss.data_ptr(), self.stream))
        self.check(self.L.fs_mlp_adam(self.p.data_ptr(), self.m.data_ptr(), self.v.data_ptr(), self.g.data_ptr(),
                                      self.q.data_ptr(), it, lr, self.stream))


def _far(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


@pytest.mark.parametrize("batch,steps,dof,rows,data", [(683, 17, 6, 5000, 17), (4062, 20, 3, 20000, 20)])
def test_train_adds_gradients_as_they_arrive(batch, steps, dof, rows, data):
    # A batch's tiles have a few usual orders of arrival, and two runs of one order differ by the
    # rounding of an Adam step, 2^-24 of a parameter, in each of at most 20 steps: 1.2e-6.  The sums
    # in the tiles' order end 1.5e-4 and 6e-5 away with these data.
    import torch
    from feynsimul_gb300.learned import LearnedProposal
    seed = 7
    x, z = _data(rows, dof, data)
    p0 = _network(dof, data)
    tx, tz = torch.from_numpy(x).cuda(), torch.from_numpy(z).cuda()
    runs, loops = [], []
    for _ in range(6):
        m = LearnedProposal(dof, 0.25, 5.0, params=p0)
        m.train(x, z, steps=steps, batch=batch, lr=1e-3, seed=seed)
        runs.append(m.params)
        s = _State(p0)
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        for it in range(steps):
            idx = torch.randint(0, x.shape[0], (batch,), device="cuda", generator=gen)
            s.step(tx.index_select(0, idx), tz.index_select(0, idx), dof, it + 1)
        torch.cuda.synchronize()
        loops.append(s.p.cpu().numpy())
    assert min(_far(a, b) for a in runs for b in loops) <= 1.2e-6


def _exact(x, z, p0, dof, batch, steps, seed):
    import torch
    flat = torch.from_numpy(p0).cuda().double().requires_grad_()
    tx, tz = torch.from_numpy(x).cuda().double(), torch.from_numpy(z).cuda().double()
    shapes = [(128, 16), (128,), (128, 128), (128,), (128, 128), (128,), (16, 128), (16,)]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    m, v = torch.zeros_like(flat), torch.zeros_like(flat)
    for it in range(1, steps + 1):
        idx = torch.randint(0, x.shape[0], (batch,), device="cuda", generator=gen)
        p = [t.reshape(s) for t, s in zip(torch.split(flat, [math.prod(s) for s in shapes]), shapes)]
        y = tx[idx]
        for i in range(0, 8, 2):
            y = y @ p[i].T + p[i + 1]
            y = torch.relu(y) if i < 6 else y
        s = 4.0 * torch.tanh(0.25 * y[:, dof:2 * dof])
        loss = (0.5 * (tz[idx, :dof] - y[:, :dof]) ** 2 * torch.exp(-s) + 0.5 * s).sum() / batch
        (g,) = torch.autograd.grad(loss, flat)
        with torch.no_grad():
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            flat -= 1e-3 * (m / (1 - 0.9 ** it)) / (torch.sqrt(v / (1 - 0.999 ** it)) + 1e-8)
    return flat.detach().cpu().numpy()


@pytest.mark.parametrize("batch,dof", [(100, 6), (1200, 3), (8192, 8)])
def test_both_orders_are_as_exact(batch, dof):
    # fifty steps: BF16 operands put both orders about 5e-3 from 64 bits, and neither further than
    # half as much again as the other
    from feynsimul_gb300.learned import LearnedProposal
    x, z = _data(20000, dof, batch)
    p0 = _network(dof, batch)

    def run(**kw):
        m = LearnedProposal(dof, 0.25, 5.0, params=p0)
        losses = m.train(x, z, steps=50, batch=batch, lr=1e-3, seed=5, **kw)
        return losses, m.params

    exact = _exact(x, z, p0, dof, batch, 50, 5)
    (l1, p1), (l2, p2) = run(reproducible=True), run(reproducible=True)
    assert np.array_equal(l1, l2) and np.array_equal(p1, p2)
    arrive = [_far(run()[1], exact) for _ in range(5)]
    ordered = _far(p1, exact)
    assert ordered <= 1.5 * max(arrive) and max(arrive) <= 1.5 * ordered


def test_ordered_steps_reuse_their_workspace():
    # more tiles than SMs, then fewer and fewer, on one workspace of NaN: every step uses only the
    # rows its own CTAs wrote, and the optimiser, launched early, the moments of the step before
    import torch
    dof = 6
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    x, z = _data(40000, dof, 3)
    tx, tz = torch.from_numpy(x).cuda(), torch.from_numpy(z).cuda()
    rng = np.random.RandomState(4)
    counts = [128 * sms + 300, 4096, 129, 1, 700, 128 * sms]
    rows = [torch.from_numpy(rng.randint(0, x.shape[0], n)).cuda() for n in counts]
    p0 = _network(dof, 3)
    one = _State(p0)
    need = ctypes.c_int64()
    one.check(one.L.fs_mlp_workspace(max(counts), ctypes.byref(need)))
    stride = need.value // sms

    def run(look):
        s, other = _State(p0), _State(p0)
        work = torch.full((need.value,), math.nan, dtype=torch.float32, device="cuda")
        out = []
        for it, idx in enumerate(rows, 1):
            if look:
                other.copy_from(s)
            s.check(s.L.fs_mlp_train_batch(s.p.data_ptr(), s.m.data_ptr(), s.v.data_ptr(), s.q.data_ptr(), tx.data_ptr(),
                                           tz.data_ptr(), idx.data_ptr(), idx.numel(), dof, s.loss.data_ptr(), it, 1e-3,
                                           work.data_ptr(), need.value, s.stream))
            out.append((s.p.clone(), s.m.clone(), s.loss.clone()))
            if look:  # the same step by atomics: FP32 sums of the same terms in another order
                other.step(tx[idx], tz[idx], dof, it)
                torch.cuda.synchronize()
                n = min(-(-idx.numel() // 128), sms)
                parts = work.cpu().numpy().astype(np.float64).reshape(sms, stride)[:n, :p0.size]
                size = np.linalg.norm(np.abs(parts).sum(axis=0))
                m, w = s.m.cpu().numpy().astype(np.float64), other.m.cpu().numpy().astype(np.float64)
                assert np.linalg.norm(m - w) <= 2.0 ** -24 * (0.1 * (2 * n + 8) * size + 4 * np.linalg.norm(w))
        torch.cuda.synchronize()
        return out

    for a, b in zip(run(True), run(False)):
        for u, w in zip(a, b):
            assert torch.equal(u, w)


@pytest.mark.parametrize("rows", [1, 300, 20000])
def test_ordered_step_without_a_loss_changes_nothing(rows):
    # as after a pass that gave up: a NaN loss in one CTA's row of the workspace, the last one's
    import torch
    from feynsimul_gb300 import _lib
    from feynsimul_gb300.learned import LearnedProposal
    dof = 6
    x, z = _data(rows, dof, 1)
    p0 = _network(dof, 1)
    s = _State(p0)
    tx, tz = torch.from_numpy(x).cuda(), torch.from_numpy(z).cuda()
    need = ctypes.c_int64()
    s.check(s.L.fs_mlp_workspace(rows, ctypes.byref(need)))
    work = torch.full((need.value,), math.nan, dtype=torch.float32, device="cuda")
    idx = torch.arange(rows, device="cuda")

    def step(it):
        s.check(s.L.fs_mlp_train_batch(s.p.data_ptr(), s.m.data_ptr(), s.v.data_ptr(), s.q.data_ptr(), tx.data_ptr(),
                                       tz.data_ptr(), idx.data_ptr(), rows, dof, s.loss.data_ptr(), it, 1e-3,
                                       work.data_ptr(), need.value, s.stream))
        torch.cuda.synchronize()

    step(1)
    before = [t.clone() for t in (s.p, s.m, s.v, s.q)]
    assert math.isfinite(float(s.loss[0])) and not np.array_equal(before[0].cpu().numpy(), p0)
    tz[rows - 1, 0] = math.nan
    step(2)
    assert math.isnan(float(s.loss[0]))
    for a, b in zip(before, (s.p, s.m, s.v, s.q)):
        assert torch.equal(a, b)

    z[rows - 1, 0] = math.nan
    m = LearnedProposal(dof, 0.25, 5.0, params=p0)
    with pytest.raises(_lib.FsError, match="NaN"):
        m.train(x, z, steps=5, batch=rows, seed=2, reproducible=True)  # 5 draws of `rows` of `rows` rows
    assert np.array_equal(m.params, p0) and m.history == []
    hist = m.train(x, z, steps=5, batch=rows, seed=2)  # as ever: NaN data give NaN parameters
    assert np.isnan(hist).any() and np.isnan(m.params).any()

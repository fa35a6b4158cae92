"""batch.autotune and the tunings that an earlier kernel left behind."""
import hashlib
import json
import os

from feynsimul_gb300 import batch


class _Sampler:
    """Times instead of a GPU: the smaller CTA is the faster one here."""

    def __init__(self, workload, op_runs, msteps, block, tpw):
        self.block, self.node_updates_per_launch, self.registers, self.smem = block, 1000, 128, 1

    def run(self, launches=1):
        return 1e-3 * self.block * launches

    def close(self):
        pass


def test_tunings_of_an_earlier_kernel_are_not_used(tmp_path, monkeypatch):
    # version 4: padded tiles of 200 KB, one CTA per SM
    wl = batch.ragged_workload(seed=0)
    old = hashlib.sha1(json.dumps([wl, 1, 4, 4], sort_keys=True).encode()).hexdigest()[:16]
    cache = tmp_path / "tune.json"
    cache.write_text(json.dumps({old: {"block_threads": 512, "tpw_target": 64}}))
    monkeypatch.setattr(batch, "BatchSampler", _Sampler)
    monkeypatch.setattr(batch.os.path, "abspath", lambda p: str(tmp_path / "no" / "batch.py"))  # nothing shipped
    best = batch.autotune(wl, candidates=[(512, 64), (256, 64)], cache_file=str(cache))
    assert best["cached"] is False and best["block_threads"] == 256


def test_shipped_tuning_is_of_this_kernel():
    shipped = os.path.join(os.path.dirname(batch.__file__), "tuned", "batch_autotune.json")
    assert batch._signature(batch.ragged_workload(seed=0), 1, 4) in json.load(open(shipped))

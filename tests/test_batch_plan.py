"""Host logic of the mixed-level batch path (no GPU): the seeded workload
sampler and the autotuner's result cache."""

import json

import pytest

from fhelium_b200 import autotune
from fhelium_b200.batch import HMULT, ROTATE, sample_mixed_workload


def test_workload_is_seeded_and_well_formed():
    levels, ops = sample_mixed_workload(35, 512, seed=7)
    again = sample_mixed_workload(35, 512, seed=7)
    assert (levels, ops) == again
    assert sample_mixed_workload(35, 512, seed=8) != (levels, ops)
    limbs = [35 - lv for lv in levels]
    assert min(limbs) >= 3 and max(limbs) <= 35
    assert len(set(limbs)) == 33  # every limb count 3..35 drawn at this size
    kinds = [op.kind for op in ops]
    assert 0.4 < kinds.count(HMULT) / len(ops) < 0.6
    for i, op in enumerate(ops):
        assert op.index == i
        if op.kind == HMULT:
            assert levels[op.partner] == levels[i]
        else:
            assert op.kind == ROTATE
            assert 1 <= abs(op.step) <= 1 << 14
    assert any(op.step < 0 for op in ops) and any(op.step > 0 for op in ops)


def test_workload_rejects_bad_ranges():
    with pytest.raises(ValueError):
        sample_mixed_workload(8, 4, min_limbs=1)
    with pytest.raises(ValueError):
        sample_mixed_workload(8, 4, max_limbs=9)


def test_cache_round_trip(tmp_path):
    path = str(tmp_path / "sub" / "tune.json")
    assert autotune._load(path) == {}
    autotune._store(path, "a", {"ks_order": 1, "streams": 2, "ms": 3.0})
    autotune._store(path, "b", {"ks_order": 0, "streams": 1, "ms": 4.0})
    data = autotune._load(path)
    assert data["a"]["streams"] == 2 and data["b"]["ks_order"] == 0
    with open(path, "w") as f:
        f.write("not json")
    assert autotune._load(path) == {}
    json.dumps(autotune.default_cache_path())


class _FakeContext:
    """Tuning values and calls of a context, without a GPU."""

    def __init__(self):
        self.values = {}

    def set_tuning(self, param, value):
        self.values[param] = value

    def get_tuning(self, param):
        return self.values.get(param, 0)

    def call(self, name, *args):
        pass


def test_saved_transforms_of_older_kernels_are_searched_again(tmp_path, monkeypatch):
    """A winner saved when 8 and 16 residues per thread named two cluster forms
    is no hit now that 8 names the column and block launches; this one's is."""
    import torch
    from types import SimpleNamespace
    from fhelium_b200 import _native as nat
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda device=None: "B200")
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: SimpleNamespace(cuda_stream=0))
    ctx = _FakeContext()
    timed = []

    def times(run, device, **kwargs):
        run()
        timed.append(dict(ctx.values))
        return 1.0 if ctx.values.get(nat.TUNE_NTT_INVERSE_EPT, ctx.values[nat.TUNE_NTT_FORWARD_EPT]) == 8 else 2.0

    monkeypatch.setattr(autotune, "time_replays", times)
    path = str(tmp_path / "tune.json")
    autotune._store(path, "B200|ntt|bits=64|N=4096|rows=3|row_start=0|batch=2",
                    {"forward_ept": 16, "inverse_ept": 16, "forward_ms": 0.1, "inverse_ms": 0.1})
    x = torch.zeros((2, 3, 4096), dtype=torch.int64)
    first = autotune.tune_ntt(ctx, x, 3, cache_path=path)
    assert not first["cached"] and len(timed) == 4
    assert ctx.get_tuning(nat.TUNE_NTT_FORWARD_EPT) == 8 and ctx.get_tuning(nat.TUNE_NTT_INVERSE_EPT) == 8
    assert autotune.tune_ntt(ctx, x, 3, cache_path=path)["cached"] and len(timed) == 4


def test_saved_batches_of_older_kernels_are_searched_again(monkeypatch):
    """So it is with the mixed batches' keys: none of the form they had before."""
    import torch
    from types import SimpleNamespace
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda device=None: "B200")
    eng = SimpleNamespace(device=0, log_n=14, num_q=8, num_p=1, moduli=[3, 5])
    groups = SimpleNamespace(groups=[SimpleNamespace(kind=HMULT, level=1, items=2)])
    op = SimpleNamespace(kind=ROTATE, index=0)
    for key in (autotune.workload_key(eng, groups),
                autotune.items_workload_key(eng, [SimpleNamespace(level=3)], [op])):
        assert key.startswith("B200|r2|logN=14|q=8|p=1|chain=") and not key.startswith("B200|logN")


def test_streaming_chunks_cover_the_batch():
    from fhelium_b200.streaming import _chunks, tapered
    assert _chunks(7, 3) == [(0, 3), (3, 5), (5, 7)]
    assert _chunks(2, 5) == [(0, 1), (1, 2)]
    assert _chunks(32, 4) == [(0, 8), (8, 16), (16, 24), (24, 32)]
    assert _chunks(5, [2, 2, 1]) == [(0, 2), (2, 4), (4, 5)]
    for bad in ([2, 2], [3, 0, 2], []):
        with pytest.raises(ValueError):
            _chunks(5, bad)
    assert tapered(32, 2, 4) == [2] * 14 + [1] * 4
    assert tapered(7, 4, 2) == [4, 1, 1, 1]
    assert tapered(3, 2, 5) == [1, 1, 1]
    assert sum(tapered(33, 4, 3)) == 33

"""The autotuner's cache on the CPU (device name and context faked): keys
bucket the atom count by powers of two and separate kernels, bin counts,
species counts and devices; the JSON file survives a round trip and is
written atomically; apply_cached sets exactly the cached variants."""
import os

import pytest

from conftest import REPO


@pytest.fixture
def tune(monkeypatch):
    from pyiid_gb300 import autotune
    path = os.path.join(REPO, 'tests', '_build', 'tuning_cache.json')
    os.makedirs(os.path.dirname(path), exist_ok=True)
    if os.path.exists(path):
        os.remove(path)
    monkeypatch.setenv('PYIID_GB300_TUNE_CACHE', path)
    monkeypatch.setattr(autotune.torch.cuda, 'get_device_name',
                        lambda *a: 'NVIDIA GB300')
    return autotune


def test_keys_bucket_atoms_and_separate_problems(tune):
    k = tune._key
    assert k('fq', 1000, 500, 1) == k('fq', 513, 500, 1)     # N <= 1024
    assert k('fq', 1000, 500, 1) != k('fq', 1025, 500, 1)
    assert k('fq', 1000, 500, 1) != k('grad_fq', 1000, 500, 1)
    assert k('fq', 1000, 500, 1) != k('fq', 1000, 498, 1)
    assert k('fq', 1000, 500, 1) != k('fq', 1000, 500, 2)
    assert k('fq', 0, 500, 1) == k('fq', 1, 500, 1)
    assert k('fq', 1000, 500, 1).startswith('NVIDIA GB300|')


def test_cache_round_trip_and_apply(tune, monkeypatch):
    assert tune._load_cache() == {}
    c = {tune._key('fq', 20000, 1475, 1): 23,
         tune._key('grad_fq', 20000, 1475, 1): 3}
    tune._save_cache(c)
    assert tune._load_cache() == c
    assert not any(f.startswith('tuning_cache.json.')
                   for f in os.listdir(os.path.dirname(tune.cache_path())))

    class FakeCtx:
        def __init__(self):
            self.set = {}

        def set_variant(self, kernel, v):
            self.set[kernel] = v

    ctx = FakeCtx()
    monkeypatch.setattr(tune, 'context', lambda device=None: ctx)
    assert tune.apply_cached(20000, 1475, 1) == {'fq': 23, 'grad_fq': 3}
    assert ctx.set == {'fq': 23, 'grad_fq': 3}
    ctx.set.clear()
    assert tune.apply_cached(20000, 1500, 1) == {} and ctx.set == {}


def test_unreadable_cache_is_empty(tune):
    with open(tune.cache_path(), 'w') as f:
        f.write('{not json')
    assert tune._load_cache() == {}


class CountingCtx:
    """A context whose calls run the kernels of ``runs`` only."""

    def __init__(self, runs):
        self.runs, self.var, self.count = runs, {'fq': 5, 'grad_fq': 2}, {}
        self.set = []

    def get_variant(self, k):
        return self.var[k]

    def set_variant(self, k, v):
        self.set.append((k, v))
        self.var[k] = v

    def variant_launches(self, k):
        return self.count.get(k, 0)

    def call(self):
        for k in self.runs:
            self.count[k] = self.count.get(k, 0) + 1


def test_a_kernel_that_does_not_run_keeps_its_variant(tune, monkeypatch):
    """tune_call times the variants of what the call runs; a kernel that it
    does not run is neither changed nor chosen by noise."""
    ctx = CountingCtx({'fq'})
    monkeypatch.setattr(tune, 'context', lambda device=None: ctx)
    monkeypatch.setattr(tune, 'variants',
                        lambda k: [(i, {}) for i in range(8)])

    def timed(fn, reps):
        fn()
        return 1.0 if ctx.var['fq'] == 3 else 2.0 - 0.1 * ctx.var['grad_fq']
    monkeypatch.setattr(tune, '_time', timed)
    r = tune.tune_call(ctx.call, kernels=('grad_fq', 'fq'))
    assert r['fq']['best'] == 3 and sorted(r['fq']['ms']) == list(range(8))
    assert r['grad_fq']['best'] == 2 and list(r['grad_fq']['ms']) == [2]
    assert ctx.var == {'fq': 3, 'grad_fq': 2}
    assert all(k == 'fq' for k, _ in ctx.set)


def test_tune_saves_what_it_timed(tune, monkeypatch):
    """Beside a timed choice, a call on the phase grid leaves the cached
    variant of its bucket as it is, and the current one where there is none."""
    import numpy as np
    import torch
    ctx = CountingCtx({'fq'})
    monkeypatch.setattr(tune, 'context', lambda device=None: ctx)
    monkeypatch.setattr(tune, 'variants',
                        lambda k: [(i, {}) for i in range(8)])
    monkeypatch.setattr(tune, '_time',
                        lambda fn, reps: (fn(), 1.0 + (ctx.var['fq'] != 6))[1])
    for name in ('fq', 'grad_fq'):
        monkeypatch.setattr(tune.debye, name, lambda *a, **k: ctx.call())
    monkeypatch.setattr(tune.debye, 'as_positions',
                        lambda x: torch.as_tensor(x))
    empty = torch.empty
    monkeypatch.setattr(tune.torch, 'empty',
                        lambda *a, **k: empty(1))
    tab = np.ones((1, 300), np.float32)
    args = (np.zeros((200, 3), np.float32), np.zeros(200, np.int32), tab, 0.05)
    key = tune._key('grad_fq', 200, 300, 1)
    tune.tune(*args, kernels=('fq',))
    ctx.var['grad_fq'] = 4
    ctx.runs = set()
    tune.tune(*args, kernels=('grad_fq',))
    assert tune._load_cache()[key] == 4
    ctx.var['grad_fq'] = 1
    tune.tune(*args, kernels=('grad_fq',))
    assert tune._load_cache() == {tune._key('fq', 200, 300, 1): 6, key: 4}

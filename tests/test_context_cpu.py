"""Context lookup on the host: which context a param_dict gets, and at what cost.  The
native context is replaced by a record of its arguments."""
import threading
import time

import numpy as np
import pytest
import torch

from ecs_mhd_2d_b200 import context


class FakeContext:
    made = []

    def __init__(self, n, dtype, nu, eta, b0, forcing=None, max_batch=1):
        time.sleep(0.01)
        self._forcing = forcing
        FakeContext.made.append(self)

    def ensure_batch(self, batch):
        pass

    def close(self):
        pass


@pytest.fixture
def lookup(monkeypatch):
    monkeypatch.setattr(context, "Context", FakeContext)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    context.clear_cache()
    FakeContext.made = []

    def get(forcing, n=8, **kw):
        return context.get_context(dict(dict(nu=0.1, eta=0.2, b0=[0.0, 0.1], forcing=forcing), **kw), n, torch.float64)

    yield get
    context.clear_cache()


def _forcings(count, n=8):
    return [torch.as_tensor(np.random.default_rng(i).standard_normal((n, n))) for i in range(count)]


def test_same_values_same_context(lookup):
    f, g = _forcings(2)
    a = lookup(f)
    assert lookup(f.clone()) is a and lookup(g) is not a and lookup(None) is not a
    assert lookup(f) is a and lookup(f, nu=0.3) is not a
    f[3, 3] += 1e-15   # another value, in place
    assert lookup(f) is not a and len(FakeContext.made) == 5


def test_many_forcings_cost_one_comparison_each(lookup, monkeypatch):
    """A sweep over forcings compares none of them with all others."""
    fs = _forcings(40)
    want = [lookup(f) for f in fs]
    calls = []
    same = context._same_bits
    monkeypatch.setattr(context, "_same_bits", lambda a, b: calls.append(1) or same(a, b))
    assert [lookup(f) for f in fs] == want
    assert len(calls) <= len(fs)


def test_threads_that_miss_together_share(lookup):
    f, got = _forcings(1)[0], []
    ts = [threading.Thread(target=lambda: got.append(lookup(f))) for _ in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert len(FakeContext.made) == 1 and all(c is got[0] for c in got)


class DeviceTensor(torch.Tensor):
    """A host tensor that says it is on the device."""
    is_cuda = True


def test_forcing_of_another_grid_is_not_staged(lookup, monkeypatch):
    """The pinned staging copy outlives the call: a forcing that is refused must not size it."""
    made = []
    empty = torch.empty

    def host_empty(*a, pin_memory=False, **kw):
        made.append(a[0])
        return empty(*a, **kw)

    monkeypatch.setattr(context, "_STAGE", threading.local())
    monkeypatch.setattr(torch, "empty", host_empty)
    with pytest.raises(ValueError, match="forcing"):
        lookup(torch.zeros((64, 64), dtype=torch.float64).as_subclass(DeviceTensor))
    assert made == []
    lookup(torch.ones((8, 8), dtype=torch.float64).as_subclass(DeviceTensor))
    assert made == [64] and np.all(FakeContext.made[-1]._forcing == 1.0)

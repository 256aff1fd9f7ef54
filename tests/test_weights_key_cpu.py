"""The key under which the executor keeps a model's packed weights: it follows every parameter and buffer, and ends where
modules hold one another."""
import signal

import pytest
import torch
from torch import nn


def _key(model, seconds=5.0):
    from ffnoml_gb300.executor import _weights_key

    def stop(*_):
        raise TimeoutError("the walk over the modules does not end")

    before = signal.signal(signal.SIGALRM, stop)
    signal.setitimer(signal.ITIMER_REAL, seconds)
    try:
        return _weights_key(model)
    finally:
        signal.setitimer(signal.ITIMER_REAL, 0)
        signal.signal(signal.SIGALRM, before)


def _model():
    m = nn.Sequential(nn.Conv3d(2, 4, 1), nn.BatchNorm3d(4), nn.Sequential(nn.Conv3d(4, 2, 1, bias=False)))
    m.shared = m[0]
    return m


def test_a_module_that_holds_the_model_ends_the_walk():
    m = _model()
    key = _key(m)
    m[2].owner = m                     # a cycle, as a trainer registered on its own model makes one
    assert _key(m) == key


@pytest.mark.parametrize("change", ["update", "buffer", "replace", "submodule"])
def test_every_change_changes_the_key(change):
    m = _model()
    key = _key(m)
    with torch.no_grad():
        if change == "update":
            m[2][0].weight.add_(1)
        elif change == "buffer":
            m[1].running_mean.add_(1)
        elif change == "replace":
            old = m[0].bias            # held, so that the new one lies elsewhere
            m[0].bias = nn.Parameter(old.clone())
        else:
            old = m[2]
            m[2] = nn.Sequential(nn.Conv3d(4, 2, 1, bias=False))
    assert _key(m) != key

"""A tensor-core pipeline whose bounded waits run out is reported by the call
that used it, not priced from what the buffers held before.

QK_B200_FAULT=timeout sets the kernels' error word, as a timed-out wait would,
before the launches of a call; nothing on the GPU waits or fails.
"""

import struct

import numpy as np
import pytest

from quantkernel_b200 import QKRuntimeError
from quantkernel_b200.surrogate import HestonSurrogate, features_of, sample_box

pytestmark = pytest.mark.gpu

MATCH = r"tensor-core pipeline timed out \(code \d+\).*\[injected\]"


def _steps(sur, tmp_path):
    """Completed optimiser steps: the first word of a checkpoint's state, after
    magic, size, base kind and the box."""
    sur.save(tmp_path / "m.qksur")
    return struct.unpack_from("<i", (tmp_path / "m.qksur").read_bytes(), 8 + 4 + 4 + 144)[0]


@pytest.fixture
def model(qk):
    sur = HestonSurrogate(qk, seed=3)
    f = features_of(**sample_box(1024, 5))
    y = np.random.default_rng(1).uniform(0.0, 0.5, 1024)
    sur.set_dataset(f, y)
    sur.train(1, batch=128, lr=1e-3, shuffle_seed=1)
    yield sur, f, y
    sur.close()


@pytest.mark.parametrize("n", (1, 700, 65536 + 3))
def test_pricing_calls(qk, model, monkeypatch, n):
    sur, _, _ = model
    b = sample_box(n, 9)
    ot = (np.arange(n) % 2).astype(np.int32)
    calls = {"predict": lambda: (sur.predict(features_of(**b)),),
             "price_batch": lambda: sur.price_batch(**b, option_type=ot)}
    for call in calls.values():
        want = call()
        monkeypatch.setenv("QK_B200_FAULT", "timeout")
        with pytest.raises(QKRuntimeError, match=MATCH):
            call()
        monkeypatch.delenv("QK_B200_FAULT")
        for g, w in zip(call(), want):  # the word is cleared with the report
            assert np.array_equal(g, w)


def test_gradients(qk, model, monkeypatch):
    sur, f, y = model
    loss, want = sur.gradients(f, y)
    monkeypatch.setenv("QK_B200_FAULT", "timeout")
    with pytest.raises(QKRuntimeError, match=MATCH):
        sur.gradients(f, y)
    monkeypatch.delenv("QK_B200_FAULT")
    again, got = sur.gradients(f, y)
    assert again == loss and np.array_equal(got, want)


def test_training_leaves_the_weights(qk, model, monkeypatch, tmp_path):
    sur, f, y = model
    before = sur.parameters()
    steps = _steps(sur, tmp_path)
    monkeypatch.setenv("QK_B200_FAULT", "timeout")
    with pytest.raises(QKRuntimeError, match=MATCH):
        sur.train(2, batch=128, lr=1e-2, shuffle_seed=4)
    monkeypatch.delenv("QK_B200_FAULT")
    assert np.array_equal(sur.parameters(), before) and _steps(sur, tmp_path) == steps
    sur.train(1, batch=128, lr=1e-3, shuffle_seed=4)
    assert _steps(sur, tmp_path) == steps + 8 and not np.array_equal(sur.parameters(), before)

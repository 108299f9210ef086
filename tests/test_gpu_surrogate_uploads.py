"""Parameters, checkpoints and datasets are on the GPU before the kernels that
read them run: calls in quick succession, alternating between two states, give
each state's results every time.
"""

import numpy as np
import pytest

from quantkernel_b200.surrogate import HestonSurrogate, features_of, sample_box

pytestmark = pytest.mark.gpu


def test_alternating_parameters(qk):
    f = features_of(**sample_box(1024, 7))
    sur = HestonSurrogate(qk, seed=3)
    rng = np.random.default_rng(2)
    states = [rng.standard_normal(sur.parameters().shape) * 0.05 for _ in range(2)]
    want = []
    for p in states:
        for _ in range(2):
            sur.set_parameters(p)
        want.append(sur.predict(f))
    assert not np.array_equal(*want)
    for i in range(400):
        sur.set_parameters(states[i % 2])
        assert np.array_equal(sur.predict(f), want[i % 2]), i
    sur.close()


def test_inference_on_the_default_stream_keeps_its_parameters(qk):
    """Parameters set while an earlier call's kernel runs on the default stream
    are for later calls only."""
    import torch

    n = 1 << 20
    f = torch.from_numpy(features_of(**sample_box(n, 7))).cuda()
    rows = torch.empty((n, 64), dtype=torch.bfloat16, device="cuda")
    base = torch.empty(n, dtype=torch.float32, device="cuda")
    y, ref = (torch.empty(n, dtype=torch.float32, device="cuda") for _ in range(2))
    sur = HestonSurrogate(qk, seed=3)
    p = np.random.default_rng(2).standard_normal(sur.parameters().shape) * 0.05
    sur.features_device(f.data_ptr(), n, rows.data_ptr(), base.data_ptr())
    torch.cuda.synchronize()
    sur.set_parameters(p)
    sur.predict_device(rows.data_ptr(), base.data_ptr(), n, ref.data_ptr())
    torch.cuda.synchronize()
    for _ in range(10):
        sur.set_parameters(p)
        sur.predict_device(rows.data_ptr(), base.data_ptr(), n, y.data_ptr())
        sur.set_parameters(-p)
        torch.cuda.synchronize()
        assert torch.equal(y, ref)
    sur.close()


def test_alternating_checkpoints(qk, tmp_path):
    f = features_of(**sample_box(1024, 7))
    want = []
    for k in range(2):
        sur = HestonSurrogate(qk, seed=3 + k)
        p = sur.parameters()
        sur.set_parameters(p + 0.01)
        sur.save(tmp_path / f"{k}.qksur")
        want.append(sur.predict(f))
        sur.close()
    sur = HestonSurrogate(qk)
    for i in range(200):
        sur.load(tmp_path / f"{i % 2}.qksur")
        assert np.array_equal(sur.predict(f), want[i % 2]), i
    sur.close()


def test_alternating_datasets(qk):
    """Gradients of two datasets of different sizes: rows, targets, order and
    the batch's place in them."""
    sur = HestonSurrogate(qk, seed=3)
    data = []
    for n in (2048, 384):
        f = features_of(**sample_box(n, n))
        data.append((f, np.random.default_rng(n).uniform(0.0, 0.5, n)))
    want = [sur.gradients(*d) for d in data]
    for i in range(100):
        loss, g = sur.gradients(*data[i % 2])
        assert loss == want[i % 2][0] and np.array_equal(g, want[i % 2][1]), i
    sur.close()

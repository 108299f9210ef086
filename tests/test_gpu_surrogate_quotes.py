"""The surrogate's host pricing call at block and chunk edges: routes, entry
checks and put-call parity on the GPU against the same call's pieces.

The network part must equal predict() on the same features (one kernel, so
the same bits), parity and intrinsic values numpy's to 1e-13 of the spot.
"""

import numpy as np
import pytest

from quantkernel_b200.surrogate import HestonSurrogate, features_of, sample_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", (1, 255, 257, 65536, 65537, 131073))
def test_price_batch_at_chunk_edges(qk, n):
    sur = HestonSurrogate(qk, seed=3)
    b = sample_box(n, 11)
    ot = (np.arange(n) % 2).astype(np.int32)
    kind = np.arange(n) % 7  # 3: bad option type, 5: expired, 6: negative variance; else in the box
    ot[kind == 3] = 2
    b["t"][kind == 5] = 0.0
    b["v0"][kind == 6] = -0.01
    price, src = sur.price_batch(**b, option_type=ot)
    net = (kind != 3) & (kind != 5) & (kind != 6)
    assert np.array_equal(src, np.where(net, 0, 2))
    y = sur.predict(features_of(**b))
    call = b["spot"] * y
    put = call - b["spot"] * np.exp(-b["q"] * b["t"]) + b["strike"] * np.exp(-b["r"] * b["t"])
    want = np.where(ot == 0, call, put)
    want[kind == 5] = np.maximum(np.where(ot == 0, b["spot"] - b["strike"], b["strike"] - b["spot"]), 0.0)[kind == 5]
    ok = kind != 3
    ok &= kind != 6
    assert np.all(np.isnan(price[~ok]))
    assert np.all(np.abs(price - want)[ok] <= 1e-13 * b["spot"][ok])
    sur.close()

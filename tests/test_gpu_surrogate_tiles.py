"""The fused inference kernel walks its tiles in pairs with the next pair's
first layer issued inside the current one's: every count of tiles per block,
even and odd, must give the bits of the layer-by-layer GEMMs."""

import numpy as np
import pytest
import torch

from quantkernel_b200.surrogate import HestonSurrogate, features_of, sample_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles", (1, 2, 3, 4, 5, 7))
@pytest.mark.parametrize("extra", (-1, 0, 1))
def test_tiles_per_block(qk, tiles, extra):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 128 * sms * tiles + 128 * (sms // 2) * extra + extra
    sur = HestonSurrogate(qk, seed=5)
    p = sur.parameters()
    sur.set_parameters(p + 0.05 * np.random.default_rng(1).standard_normal(p.size))
    f = torch.from_numpy(features_of(**sample_box(4099, 3))).cuda().repeat(n // 4099 + 1, 1)[:n].contiguous()
    rows = torch.empty((n, 64), dtype=torch.bfloat16, device="cuda")
    base = torch.empty(n, dtype=torch.float32, device="cuda")
    y = torch.full((2, n + 1), float("nan"), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    sur.features_device(f.data_ptr(), n, rows.data_ptr(), base.data_ptr())
    torch.cuda.synchronize()
    for k in (0, 1):
        sur.predict_device(rows.data_ptr(), base.data_ptr(), n, y[k].data_ptr(), layered=bool(k))
    torch.cuda.synchronize()
    assert torch.isfinite(y[:, :n]).all() and torch.isnan(y[:, n]).all()
    assert torch.equal(y[0, :n], y[1, :n])

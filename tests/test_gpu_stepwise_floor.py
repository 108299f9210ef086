"""The one-factor step loop with its per-block floor check against the loop
that floors every step (step unrolling 2), bit for bit: volatilities from where
the floor never binds to where most paths end on it or overflow, step counts
around the six-step block, ragged path counts.
"""

import numpy as np
import pytest

from quantkernel_b200 import QK_PLAN_NO_ANTITHETIC, QK_PLAN_STEP_UNROLL2

pytestmark = pytest.mark.gpu

VOLS = (0.0, 0.2, 0.9, 1.6, 2.4, 4.0, 9.0, 1e3, 1e19)
STEPS = (1, 5, 6, 7, 12, 61)


@pytest.mark.parametrize("anti", (True, False))
@pytest.mark.parametrize("model", (2, 3, 4))
def test_block_floor_check_gives_the_floored_bits(qk, model, anti):
    grid = [(v, s, p) for v in VOLS for s in STEPS for p in (3, 1025, 4097)]
    n = len(grid)
    cols = dict(model=np.full(n, model, np.int32), spot=np.full(n, 100.0), strike=np.full(n, 95.0),
                t=np.full(n, 1.7), vol=np.array([g[0] for g in grid]), r=np.full(n, 0.03),
                q=np.where(np.arange(n) % 2, 0.01, 2.5),
                option_type=(np.arange(n) % 2).astype(np.int32),
                paths=np.array([g[2] for g in grid], np.int32),
                steps=np.array([g[1] for g in grid], np.int32),
                seed=np.arange(n, dtype=np.uint64) + np.uint64(900))
    out = []
    for flags in (0, QK_PLAN_STEP_UNROLL2):
        plan = qk.plan(**cols, flags=flags | (0 if anti else QK_PLAN_NO_ANTITHETIC))
        assert plan.config()["step_unroll"] == (2 if flags else 1)
        plan.execute()
        out.append(plan.results())
        plan.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b, equal_nan=True), np.flatnonzero(~((a == b) | (np.isnan(a) & np.isnan(b))))

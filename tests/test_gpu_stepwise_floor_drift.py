"""The one-factor step loop's per-block floor check where the spot is near or
below the floor of 1e-12 and the drift of a step is large, at each number of
units per thread, against the loop that floors every step (step unrolling 2),
bit for bit.  A growing state can lie above the block's limit and still meet a
floor above one inside the block.
"""

import numpy as np
import pytest

from quantkernel_b200 import QK_PLAN_NO_ANTITHETIC, QK_PLAN_STEP_UNROLL2

pytestmark = pytest.mark.gpu

SPOTS = (5e-14, 2e-13, 9e-13, 1e-12, 3e-12, 1e-11, 4e-10, 100.0)
DRIFTS = (-0.5, 0.0, 0.7, 2.0, 3.0, 9.0)  # r dt of a step
VOLS = (0.0, 0.2, 1.5)               # vol sqrt(dt) of a step


@pytest.mark.parametrize("anti", (True, False))
@pytest.mark.parametrize("model", (2, 3, 4))
@pytest.mark.parametrize("upt,paths,steps", ((1, 1001, 12), (1, 130, 61), (2, 3001, 78), (4, 6001, 13)))
def test_floor_near_the_spot(qk, model, anti, upt, paths, steps):
    grid = [(s, d, v) for s in SPOTS for d in DRIFTS for v in VOLS]
    # one option alone where the batch must not fill the chip
    for cases in ([[g] for g in grid] if upt == 1 else [grid]):
        n = len(cases)
        s, d, v = (np.array(c) for c in zip(*cases))
        cols = dict(model=np.full(n, model, np.int32), spot=s, strike=0.9 * s, t=np.full(n, 0.01 * steps),
                    vol=10.0 * v, r=100.0 * d, q=np.zeros(n), option_type=np.zeros(n, np.int32),
                    paths=np.full(n, paths if anti else (paths + 1) // 2, np.int32),
                    steps=np.full(n, steps, np.int32),
                    seed=np.arange(n, dtype=np.uint64) + np.uint64(17))
        out = []
        for flags in (0, QK_PLAN_STEP_UNROLL2):
            plan = qk.plan(**cols, flags=flags | (0 if anti else QK_PLAN_NO_ANTITHETIC))
            config = plan.config()
            assert config["step_unroll"] == (2 if flags else 1)
            assert flags or config["units_per_thread"] == upt
            plan.execute()
            out.append(plan.results())
            plan.close()
        for a, b in zip(*out):
            same = (a == b) | (np.isnan(a) & np.isnan(b))
            assert np.all(same), [cases[i] for i in np.flatnonzero(~same)]

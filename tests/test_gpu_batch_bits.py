"""A stepwise option's price is the same bits alone, in a book of any size and
in a mixed plan, however many units a thread takes there.

Payoffs are whole multiples of a quarter of the strike's last bit (S_T above the
strike is a multiple of that bit, K - S_T is rounded to it or finer), so their
double-double sums are exact below 2^50 strikes and no grouping changes them.
Squares have more bits than that: standard errors may differ in their last one.
"""

import numpy as np
import pytest

from quantkernel_b200 import QK_MC_EULER, QK_MC_HESTON, QK_MC_LOCAL_VOL, QK_MC_MILSTEIN, workloads

pytestmark = pytest.mark.gpu

MODELS = {"heston_monte_carlo": QK_MC_HESTON, "euler_maruyama": QK_MC_EULER, "milstein": QK_MC_MILSTEIN,
          "local_vol_monte_carlo": QK_MC_LOCAL_VOL}


def _book(name, n, paths, steps):
    if name == "heston_monte_carlo":
        b = workloads.heston(n, paths, steps, seed=6)
        b["option_type"] = (np.arange(n) % 2).astype(np.int32)
        return b
    b = workloads.bsm_terminal(n, paths, seed=6)
    b["steps"] = np.full(n, steps, np.int32)
    return b


def _same(got, want):
    assert np.array_equal(got[0], want[0], equal_nan=True), got[0] - want[0]
    np.testing.assert_allclose(got[1], want[1], rtol=1e-14, atol=0)


@pytest.mark.parametrize("paths,steps", ((1, 7), (999, 13), (5000, 75)))
@pytest.mark.parametrize("name", MODELS)
def test_books_of_every_size(qk, name, paths, steps):
    fn = getattr(qk, name + "_price_se_batch")
    full = _book(name, 1100, paths, steps)
    want = fn(**full)
    # results straight to pinned memory up to 1024 options, copied beyond
    for n in (1, 3, 40, 65, 500, 1023, 1024, 1025):
        _same(fn(**{k: v[:n] for k, v in full.items()}), [w[:n] for w in want])
    # the same options among others of another family: the persistent kernel
    other = _book("heston_monte_carlo" if name != "heston_monte_carlo" else "milstein", 200, 3000, 9)
    cols = {}
    for k in {**full, **other}:
        parts = [b.get(k, np.zeros(len(b["spot"]))) for b in (full, other)]
        cols[k] = np.concatenate(parts).astype(parts[0].dtype)
    model = np.full(1300, MODELS[name], np.int32)
    model[1100:] = QK_MC_HESTON if name != "heston_monte_carlo" else QK_MC_MILSTEIN
    plan = qk.plan(model=model, **cols)
    plan.execute()
    _same([r[:1100] for r in plan.results()], want)
    plan.close()


@pytest.mark.parametrize("steps", (179, 180))
@pytest.mark.parametrize("paths", (1024 * 124 - 3, 1024 * 126 + 1))  # 5952 and 6096 tiles of 512 pairs
@pytest.mark.parametrize("name", ("euler_maruyama", "milstein"))
def test_long_paths_on_either_side_of_the_limits(qk, name, paths, steps):
    b = _book(name, 48, paths, steps)
    fn = getattr(qk, name + "_price_se_batch")
    full = fn(**b)
    for i in (0, 47):
        _same(fn(**{k: v[i:i + 1] for k, v in b.items()}), [f[i:i + 1] for f in full])

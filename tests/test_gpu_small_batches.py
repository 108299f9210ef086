"""One-shot batches around the sizes where the plan changes: fewer units per
thread while the tiles do not fill the chip, results written straight to the
pinned buffer up to 64 options.  An option's price and standard error must not
depend on the batch it is in (double-double sums: 1e-14 allows their final
rounding only), and read-only or sliced columns must serve like owned ones.
"""

import numpy as np
import pytest

from quantkernel_b200 import workloads

pytestmark = pytest.mark.gpu


def _batch(kind, n, paths):
    if kind == "heston":
        return workloads.heston(n, paths, 20, seed=4)
    b = workloads.bsm_terminal(n, paths, seed=4)
    if kind != "antithetic_variates":
        b["steps"] = np.full(n, 20, np.int32)
    return b


@pytest.mark.parametrize("paths", (999, 4097))
@pytest.mark.parametrize("kind", ("heston", "euler_maruyama", "milstein", "antithetic_variates"))
def test_price_does_not_depend_on_the_batch(qk, kind, paths):
    fn = getattr(qk, "heston_monte_carlo_price_se_batch" if kind == "heston" else kind + "_price_se_batch")
    full = _batch(kind, 700, paths)
    want = fn(**full)
    for n in (1, 2, 36, 63, 64, 65, 150):
        got = fn(**{k: v[:n] for k, v in full.items()})
        for g, w in zip(got, want):
            np.testing.assert_allclose(g, w[:n], rtol=1e-14, atol=0)


@pytest.mark.parametrize("steps", (71, 72))
@pytest.mark.parametrize("paths", (1024 * 124 - 3, 1024 * 125 + 1))
@pytest.mark.parametrize("kind", ("euler_maruyama", "milstein", "local_vol_monte_carlo"))
def test_long_one_factor_paths(qk, kind, paths, steps):
    """Two or four units a thread, on either side of 72 steps and of 6000 tiles:
    options of a batch of 48 against the same options priced alone."""
    b = workloads.bsm_terminal(48, paths, seed=9)
    b["steps"] = np.full(48, steps, np.int32)
    fn = getattr(qk, kind + "_price_se_batch")
    full = fn(**b)
    for i in (0, 31, 47):
        for g, w in zip(fn(**{k: v[i:i + 1] for k, v in b.items()}), full):
            np.testing.assert_allclose(g, w[i:i + 1], rtol=1e-14, atol=0)


def test_read_only_and_strided_columns(qk):
    b = _batch("heston", 12, 1001)
    want = qk.heston_monte_carlo_price_batch(**b)
    odd = {}
    for i, (k, v) in enumerate(b.items()):
        if i % 2:
            v = np.repeat(v, 2)[::2]
        v = v.copy() if i % 3 else v
        v.flags.writeable = bool(i % 3)
        odd[k] = v
    assert np.array_equal(qk.heston_monte_carlo_price_batch(**odd), want)


class _Device:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f8", data=(ptr, False), version=3)


def test_unknown_plan_flags_keep_device_results(qk):
    """A plan built with a flag bit that means nothing to callers is read and
    run again like any other: its results stay on the device too."""
    import torch

    b = workloads.mixed(8, seed=3, log2_paths=(10, 11), log2_steps=(3, 4))
    plan = qk.plan(**b, flags=0x10000)
    want = qk.plan(**b)
    for p in (want, plan, plan):
        p.execute()
    w, g = want.results(), plan.results()
    for a, c in zip(g, w):
        assert np.array_equal(a, c)
    for ptr, a in zip(plan.device_results(), w):
        assert np.array_equal(torch.as_tensor(_Device(ptr, 8), device="cuda").cpu().numpy(), a)

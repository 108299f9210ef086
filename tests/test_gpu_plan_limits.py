"""Plans at the limits of their host arithmetic and layout: path counts next to
the largest 32-bit integer, and the alignment of the device result arrays.
"""

import numpy as np
import pytest

from quantkernel_b200 import QK_MC_HESTON, QK_PLAN_NO_ANTITHETIC, workloads

pytestmark = pytest.mark.gpu

INT_MAX = 2**31 - 1


@pytest.mark.parametrize("paths", (INT_MAX, INT_MAX - 255, INT_MAX - 510, INT_MAX - 511, INT_MAX - 600))
@pytest.mark.parametrize("model,upt", ((2, 4), (3, 4), (4, 4), (QK_MC_HESTON, 2)))
def test_units_per_thread_at_the_largest_path_counts(qk, model, upt, paths):
    """One unpaired option fills the chip many times over: its family's own
    units per thread.  The plan is built and not run."""
    one = np.ones(1)
    plan = qk.plan(model=np.full(1, model, np.int32), spot=100 * one, strike=95 * one, t=one, vol=0.2 * one,
                   r=0.02 * one, q=0 * one, v0=0.04 * one, kappa=one, theta=0.04 * one, sigma=0.3 * one,
                   rho=-0.5 * one, option_type=np.zeros(1, np.int32), paths=np.full(1, paths, np.int32),
                   steps=np.ones(1, np.int32), seed=np.ones(1, np.uint64), flags=QK_PLAN_NO_ANTITHETIC)
    assert plan.config()["units_per_thread"] == upt
    plan.close()


class _Device:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f8", data=(ptr, False), version=3)


@pytest.mark.parametrize("n", (1, 2, 3, 31, 33, 65, 1001))
def test_device_results_are_aligned_like_allocations(qk, n):
    import torch

    plan = qk.plan(**workloads.mixed(n, seed=5, log2_paths=(8, 9), log2_steps=(2, 3)))
    plan.execute()
    host = plan.results()
    for ptr, a in zip(plan.device_results(), host):
        assert ptr % 256 == 0
        assert np.array_equal(torch.as_tensor(_Device(ptr, n), device="cuda").cpu().numpy(), a, equal_nan=True)
    plan.close()

"""The surrogate's host pricing call where its routes meet: options that the
entry checks decide do not depend on the network, and outputs may share memory
with the inputs they replace.
"""

import ctypes as ct

import numpy as np
import pytest

from quantkernel_b200.surrogate import N_PARAMS, HestonSurrogate, sample_box

pytestmark = pytest.mark.gpu


def _quotes(n):
    """In the box, expired, outside the box (Monte Carlo) and refused, in turn."""
    b = sample_box(n, 23)
    ot = (np.arange(n) % 2).astype(np.int32)
    kind = np.arange(n) % 4 if n < 100 else np.where(np.arange(n) % 5000 < 8, np.arange(n) % 4, 0)
    b["t"][kind == 1] = 0.0
    b["strike"][kind == 2] *= 3.0
    b["v0"][kind == 3] = -0.01
    return b, ot, kind


@pytest.mark.parametrize("value", (np.nan, np.inf))
def test_decided_options_do_not_depend_on_the_network(qk, value):
    sur = HestonSurrogate(qk, seed=3)
    b, ot, kind = _quotes(64)
    want, src = sur.price_batch(**b, option_type=ot, fallback_paths=1000, fallback_steps=8)
    sur.set_parameters(np.full(N_PARAMS, value))
    got, src2 = sur.price_batch(**b, option_type=ot, fallback_paths=1000, fallback_steps=8)
    assert np.array_equal(src, src2)
    assert np.array_equal(src, np.array([0, 2, 1, 2])[kind])
    decided = kind != 0
    assert np.array_equal(got[decided], want[decided], equal_nan=True)
    assert np.all(np.isfinite(got[kind == 1])) and np.all(np.isfinite(got[kind == 2]))
    sur.close()


@pytest.mark.parametrize("n", (40, 65536 + 21))
@pytest.mark.parametrize("column", (0, 1, 6, 9))
def test_outputs_in_the_inputs_memory(qk, n, column):
    """out_prices over one of the ten columns, out_source over option_type."""
    sur = HestonSurrogate(qk, seed=3)
    b, ot, kind = _quotes(n)
    want, src = sur.price_batch(**b, option_type=ot, fallback_paths=500, fallback_steps=8, fallback_seed=5)
    cols = [np.ascontiguousarray(b[k], np.float64) for k in ("spot", "strike", "t", "r", "q", "v0", "kappa",
                                                             "theta", "sigma", "rho")]
    pd, pi = ct.POINTER(ct.c_double), ct.POINTER(ct.c_int32)
    typ = ot.copy()
    rc = sur.lib.qk_sur_heston_price_batch(
        sur._h, *[c.ctypes.data_as(pd) for c in cols], typ.ctypes.data_as(pi), n, 500, 8, 5,
        cols[column].ctypes.data_as(pd), typ.ctypes.data_as(pi))
    assert rc == 0
    assert np.array_equal(cols[column], want, equal_nan=True)
    assert np.array_equal(typ, src)
    sur.close()

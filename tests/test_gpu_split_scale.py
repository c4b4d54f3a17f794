"""The FP16 pairs of the mixed factorisation's panel slices, scaled by one
power of two per tensor: the factor is FP32-class whatever the tensor's
magnitude, and rows whose diagonal is 10^6 below the largest keep their own
relative accuracy (a pair holds values down to 2^-34 of the largest row's).

Tolerance: the mixed factor's own bound (1e-5, FP32 class) per row, relative
to the row's largest entry sqrt(D_ii)."""
import copy

import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mag", [1e-12, 1.0, 1e12])
@pytest.mark.parametrize("spread", [1.0, 1e-6])
def test_factor_at_any_magnitude(mag, spread):
    from brownian_dynamics_cuda_gb300 import PREC_FP64, PREC_MIXED, Context
    fib, _ = load_golden("syn_4nuc_lh")
    f = copy.deepcopy(fib)
    f.scalars["a1"] *= mag
    f.scalars["a2"] *= mag
    # far from the others, so that only its own diagonal changes scale
    f.state["r_t"] = f.state["r_t"].copy()
    f.arrays["t_rad"] = f.arrays["t_rad"].copy()
    f.state["r_t"][21:24] = (0.0, 0.0, 1e9)
    f.arrays["t_rad"][7] /= spread
    L64 = Context(f, precision=PREC_FP64).cholesky()
    c = Context(f, precision=PREC_MIXED)
    Lm = c.cholesky()
    assert c.negative_pivots() == 0
    row = np.sqrt((L64 * L64).sum(1))            # sqrt(D_ii)
    assert (np.abs(Lm - L64).max(1) / row).max() <= 1e-5

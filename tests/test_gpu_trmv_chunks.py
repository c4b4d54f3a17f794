"""The noise displacement's partial sums go in runs of 32 columns up to 3N = 2,048,
of 128 up to 8,192, of 512 beyond: beside both lines it has to be s2dt L p with the
factor that the library itself returns.

Tolerances, against the product in NumPy with the same factor: FP64 sums 2 (m + 2)
u sum_k |L_ik p_k| s2dt, u = 2^-53; the mixed path's double-float sums keep 40 bits:
2^-40 of the same sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 3N -> linker beads of each nucleosome (tails of 5 beads)
SIZES = {2046: (17,) * 8 + (18,) * 2, 2049: (17,) * 7 + (18,) * 3, 8190: (17,) * 30 + (18,) * 10,
         8193: (17,) * 29 + (18,) * 11}


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("m", sorted(SIZES))
def test_displacement_is_factor_times_noise(m, mixed, tmp_path):
    from brownian_dynamics_cuda_gb300 import PREC_FP64, PREC_MIXED, Context
    from brownian_dynamics_cuda_gb300.fiber_gen import FiberSpec, linker_beads, make_fiber
    bp = [next(b for b in range(1, 400) if linker_beads(b) == w) for w in SIZES[m]]
    fib = make_fiber(FiberSpec(len(bp), bp, tail_len=5, seed=3), str(tmp_path))
    assert fib.m == m
    c = Context(fib, precision=PREC_MIXED if mixed else PREC_FP64)
    L = c.cholesky()
    p = np.random.default_rng(m).normal(size=m)
    s2dt = fib.scalars["s2dt"]
    bound = np.abs(L) @ np.abs(p) * s2dt
    err = np.abs(c.noise_displacement(p) - s2dt * (L @ p))
    assert np.all(err <= (2.0**-40 if mixed else 2 * (m + 2) * 2.0**-53) * bound)

"""The matrix-free Krylov product at the edges of its splits: bead counts n_D on and off
multiples of its 4 beads a block, one run of 1,024 beads a warp and the 4,096 of a
round, against FP64's product with the stored tensor.

Tolerance: both run to a relative change of 1e-9, so the difference is that of the
products: FP32 blocks (4e-7 of an entry) through D^{1/2}, 1e-5 of the largest
component at these condition numbers (the mixed path's noise class is 1e-6 a
product)."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

# n_D -> (linker beads per nucleosome, tail length)
SIZES = {13: ((2,), 1), 22: ((11,), 1), 1023: ((21,) * 7 + (22,) * 3, 8), 1024: ((21,) * 6 + (22,) * 4, 8),
         1025: ((21,) * 5 + (22,) * 5, 8), 4097: ((21,) * 23 + (22,) * 17, 8)}


@pytest.mark.parametrize("n_D", sorted(SIZES))
def test_matrix_free_product_edges(n_D, tmp_path):
    from brownian_dynamics_cuda_gb300 import PREC_FP64, PREC_MIXED, Context
    from brownian_dynamics_cuda_gb300.fiber_gen import FiberSpec, linker_beads, make_fiber
    beads, tail_len = SIZES[n_D]
    bp = [next(b for b in range(1, 400) if linker_beads(b) == w) for w in beads]
    fib = make_fiber(FiberSpec(len(beads), bp, tail_len=tail_len, seed=3), str(tmp_path))
    assert fib.m == 3 * n_D
    p = np.random.default_rng(n_D).normal(size=fib.m)
    out = []
    for prec in (PREC_FP64, PREC_MIXED):
        c = Context(fib, precision=prec)
        c.set_noise_mode(1, tol=1e-9, kmax=min(3 * n_D, 200))
        out.append(c.noise_displacement(p))
        if prec == PREC_MIXED:
            assert np.array_equal(c.noise_displacement(p), out[1])
    assert rel_err(out[1], out[0]) <= 1e-5

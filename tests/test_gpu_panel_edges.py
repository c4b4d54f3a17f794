"""The mixed factorisation at the edges of its 128-column panels: one panel or
less, exact multiples, and a last panel of a few rows (so that the chain of
diagonal blocks, their inverses and the tile products meet padded rows), up to
sizes with many tiles.

Tolerances are the mixed path's own: the factor 1e-5 and the noise
displacement 1e-6 (max norm, relative to the FP64 path's); a second
factorisation on the same buffers gives the same bits."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

# (linker beads per nucleosome, tail length) -> 3N
SIZES = {63: ((10,), 1), 126: ((11,), 3), 129: ((12,), 3), 384: ((13, 13), 5), 387: ((13, 14), 5), 513: ((6, 6, 6), 5),
         762: ((25, 27), 10), 1212: ((8,) * 7 + (20,), 4)}


def _fiber(beads, tail_len, path):
    from brownian_dynamics_cuda_gb300.fiber_gen import FiberSpec, linker_beads, make_fiber
    bp = [next(b for b in range(1, 400) if linker_beads(b) == w) for w in beads]
    return make_fiber(FiberSpec(len(beads), bp, tail_len=tail_len, seed=3), str(path))


@pytest.mark.parametrize("m", sorted(SIZES))
def test_factor_at_panel_edges(m, tmp_path):
    from brownian_dynamics_cuda_gb300 import PREC_FP64, PREC_MIXED, Context
    fib = _fiber(*SIZES[m], tmp_path)
    assert fib.m == m
    p = np.random.default_rng(m).normal(size=m)
    a, c = Context(fib, precision=PREC_FP64), Context(fib, precision=PREC_MIXED)
    L64 = a.cholesky()
    Lm = c.cholesky()
    assert c.negative_pivots() == 0
    assert np.all(np.triu(Lm, 1) == 0.0)
    assert rel_err(Lm, L64) <= 1e-5
    assert np.array_equal(c.cholesky(), Lm)
    assert rel_err(c.noise_displacement(p), a.noise_displacement(p)) <= 1e-6

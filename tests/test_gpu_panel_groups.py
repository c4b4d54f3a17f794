"""The mixed factorisation's groups of panels (four, six or six panels to a pass, by the
tile rows left) where their kind changes: sizes whose first group is of single
panels' sums, of pairs' (27 tile rows) and of triples' (44), and one tile row more
and less, with full and three-row last tile rows.

Tolerances are the mixed path's own: the factor 1e-5 and the noise displacement
1e-6 (max norm, relative to the FP64 path's), at every setting of
`set_mixed_passes`; a second factorisation on the same buffers gives the same
bits."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

# 3N -> linker beads of each nucleosome (tails of 5 beads, 10 a nucleosome)
SIZES = {3327: (18,) * 11 + (19,) * 5, 3456: (21,) * 16, 3459: (21,) * 15 + (22,),
         5502: (14,) * 14 + (15,) * 14, 5505: (14,) * 13 + (15,) * 15, 5763: (13,) * 29 + (14,)}


@pytest.mark.parametrize("m", sorted(SIZES))
def test_groups_match_fp64(m, tmp_path):
    from brownian_dynamics_cuda_gb300 import PREC_FP64, PREC_MIXED, Context
    from brownian_dynamics_cuda_gb300.fiber_gen import FiberSpec, linker_beads, make_fiber
    bp = [next(b for b in range(1, 400) if linker_beads(b) == w) for w in SIZES[m]]
    fib = make_fiber(FiberSpec(len(bp), bp, tail_len=5, seed=3), str(tmp_path))
    assert fib.m == m
    p = np.random.default_rng(m).normal(size=m)
    a, c = Context(fib, precision=PREC_FP64), Context(fib, precision=PREC_MIXED)
    L64, rd64 = a.cholesky(), a.noise_displacement(p)
    Lm = c.cholesky()
    assert c.negative_pivots() == 0
    assert rel_err(Lm, L64) <= 1e-5
    assert np.array_equal(c.cholesky(), Lm)
    for passes in (1, 2, 3):
        c.set_mixed_passes(passes)
        assert rel_err(c.noise_displacement(p), rd64) <= 1e-6

"""From 256 tile rows on the mixed factorisation updates the bulk with six panels at a
time, beside the next six panels; `set_mixed_passes(1 or 2)` takes the general path
(one or two panels a pass) over the same matrix.  At the first such size and one
tile row more, both with a last tile row of three rows, the displacements have to
agree within twice the mixed path's 1e-6 (max norm, each against FP64), and a
second factorisation on the same buffers has to give the same bits."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

# 3N -> linker beads of 140 nucleosomes (tails of 5 beads)
SIZES = {32643: (26,) * 39 + (27,) * 101, 32769: (27,) * 137 + (28,) * 3}


@pytest.mark.parametrize("m", sorted(SIZES))
def test_six_panel_groups_match_the_general_path(m, tmp_path):
    from brownian_dynamics_cuda_gb300 import PREC_MIXED, Context
    from brownian_dynamics_cuda_gb300.fiber_gen import FiberSpec, linker_beads, make_fiber
    bp = [next(b for b in range(1, 400) if linker_beads(b) == w) for w in SIZES[m]]
    fib = make_fiber(FiberSpec(len(bp), bp, tail_len=5, seed=3), str(tmp_path))
    assert fib.m == m
    p = np.random.default_rng(m).normal(size=m)
    c = Context(fib, precision=PREC_MIXED)
    wide = c.noise_displacement(p)
    assert c.negative_pivots() == 0
    assert np.array_equal(c.noise_displacement(p), wide)
    for passes in (2, 1):
        c.set_mixed_passes(passes)
        assert rel_err(c.noise_displacement(p), wide) <= 2e-6
    c.set_mixed_passes(3)
    assert np.array_equal(c.noise_displacement(p), wide)

"""FP64 path: the factorisation at the edges of its 32-column panels (64-column
blocks, 32-row tiles), and pair forces beside the cut-offs (7, 4 nm) and beside
the distance at which a pair is skipped by its FP32 distance (sqrt 50 nm).

Tolerances.  Factor: the backward error of Cholesky, |L L^T - D| <= (m + 1) u
max D, u = 2^-53, with as much again for NumPy's product and a factor 2 for the
pivots' reciprocal roots (2 ulp).  Forces: 1e-10 of the largest, the FP64 parity
class."""
import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu

# (linker beads per nucleosome, tail length) -> 3N
SIZES = {39: ((2,), 1), 63: ((10,), 1), 66: ((11,), 1), 96: ((21,), 1), 99: ((22,), 1), 129: ((12,), 3),
         387: ((13, 14), 5)}


@pytest.mark.parametrize("m", sorted(SIZES))
def test_fp64_factor_at_panel_edges(m, tmp_path):
    from brownian_dynamics_cuda_gb300 import PREC_FP64, Context
    from brownian_dynamics_cuda_gb300.fiber_gen import FiberSpec, linker_beads, make_fiber
    beads, tail_len = SIZES[m]
    bp = [next(b for b in range(1, 400) if linker_beads(b) == w) for w in beads]
    c = Context(make_fiber(FiberSpec(len(beads), bp, tail_len=tail_len, seed=3), str(tmp_path)), precision=PREC_FP64)
    assert c.m == m
    D = np.tril(c.diffusion_tensor())
    D = D + np.tril(D, -1).T
    L = c.cholesky()
    assert np.all(np.triu(L, 1) == 0.0) and c.negative_pivots() == 0
    assert np.abs(L @ L.T - D).max() <= 4 * (m + 1) * 2.0**-53 * np.abs(D).max()


@pytest.mark.parametrize("d", [7.0 - 4e-9, 7.0 + 4e-9, 4.0 - 4e-9, 4.0 + 4e-9, 50**0.5 - 1e-6, 50**0.5 + 1e-6])
@pytest.mark.parametrize("partner", ["tail", "linker", "lh"])
def test_fp64_pairs_beside_cutoffs_match_oracle(partner, d):
    from brownian_dynamics_cuda_gb300 import PREC_FP64, Context
    from oracle.pyoracle import Oracle
    fib, _ = load_golden("syn_4nuc_lh")
    rt = fib.state["r_t"].reshape(-1, 3).copy()
    grp = fib.arrays["t_grp"]
    if partner == "tail":
        p = rt[int(np.nonzero(grp != grp[0])[0][-1])]
    elif partner == "linker":
        p = fib.state["r"].reshape(-1, 3)[int(np.nonzero(fib.arrays["type"] == 0)[0][0])]
    else:
        p = fib.state["r_lh"].reshape(-1, 3)[0]
    rt[0] = p + np.array([0.0, d, 0.0])
    fib.state["r_t"] = rt.ravel()
    c, o = Context(fib, precision=PREC_FP64), Oracle(fib)
    got, ref = c.forces(), o.forces()
    for k in ("force", "torque", "t_force", "LH_force"):
        assert np.abs(got[k] - ref[k]).max() <= 1e-10 * np.abs(ref[k]).max(), k

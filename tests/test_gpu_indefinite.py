"""Mixed factors of indefinite tensors.  A bead with a negative radius makes
negative pivots; the reference replaces them by |f| (func.cpp:827-833), and the
factor may grow far past sqrt(max D_ii), which the FP16 slices' common scale is
chosen by.  Such a factor is as close to FP64's as any FP32 factor, or not
finite where FP32 cannot hold it: never finite and wrong.

Bounds: 1e-5 for a row relative to its 2-norm and for the displacement in the
2-norm, the mixed factor's own (FP32 class).  A NumPy model of FP32 arithmetic
with 24-bit slices gives at most 1.3e-6 and 5e-7 for these fibers; with slices
cut off at FP16's largest value it gives 3e-2 to 4e-1."""
import copy
import tempfile

import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


def _bad(fib, key, i, radius):
    f = copy.deepcopy(fib)
    f.arrays[key] = f.arrays[key].copy()
    f.arrays[key][i] = radius
    return f


def _ctx(f, mixed, passes=3):
    from brownian_dynamics_cuda_gb300 import PREC_FP64, PREC_MIXED, Context
    c = Context(f, precision=PREC_MIXED if mixed else PREC_FP64)
    if mixed:
        c.set_mixed_passes(passes)
    return c


# the bead in the first and in a middle tile, at the end, in a tile row's last columns
GROWN = [("syn_4nuc_lh", "rad", 2, -1.5), ("syn_4nuc_lh", "lh_rad", 9, -11.6),  # little growth, all rows fit
         ("syn_4nuc_lh", "lh_rad", 12, -12.0), ("syn_4nuc_lh", "lh_rad", 3, -300.0),
         ("syn_4nuc_lh", "lh_rad", 40, -300.0), ("syn_4nuc_lh", "lh_rad", -1, -300.0),
         ("syn_4nuc_lh", "lh_rad", 40, -1e4), ("syn_4nuc_lh", "t_rad", 2, -300.0),
         ("syn_4nuc_lh", "t_rad", -1, -300.0), ("cfg0_12nuc", "t_rad", -1, -300.0),
         ("cfg0_12nuc", "t_rad", -1, -1e4)]


@pytest.mark.parametrize("name,key,i,radius", GROWN)
def test_grown_factor_follows_fp64(name, key, i, radius):
    f = _bad(load_golden(name)[0], key, i, radius)
    c64, c = _ctx(f, False), _ctx(f, True)
    L64, L = c64.cholesky(), c.cholesky()
    assert c.negative_pivots() == c64.negative_pivots() > 0
    row = np.sqrt((L64 * L64).sum(1))
    assert (np.abs(L - L64).max(1) / row).max() <= 1e-5
    p = np.random.default_rng(0).standard_normal(f.m)
    rd64, rd = c64.noise_displacement(p), c.noise_displacement(p)
    assert np.linalg.norm(rd - rd64) <= 1e-5 * np.linalg.norm(rd64)


# 31, 43 and 90 tile rows: passes of one, two and three panels an accumulator, the
# grown rows among those of every panel before their own tile's
@pytest.mark.parametrize("passes", [1, 2, 3])
@pytest.mark.parametrize("nuc,lh,bad", [(24, False, [("t_rad", -1, -300.0)]),
                                        (24, True, [("lh_rad", 52, -1e4), ("lh_rad", 211, -300.0),
                                                    ("lh_rad", 369, -12.0), ("lh_rad", -1, -1e4)]),
                                        (50, True, [("lh_rad", -1, -300.0)])])
def test_grown_rows_in_every_schedule(nuc, lh, bad, passes):
    from brownian_dynamics_cuda_gb300.fiber_gen import FiberSpec, make_fiber
    with tempfile.TemporaryDirectory() as d:
        fib = make_fiber(FiberSpec(nuc, [30] * nuc, lh=lh, cs=0.15, seed=5), d)
    p = np.random.default_rng(0).standard_normal(fib.m)
    for key, i, radius in bad:
        f = _bad(fib, key, i, radius)
        c64, c = _ctx(f, False), _ctx(f, True, passes)
        rd64, rd = c64.noise_displacement(p), c.noise_displacement(p)
        assert c.negative_pivots() == c64.negative_pivots() > 0
        assert np.linalg.norm(rd - rd64) <= 1e-5 * np.linalg.norm(rd64)
        assert np.array_equal(rd, c.noise_displacement(p))  # the same bits again


def test_grown_replica_of_a_batch():
    from brownian_dynamics_cuda_gb300 import PREC_MIXED, Batch, Context, Noise
    good, _ = load_golden("syn_4nuc_lh")
    fibers = [good, _bad(good, "lh_rad", -1, -300.0), load_golden("cfg0_12nuc")[0]]
    nz = [Noise(7 + i).step(0, f.arrays["r_var"], f.m) for i, f in enumerate(fibers)]
    b = Batch(fibers, precision=PREC_MIXED)
    b.step([n[0] for n in nz], [n[1] for n in nz])
    for f, n, view in zip(fibers, nz, b.contexts):
        c = Context(f, precision=PREC_MIXED)
        c.step(*n)
        for k in ("r", "r_t", "r_lh", "rd"):
            assert np.array_equal(view.get(k), c.get(k)), k


@pytest.mark.parametrize("key,i,radius", [("rad", 11, -5.08), ("rad", 1, -5.74), ("t_rad", 54, -1.52),
                                          ("t_rad", 51, -8.1), ("lh_rad", 44, -4.92)])
def test_factor_past_fp32_is_not_finite(key, i, radius):
    from brownian_dynamics_cuda_gb300 import BDError, Context, PREC_MIXED
    fib, z = load_golden("syn_4nuc_lh")
    f = _bad(fib, key, i, radius)
    c = _ctx(f, True)
    assert not np.isfinite(c.cholesky()).all()
    assert not np.isfinite(c.noise_displacement(z["noise0_p"])).all()
    c = Context(f, precision=PREC_MIXED)
    c.step(z["noise0_rr"], z["noise0_p"])       # (its energy is that of the positions before the move)
    assert not all(np.isfinite(c.get(k)).all() for k in ("r", "r_t", "r_lh"))
    with pytest.raises(BDError) as ei:
        c.step(z["noise0_rr"], z["noise0_p"])
    assert ei.value.code == 5
    g = Context(fib, precision=PREC_MIXED)      # a context of its own is not touched
    g.step(z["noise0_rr"], z["noise0_p"])
    assert np.isfinite(g.get("r")).all()

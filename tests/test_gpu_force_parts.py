"""A force pass in parts beside each other against the same pass in one row, and
steps that keep their tensor and factor (frequency_RP > 1), where the first force
pass runs beside the noise displacement alone: bit for bit, as the kernels and
their operands are the same.  A replica of a batch runs its passes in one row;
so does a context whose phases are timed."""
import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["syn_4nuc_lh", "cfg0_12nuc"])
@pytest.mark.parametrize("mixed", [True, False])
def test_parts_equal_the_row(name, mixed):
    from brownian_dynamics_cuda_gb300 import PREC_FP64, PREC_MIXED, Batch, Context
    fib, z = load_golden(name)
    prec = PREC_MIXED if mixed else PREC_FP64
    b = Batch([fib], precision=prec)
    c = Context(fib, precision=prec)
    for _ in range(3):
        row, parts = b.contexts[0].forces(), c.forces()
        assert row.keys() == parts.keys()
        for k in row:
            assert np.array_equal(row[k], parts[k]), k
        b.step([z["noise0_rr"]], [z["noise0_p"]])
        c.step(z["noise0_rr"], z["noise0_p"])


@pytest.mark.parametrize("name", ["syn_4nuc_lh", "cfg0_12nuc"])
@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("freq", [2, 10])
def test_steps_without_a_factorisation(name, mixed, freq):
    from brownian_dynamics_cuda_gb300 import PREC_FP64, PREC_MIXED, Context, Noise
    fib, _ = load_golden(name)
    out = []
    for timed in (True, False):
        c = Context(fib, precision=PREC_MIXED if mixed else PREC_FP64, frequency_RP=freq)
        if timed:
            c.phase_times()  # from here on phases are timed, one after the other
        nz = Noise(11)
        e = [c.step(*nz.step(s, fib.arrays["r_var"], fib.m)) for s in range(5)]
        out.append((e, {k: np.array(c.get(k)) for k in ("r", "a", "b", "c", "r_t", "r_lh", "rd")}))
    assert out[0][0] == out[1][0]
    for k in out[0][1]:
        assert np.array_equal(out[0][1][k], out[1][1][k]), k

"""A step's first force pass runs on a side stream beside the factorisation, and a
force pass's independent parts beside each other: the same kernels in another
order.  A context whose phases are timed runs them one after the other, so its
state has to match bit for bit; so do contexts stepped from several threads at
once (each has its own side streams)."""
import threading

import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu
KEYS = ("r", "a", "b", "c", "r_t", "r_lh")


def _run(fib, precision, use_graph, timed, steps=4, krylov=False):
    from brownian_dynamics_cuda_gb300 import Context, Noise
    c = Context(fib, precision=precision, use_graph=use_graph)
    if krylov:
        c.set_noise_mode(1)
    if timed:
        c.phase_times()  # from here on phases are timed
    nz = Noise(11)
    for s in range(steps):
        c.step(*nz.step(s, fib.arrays["r_var"], fib.m))
    out = {k: np.array(c.get(k)) for k in KEYS}
    out.update({"f_" + k: np.array(v) for k, v in c.forces().items()})
    c.close()
    return out


@pytest.mark.parametrize("name", ["syn_4nuc_lh", "cfg0_12nuc"])
@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("mode", ["stream", "graph", "krylov", "threads"])
def test_overlapped_steps_equal_serial_ones(name, mixed, mode):
    from brownian_dynamics_cuda_gb300 import PREC_FP64, PREC_MIXED
    fib, _ = load_golden(name)
    prec = PREC_MIXED if mixed else PREC_FP64
    ref = _run(fib, prec, False, True, krylov=mode == "krylov")
    if mode == "threads":
        got = [None] * 3

        def work(k):
            got[k] = _run(fib, prec, k == 1, False)
        ts = [threading.Thread(target=work, args=(k,)) for k in range(3)]
        [t.start() for t in ts]
        [t.join() for t in ts]
    else:
        got = [_run(fib, prec, mode == "graph", False, krylov=mode == "krylov")]
    for g in got:
        for k in ref:
            assert np.array_equal(g[k], ref[k]), k

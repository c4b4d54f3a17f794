"""The core pairs' adjoint (a closed form) on fibers whose cores lie close: site
pairs on both sides of the Lennard-Jones cut-off at 8 nm and next to it, within
25 nm and past it.  FP64 adjoint against central differences of the FP64
rollout, with the bound of the other gradients (1e-6 of the largest component)."""
import tempfile

import numpy as np
import pytest

from test_gpu_adjoint import fd_grad, noise_rows, rel_vec

pytestmark = pytest.mark.gpu


def _sites(fib):
    s = {k: fib.state[k].reshape(-1, 3) for k in ("r", "a", "b", "c")}
    pos = fib.arrays["core_pos"].reshape(-1, 3)
    cores = np.nonzero(fib.arrays["type"] == 1)[0]
    return [s["r"][i] + pos @ np.stack([s["a"][i], s["b"][i], s["c"][i]]) for i in cores]


@pytest.mark.parametrize("nuc,bp,seed", [(2, 20, 5), (3, 20, 7), (4, 22, 11)])
def test_close_cores(nuc, bp, seed):
    from brownian_dynamics_cuda_gb300 import Context, PREC_FP64
    from brownian_dynamics_cuda_gb300.fiber_gen import FiberSpec, make_fiber
    fib = make_fiber(FiberSpec(nuc, [bp] * nuc, lh=False, seed=seed), tempfile.mkdtemp())
    x = _sites(fib)
    d = np.concatenate([np.linalg.norm(x[i][:, None] - x[j][None], axis=2).ravel()
                        for i in range(nuc) for j in range(i)])
    assert (d < 8).sum() > 100 and (d > 8).sum() > 100 and (np.abs(d - 8) < 0.05).sum() > 10
    rr, p = noise_rows(fib, 4, seed)
    loss_fd, g_fd = fd_grad(fib, rr, p, 2)
    loss, g = Context(fib, precision=PREC_FP64).adjoint(rr, p, window=2, checkpoint_every=2)
    assert abs(loss - loss_fd) <= 1e-12 * abs(loss_fd)
    assert rel_vec(g, g_fd) <= 1e-6, (g, g_fd)

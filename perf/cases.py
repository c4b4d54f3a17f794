"""The framework's work in performance cases: what a program of its user runs.

A simulation is a loop of Brownian-dynamics steps of one fiber (the host draws
the step's noise, the step runs on the GPU, the state is sampled), a batch of
replicas advanced together, or a gradient of a rollout; around it stand single
calls (the forces of a state, a noise displacement).  Sizes follow the
benchmark fibers of brownian_dynamics_cuda_gb300/fiber_gen.py: 12, 24, 50 and
200 nucleosomes, linkers of 20 to 60 bp, with and without linker histones, at
50, 100 or 150 mM salt; the smallest fiber is the 4-nucleosome one of the tests.

``prepare`` builds the fiber and the handle that a program keeps; ``run`` is
one pass through the public entry points and returns everything that the call
computes.  Fibers, charges and noise are made from the seed alone.
"""
import math
import tempfile

import numpy as np

from brownian_dynamics_cuda_gb300 import NOISE_KRYLOV, PREC_FP64, PREC_MIXED, Batch, Context, Noise
from brownian_dynamics_cuda_gb300.fiber_gen import FiberSpec, linker_beads, make_fiber

TAILS, LH_BEADS, SITES = 50, 22, 300  # per nucleosome: tail beads, mobile linker-histone beads, core charges
STATE = ("r", "a", "b", "c", "r_t", "r_lh")


def listed():
    return [
        # The smallest calls: a four-nucleosome fiber with linker histones, where launches and latency count.
        dict(name="step_mixed_4nuc_lh", kind="step", precision="mixed", nuc=4, bp_lo=30, bp_hi=30, lh=True, cs=0.15),
        # The ordinary simulations in mixed precision: the 12-, 24- and 50-nucleosome benchmark fibers.
        dict(name="step_mixed_12nuc", kind="step", precision="mixed", nuc=12, bp_lo=26, bp_hi=26, lh=False, cs=0.15),
        dict(name="step_mixed_24nuc", kind="step", precision="mixed", nuc=24, bp_lo=30, bp_hi=30, lh=False, cs=0.15),
        dict(name="step_mixed_50nuc_lh", kind="step", precision="mixed", nuc=50, bp_lo=44, bp_hi=44, lh=True, cs=0.15),
        # The largest fiber: 200 nucleosomes, alternating linkers, 3N = 46,200.
        dict(name="step_mixed_200nuc_lh", kind="step", precision="mixed", nuc=200, bp_lo=26, bp_hi=44,
             alternate=True, lh=True, cs=0.15),
        # An ensemble of uneven replicas, one call a step, the noise drawn on the device.
        dict(name="batch_mixed_24rep", kind="batch", replicas=24, nuc_lo=12, nuc_hi=48, bp_lo=20, bp_hi=60),
        # The same dynamics with the Lanczos noise in place of the factorisation.
        dict(name="krylov_mixed_50nuc_lh", kind="krylov", nuc=50, bp_lo=44, bp_hi=44, lh=True, cs=0.15),
        # The FP64 parity path, small and at the 50-nucleosome size.
        dict(name="step_fp64_12nuc", kind="step", precision="fp64", nuc=12, bp_lo=26, bp_hi=26, lh=False, cs=0.15),
        dict(name="step_fp64_50nuc_lh", kind="step", precision="fp64", nuc=50, bp_lo=44, bp_hi=44, lh=True, cs=0.15),
        # Single FP64 calls of an analysis: the forces of a state, and a noise displacement sqrt(2 dt) L p.
        dict(name="forces_fp64_50nuc_lh", kind="forces", nuc=50, bp_lo=44, bp_hi=44, lh=True, cs=0.15),
        dict(name="noise_fp64_24nuc", kind="noise", nuc=24, bp_lo=30, bp_hi=30, lh=False, cs=0.15),
        # A parameter fit's backward pass: the gradient of a short FP64 rollout.
        dict(name="gradient_fp64_6nuc", kind="gradient", nuc=6, bp_lo=26, bp_hi=30, cs=0.15, steps=8, window=4,
             checkpoint=4),
    ]


def draw(rng):
    def log_int(lo, hi):
        return min(hi, int(lo * math.exp(rng.random() * math.log((hi + 1) / lo))))

    bp = sorted((rng.randint(20, 60), rng.randint(20, 60)))
    common = dict(bp_lo=bp[0], bp_hi=bp[1], alternate=rng.random() < 0.25, cs=rng.choice([0.05, 0.10, 0.15]))
    kind = rng.choice(["mixed"] * 5 + ["fp64"] * 2 + ["batch", "krylov", "forces", "noise", "gradient"])
    if kind == "mixed":
        return dict(common, kind="step", precision="mixed", nuc=log_int(4, 190), lh=rng.random() < 0.5)
    if kind == "fp64":
        return dict(common, kind="step", precision="fp64", nuc=log_int(4, 46), lh=rng.random() < 0.5)
    if kind == "batch":
        lo = rng.randint(8, 16)
        return dict(kind="batch", replicas=log_int(3, 24), nuc_lo=lo, nuc_hi=rng.randint(lo + 4, 48), bp_lo=bp[0],
                    bp_hi=bp[1])
    if kind == "krylov":
        return dict(common, kind="krylov", nuc=log_int(12, 100), lh=rng.random() < 0.5)
    if kind == "forces":
        return dict(common, kind="forces", nuc=log_int(4, 100), lh=rng.random() < 0.5)
    if kind == "noise":
        return dict(common, kind="noise", nuc=log_int(4, 40), lh=rng.random() < 0.5)
    return dict(common, kind="gradient", nuc=rng.randint(3, 7), steps=rng.randint(4, 8), window=rng.randint(1, 4),
                checkpoint=rng.randint(1, 8))


def _linkers(case, nuc, rng):
    """Linker lengths: the case's own, so that every seed gives arrays of the same sizes."""
    lo, hi = case["bp_lo"], case["bp_hi"]
    if case.get("alternate", False):
        return [lo if k % 2 == 0 else hi for k in range(nuc)]
    return [int(b) for b in rng.integers(lo, hi + 1, size=nuc)]


def _fiber(nuc, linkers, lh, cs, seed):
    """The seeded fiber; a seed whose random geometry clashes gives way to the next."""
    for k in range(20):
        spec = FiberSpec(nuc, linkers, lh=lh, cs=cs, seed=seed + 7919 * k, lh_charge_range=(0.0, 1.0) if lh else None)
        with tempfile.TemporaryDirectory() as d:
            try:
                return make_fiber(spec, d)
            except RuntimeError:
                continue
    raise RuntimeError("no geometry without clashes")


def _one(case, seed):
    rng = np.random.default_rng([case["nuc"], case["bp_lo"], case["bp_hi"]])
    return _fiber(case["nuc"], _linkers(case, case["nuc"], rng), case.get("lh", False), case["cs"], seed % 1_000_003)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        rng = np.random.default_rng([case["replicas"], case["nuc_lo"], case["nuc_hi"], case["bp_lo"], case["bp_hi"]])
        fibers = []
        for i in range(case["replicas"]):
            nuc = int(rng.integers(case["nuc_lo"], case["nuc_hi"] + 1))
            cs = float(rng.choice([0.05, 0.10, 0.15]))
            fibers.append(_fiber(nuc, _linkers(case, nuc, rng), False, cs, seed % 1_000_003 + i))
        return dict(kind=kind, batch=Batch(fibers, precision=PREC_MIXED, use_graph=True), seed=seed % 1_000_000)
    fib = _one(case, seed)
    state = dict(kind=kind, fiber=fib, noise=Noise(seed % 1_000_000), at=0)
    if kind in ("step", "krylov"):
        mixed = kind == "krylov" or case["precision"] == "mixed"
        state["ctx"] = Context(fib, precision=PREC_MIXED if mixed else PREC_FP64, use_graph=True)
        if kind == "krylov":
            state["ctx"].set_noise_mode(NOISE_KRYLOV, 1e-6, 128)
        state["out"] = {k: np.zeros(v.size) for k, v in fib.state.items()}
        return state
    state["ctx"] = Context(fib, precision=PREC_FP64)
    if kind == "noise":
        state["p"] = np.random.default_rng(seed).standard_normal(fib.m)
    elif kind == "gradient":
        rows = [state["noise"].step(s, fib.arrays["r_var"], fib.m) for s in range(case["steps"])]
        state["rr"], state["p"] = (np.array([r[k] for r in rows]) for k in (0, 1))
        state["window"], state["checkpoint"] = case["window"], case["checkpoint"]
    return state


def run(s):
    kind = s["kind"]
    if kind == "batch":
        b = s["batch"]
        energies = b.run_device(1, s["seed"])  # the generators go on from call to call
        return dict(energy=energies, **{k: np.concatenate([c.get(k) for c in b.contexts]) for k in STATE[:5]})
    if kind in ("step", "krylov"):
        # one pass of the main loop: the host draws the noise, the step runs, the state is sampled
        rr, p = s["noise"].step(s["at"], s["fiber"].arrays["r_var"], s["ctx"].m)
        e = s["ctx"].step_reference(s["at"], 1 << 30, 1, rr, p, s["out"])
        s["at"] += 1
        return dict(energy=e, **{k: v.copy() for k, v in s["out"].items() if v.size})
    if kind == "forces":
        return {k: v for k, v in s["ctx"].forces().items() if np.size(v)}
    if kind == "noise":
        return s["ctx"].noise_displacement(s["p"])
    loss, grad = s["ctx"].adjoint(s["rr"], s["p"], s["window"], s["checkpoint"])
    return dict(loss=loss, gradient=grad)


# ---------------------------------------------------------------- work
def _sizes(case, nuc):
    mean = 0.5 * (linker_beads(case["bp_lo"]) + linker_beads(case["bp_hi"]))
    n = nuc * (1 + mean)
    return n, n + nuc * (TAILS + (LH_BEADS if case.get("lh", False) else 0))


def _force_flops(nuc, n, nD):
    """One force pass: every core sees about four other cores' charges, its linkers' beads and, per bead, the ~200
    beads within the cut-off; about 20 operations a pair."""
    return 20.0 * (2 * nuc * SITES * SITES + 8 * n * SITES + 100 * nD)


def _step_work(case, nuc, word, factor):
    n, nD = _sizes(case, nuc)
    m = 3 * nD
    # state and noise in, state out; the lower factor does not fit on the chip beside the rest: written and read once
    by = 8 * (2 * (9 * n + m) + 3 * n + m) + (word * m * m if factor else 0)
    fl = 2 * _force_flops(nuc, n, nD) + (m ** 3 / 3 + m * m if factor else 30 * 25.0 * nD * nD) + 2 * 25.0 * nD * nD / 2
    return by, fl


def work(case):
    kind = case["kind"]
    if kind == "batch":
        by = fl = 0.0
        R, lo, hi = case["replicas"], case["nuc_lo"], case["nuc_hi"]
        for i in range(R):  # the replicas' sizes, evenly spread
            x, y = _step_work(case, lo + (hi - lo) * (i + 0.5) / R, 4, True)
            by, fl = by + x, fl + y
        return {"bytes": by, "flops": fl}
    nuc = case["nuc"]
    n, nD = _sizes(case, nuc)
    m = 3 * nD
    if kind == "forces":
        return {"bytes": 8.0 * (2 * 12 * n + 2 * 3 * (nD - n)), "flops": _force_flops(nuc, n, nD)}
    if kind == "noise":
        return {"bytes": 8.0 * (m * m + 3 * m), "flops": m ** 3 / 3 + m * m + 25.0 * nD * nD / 2}
    if kind == "gradient":  # each step forward (twice, from its checkpoint) and back (two to three times its work)
        by, fl = _step_work(case, nuc, 8, True)
        return {"bytes": 3 * case["steps"] * by, "flops": 4 * case["steps"] * fl}
    by, fl = _step_work(case, nuc, 8 if case.get("precision") == "fp64" else 4, kind == "step")
    return {"bytes": float(by), "flops": float(fl)}


# --------------------------------------------------------------- exact
def _rpy(r, rad, a1, a2):
    """The Rotne-Prager-Yamakawa tensor of beads r [N, 3] with radii rad."""
    N = len(rad)
    d = r[:, None] - r[None]
    s2 = (d * d).sum(-1)
    s2[np.diag_indices(N)] = 1.0
    s = np.sqrt(s2)
    far = s >= rad[:, None] + rad[None]
    f = (rad[:, None] ** 2 + rad[None] ** 2) / s2
    se = np.cbrt((rad[:, None] ** 3 + rad[None] ** 3) / 2)
    iso = np.where(far, a2 / s * (1 + f / 3), a1 / se * (1 - 9 * s / (32 * se)))
    dyad = np.where(far, a2 / s * (1 - f) / s2, 3 * a1 / (32 * se * se * s))
    iso[np.diag_indices(N)] = a1 / rad
    dyad[np.diag_indices(N)] = 0.0
    D = dyad[:, None, :, None] * d.transpose(0, 2, 1)[:, :, :, None] * d[:, None]
    D += iso[:, None, :, None] * np.eye(3)[None, :, None, :]
    return D


def exact(case, seed):
    """sqrt(2 dt) L p from the model's definition; the other cases' outputs follow from the whole force field."""
    if case["kind"] != "noise":
        return None
    import torch
    fib = _one(case, seed)
    r = np.concatenate([fib.state[k].reshape(-1, 3) for k in ("r", "r_t", "r_lh")])
    rad = np.concatenate([fib.arrays[k] for k in ("rad", "t_rad", "lh_rad")])
    N = len(rad)
    D = _rpy(r, rad, fib.scalars["a1"], fib.scalars["a2"]).reshape(N, 3, N, 3).reshape(3 * N, 3 * N)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    L = torch.linalg.cholesky(torch.from_numpy(D).to(dev))
    p = torch.from_numpy(np.random.default_rng(seed).standard_normal(3 * N)).to(dev)
    return (fib.scalars["s2dt"] * (L @ p)).cpu().numpy()

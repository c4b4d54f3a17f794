"""Device memory of a context, on the CPU (fake_cudart.c logs the allocations):
the slots of the core pairs' partial sums are the precision's own - 15 a pair in
FP64, 4 mixed - and otherwise both precisions' arenas are alike."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

PROBE = r"""
import ctypes, sys
sys.path[:0] = [%r, %r]
from conftest import load_golden
from brownian_dynamics_cuda_gb300 import Context, PREC_FP64, PREC_MIXED
fake = ctypes.CDLL(%r)
fake.fake_fail.argtypes = [ctypes.c_char, ctypes.c_int]
fib, _ = load_golden(sys.argv[1])
arena = []
for prec in (PREC_FP64, PREC_MIXED):
    fake.fake_fail(b"R", -1)
    c = Context(fib, precision=prec)
    ops, st = ctypes.create_string_buffer(1 << 16), (ctypes.c_long * (1 << 16))()
    n = fake.fake_log(ops, st, 1 << 16)
    arena.append(next(st[i] for i in range(n) if ops.raw[i:i + 1] == b"M"))
print(c.n_c, *arena)
"""


@pytest.mark.parametrize("name", ["syn_4nuc_lh", "cfg0_12nuc"])
def test_core_pair_slots_by_precision(tmp_path, name):
    so = str(tmp_path / "fake_cudart.so")
    subprocess.run(["gcc", "-O1", "-w", "-shared", "-fPIC", os.path.join(ROOT, "tests", "fake_cudart.c"), "-o", so],
                   check=True)
    p = subprocess.run([sys.executable, "-c", PROBE % (ROOT, os.path.join(ROOT, "tests"), so), name],
                       env=dict(os.environ, LD_PRELOAD=so), capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout + p.stderr
    nc, fp64, mixed = map(int, p.stdout.split())
    slots = [(k * nc * nc * 10 * 8 + 255) // 256 * 256 for k in (15, 4)]
    assert fp64 - mixed == slots[0] - slots[1]

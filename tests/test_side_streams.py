"""A step's and a force pass's forks and joins, on the CPU: the library runs
against a runtime that logs its calls (fake_cudart.c), and each event call is
made to fail in turn.  Work on a side stream that is not joined would run
beside whatever comes next, so after the failure nothing is launched, both
side streams are waited for, the call reports it, and the next call is as if
it had not happened."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

PROBE = r"""
import ctypes, sys
sys.path[:0] = [%r, %r]
from conftest import load_golden
import numpy as np
from brownian_dynamics_cuda_gb300 import BDError, Context, PREC_FP64, PREC_MIXED
fake = ctypes.CDLL(%r)
fake.fake_fail.argtypes = [ctypes.c_char, ctypes.c_int]

def log():
    ops, st = ctypes.create_string_buffer(1 << 16), (ctypes.c_long * (1 << 16))()
    n = fake.fake_log(ops, st, 1 << 16)
    return [(ops.raw[i:i + 1].decode(), st[i]) for i in range(n)]

name, mixed, call = sys.argv[1], sys.argv[2] == "mixed", sys.argv[3]
fib, z = load_golden(name)
c = Context(fib, precision=PREC_MIXED if mixed else PREC_FP64)
run = c.forces if call == "forces" else (lambda: c.step(z["noise0_rr"], z["noise0_p"]))
fake.fake_fail(b"R", -1)
run()
whole = log()
side = {s for op, s in whole if op == "L"} - {next(s for op, s in whole if op == "S")}
assert len(side) == 2 and not any(op == "F" for op, _ in whole)
tried = 0
for op in "RW":
    for nth in range(sum(o == op for o, _ in whole)):
        fake.fake_fail(op.encode(), nth)
        try:
            run()
            raise SystemExit("%%s %%d: no error reported" %% (op, nth))
        except BDError as e:
            assert e.code == 3, e.code
        seen = log()
        at = [o for o, _ in seen].index("F")
        after = seen[at + 1:]
        assert not [s for o, s in after if o == "L"], (op, nth, "launches after the failure")
        busy = {s for o, s in seen[:at] if o == "L"} & side
        assert busy <= {s for o, s in after if o == "S"}, (op, nth, "a side stream left running")
        fake.fake_fail(b"R", -1)
        run()
        assert log() == whole, (op, nth, "the next call")
        tried += 1
print("tried", tried)
"""


@pytest.mark.parametrize("call", ["forces", "step"])
@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("name", ["syn_4nuc_lh", "cfg0_12nuc"])
def test_failed_fork_or_join(tmp_path, name, prec, call):
    so = str(tmp_path / "fake_cudart.so")
    src = os.path.join(ROOT, "tests", "fake_cudart.c")
    subprocess.run(["gcc", "-O1", "-w", "-shared", "-fPIC", src, "-o", so], check=True)
    env = dict(os.environ, LD_PRELOAD=so)
    p = subprocess.run([sys.executable, "-c", PROBE % (ROOT, os.path.join(ROOT, "tests"), so), name, prec, call],
                       env=env, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout + p.stderr
    assert int(p.stdout.split()[-1]) >= 8

"""Passes of gate runs around 48 KB of shared memory, launched first in a process: the kernel's static block counts
towards the limit above which the launch has to ask.  Layers of H + T with a CNOT ladder every fourth make FP32
passes of 47-48 KB on 20 to 23 qubits (14 layers: 49088 bytes); the layer counts around them go below and above."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import sys
sys.path.insert(0, %(root)r)
import numpy as np
import __graft_entry__
qi = __graft_entry__.load_package()
from quant_iron_gb300.workloads import GateList
n, gl = %(n)d, GateList()
for layer in range(%(layers)d):
    for q in range(n):
        gl.add("H", [q]).add("T", [q])
    if layer %% 4 == 3:
        for q in range(n - 1):
            gl.add("CNOT", [q + 1], [q])
gates = gl.array()
with qi.DeviceState(n, qi.F32) as a, qi.DeviceState(n, qi.F64) as b:
    a.set_zero()
    b.set_zero()
    qi.Plan(n, qi.F32, gates).execute(a)
    for g in gates:
        b.apply_gate(g)
    # a gate rounds each amplitude by a few 2^-24 of the state's norm
    assert a.compare(b)["max_abs_err"] <= 8 * len(gates) * 2.0 ** -24
print("same state")
"""


@pytest.mark.parametrize("n,layers", [(20, 14), (20, 13), (20, 15), (23, 14)])
def test_first_launch_of_a_process(n, layers):
    import __graft_entry__
    r = subprocess.run([sys.executable, "-c", PROGRAM % {"root": __graft_entry__.ROOT, "n": n, "layers": layers}],
                       stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0 and "same state" in r.stdout, r.stdout[-2000:]

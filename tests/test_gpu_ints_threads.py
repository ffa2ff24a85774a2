"""First calls of corr_ri_integrals in several threads at once, in a process of their
own (the Boys table is built and uploaded by the first of them)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import threading
import numpy as np
import corr_gb300

S = np.load("tests/golden/systems.npz")
names = ("l", "nprim", "poff", "center", "exps", "coefs")
obs, aux = (corr_gb300.Basis(*(S[f"c1_{k}_{n}"] for n in names)) for k in ("obs", "aux"))
contexts = [corr_gb300.Context(0) for _ in range(6)]
gate = threading.Barrier(len(contexts))
first = [None] * len(contexts)

def work(k):
    gate.wait()
    first[k] = contexts[k].ri_integrals(obs, aux, device="cpu")

threads = [threading.Thread(target=work, args=(k,)) for k in range(len(contexts))]
for t in threads:
    t.start()
for t in threads:
    t.join()
J, P = contexts[0].ri_integrals(obs, aux, device="cpu")
assert all(np.array_equal(a, J) and np.array_equal(b, P) for a, b in first)
"""


def test_first_calls():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=root, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]

"""Entry points that take their scratch from the library's own pool, as the first
call of a process under a stream capture: the graph's replays give the bits of the
calls run at once.  Each case in a process of its own, so that the pool is new."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEAD = """
import numpy as np, torch
from lacmopy_gb300 import _lib
from lacmopy_gb300.device import _ptr, _stream
lib = _lib.load()
"""
# 600 SIPs: more pairs than one CTA screens itself
BOX = """
rng = np.random.default_rng(1)
s0 = [torch.tensor(rng.uniform(1e3, 1e5, 600), device="cuda"),
      torch.tensor(10 ** rng.uniform(0, 6, 600), device="cuda"),
      torch.zeros(2, dtype=torch.int64, device="cuda")]
def calls(s):
    for q in range(3):
        _lib.check(lib.lacmo_collision_step_golovin(_ptr(s[0]), _ptr(s[1]), 600, 100.0,
                                                    _ptr(s[2]), None, 7, q, _stream()), "golovin")
"""
ADJOINT = """
from lacmopy_gb300 import adjoint, synthetic
st = synthetic.make_icmw_state(Nx=4, Nz=6, no_spcm=(3, 4), seed=6, kernel_type="Long_Bott")
# one SIP a cell: a cell's sum has one term, in no order
first = np.unique(st["cells"][0].astype(np.int64) * 6 + st["cells"][1], return_index=True)[1]
st["xi"][np.setdiff1d(np.arange(st["xi"].size), first)] = 0.0
model = adjoint.StepModel(st, 1, collisions=False)
s0 = model.initial_state()
def calls(s):
    m_w, m_s, xi, Th, rv = s
    model._sub_steps(m_w, m_s, Th, rv, 0.6, model.cells[0], model.n, 2, None, 3)
"""
TAIL = """
a, b = [t.clone() for t in s0], [t.clone() for t in s0]
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    calls(b)
calls(a)
assert not torch.equal(a[0], s0[0])
for replay in range(2):
    for t, u in zip(b, s0):
        t.copy_(u)
    g.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(a, b))
"""


@pytest.mark.parametrize("calls", [BOX, ADJOINT], ids=["box", "adjoint"])
def test_first_call_under_capture(calls):
    r = subprocess.run([sys.executable, "-c", HEAD + calls + TAIL], cwd=ROOT, timeout=300,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]

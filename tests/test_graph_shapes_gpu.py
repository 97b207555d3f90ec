"""CUDA-graph replay of the matvec at shapes beyond the one-launch product, which records no graph: real and complex, D = 3 and 9,
plans with a cluster split and with a tail split, an eigensolve, and sweeps that rebind the shape.  A child process runs them with
the graph path's step trace on: its lines on stderr show that graphs were replayed and not given up."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import sys
import torch
import dmrg_b200 as hb
from oracle import physics as ph

mark = lambda s: (sys.stderr.write("MARK " + s + "\n"), sys.stderr.flush())
st = torch.cuda.Stream()
for chi, chiR, D, c in [(130, 128, 3, False), (200, 150, 3, False), (313, 569, 3, False), (72, 70, 9, True), (130, 128, 9, True)]:
    mark(f"{chi}x{chiR}")
    th, W, L, R = ph.heff_inputs(chi, D=D, cplx=c, seed=chi + D, chiR=chiR)
    opg, opp = (hb.MatVecMPOS([W], L, R, cplx=c, stream=st) for _ in range(2))
    opg.set_graphs(True)
    opp.set_graphs(False)
    dt = torch.complex128 if c else torch.float64
    xs = [torch.randn(th.size, dtype=dt, device="cuda") for _ in range(3)]
    yg = [torch.full((th.size,), float("nan"), dtype=dt, device="cuda") for _ in xs]
    yp = [torch.empty(th.size, dtype=dt, device="cuda") for _ in xs]
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        for k in range(3):  # the first product records, the next two replay
            opg.MultAx(xs[k], yg[k])
            opp.MultAx(xs[k], yp[k])
    st.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(yg, yp)), (chi, chiR)
    opg.close()
    opp.close()
mark("eigs")
th, W, L, R = ph.heff_inputs(130, D=3, cplx=False, seed=9, chiR=128)
out = []
for g in (True, False):
    op = hb.MatVecMPOS([W], L, R, stream=st)
    op.set_graphs(g)
    with torch.cuda.stream(st):
        e, r = op.eigs(x0=hb.to_device(th), tol=1e-10, mixed=False)
    st.synchronize()
    out.append((e, r["num_mv"]))
    op.close()
assert out[0] == out[1], out
mark("sweep")
h = ph.random_fields(11, 16)
a = hb.fdmrg(h, chi_max=128, sweeps=5, trunc_lim=1e-20, stream=st)
mark("end")
b = hb.fdmrg(h, chi_max=128, sweeps=5, trunc_lim=1e-20)
assert a["energy"] == b["energy"]
"""


def test_replay_beyond_the_fused_rule(cuda):
    env = dict(os.environ, HEFF_GRAPHS="1", HEFF_GRAPHS_TRACE="1")
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=os.path.join(os.path.dirname(__file__), ".."), env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    parts = {s.split("\n", 1)[0]: s.count("replay: launch") for s in r.stderr.split("MARK ")[1:]}
    for name in ("130x128", "200x150", "313x569", "72x70"):
        assert parts[name] >= 2, parts
    assert parts["eigs"] > 0 and parts["sweep"] > 0, parts

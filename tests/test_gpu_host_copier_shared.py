"""The threads and the pinned ring of large results: one set per device however many
contexts there are, none for a program's first 32 MB, gone with the last context; and
the same bits before and after they are made, and while another call holds them.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
import os, threading
import numpy as np
from atlas12_b200 import _lib, atlas, operators, surrogate, synthetic
from atlas12_b200._lib import ptr

tasks = lambda: len(os.listdir("/proc/self/task"))
m = surrogate.grey_model(9000.0, 4.0, nrhox=56, ross=surrogate.RossTable(nt=48, np_=48, nwave=300))
e = surrogate.eos(m["t"], m["p"])
ws, _ = synthetic.geometric_waveset(9.0, 160000.0, 8000)
vec = [np.ascontiguousarray(v) for v in (m["t"], e["xne"], e["rho"], e["nh"] * (1 - e["xh"]) / 2, e["nh"] * e["xh"])]

def make():
    ctx = _lib.Context(0, _lib.PREC_FP64)
    A = atlas.Atlas(ctx, operators.load())
    A.set_kapp_tables(operators.load())
    return ctx, A

def run(ctx):  # 13.8 MB of results
    out = [np.full((8000, 72), 7.0) for _ in range(3)]
    ctx.call("atlasgpu_atlas_kapp_hydrogen", 8000, ptr(ws), 56, 72, *[ptr(v) for v in vec], None, None,
             *[ptr(o) for o in out], None)
    return np.stack(out)

ctxs = [make() for _ in range(4)]
none = tasks()
first = run(ctxs[0][0])
assert tasks() == none, "threads made for one call"
for k in range(3):
    for c, _ in ctxs:
        assert np.array_equal(run(c), first)
one = tasks() - none
assert 1 <= one <= 7, one
got = [[], [], [], []]
def work(i):
    for _ in range(4):
        got[i].append(np.array_equal(run(ctxs[i][0]), first))
th = [threading.Thread(target=work, args=(i,)) for i in range(4)]
for t in th: t.start()
for t in th: t.join()
assert got == [[True] * 4] * 4
assert tasks() - none == one, (tasks(), none, one)
for c, _ in ctxs[1:]:
    c.close()
assert tasks() - none == one
assert np.array_equal(run(ctxs[0][0]), first)
ctxs[0][0].close()
assert tasks() == none, (tasks(), none)
c, A = make()
assert np.array_equal(run(c), first) and tasks() == none
c.close()
print("done", one)
"""


def test_one_set_of_threads():
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, env=dict(os.environ, PYTHONPATH=ROOT),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, r.stdout + r.stderr[-3000:]

"""The kernels that walk fields by pointers, in the bounds-checked and NaN-poisoned build
(MPDX_LIBRARY=debug, a separate process): staged step, several 1D steps per launch,
Boussinesq step with its one-launch pressure solve, refilled advector halos, field views;
and the fused kernels, for the NaN.  They finish without an access outside a field and without NaN, and equal the oracle."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = r"""
import ctypes, json, sys
sys.path.insert(0, ROOT); sys.path.insert(0, ROOT + "/tests"); sys.path.insert(0, ROOT + "/oracle")
import numpy as np
from libmpdataxx_b200 import _lib
from libmpdataxx_b200 import opts as o
from oracle import Oracle
from runners import load, bq_run, bq_oracle
from test_gpu_edges import NO_DIV, random_problem
from test_gpu_fused import periodic_setup
from test_gpu_parity import make_run
from test_gpu_boussinesq import random_bq

assert _lib.SO_PATH.endswith("libmpdx_debug.so"), _lib.SO_PATH
C, O, R = "cyclic", "open", "rigid"
out = []
def rel(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))
"""

SCRIPT = HEAD + r"""
cases = [((9, 13), [C, C, O, O], o.iga | o.fct, 3, 1, "general"), ((11, 12), [O, R, R, O], o.tot | o.fct, 3, 6, "general"),
         ((8, 9, 7), [C, C, O, O, R, R], o.iga | o.tot | o.fct, 2, 1, "general"), ((9, 7, 8), [R, O, C, C, O, O], o.fct, 3, 2, "general"),
         ((6, 21, 69), [O] * 6, 0, 3, 1, "general"), ((37,), [O, O], o.tot | o.fct, 3, 1, "general"),
         ((300,), [O, O], o.fct, 3, 2, "auto"), ((23, 110, 120), [O, O, R, R, C, C], o.iga | o.fct, 2, 1, "general")]
for grid, bcs, opts, iters, n_eqns, path in cases:
    s = random_problem(grid, seed=sum(grid), n_eqns=n_eqns)
    run = make_run(grid, opts, n_iters=iters, n_eqns=n_eqns, bcs=bcs, max_abs_div_eps=NO_DIV, path=path)
    orc = Oracle(grid, opts, n_iters=iters, n_eqns=n_eqns, bcs=bcs, max_abs_div_eps=NO_DIV)
    load(run, s)
    load(orc, s)
    run.advance(2)
    orc.advance(2)
    got = [np.array(run.advectee(e)) for e in range(n_eqns)]
    out.append([str(grid), run.stats()["kernels"], all(bool(np.isfinite(a).all()) for a in got),
                max(rel(a, orc.advectee(e)) for e, a in enumerate(got))])
# periodic: staged on the automatic path, a second advector; 1D steps in registers
for grid, opts, iters in [((24, 22, 41), o.iga | o.fct, 2), ((40, 51), o.fct, 3)]:
    run = None
    for k in range(2):
        s = periodic_setup(grid, seed=k + 1)
        if run is None:
            run = make_run(grid, opts, n_iters=iters, max_abs_div_eps=1e-6, path="auto")
        load(run, s)
        run.advance(2)
        orc = Oracle(grid, opts, n_iters=iters, max_abs_div_eps=1e-6)
        load(orc, s)
        orc.advance(2)
        got = np.array(run.advectee())
        out.append([str(grid) + str(k), run.stats()["kernels"], bool(np.isfinite(got).all()), rel(got, orc.advectee())])
# the fused kernels by name, and the one-block 1D steps: nothing that was not written is read
for grid, opts, iters in [((24, 22, 41), o.iga | o.fct, 2), ((24, 22, 41), o.fct, 2), ((23, 19), o.iga | o.fct, 2), ((40, 51), o.fct, 3)]:
    s = periodic_setup(grid, seed=5)
    run, orc = make_run(grid, opts, n_iters=iters, max_abs_div_eps=1e-6, path="fused"), Oracle(grid, opts, n_iters=iters, max_abs_div_eps=1e-6)
    for r in (run, orc):
        load(r, s)
        r.advance(3)
    got = np.array(run.advectee())
    out.append(["fused " + str(grid), run.stats()["kernels"], bool(np.isfinite(got).all()), rel(got, orc.advectee())])
for opts in (0, o.iga | o.fct, o.abs):
    run, orc = make_run((40,), opts, path="auto"), Oracle((40,), opts)
    psi = np.random.default_rng(1).uniform(0.5, 2.0, 40)
    psi[-1] = psi[0]
    for r in (run, orc):
        r.set_advectee(psi, 0)
        r.set_advector(np.full(40, 0.4), 0)
        r.advance(30)
    got = np.array(run.advectee())
    out.append(["40 " + str(opts), run.stats()["kernels"], bool(np.isfinite(got).all()), rel(got, orc.advectee(0))])
for grid, bcs, k in [((33, 29), [C, C, R, R], 1), ((9, 8, 7), [C] * 4 + [R] * 2, 3), ((45, 43, 41), [R] * 6, 2), ((300, 254), [C] * 4, 4)]:
    s = random_bq(grid, bcs, seed=sum(grid) + k, prs_k=k)
    run, orc = bq_run(s), bq_oracle(s)
    run.advance(1)
    orc.advance(1)
    got = [np.array(run.advectee(e)) for e in range(len(grid) + 1)]
    out.append(["bq " + str(grid), run.stats()["kernels"], all(bool(np.isfinite(a).all()) for a in got),
                max(rel(a, orc.advectee(e)) for e, a in enumerate(got))])
print(json.dumps(out))
"""


def debug_process(script):
    so = os.path.join(ROOT, "libmpdataxx_b200", "libmpdx_debug.so")
    assert os.path.exists(so), "the debug library is built with the rest (make -C libmpdataxx_b200/csrc)"
    p = subprocess.run([sys.executable, "-c", "ROOT = " + repr(ROOT) + "\n" + script], env=dict(os.environ, MPDX_LIBRARY="debug"),
                       capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr[-3000:]
    return json.loads(p.stdout.strip().splitlines()[-1])


def test_walking_kernels_run_clean():
    stages, fused, line, block = 2, 3, 4, 5
    for name, kernels, finite, err in debug_process(SCRIPT):
        want = fused if name.startswith("fused") else line if name in ("(300,)", "40 0", "40 33") else block if name == "40 2" else stages
        assert kernels == want, (name, kernels)
        assert finite, name
        assert err <= 1e-12, (name, err)


def test_walking_pointers_record_what_is_outside(tmp_path):
    exe = str(tmp_path / "elem_check")
    subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe,
                    os.path.join(ROOT, "tests", "cuda", "elem_check.cu")], check=True)
    p = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0 and p.stdout.strip() == "ok", p.stdout + p.stderr

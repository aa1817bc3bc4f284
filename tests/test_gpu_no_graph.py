"""KIELFLOW_B200_NO_GRAPH=1: steps, solves and gradients launched kernel by kernel,
with the results of the captured graphs."""
import os
import subprocess
import sys

import numpy as np
import pytest

import kielflow_b200 as kf
from kielflow_b200 import configs as C

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def everything():
    n, out = 32, {}
    for name in ("fas128", "jacobi32"):
        w = dict(C.WORKLOADS[name], Q=-5.0)
        st, nd, mask, dt = C.make_inputs(w, n)
        with kf.Context(C.config_for(w, n)) as ctx:
            ctx.set_sources(nd, mask)
            for k in range(3):  # a context's first adaptive FAS solve is launched singly in any case
                l0 = ctx.launch_count()
                out[f"{name} phi {k}"] = ctx.poisson(np.zeros((n, n, n)), 1.0 + nd)
                out[f"{name} launches {k}"] = np.array(ctx.launch_count() - l0)
            ctx.set_state(*st)
            ctx.rk4(dt, 1)
            out[f"{name} step"] = np.array(ctx.get_state())
    w = dict(C.WORKLOADS["adj128"], Q=-5.0)
    st, nd, mask, dt = C.make_inputs(w, n)
    with kf.Context(C.config_for(w, n)) as ctx:
        ctx.set_sources(nd, mask)
        ctx.set_state(*st)
        g = ctx.adjoint(C.wake_window(n), 2, dt, ckpt_every=2)
        out["dn0"] = g["dn0"]
    return out


def test_same_results_without_graphs(tmp_path):
    code = ("import sys; sys.path[:0] = [%r, %r]; import numpy as np, test_gpu_no_graph as t; "
            "np.savez(%r, **t.everything())" % (ROOT, os.path.dirname(os.path.abspath(__file__)), str(tmp_path / "a.npz")))
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300, cwd=ROOT,
                   env=dict(os.environ, KIELFLOW_B200_NO_GRAPH="1"))
    a, b = np.load(tmp_path / "a.npz"), everything()
    for k in b:
        if "launches" not in k:
            assert np.array_equal(a[k], b[k]), k
    # the graphs' control kernels are counted: none of them here
    assert a["fas128 launches 0"] == a["fas128 launches 1"] == a["fas128 launches 2"] < b["fas128 launches 1"]

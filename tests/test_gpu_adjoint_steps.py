"""Steps and solves before and after a context's first gradient: graphs captured
before it stay valid (their job lists live as long as the context)."""
import numpy as np
import pytest

import kielflow_b200 as kf
from kielflow_b200 import configs as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("host_call", [False, True])
@pytest.mark.parametrize("n", [32, 64])
def test_steps_around_an_adjoint(n, host_call):
    """Captured step, gradient, the same captured step; against a context whose
    first step is launched kernel by kernel, so that it captures its step after
    the gradient: identical states, potentials and gradients."""
    w = dict(C.WORKLOADS["adj128"], Q=-5.0)
    st, nd, mask, dt = C.make_inputs(w, n)
    out = []
    for before in (True, False):
        with kf.Context(C.config_for(w, n)) as ctx:
            ctx.set_sources(nd, mask)

            def step(arrays):
                if host_call:
                    ctx.step_host(arrays, dt, 1)
                    return arrays
                ctx.set_state(*arrays)
                ctx.rk4(dt, 1)
                return ctx.get_state()

            a = [np.ascontiguousarray(x).copy() for x in st]
            ctx.profile(not before)
            a = step(a)
            ctx.profile(False)
            ctx.set_state(*a)
            g = ctx.adjoint(C.wake_window(n), 2, dt, ckpt_every=1)
            ctx.set_state(*a)
            a = step(a)
            out.append((a, ctx.get_phi(), g))
    (a, p, g), (b, q, h) = out
    assert all(np.array_equal(x, y) for x, y in zip(a, b)) and np.array_equal(p, q)
    assert np.array_equal(g["dn0"], h["dn0"]) and all(g[k] == h[k] for k in ("J", "dJ_dM", "dJ_dtau", "dJ_dnd"))
    assert all(np.isfinite(x).all() for x in a)

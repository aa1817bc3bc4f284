"""The same calls on pageable and on page-locked host arrays, once more than 64 MB
of pageable ones have gone through a context (from there on several threads
share each copy): identical results."""
import ctypes

import numpy as np
import pytest
import torch

import kielflow_b200 as kf
from kielflow_b200 import configs as C

pytestmark = pytest.mark.gpu

D = ctypes.POINTER(ctypes.c_double)


def array(a, pinned):
    """A copy of a in fresh memory of the kind asked for."""
    if not pinned:
        return np.array(a, order="C", copy=True)
    h = torch.empty(a.shape, dtype=torch.complex128 if a.dtype.kind == "c" else torch.float64, pin_memory=True).numpy()
    h[...] = a
    return h


def ptr(a):
    return a.ctypes.data_as(D)


@pytest.mark.parametrize("n,name,nsteps", [(96, "fas128", 2), (128, "fas128", 1), (128, "fp32bulk256", 2)])
def test_calls_on_both_kinds(n, name, nsteps):
    w = dict(C.WORKLOADS[name], Q=-5.0, sigma=0.5)
    st, nd, mask, dt = C.make_inputs(w, n)
    rng = np.random.default_rng(n)
    guess = 1e-2 * rng.standard_normal((n, n, n))
    out = []
    for pinned in (False, True):
        with kf.Context(C.config_for(w, n)) as ctx:
            for _ in range(-(-(80 << 20) // (8 * n ** 3))):  # 80 MB of pageable arrays
                ctx.set_phi(np.zeros((n, n, n)))
            src = array(nd, pinned), array(mask, pinned)
            ctx._check(ctx.L.kf_set_sources(ctx.h, ptr(src[0]), ptr(src[1])))
            a = [array(f, pinned) for f in st]
            got = []
            for _ in range(2):
                ctx.step_host(a, dt, nsteps)
                got += [f.copy() for f in a]
            ctx._check(ctx.L.kf_set_state(ctx.h, *[ptr(f) for f in a]))
            b = [array(np.zeros_like(f), pinned) for f in a]
            ctx._check(ctx.L.kf_get_state(ctx.h, *[ptr(f) for f in b]))
            phi = array(np.full((n, n, n), np.nan), pinned)
            g = array(guess, pinned)
            ctx._check(ctx.L.kf_poisson_solve_to(ctx.h, ptr(g), ptr(array(1.0 + nd, pinned)), ptr(phi)))
            assert np.array_equal(g, guess)
            out.append(got + b + [phi, ctx.get_phi()])
    assert all(np.array_equal(x, y) for x, y in zip(*out))
    assert np.array_equal(out[0][-1], out[0][-2]) and all(np.isfinite(x).all() for x in out[0])

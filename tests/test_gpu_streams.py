"""A context on a caller's stream: host arrays, steps and solves give what they
give on the context's own stream."""
import numpy as np
import pytest
import torch

import kielflow_b200 as kf
from kielflow_b200 import configs as C
from kielflow_b200 import inputs as I

pytestmark = pytest.mark.gpu

PER_THREAD = 2  # cudaStreamPerThread


@pytest.mark.parametrize("prec", [kf.KF_FP64, kf.KF_FP32_BULK])
@pytest.mark.parametrize("stream", ["own", "torch", "per thread"])
def test_pageable_arrays_on_a_stream(stream, prec):
    """More than 64 MB of pageable arrays of 16.8 MB each, both ways and through a
    transform between them, several times over."""
    n = 128
    rng = np.random.default_rng(3)
    x = [rng.standard_normal((n, n, n)) for _ in range(2)]
    st = [np.fft.rfftn(rng.standard_normal((n, n, n))) for _ in range(4)]
    bulk = np.complex64 if prec == kf.KF_FP32_BULK else np.complex128
    own = torch.cuda.Stream()
    with kf.Context(kf.Config.make(n, I.L_DEFAULT, 0.8, precision=prec)) as ctx:
        want = [ctx.r2c(a) for a in x]
        if stream != "own":
            ctx.set_stream(own.cuda_stream if stream == "torch" else PER_THREAD)
        for rep in range(3):
            src = [(1.0 + rep) * a for a in st]
            ctx.set_state(*src)
            for a in src:
                a[...] = np.nan
            got = ctx.get_state()
            assert all(np.array_equal(((1.0 + rep) * a).astype(bulk).astype(np.complex128), b) for a, b in zip(st, got))
            assert all(np.array_equal(ctx.r2c(a), w) for a, w in zip(x, want))
        ctx.set_stream(0)


@pytest.mark.parametrize("stream", ["torch", "per thread"])
def test_steps_on_a_stream(stream):
    n, w = 32, C.WORKLOADS["fas128"]
    st, nd, mask, dt = C.make_inputs(w, n)
    own = torch.cuda.Stream()
    out = []
    for handle in (None, own.cuda_stream if stream == "torch" else PER_THREAD):
        with kf.Context(C.config_for(w, n)) as ctx:
            if handle is not None:
                ctx.set_stream(handle)
            ctx.set_state(*st)
            ctx.set_sources(nd, mask)
            ctx.rk4(dt, 2)
            a = [np.ascontiguousarray(f).copy() for f in ctx.get_state()]
            ctx.step_host(a, dt, 1)
            out.append(a + [ctx.get_phi(), ctx.poisson(np.zeros((n, n, n)), 1.0 + nd)])
            ctx.set_stream(0)
    assert all(np.array_equal(a, b) for a, b in zip(*out))

"""The right-hand side at the production size, 256^3 (radix plans and block shapes
of its own), on full spectra against the CPU oracle."""
import functools

import numpy as np
import pytest

import kielflow_b200 as kf
from kielflow_b200 import configs as C
from kielflow_b200 import inputs as I
from oracle import bind

pytestmark = pytest.mark.gpu

N = 256
NO_PHI = kf.KF_T_ALL & ~(kf.KF_T_POISSON | kf.KF_T_E_INT)


@functools.lru_cache(maxsize=1)
def fields():
    rng = np.random.default_rng(N)
    st = [1e-2 * np.fft.rfftn(rng.standard_normal((N, N, N))) for _ in range(4)]
    return st, I.gauss_charge(N, C.L_BOX, -50.0, 0.3), I.sphere_mask(N, C.L_BOX, 2.0)


def config(stretched, prec):
    return C.config_for(C.WORKLOADS["fp64_256"], n=N, precision=prec, terms=NO_PHI,
                        stretch_m=C.STRETCH_FRONTEND if stretched else 0.0)


@functools.lru_cache(maxsize=1)
def reference(stretched):
    st, nd, mask = fields()
    cfg = config(stretched, kf.KF_FP64)
    o = bind.Oracle(bind.KfoConfig(*[getattr(cfg, f) for f, _ in bind.KfoConfig._fields_]))
    o.set_state(st)
    o.set_sources(nd, mask)
    o.rhs()
    return o.get_state()


@pytest.mark.parametrize("plan", [0, 1])
@pytest.mark.parametrize("prec", [kf.KF_FP64, kf.KF_FP32_BULK])
@pytest.mark.parametrize("stretched", [False, True])
def test_rhs_vs_oracle(stretched, prec, plan):
    """1e-12 and 1e-5 of the largest element, as at the smaller sizes."""
    st, nd, mask = fields()
    with kf.Context(config(stretched, prec)) as ctx:
        ctx.set_tuning(plan, 8)
        ctx.set_state(*st)
        ctx.set_sources(nd, mask)
        ctx.rhs()
        g = ctx.get_state()
    r = reference(stretched)
    scale = max(np.abs(x).max() for x in r)
    assert max(np.abs(a - b).max() for a, b in zip(g, r)) / scale < (1e-12 if prec == kf.KF_FP64 else 1e-5)

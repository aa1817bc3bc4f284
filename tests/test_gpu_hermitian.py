"""States that are no spectra of real fields: their kz = 0 and kz = n/2 planes
are not Hermitian.  With penalization the reference takes the right-hand side
through physical space, which keeps the Hermitian part of those planes."""
import numpy as np
import pytest

import kielflow_b200 as kf
from kielflow_b200 import configs as C
from kielflow_b200 import inputs as I
from oracle import bind

pytestmark = pytest.mark.gpu

NO_PHI = kf.KF_T_ALL & ~(kf.KF_T_POISSON | kf.KF_T_E_INT)


@pytest.mark.parametrize("prec", [kf.KF_FP64, kf.KF_FP32_BULK])
@pytest.mark.parametrize("stretched", [False, True])
@pytest.mark.parametrize("mask", ["none", "ball"])
@pytest.mark.parametrize("pen", [True, False])
@pytest.mark.parametrize("n", [16, 32, 96])
def test_rhs_vs_oracle(n, pen, mask, stretched, prec):
    w = C.WORKLOADS["fas128"]
    cfg = C.config_for(w, n=n, precision=prec, terms=NO_PHI if pen else NO_PHI & ~kf.KF_T_PENALIZATION,
                       stretch_m=C.STRETCH_FRONTEND if stretched else 0.0)
    rng = np.random.default_rng(n)
    st = [1e-2 * n ** 1.5 * (rng.standard_normal((n, n, n // 2 + 1)) + 1j * rng.standard_normal((n, n, n // 2 + 1)))
          for _ in range(4)]
    nd = I.gauss_charge(n, C.L_BOX, w["Q"], w["sigma"])
    H = I.sphere_mask(n, C.L_BOX, 2.0) if mask == "ball" else np.zeros((n, n, n))
    with kf.Context(cfg) as ctx:
        ctx.set_state(*st)
        ctx.set_sources(nd, H)
        ctx.rhs()
        g = ctx.get_state()
    o = bind.Oracle(bind.KfoConfig(*[getattr(cfg, f) for f, _ in bind.KfoConfig._fields_]))
    o.set_state(st)
    o.set_sources(nd, H)
    o.rhs()
    r = o.get_state()
    scale = max(np.abs(x).max() for x in r)
    assert max(np.abs(a - b).max() for a, b in zip(g, r)) / scale < (1e-12 if prec == kf.KF_FP64 else 1e-5)

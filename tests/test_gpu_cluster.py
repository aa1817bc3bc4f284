"""The coarse levels of a V-cycle in one thread-block cluster (kf_set_coarse_block)
against the level-by-level kernels, bit for bit: every cluster size that the
supported grids give (the largest divisor of the coarsest n up to 16), one to
four levels held, both smoother
orders, and the adjoint's linear system."""
import numpy as np
import pytest

import kielflow_b200 as kf
from kielflow_b200 import configs as C
from kielflow_b200 import inputs as I

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,levels,stretched", [(16, 2, False), (16, 4, False), (32, 2, False), (32, 4, True), (64, 3, False),
                                                (64, 5, True), (96, 4, False), (96, 5, False), (128, 4, True),
                                                (128, 5, False)])
def test_poisson_bit_identical(n, levels, stretched):
    m = C.STRETCH_FRONTEND if stretched else 0.0
    rng = np.random.default_rng(n + levels)
    rho = np.exp(0.1 * rng.standard_normal((n, n, n))) + I.gauss_charge(n, C.L_BOX, -10.0, 0.5, m)
    cfg = kf.Config.make(n, C.L_BOX, 0.8, poisson_mode=kf.KF_PS_FAS, mg_levels=levels, mg_pre=1 + levels % 2, mg_post=2,
                         res_tol=0.0, max_cycles=4, mg_omega=1.25, stretch_m=m)
    res = []
    for on in (False, True):
        with kf.Context(cfg) as ctx:
            ctx.set_coarse_block(on)
            res.append(ctx.poisson(np.zeros((n, n, n)), rho))
    assert np.array_equal(*res) and np.isfinite(res[0]).all()


@pytest.mark.parametrize("n,levels", [(32, 2), (64, 3), (64, 4)])
def test_adjoint_bit_identical(n, levels):
    w = dict(C.WORKLOADS["adj128"], Q=-5.0)
    st, nd, mask, dt = C.make_inputs(w, n=n)
    cfg = C.config_for(w, n=n, mg_levels=levels)
    res = []
    for on in (False, True):
        with kf.Context(cfg) as ctx:
            ctx.set_coarse_block(on)
            ctx.set_state(*st)
            ctx.set_sources(nd, mask)
            res.append(ctx.adjoint(C.wake_window(n), 2, dt, ckpt_every=2))
    a, b = res
    assert np.array_equal(a["dn0"], b["dn0"]) and a["adj_cycles"] == b["adj_cycles"]
    assert all(a[k] == b[k] for k in ("J", "dJ_dM", "dJ_dtau", "dJ_dnd"))

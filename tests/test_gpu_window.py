"""The mask's window of rows is read on the device: a context whose mask moves,
grows or goes between captured steps gives what a new context with that mask
gives, bit for bit."""
import numpy as np
import pytest

import kielflow_b200 as kf
from kielflow_b200 import configs as C
from kielflow_b200 import inputs as I

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [kf.KF_FP64, kf.KF_FP32_BULK])
@pytest.mark.parametrize("stretched", [False, True])
@pytest.mark.parametrize("poisson", [True, False])
@pytest.mark.parametrize("n", [16, 32])
def test_masks_in_turn(n, poisson, stretched, prec):
    w = dict(C.WORKLOADS["fas128"], Q=-5.0)
    st, nd, ball, dt = C.make_inputs(w, n)
    ball = I.sphere_mask(n, C.L_BOX, 3.0)
    one = np.zeros((n, n, n))
    one[n - 1, 0, n // 2] = 1.0
    masks = [0.0 * ball, ball, np.roll(ball, (n // 2, 3), (0, 1)), one, np.ones((n, n, n)), 0.0 * ball, ball]
    terms = kf.KF_T_ALL if poisson else kf.KF_T_ALL & ~kf.KF_T_POISSON
    cfg = C.config_for(w, n=n, precision=prec, terms=terms, stretch_m=C.STRETCH_FRONTEND if stretched else 0.0,
                       phi_extrap=0)  # the start of a solve does not depend on the time reached

    def step(ctx, mask):
        ctx.set_phi(np.zeros((n, n, n)))
        ctx.set_state(*st)
        ctx.set_sources(nd, mask)
        ctx.rk4(0.1 * dt, 1)
        return ctx.get_state()

    with kf.Context(cfg) as ctx:
        first = step(ctx, masks[1])
        for m in masks:
            got = step(ctx, m)
            with kf.Context(cfg) as new:
                assert all(np.array_equal(a, b) for a, b in zip(got, step(new, m)))
        assert all(np.array_equal(a, b) for a, b in zip(got, first))

"""The FAS stop test's maximum |residual| against the residual of the potential
that the solve returns, formed on the host."""
import numpy as np
import pytest

import kielflow_b200 as kf
from kielflow_b200 import configs as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [4, 8, 16])
@pytest.mark.parametrize("n,levels", [(64, 3), (96, 4), (128, 4)])
def test_stop_test_sees_every_row(n, levels, rows):
    """A solve that may stop at once returns the pre-smoothed potential and its
    max |f|, found at a spike of rho: in rows of every block and lane (96^3: blocks
    of 24 threads a row, the last ones cut off by the level's end).  The residual
    is a difference of terms of about |phi| / h^2 and rho: 1e-12 of the spike."""
    cfg = kf.Config.make(n, C.L_BOX, 0.8, poisson_mode=kf.KF_PS_FAS, mg_levels=levels, mg_pre=1, mg_post=1, res_tol=1e30,
                         max_cycles=5)
    h2 = (C.L_BOX / n) ** -2
    rng = np.random.default_rng(n)
    with kf.Context(cfg) as ctx:
        ctx.set_tuning(0, rows)
        for j in [0, 1, 4, 5, 9, 10, 31, n // 2 + 1, n - 6, n - 5, n - 2, n - 1]:
            rho = np.exp(0.1 * rng.standard_normal((n, n, n)))
            rho[rng.integers(n), j, rng.integers(n)] += 1e3
            phi = ctx.poisson(np.zeros((n, n, n)), rho)
            lap = sum(np.roll(phi, s, a) for s in (1, -1) for a in range(3)) - 6.0 * phi
            want = np.abs(h2 * lap + rho - np.exp(phi)).max()
            assert abs(ctx.diag().last_residual - want) <= 1e-9

"""The Jacobi relaxation, whose sweep loop and stop test run on the device,
against the CPU oracle."""
import numpy as np
import pytest

import kielflow_b200 as kf
from kielflow_b200 import configs as C
from kielflow_b200 import inputs as I
from oracle import bind

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [kf.KF_PS_JACOBI_RES, kf.KF_PS_CASCADIC])
@pytest.mark.parametrize("n", [16, 32, 64, 96])
def test_jacobi_vs_oracle(n, mode):
    """The oracle's sweeps, one for one, and its potential: levels of less than a
    block (2^3) to several points a thread (96^3)."""
    if mode == kf.KF_PS_JACOBI_RES and n > 32:
        pytest.skip("thousands of sweeps on the oracle")
    rng = np.random.default_rng(n)
    rho = np.exp(0.1 * rng.standard_normal((n, n, n))) + I.gauss_charge(n, C.L_BOX, -10.0, 1.0)
    cfg = kf.Config.make(n, C.L_BOX, 0.8, poisson_mode=mode, nlj_max_it=500, res_tol=1e-8, mg_levels=1)
    with kf.Context(cfg) as ctx:
        phi = ctx.poisson(np.zeros((n, n, n)), rho)
        its = ctx.diag().total_iterations
    o = bind.Oracle(bind.KfoConfig(*[getattr(cfg, f) for f, _ in bind.KfoConfig._fields_]))
    ref = o.poisson(np.zeros((n, n, n)), rho)
    assert np.abs(phi - ref).max() <= 1e-12 * np.abs(ref).max()
    assert its == o.stats().total_iterations

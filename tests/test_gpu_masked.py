"""Masked transform passes (only what the 2/3 rule keeps is moved): right-hand
sides of states whose spectra are full, against the CPU oracle.  White noise
puts as much into the removed wave numbers as into the kept ones, so a wrong
bound of a pass, a stale value outside one or a missing edge element shows."""
import numpy as np
import pytest

import kielflow_b200 as kf
from kielflow_b200 import configs as C
from kielflow_b200 import inputs as I
from oracle import bind

pytestmark = pytest.mark.gpu

NO_PHI = kf.KF_T_ALL & ~(kf.KF_T_POISSON | kf.KF_T_E_INT)


def noise_state(n, seed):
    rng = np.random.default_rng(seed)
    return [1e-2 * bind.r2c(rng.standard_normal((n, n, n))) for _ in range(4)]


def oracle_rhs(cfg, st, nd, mask):
    o = bind.Oracle(bind.KfoConfig(*[getattr(cfg, f) for f, _ in bind.KfoConfig._fields_]))
    o.set_state(st)
    o.set_sources(nd, mask)
    o.rhs()
    return o.get_state()


@pytest.mark.parametrize("plan", [0, 1])
@pytest.mark.parametrize("prec", [kf.KF_FP64, kf.KF_FP32_BULK])
@pytest.mark.parametrize("pen", [True, False])
@pytest.mark.parametrize("n", [16, 32, 64, 96, 128])
def test_full_spectrum_rhs_vs_oracle(n, pen, prec, plan):
    w = C.WORKLOADS["fas128"]
    terms = NO_PHI if pen else NO_PHI & ~kf.KF_T_PENALIZATION
    cfg = C.config_for(w, n=n, precision=prec, terms=terms)
    nd = I.gauss_charge(n, C.L_BOX, w["Q"], w["sigma"])
    mask = I.sphere_mask(n, C.L_BOX, 2.0)
    st = noise_state(n, n)
    with kf.Context(cfg) as ctx:
        ctx.set_tuning(plan, 8)
        ctx.set_state(*noise_state(n, n + 1))  # another state first: whatever it leaves outside the
        ctx.set_sources(nd, mask)              # bounds must not reach the second result
        ctx.rhs()
        ctx.set_state(*st)
        ctx.rhs()
        g = ctx.get_state()
    r = oracle_rhs(cfg, st, nd, mask)
    scale = max(np.abs(x).max() for x in r)
    err = max(np.abs(a - b).max() for a, b in zip(g, r)) / scale
    assert err < (1e-12 if prec == kf.KF_FP64 else 1e-5)


MASKS = {
    "none": lambda n: np.zeros((n, n, n)),
    "one point": lambda n: np.eye(1, n ** 3, 5 * n * n + 3 * n + n - 1).reshape(n, n, n),
    "ball": lambda n: I.sphere_mask(n, C.L_BOX, 2.0),
    "across the box edge": lambda n: np.roll(I.sphere_mask(n, C.L_BOX, 2.0), (n // 2, n // 2, n // 3), (0, 1, 2)),
    "smooth, everywhere": lambda n: np.random.default_rng(n).uniform(0.0, 1.0, (n, n, n)),
}


@pytest.mark.parametrize("prec", [kf.KF_FP64, kf.KF_FP32_BULK])
@pytest.mark.parametrize("kind", list(MASKS))
def test_penalization_masks_vs_oracle(kind, prec):
    """The linear terms are transformed on the mask's window of rows only."""
    n, w = 32, C.WORKLOADS["fas128"]
    cfg = C.config_for(w, n=n, precision=prec, terms=NO_PHI)
    nd = I.gauss_charge(n, C.L_BOX, w["Q"], w["sigma"])
    st, dt = noise_state(n, 7), 1e-3
    o = bind.Oracle(bind.KfoConfig(*[getattr(cfg, f) for f, _ in bind.KfoConfig._fields_]))
    with kf.Context(cfg) as ctx:
        for k in ("ball", kind):  # the window changes under a captured step
            ctx.set_sources(nd, MASKS[k](n))
            ctx.set_state(*st)
            ctx.rk4(dt, 2)
        g = ctx.get_state()
    o.set_state(st)
    o.set_sources(nd, MASKS[kind](n))
    o.rk4(dt, 2)
    r = o.get_state()
    scale = max(np.abs(x).max() for x in r)
    err = max(np.abs(a - b).max() for a, b in zip(g, r)) / scale
    assert err < (1e-12 if prec == kf.KF_FP64 else 1e-5)


@pytest.mark.parametrize("plan", [0, 1])
@pytest.mark.parametrize("prec", [kf.KF_FP64, kf.KF_FP32_BULK])
@pytest.mark.parametrize("filtered", [True, False])
@pytest.mark.parametrize("n", [16, 64, 96, 128])
def test_given_potential_vs_oracle(n, filtered, prec, plan):
    """Of phi^ only the columns on which the phi filter is not 0 are formed (with
    the pressure term, which applies it; all of them without): a white-noise
    potential, taken as given."""
    w = C.WORKLOADS["fas128"]
    terms = kf.KF_T_ALL & ~kf.KF_T_POISSON & (-1 if filtered else ~kf.KF_T_PRESSURE)
    cfg = C.config_for(w, n=n, precision=prec, terms=terms)
    nd = I.gauss_charge(n, C.L_BOX, w["Q"], w["sigma"])
    mask = I.sphere_mask(n, C.L_BOX, 2.0)
    phi = 1e-2 * np.random.default_rng(n).standard_normal((n, n, n))
    st = noise_state(n, n)
    o = bind.Oracle(bind.KfoConfig(*[getattr(cfg, f) for f, _ in bind.KfoConfig._fields_]))
    o.set_phi(phi)
    o.set_state(st)
    o.set_sources(nd, mask)
    o.rhs()
    r = o.get_state()
    with kf.Context(cfg) as ctx:
        ctx.set_tuning(plan, 8)
        ctx.set_state(*st)
        ctx.set_sources(nd, mask)
        ctx.set_phi(phi)
        ctx.rhs()
        g = ctx.get_state()
    scale = max(np.abs(x).max() for x in r)
    err = max(np.abs(a - b).max() for a, b in zip(g, r)) / scale
    assert err < (1e-12 if prec == kf.KF_FP64 else 1e-5)


@pytest.mark.parametrize("plan", [0, 1])
@pytest.mark.parametrize("prec", [kf.KF_FP64, kf.KF_FP32_BULK])
@pytest.mark.parametrize("kind", [None, "ball", "across the box edge"])
@pytest.mark.parametrize("n", [16, 32, 96, 128])
def test_full_spectrum_stretched_rhs_vs_oracle(n, kind, prec, plan):
    """On stretched axes: the filtered derivatives' passes (k_x_filter), the sums in
    physical space and the penalization on the mask's window (kind None: without).
    Four transforms follow one another, each good to a few rounding units of the
    field's scale: 1e-5 and 1e-12 as above."""
    w = C.WORKLOADS["fas128"]
    L = I.L_DEFAULT
    terms = NO_PHI if kind else NO_PHI & ~kf.KF_T_PENALIZATION
    cfg = C.config_for(w, n=n, precision=prec, terms=terms, stretch_m=I.frontend_stretch(L))
    nd = I.gauss_charge(n, C.L_BOX, w["Q"], w["sigma"])
    mask = MASKS[kind or "ball"](n)
    st = noise_state(n, n)
    with kf.Context(cfg) as ctx:
        ctx.set_tuning(plan, 8)
        ctx.set_state(*noise_state(n, n + 1))
        ctx.set_sources(nd, mask)
        ctx.rhs()
        ctx.set_state(*st)
        ctx.rhs()
        g = ctx.get_state()
    r = oracle_rhs(cfg, st, nd, mask)
    scale = max(np.abs(x).max() for x in r)
    err = max(np.abs(a - b).max() for a, b in zip(g, r)) / scale
    assert err < (1e-12 if prec == kf.KF_FP64 else 1e-5)

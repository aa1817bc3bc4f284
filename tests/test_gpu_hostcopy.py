"""Pageable host arrays through the threaded copies (4 MB and up), against the
same calls on page-locked arrays: sizes that are no multiple of a thread's range
or of a pinned piece, both directions, several contexts at once."""
import threading

import numpy as np
import pytest

import kielflow_b200 as kf
from kielflow_b200 import inputs as I

pytestmark = pytest.mark.gpu


def noise(n, seed):
    rng = np.random.default_rng(seed)
    return [np.fft.rfftn(rng.standard_normal((n, n, n))) for _ in range(4)]


@pytest.mark.parametrize("prec", [kf.KF_FP64, kf.KF_FP32_BULK])
@pytest.mark.parametrize("n", [64, 96, 128])
def test_state_round_trip(n, prec):
    st = noise(n, n)
    with kf.Context(kf.Config.make(n, I.L_DEFAULT, 0.8, precision=prec)) as ctx:
        for rep in range(2):  # the pieces are used again
            src = [a + rep for a in st]
            keep = [a.copy() for a in src]
            ctx.set_state(*src)
            for a in src:
                a[...] = np.nan  # an upload's source may change on return
            got = ctx.get_state()
            want = keep if prec == kf.KF_FP64 else [a.astype(np.complex64).astype(np.complex128) for a in keep]
            assert all(np.array_equal(a, b) for a, b in zip(got, want))
        phi = np.random.default_rng(1).standard_normal((n, n, n))
        ctx.set_phi(phi)
        assert np.array_equal(ctx.get_phi(), phi)


def test_contexts_in_threads():
    n, res = 96, {}

    def work(k):
        st = noise(n, k)
        with kf.Context(kf.Config.make(n, I.L_DEFAULT, 0.8)) as ctx:
            for _ in range(3):
                ctx.set_state(*st)
                res[k] = all(np.array_equal(a, b) for a, b in zip(ctx.get_state(), st))

    th = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert res == {k: True for k in range(4)}


def test_poisson_solve_leaves_its_guess():
    n = 128
    rho = 1.0 + I.gauss_charge(n, I.L_DEFAULT, -5.0, 0.5)
    guess = np.zeros((n, n, n))
    cfg = kf.Config.make(n, I.L_DEFAULT, 0.8, poisson_mode=kf.KF_PS_FAS, mg_levels=4)
    with kf.Context(cfg) as ctx:
        a = ctx.poisson(guess, rho)
        assert not guess.any() and np.isfinite(a).all() and a.any()
        assert np.array_equal(a, ctx.get_phi())

"""FP32-bulk steps through kf_step_host against recorded ones.  The call returns
FP64 arrays, so its FP32 rounding errors (1e-7 of the result) are part of what a
caller compares from one version to the next: a kernel that forms the same sums
in another order shows here, at far below its error against the exact result.

golden/fp32_step.npz holds elements of each field inside the 2/3 rule, and the
fields' norms, after one step of the library that ran the right-hand side pass by
pass (separate z transforms, products and RK4 update) on a B200."""
import os

import numpy as np
import pytest

import kielflow_b200 as kf
from kielflow_b200 import configs as C

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "fp32_step.npz")
CASES = [(32, "all"), (32, "no penalization"), (64, "all"), (96, "all"), (128, "all"), (256, "all")]


def step(n, terms):
    w = C.WORKLOADS["fp32bulk256"]
    over = {} if terms == "all" else {"terms": kf.KF_T_ALL & ~kf.KF_T_PENALIZATION}
    st, nd, mask, dt = C.make_inputs(w, n)
    with kf.Context(C.config_for(w, n, **over)) as ctx:
        ctx.set_sources(nd, mask)
        arrays = [np.ascontiguousarray(x).copy() for x in st]
        ctx.step_host(arrays, dt, 1)
    return arrays


def samples(n, arrays):
    k = np.minimum(np.arange(n), n - np.arange(n)) / (n / 2)
    kz = np.arange(n // 2 + 1) / (n / 2)
    inside = np.flatnonzero(k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz ** 2 < 0.44)
    low = np.flatnonzero(k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz ** 2 < (10.0 / n) ** 2)
    at = np.concatenate([low, inside[:: max(1, inside.size // 1500)]])
    return np.array([a.reshape(-1)[at] for a in arrays])


@pytest.mark.parametrize("n,terms", CASES)
def test_step_host_fp32_as_recorded(n, terms):
    """Relative 2-norm of each field to 1e-9: equal bits but for the inputs' FP64
    rounding, which the host's FFT may form differently (1e-16 of an element, and
    so another FP32 value for about one in 10^8)."""
    rec = np.load(GOLDEN)[f"{n} {terms}"]
    got = samples(n, step(n, terms))
    for a, b in zip(got, rec):
        assert np.linalg.norm(a - b) <= 1e-9 * np.linalg.norm(b)

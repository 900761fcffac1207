"""The bound on a host wait is one for a single replay, whatever the pair terms take."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_wait_bound_without_fixed_point(gb, torch_cuda):
    """Bodies far inside the softening (FP64 terms): with a bound of three replays' time, 160
    attempts end at their budget and not at the bound."""
    n = 2048
    r = np.random.default_rng(1)
    x0 = np.concatenate([1e-6 * r.standard_normal(3 * n), 1e-7 * r.standard_normal(3 * n)])
    ode = gb.NBodyODE(n, 1.0, 1.0 / n)

    def run(max_attempts, timeout):
        it = gb.Integrator("DOPRI5", ode, gb.Gb300Executor(max_attempts=max_attempts,
                                                           host_wait_timeout_s=timeout))
        it.start(x0, 0.0, 1e6, 1e-18, 1e-13)
        t = time.perf_counter()
        rc = it.advance()
        t = time.perf_counter() - t
        attempts = it.stats()["n_attempts"]
        it.close()
        return rc, t, attempts

    budget, one, attempts = run(16, 600.0)
    assert attempts == 16
    rc, _, attempts = run(160, 3.0 * one)
    assert (rc, attempts) == (budget, 160)

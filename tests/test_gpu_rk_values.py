"""The element-wise kernels on values that the integer products leave to the FP64 unit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPECIAL = np.array([0.0, -0.0, 5e-324, -3e-310, 2.2250738585072014e-308, 1e-300, -1e300,
                    1.7976931348623157e308, np.inf, -np.inf, np.nan, 1.0, -1.5, 3.0, 1e-160])


@pytest.mark.parametrize("n", [1, 2, 511, 1026])
@pytest.mark.parametrize("dt", [0.0137, 1e-308, 5e-324, 0.0, 1e300])
@pytest.mark.parametrize("name", ["DOPRI5", "RKF78"])
def test_special_values_bit_for_bit(gb, torch_cuda, name, dt, n):
    """Zeros, subnormals, huge values, infinities and NaN among ordinary ones, step sizes that are
    not normal: the IEEE operations in the reference's order (a zero's sign aside)."""
    torch = torch_cuda
    t = gb.tableau(name)
    S = t.n_stages
    rng = np.random.default_rng(n)
    x0 = rng.standard_normal(n)
    ks = rng.standard_normal((S, n)) * 10.0 ** rng.integers(-20, 20, (S, n))
    pick = rng.random((S, n)) < 0.1
    ks[pick] = rng.choice(SPECIAL, pick.sum())
    dx0, dks = gb.to_device(x0), gb.to_device(ks.reshape(-1))
    out, err = torch.empty(n, dtype=torch.float64, device="cuda"), torch.empty_like(dx0)

    def total(coef):
        v = np.zeros(n)
        for j, c in enumerate(coef):
            if c != 0.0:
                v = v + c * ks[j]
        return v * dt

    with np.errstate(all="ignore"):
        for stage in range(1, S):
            gb.rk_stage(t, stage, dt, dx0, dks, out, n)
            want = x0 + total([t.a[stage - 1][j] for j in range(stage)])
            np.testing.assert_array_equal(out.cpu().numpy(), want)
        gb.rk_update(t, dt, dx0, dks, out, err, n)
        np.testing.assert_array_equal(out.cpu().numpy(), x0 + total([t.b[j] for j in range(S)]))
        np.testing.assert_array_equal(err.cpu().numpy(),
                                      total([t.b[j] - t.bt[j] for j in range(S)]))

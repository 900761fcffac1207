"""FP64 right-hand side, leapfrog and energy of systems with one dominant mass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(n, heavy, light, seed=0):
    r = np.random.default_rng(1000 * n + seed)
    x = r.standard_normal(6 * n)
    m = light * r.uniform(0.5, 2.0, n)
    m[heavy] = 1.0
    return x, m


def _exact(x, m, soft):
    n = len(m)
    p = x[: 3 * n].reshape(n, 3).astype(np.longdouble)
    ml = m.astype(np.longdouble)
    d = p[None, :, :] - p[:, None, :]
    r2 = (d * d).sum(2) + np.longdouble(soft * soft)
    np.fill_diagonal(r2, 1)
    s = ml[None, :] / (r2 * np.sqrt(r2))
    np.fill_diagonal(s, 0)
    r = np.sqrt(r2)
    np.fill_diagonal(r, np.inf)
    return ((d * s[:, :, None]).sum(1), (np.sqrt((d * d).sum(2)) * s).sum(1).astype(float),
            -0.5 * (ml[:, None] * ml[None, :] / r).sum())


@pytest.mark.parametrize("light", [1e-3, 1e-6, 1e-9, 1e-15, 1e-20, 1e-100, 5e-311])
@pytest.mark.parametrize("n", [2, 33, 129, 517])
def test_one_dominant_mass(gb, torch_cuda, n, light):
    """The heavy body feels the light ones alone: every body within 16 2^-53 of the sum of its
    terms' sizes, the potential energy within 24 2^-53 of itself, as with equal masses."""
    soft = 0.01
    for heavy in (0, n // 2, n - 1):
        x, m = _system(n, heavy, light)
        acc, scale, pe = _exact(x, m, soft)
        mt = gb.to_device(m)
        for tile in (None, gb.tiling(f64_pair=1), gb.tiling(2, 4, 32, f64_pair=1)):
            got = gb.nbody_rhs_f64(x, n, soft, 1.0, mt, tile=tile).cpu().numpy()[3 * n:]
            err = np.abs((got.reshape(n, 3) - acc).astype(float)).max(axis=1)
            # denormal terms: at most 4 units of the last place each
            bound = 16 * 2.0 ** -53 * scale + 4 * n * 5e-324
            assert np.all(err <= bound), (err / bound).max()
        e = gb.energy(x, n, soft, 1.0, mt)
        assert abs(e["pe"] - pe) <= 24 * 2.0 ** -53 * abs(pe) + n * 5e-324


def test_mass_spectrum(gb, torch_cuda):
    """Masses over 30 decades in any order, with bodies of no mass among them: the same bounds."""
    n, soft = 700, 0.01
    r = np.random.default_rng(8)
    x, m = r.standard_normal(6 * n), 10.0 ** r.uniform(-30.0, 0.0, n)
    m[::5] = 0.0
    acc, scale, pe = _exact(x, m, soft)
    mt = gb.to_device(m)
    # a rounded sum for each class of masses in a tile
    got = gb.nbody_rhs_f64(x, n, soft, 1.0, mt).cpu().numpy()[3 * n:]
    err = np.linalg.norm((got.reshape(n, 3) - acc).astype(float), axis=1)
    assert np.all(err <= 64 * 2.0 ** -53 * scale), (err / scale).max() * 2.0 ** 53
    assert abs(gb.energy(x, n, soft, 1.0, mt)["pe"] - pe) <= 64 * 2.0 ** -53 * abs(pe)


def test_heavy_body_in_leapfrog(gb, torch_cuda):
    """Leapfrog from rest: the heavy body's momentum is the light ones' with the sign turned."""
    n = 129
    x, m = _system(n, n // 3, 1e-12, seed=4)
    x[3 * n:] = 0.0
    ode = gb.NBodyODE(n, 0.05, 1.0, gb.to_device(m))
    y, _ = gb.ParallelLeapfrogIntegrator.integrate(x, 0.0, 2.0 ** -10, 2.0 ** -10, ode, None,
                                                   gb.Gb300Executor())
    p = m[:, None] * y.cpu().numpy()[3 * n:].reshape(n, 3)
    # light-light forces are 1e-12 of the others; sums of 128 terms in FP64
    assert np.abs(p.sum(0)).max() <= 1e-13 * np.abs(p).sum()

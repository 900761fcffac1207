"""The FP64 right-hand side's fixed-point pair terms against extended precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(kind, n):
    r = np.random.default_rng(n)
    x = r.standard_normal(6 * n)
    soft, m = 0.01, None
    p = x[: 3 * n].reshape(n, 3)
    if kind == "far from the origin":
        p += (1.0e6, -3.0e5, 7.0)
    elif kind == "masses":
        m = 10.0 ** r.uniform(-9.0, 0.0, n)
        m[:: 7] = 0.0
        m[-1] = 1.0
    elif kind == "close pairs":  # below the window: FP64 terms
        soft = 1e-7
        p[1::2] = p[: 2 * (n // 2): 2] + 1e-6 * r.standard_normal((n // 2, 3))
    elif kind == "no softening":
        soft = 0.0
    elif kind == "one far body":  # nearly every other pair is below the window
        p[n // 2] = (3.0e7, 1.0, -2.0e6)
    elif kind == "tiny":  # the extent is far below the softening: no fixed point
        p *= 1e-9
    elif kind == "scaled down":
        p *= 2.0 ** -200
        soft *= 2.0 ** -200
    elif kind == "grid":  # exact symmetry, many equal distances
        p[:] = np.stack([np.arange(n) % 5, np.arange(n) // 5 % 7, np.arange(n) // 35], 1)
        soft = 0.25
    return x, soft, m


@pytest.mark.parametrize("kind", ["plain", "far from the origin", "masses", "close pairs",
                                  "no softening", "one far body", "tiny", "scaled down", "grid"])
@pytest.mark.parametrize("n", [2, 33, 128, 129, 517])
def test_rhs_f64_default_against_extended_precision(gb, torch_cuda, kind, n):
    """Every body's acceleration within 16 2^-53 of the sum of its terms' sizes: a term is within
    2^-55 (fixed point) or 6 2^-53 (FP64), a CTA's sum exact in fixed point, and at most 8
    partial sums, a conversion and the mass are rounded."""
    x, soft, m = _system(kind, n)
    p = x[: 3 * n].reshape(n, 3).astype(np.longdouble)
    ml = np.full(n, np.longdouble(1.0) / n) if m is None else m.astype(np.longdouble)
    d = p[None, :, :] - p[:, None, :]
    r2 = (d * d).sum(2) + np.longdouble(soft * soft)
    np.fill_diagonal(r2, 1)
    s = ml[None, :] / (r2 * np.sqrt(r2))
    np.fill_diagonal(s, 0)
    ref = (d * s[:, :, None]).sum(1)
    scale = (np.sqrt((d * d).sum(2)) * s).sum(1).astype(float)
    mt = None if m is None else gb.to_device(m)
    for tile in (None, gb.tiling(f64_pair=1), gb.tiling(2, 4, 32, f64_pair=1)):
        got = gb.nbody_rhs_f64(x, n, soft, 1.0 / n, mt, tile=tile).cpu().numpy()
        np.testing.assert_array_equal(got[: 3 * n], x[3 * n:])
        err = np.linalg.norm((got[3 * n:].reshape(n, 3) - ref).astype(float), axis=1)
        assert np.all(err <= 16 * 2.0 ** -53 * scale), (err / scale).max() * 2.0 ** 53


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("pair", [0, 1])
def test_rhs_f64_not_finite(gb, torch_cuda, bad, pair):
    """A coordinate that is not finite gives the FP64 loop's result."""
    n = 200
    x = np.random.default_rng(3).standard_normal(6 * n)
    x[3 * 77 + 1] = bad
    got = gb.nbody_rhs_f64(x, n, 0.01, 1.0 / n, tile=gb.tiling(f64_pair=pair)).cpu().numpy()
    ref = gb.nbody_rhs_f64(x, n, 0.01, 1.0 / n, tile=gb.tiling(f64_pair=2)).cpu().numpy()
    if pair == 0:
        np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
    assert np.isnan(got[3 * n + 3 * 77 + 1])
    np.testing.assert_array_equal(got[: 3 * n], x[3 * n:])


@pytest.mark.parametrize("kind", ["plain", "far from the origin", "masses", "close pairs",
                                  "one far body", "tiny", "grid"])
@pytest.mark.parametrize("n", [2, 31, 33, 129, 517])
def test_potential_energy_against_extended_precision(gb, torch_cuda, kind, n):
    """The potential energy within 24 2^-53 of itself (its terms have one sign): a term is within
    2^-55 (fixed point) or 4 2^-53 (FP64), a CTA's sum per body exact in fixed point; the sums
    over 8 ranks, 128 bodies (tree) and the tiles, the masses and a half are rounded."""
    x, soft, m = _system(kind, n)
    p = x[: 3 * n].reshape(n, 3).astype(np.longdouble)
    ml = np.full(n, np.longdouble(1.0 / n)) if m is None else m.astype(np.longdouble)
    d = p[None, :, :] - p[:, None, :]
    r = np.sqrt((d * d).sum(2) + np.longdouble(soft * soft))
    np.fill_diagonal(r, np.inf)
    ref = -0.5 * (ml[:, None] * ml[None, :] / r).sum()
    e = gb.energy(x, n, soft, 1.0 / n, None if m is None else gb.to_device(m))
    assert abs(e["pe"] - ref) <= 24 * 2.0 ** -53 * abs(ref), float((e["pe"] - ref) / ref * 2 ** 53)

"""The FP64 right-hand side, component by component, of systems that are thin along one axis."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(gb, x, n, soft, m=None):
    """Every component of every acceleration within (24 + n / 8) 2^-53 of the sum of its terms'
    sizes in that component: a term is within 2^-55 (fixed point) or 6 2^-53 (FP64) of itself in
    each, a CTA's sums are exact in fixed point, a lane adds at most n / 8 terms in FP64, and
    the partial sums (lanes, ranks, classes of masses), the conversion and the mass are rounded."""
    p = x[: 3 * n].reshape(n, 3).astype(np.longdouble)
    ml = np.full(n, np.longdouble(1.0 / n)) if m is None else m.astype(np.longdouble)
    d = p[None, :, :] - p[:, None, :]
    r2 = (d * d).sum(2) + np.longdouble(soft * soft)
    np.fill_diagonal(r2, 1)
    s = ml[None, :] / (r2 * np.sqrt(r2))
    np.fill_diagonal(s, 0)
    t = d * s[:, :, None]
    ref, scale = t.sum(1), np.abs(t).sum(1).astype(float)
    mt = None if m is None else gb.to_device(m)
    for tile in (None, gb.tiling(f64_pair=1), gb.tiling(2, 4, 32, f64_pair=1)):
        got = gb.nbody_rhs_f64(x, n, soft, 1.0 / n, mt, tile=tile).cpu().numpy()[3 * n:]
        err = np.abs((got.reshape(n, 3) - ref).astype(float))
        bound = (24 + n / 8) * 2.0 ** -53 * scale + n * 1e-320
        assert np.all(err <= bound), (err / np.maximum(bound, 1e-300)).max()


@pytest.mark.parametrize("thickness", [1.0, 1e-3, 1e-6, 1e-7, 1e-8, 1e-9, 1e-12, 1e-15, 1e-40])
@pytest.mark.parametrize("n", [2, 33, 129, 517])
def test_thin_systems(gb, torch_cuda, n, thickness):
    r = np.random.default_rng(n)
    for axis in range(3):
        x = r.standard_normal(6 * n)
        x[axis:3 * n:3] *= thickness
        _check(gb, x, n, 0.01)


@pytest.mark.parametrize("separation", [1e-2, 1e-5, 1e-8])
@pytest.mark.parametrize("n", [2, 40])
def test_pairs_far_closer_than_the_softening(gb, torch_cuda, n, separation):
    """All bodies on a line, a thousandth of the softening and less beside it."""
    r = np.random.default_rng(n)
    x = r.standard_normal(6 * n) * separation
    x[0:3 * n:3] = r.uniform(-0.2, 0.2, n)
    _check(gb, x, n, 0.25)


def test_heavy_thin_disc_in_a_light_halo(gb, torch_cuda):
    """The halo is as thick as the disc is wide, so the grid is; a disc body's force across the
    disc is 1e-9 of the one along it, or the halo's few bodies'."""
    n = 300
    r = np.random.default_rng(2)
    x = r.standard_normal(6 * n)
    x[2:3 * n:3] *= 1e-9
    m = np.full(n, 1.0 / n)
    for j, light in ((7, 1e-3), (150, 1e-13), (299, 0.0)):
        x[3 * j + 2], m[j] = 0.7, light
    _check(gb, x, n, 0.01, m)


def test_coordinates_below_the_grid(gb, torch_cuda):
    """A plane whose thickness is 1e-35: the grid has nothing of it."""
    n = 130
    r = np.random.default_rng(3)
    x = r.standard_normal(6 * n)
    x[2:3 * n:3] *= 1e-35
    x[3 * 5 + 2] = x[3 * 77 + 2] = 0.0
    _check(gb, x, n, 0.01)


def test_plane(gb, torch_cuda):
    """No component across an exact plane."""
    n = 517
    x = np.random.default_rng(4).standard_normal(6 * n)
    x[1:3 * n:3] = 0.375
    got = gb.nbody_rhs_f64(x, n, 0.01, 1.0 / n).cpu().numpy()
    assert np.all(got[3 * n:].reshape(n, 3)[:, 1] == 0.0)
    _check(gb, x, n, 0.01)


def test_many_close_pairs_on_one_side(gb, torch_cuda):
    """Sums beyond 128 bits: 20000 bodies in a point, 2^-12.6 of the extent from body 0 (the other
    bodies of its warp are farther from that point)."""
    n = 20033
    x = np.zeros(6 * n)
    p = x[: 3 * n].reshape(n, 3)
    p[:32, 0] = -0.01 * np.arange(32)
    p[32:-1, 0] = 2.0 ** -12.6
    p[-1, 0] = 0.6
    soft = 2.0 ** -14
    got = gb.nbody_rhs_f64(x, n, soft, 1.0).cpu().numpy()[3 * n:3 * n + 3]
    d = p[1:, 0].astype(np.longdouble)
    r2 = d * d + np.longdouble(soft * soft)
    t = d / (r2 * np.sqrt(r2))
    assert got[1] == got[2] == 0.0
    assert abs(got[0] - t.sum()) <= 16 * 2.0 ** -53 * np.abs(t).sum()

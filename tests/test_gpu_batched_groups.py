"""Small FP64 systems that share a CTA keep to their own shared memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spc", [2, 4])
def test_groups_do_not_touch_each_other(gb, torch_cuda, spc):
    """400 systems with separations over the whole fixed-point window (every row of each group's
    softening table): bit for bit the batch with one system per CTA."""
    r = np.random.default_rng(spc)
    sizes = r.integers(2, 128 // spc + 1, 400)
    xs = []
    for n in sizes:
        x = np.zeros(6 * n)
        d = r.standard_normal((n, 3))
        d *= (2.0 ** r.uniform(-9.0, 0.0, n) / np.linalg.norm(d, axis=1))[:, None]
        x[: 3 * n] = d.ravel()
        xs.append(x)
    x0 = np.concatenate(xs)
    out = []
    for g in (1, spc):
        b = gb.Batch("DOPRI5", sizes, 2.0 ** -10, precision="f64", max_attempts=40,
                     tiling=gb.GbBatchTiling(128, 1, 1, 0, g))
        assert b.geometry()["systems_per_cta"] == g
        b.start(x0, 0.0, 1e-3, 1e-9, 1e-9)
        b.advance()
        x, t = b.state()
        out.append((x.cpu().numpy(), t))
        b.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])

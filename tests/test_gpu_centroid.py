"""The mixed right-hand side's reference point: the centroid in its fixed order of additions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 127, 1023, 1024, 1025, 4096, 4097, 9001])
def test_centroid_in_order(gb, torch_cuda, n):
    """1024 chains (body t, t + 1024, ...), then a tree with halving distance: bit for bit, on
    both sides of the size up to which the cluster packs the bodies itself."""
    torch = torch_cuda
    x = np.random.default_rng(n).standard_normal(6 * n) + 3.0
    size = gb.lib().gb_nbody_mixed_workspace_bytes(n)
    work = torch.zeros(size, dtype=torch.uint8, device="cuda")
    gb.nbody_rhs_mixed(x, n, 0.05, 1.0 / n, work=work)
    got = work[(32 * n + 255) // 256 * 256:][:24].cpu().numpy().view(np.float64)
    p = x[: 3 * n].reshape(n, 3)
    v = np.zeros((1024, 3))
    for i in range(0, n, 1024):
        rows = p[i: i + 1024]
        v[: len(rows)] += rows
    st = 512
    while st:
        v[:st] += v[st: 2 * st]
        st //= 2
    np.testing.assert_array_equal(got, v[0] / n)
    # the packed positions: hi + lo parts of x - c
    packed = work[: 32 * n].cpu().numpy().view(np.float32).reshape(n, 8)
    d = p - got
    hi = d.astype(np.float32)
    np.testing.assert_array_equal(packed[:, :3], hi)
    np.testing.assert_array_equal(packed[:, 4:7], (d - hi).astype(np.float32))

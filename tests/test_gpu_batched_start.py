"""Start of a batch: a system's first step does not depend on the systems beside it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("sizes", [[2, 7, 41, 42], [43, 44, 300], [2, 42, 43, 5, 171, 41, 64, 1000]])
def test_first_step_of_a_system(gb, torch_cuda, precision, sizes):
    """Norms by a warp up to 42 bodies and by a cluster above: the same bits as the system alone in
    a batch."""
    xs = [gb.ic_plummer(n, 50 + n) for n in sizes]
    til = gb.GbBatchTiling(128, 2, 1, 0, 1)

    def first(ns, x):
        b = gb.Batch("DOPRI5", ns, 0.05, precision=precision, tiling=til)
        b.start(np.concatenate(x), 0.0, 0.1, 1e-9, 1e-9)
        b.sync()
        dt = [s["dt_initial"] for s in b.stats(per_system=True)["systems"]]
        b.close()
        return dt

    together = first(sizes, xs)
    assert all(np.isfinite(together)) and min(together) > 0.0
    assert together == [first([n], [x])[0] for n, x in zip(sizes, xs)]

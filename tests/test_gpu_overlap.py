"""Launches that overlap the kernel before them in the stream: a chain of dependent calls gives
the same bits as with a synchronisation after each call, and as the same chain captured."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chain(gb, torch, n, mixed, masses, after, steps=3):
    """steps of DOPRI5 by single calls, each reading what the ones before it wrote."""
    x = gb.to_device(np.random.default_rng(n).standard_normal(6 * n)).clone()
    nv = 6 * n
    m = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda") if masses else None
    f = gb.nbody_rhs_mixed if mixed else gb.nbody_rhs_f64
    kw = {"masses": m}
    if mixed:
        kw["work"] = torch.empty(gb.lib().gb_nbody_mixed_workspace_bytes(n), dtype=torch.uint8,
                                 device="cuda")
    ks = torch.zeros(7, nv, dtype=torch.float64, device="cuda")
    temp, err, target, xn = (torch.empty_like(x) for _ in range(4))
    tol = torch.full_like(x, 1e-9)

    def run():
        norms = []
        y, z = x.clone(), xn
        after()
        f(y, n, 0.05, 1.0 / n, out=ks[0], **kw)
        after()
        for _ in range(steps):
            for s in range(1, 7):
                gb.rk_stage("DOPRI5", s, 1e-3, y, ks, temp, nv)
                after()
                f(temp, n, 0.05, 1.0 / n, out=ks[s], **kw)
                after()
            gb.rk_update("DOPRI5", 1e-3, y, ks, z, err, nv)
            after()
            gb.rk_error_target(tol, tol, z, y, target, nv)
            after()
            norms.append(gb.rk_norm(err, target, nv))
            after()
            y.copy_(z)
            ks[0].copy_(ks[6])
            after()
        return y, torch.stack([v.reshape(()) for v in norms]), ks

    return run


# 304 / 305: the FP64 grids of 76 and 80 CTAs; 4863 ... 4865, 9729: on both sides of 4 CTAs per SM
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("masses", [False, True])
@pytest.mark.parametrize("n", [1, 64, 304, 305, 767, 768, 3001, 4097, 4864, 4865, 9729])
def test_chained_calls_equal_synchronised_ones(gb, torch_cuda, n, mixed, masses):
    torch = torch_cuda
    want = [t.clone() for t in chain(gb, torch, n, mixed, masses, torch.cuda.synchronize)()]
    run = chain(gb, torch, n, mixed, masses, lambda: None)
    for got in (run(), run()):
        for a, b in zip(want, got):
            assert torch.equal(a, b)


def test_captured_chain(gb, torch_cuda):
    torch = torch_cuda
    n = 257
    want = [t.clone() for t in chain(gb, torch, n, False, False, torch.cuda.synchronize)()]
    run = chain(gb, torch, n, False, False, lambda: None)
    run()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = run()
    for _ in range(2):
        g.replay()
    torch.cuda.synchronize()
    for a, b in zip(want, got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("n", [1, 304, 1365, 1366, 3001])
def test_leapfrog_equals_single_steps(gb, torch_cuda, n, precision):
    """1365 / 1366 bodies: 16 and 17 CTAs of the drift and kick kernels.  A step at a time starts
    from a fresh a(x), the same bits as the a(x) kept from the step before."""
    x0 = gb.to_device(np.random.default_rng(n).standard_normal(6 * n))
    ode, exe = gb.NBodyODE(n, 0.05, 1.0 / n), gb.Gb300Executor(precision=precision)
    step = gb.ParallelLeapfrogIntegrator.integrate
    want = x0
    for _ in range(6):
        want, _ = step(want, 0.0, 1 / 64, 1 / 64, ode, None, exe)
        torch_cuda.cuda.synchronize()
    got, _ = step(x0, 0.0, 6 / 64, 1 / 64, ode, None, exe)
    assert torch_cuda.equal(got, want)

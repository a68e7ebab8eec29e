"""CG(Prec::di) with tree sums at the sizes where its form changes: one block
(2048 cells), one cluster (16384), kernels per pass above, with 16-byte or,
for an x that is only 8-byte aligned, scalar updates. Against the oracle after
a fixed number of steps: the sums are in another order, and each step carries
their relative difference (a few units of 2^-53 times sqrt(N)) on, well below
1e-11 after a dozen steps."""
import numpy as np
import pytest

from test_gpu_sweeps import problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(2, 3, 5), (4, 16, 32), (2, 33, 32), (16, 32, 32), (5, 29, 113), (17, 33, 30)])
def test_cg_forms(engine, oracle, dims):
    P = problem(dims, False)
    steps = min(12, P.N // 2)
    xo, st = oracle.cg(P, maxit=steps, res_rat=1e-30, res_tol=1e-30)
    with engine.Session(*dims, P.h) as s:
        s.upload_matrix(P.A)
        kr = engine.CG(s)
        x = np.zeros(P.N)
        kr.solve(x, P.b.copy(), 1, steps, None, 1e-30, 1e-30)
        assert kr.last.status == engine.MAXITER and kr.last.iterations == steps
        assert len(s.history()) == steps
        assert kr.last.res0 == pytest.approx(st["res0"], rel=1e-12)
        assert np.linalg.norm(x - xo) <= 1e-11 * np.linalg.norm(xo)
        # the staleness window ends a run where the oracle's ends
        xs, ss = oracle.cg(P, maxit=200, res_rat=1e-30, res_tol=1e-30, stalecount=4)
        x[:] = 0.0
        kr.solve(x, P.b.copy(), 1, 200, None, 1e-30, 1e-30, 1.0, 4)
        if kr.last.status == engine.STALE and ss["iterations"] < 20:
            assert abs(kr.last.iterations - ss["iterations"]) <= 1
        # converges, and a converged start returns at once with x unchanged
        assert kr.solve(x, P.b.copy(), 1, 20000, None, 1e-9, 1e-30)
        y = x.copy()
        kr.solve(y, P.b.copy(), 1, 10, None, 1e-9, kr.last.res * 2.0)
        assert kr.last.status == engine.INITIAL and np.array_equal(x, y)


@pytest.mark.parametrize("dims", [(4, 16, 32), (17, 33, 30)])
@pytest.mark.parametrize("solver", ["cg", "gs", "engine"])
def test_unaligned_device_vectors(engine, oracle, dims, solver):
    """x and b as slices that start 8 bytes into an allocation: the results of
    aligned ones."""
    torch = pytest.importorskip("torch")
    P = problem(dims, False)
    out = []
    with engine.Session(*dims, P.h) as s:
        s.upload_matrix(P.A)
        for shift in (0, 1):
            x = torch.zeros(P.N + shift, dtype=torch.float64, device="cuda")[shift:]
            b = torch.zeros(P.N + shift, dtype=torch.float64, device="cuda")[shift:]
            b.copy_(torch.from_numpy(P.b))
            if solver == "engine":
                assert engine.Engine(s).solve(x, b, precision=engine.MIXED)
            else:
                kr = engine.CG(s) if solver == "cg" else engine.GaussSeidel(s)
                kr.solve(x, b, 1, 10, None, 1e-30, 1e-30)
            out.append(x.cpu().numpy())
    assert np.linalg.norm(out[0] - out[1]) <= 1e-12 * np.linalg.norm(out[0])

"""CG(Prec::di) with tree sums at the sizes where its form changes: one block
(2048 cells), one cluster (16384), kernels per pass above, with 16-byte or,
for an x that is only 8-byte aligned, scalar updates. Against the oracle after
a fixed number of steps: the sums are in another order, and each step carries
their relative difference (a few units of 2^-53 times sqrt(N)) on, well below
1e-11 after a dozen steps."""
import numpy as np
import pytest

from golden_util import bc_of
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
        x[:] = 0.0
        # converges, and a converged start returns at once with x unchanged
        assert kr.solve(x, P.b.copy(), 1, 20000, None, 1e-9, 1e-30)
        y = x.copy()
        kr.solve(y, P.b.copy(), 1, 10, None, 1e-9, kr.last.res * 2.0)
        assert kr.last.status == engine.INITIAL and np.array_equal(x, y)


def window_margin(st, stalecount):
    """Smallest relative distance of any residual from the comparison of the
    staleness window that decides on it (cg.cpp:138-160)."""
    win = [1e24] * (stalecount - 1) + [st["res0"]]
    margin = np.inf
    for r in st["hist"]:
        if all(r >= w for w in win):
            return min(margin, r / max(win) - 1.0)
        margin = min(margin, max(win) / r - 1.0)
        win = win[1:] + [r]
    return 0.0   # never stale


@pytest.mark.parametrize("dims,stalecount", [
    ((2, 3, 5), 1), ((2, 3, 5), 2), ((4, 16, 32), 1), ((4, 16, 32), 6),      # one block
    ((2, 33, 32), 1), ((16, 32, 32), 1), ((16, 32, 32), 6), ((5, 29, 113), 4),   # one cluster
    ((17, 33, 30), 1), ((17, 33, 30), 3), ((17, 33, 31), 6)])                # kernels per pass
def test_cg_staleness_window(engine, oracle, dims, stalecount):
    """A run that goes stale ends there, in the oracle's iteration: the
    residuals differ by the order of the sums (below 1e-7 after these steps),
    the comparisons that end the run are further apart than 1e-4."""
    P = problem(dims, False)
    xo, st = oracle.cg(P, maxit=200, res_rat=1e-30, res_tol=1e-30, stalecount=stalecount, hist=True)
    assert st["status"] == 2 and window_margin(st, stalecount) > 1e-4
    with engine.Session(*dims, P.h) as s:
        s.upload_matrix(P.A)
        kr = engine.CG(s)
        x = np.zeros(P.N)
        assert not kr.solve(x, P.b.copy(), 1, 200, None, 1e-30, 1e-30, 1.0, stalecount)
        assert kr.last.status == engine.STALE
        assert kr.last.iterations == st["iterations"]
        assert np.allclose(s.history(), st["hist"], rtol=1e-7, atol=0.0)
        assert np.linalg.norm(x - xo) <= 1e-7 * np.linalg.norm(xo)


@pytest.mark.parametrize("n", [8, 12, 13, 20, 25, 27])   # 512 to 19683 cells: every form
@pytest.mark.parametrize("periodic", [1, 2, 4, 7])
def test_cg_forms_periodic(engine, oracle, n, periodic):
    """Neighbours across a periodic face: in the block's own shared memory, in
    another block's, or in global memory."""
    P = oracle.Problem(0, 3, n=n, periodic=periodic)
    xo, st = oracle.cg(P, maxit=12, res_rat=1e-30, res_tol=1e-30, hist=True)
    with engine.Session(*P.dims, P.h, bc=bc_of(P)) as s:
        s.upload_matrix(P.A)
        kr = engine.CG(s)
        x = np.zeros(P.N)
        kr.solve(x, P.b.copy(), 1, 12, None, 1e-30, 1e-30)
        assert kr.last.iterations == 12
        assert np.allclose(s.history(), st["hist"], rtol=1e-9, atol=0.0)
        assert np.linalg.norm(x - xo) <= 1e-9 * np.linalg.norm(xo)


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

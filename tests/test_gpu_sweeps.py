"""The one-launch lexicographic sweeps (IC0, IC2, Gauss-Seidel) on grids that
cut their 8 x 8 column tiles unevenly, with columns shorter and longer than
the march's skew and on one k plane: bit for bit the oracle's results after a
fixed number of steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(7, 9, 5), (8, 8, 8), (9, 17, 33), (24, 16, 31), (2, 30, 67), (33, 3, 2), (17, 25, 1), (40, 41, 32),
        (1, 20, 33), (19, 1, 33), (1, 1, 44), (3, 5, 33)]


def problem(dims, convect, solids=0.1):
    import flow
    g = np.random.default_rng(sum(dims))
    nx, ny, nz = dims
    bc = [0] * 6
    bc[5 if nz > 1 else 3] = 1
    h = 1.0 / max(dims)
    col = g.random(dims)
    solid = (g.random(dims) < solids).astype(np.uint8)
    A = flow.assemble_mix(dims, h, bc, col, 100.0, 1.0, solid=solid)
    if convect:  # first-order upwind convection along x: a non-symmetric matrix
        ok = (solid[1:] == 0) & (solid[:-1] == 0)
        F = np.zeros(dims)
        F[1:] = 0.002 * convect * h * ok
        A["w"] = A["w"] + F.reshape(-1)
        A["c"] = A["c"] + F.reshape(-1)
        A["ci"] = 1.0 / A["c"]
    b = (g.random(dims) - 0.5) * (solid == 0)
    P = flow.StepProblem(dims, h, A, b.reshape(-1))
    P.ci = A["ci"]
    P.solid = solid.reshape(-1)
    P.periodic = 0
    return P


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("solver,prec,steps,convect", [("cg", "ic0", 4, False), ("cg", "ic2", 4, False),
                                                       ("bicgs", "ic2", 2, True), ("gs", "di", 3, False),
                                                       ("gs", "di", 3, True)])
def test_sweeps_bit_exact(engine, oracle, dims, solver, prec, steps, convect):
    P = problem(dims, convect)
    xo, _ = oracle.cg(P, solver=solver, prec=prec, maxit=steps, res_rat=1e-30, res_tol=1e-30)
    assert np.all(np.isfinite(xo))
    with engine.Session(*dims, P.h) as s:
        s.upload_matrix(P.A)
        s.upload_ci(P.ci)
        kr = {"cg": engine.CG, "bicgs": engine.BiCGS, "gs": engine.GaussSeidel}[solver]
        kr = kr(s, exact_sums=True) if solver == "gs" else kr(s, prec=prec, exact_sums=True)
        x = np.zeros(P.N)
        for _ in range(2):  # the second solve finds the exchange words of the first
            x[:] = 0.0
            kr.solve(x, P.b.copy(), 1, steps, None, 1e-30, 1e-30)
            assert np.array_equal(x, xo)


@pytest.mark.parametrize("dims", [(1, 700, 800), (700, 1, 800), (1, 1, 200000), (3, 400, 400)])
@pytest.mark.parametrize("solver,prec", [("cg", "ic2"), ("gs", "di")])
def test_thin_grids_take_memory_by_their_cells(engine, dims, solver, prec):
    """The sweeps' storage holds the columns that exist: a grid of one or few
    columns along i or j takes no more than 1.5 times the memory per cell of
    one whose tiles are full (8, 8, 64 and 2.7 times with whole tiles)."""
    torch = pytest.importorskip("torch")

    def mem(d):
        n = d[0] * d[1] * d[2]
        rho = torch.ones(n, dtype=torch.float64, device="cuda")
        solid = torch.zeros(n, dtype=torch.uint8, device="cuda")
        b = torch.sin(torch.arange(n, dtype=torch.float64, device="cuda"))
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        with engine.Session(*d, 1.0) as s:
            s.assemble_pressure(rho, solid)
            kr = engine.GaussSeidel(s) if solver == "gs" else engine.CG(s, prec=prec)
            torch.cuda.synchronize()
            free = torch.cuda.mem_get_info()[0]
            kr.solve(x, b, 1, 2, None, 1e-30, 1e-30)
            torch.cuda.synchronize()
            return (free - torch.cuda.mem_get_info()[0]) / n
    assert mem(dims) <= 1.5 * mem((40, 40, 800))

"""The engine's hierarchy as the caller sees it: which levels there are, what
an explicit coarse_max does, and that a solve depends on its matrix and its
options alone, not on the calls before it on the same session."""
import numpy as np
import pytest

from test_gpu_sweeps import problem

pytestmark = pytest.mark.gpu


def solve(engine, E, P, **kw):
    x = np.zeros(P.N)
    assert E.solve(x, P.b.copy(), tol=1e-9, **kw)
    assert np.linalg.norm(x) > 0.0
    return x


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("before", [None, 0, 4096])
def test_explicit_coarse_max_is_a_limit(engine, precision, before):
    """20x16x18 coarsens to 720 and 100 cells: asked for at most 512 the
    hierarchy goes down to 100, whatever an earlier call on the session asked
    for (None: no earlier call; 0: the engine's choice)."""
    P = problem((20, 16, 18), False)
    with engine.Session(*P.dims, P.h) as s:
        s.upload_matrix(P.A)
        E = engine.Engine(s)
        ref = solve(engine, E, P, precision=precision, coarse_max=511)
        assert s.levels(1) == [(20, 16, 18), (10, 8, 9), (5, 4, 5)]
    with engine.Session(*P.dims, P.h) as s:
        s.upload_matrix(P.A)
        E = engine.Engine(s)
        if before is not None:
            solve(engine, E, P, precision=precision, coarse_max=before)
        x = solve(engine, E, P, precision=precision, coarse_max=512)
        assert E.last.levels == 3
        assert np.array_equal(x, ref)


@pytest.mark.parametrize("dims,coarse_max,levels", [
    ((20, 16, 18), 0, [(20, 16, 18), (10, 8, 9)]),                    # 720 cells are the coarsest
    ((20, 16, 18), 100, [(20, 16, 18), (10, 8, 9), (5, 4, 5)]),
    ((17, 33, 30), 0, [(17, 33, 30), (9, 17, 15), (5, 9, 8)]),        # padded rows
    ((66, 71, 1), 0, [(66, 71, 1), (33, 36, 1), (17, 18, 1)]),        # 2-D, padded
    ((24, 18, 17), 0, [(24, 18, 17), (12, 9, 9), (6, 5, 5)]),         # 972 cells on level 1: coarsened
    ((36, 33, 38), 0, [(36, 33, 38), (18, 17, 19), (9, 9, 10)]),      # 810 cells on level 2: the coarsest
    ((41, 31, 35), 0, [(41, 31, 35), (21, 16, 18), (11, 8, 9)]),      # 792 cells, stored as 880
    ((12, 8, 8), 0, [(12, 8, 8)]),
    ((10, 10, 10), 0, [(10, 10, 10), (5, 5, 5)]),
    ((31, 32, 35), 4096, [(31, 32, 35), (16, 16, 18), (8, 8, 9)]),
    ((64, 64, 2), 0, [(64, 64, 2), (32, 32, 1), (16, 16, 1)]),        # thin
    ((9, 5, 7), 0, [(9, 5, 7)]),
])
def test_levels_are_those_of_the_hierarchy(engine, dims, coarse_max, levels):
    """pbg_levels and pbg_result.levels: the levels that are solved on, with
    the extents of the caller's grid halved (no pad cells)."""
    P = problem(dims, False, solids=0.0)
    with engine.Session(*dims, P.h) as s:
        s.upload_matrix(P.A)
        E = engine.Engine(s)
        for precision in (0, 1):
            solve(engine, E, P, precision=precision, coarse_max=coarse_max)
            assert E.last.levels == len(levels)
            assert s.levels(1) == levels


@pytest.mark.parametrize("dims", [(16, 16, 18), (16, 18, 17), (30, 31, 6), (66, 70, 1)])
def test_fp64_solve_does_not_depend_on_a_mixed_one_before(engine, dims):
    """The hierarchy that a mixed solve leaves serves FP64 solves too: its
    rows, and with them the bits, are the same for both."""
    P = problem(dims, False)
    with engine.Session(*dims, P.h) as s:
        s.upload_matrix(P.A)
        ref = solve(engine, engine.Engine(s), P, precision=engine.FP64)
    with engine.Session(*dims, P.h) as s:
        s.upload_matrix(P.A)
        E = engine.Engine(s)
        solve(engine, E, P, precision=engine.MIXED)
        assert np.array_equal(solve(engine, E, P, precision=engine.FP64), ref)


def relres(oracle, P, x):
    return np.linalg.norm(oracle.resid(P, x, P.b)) / np.linalg.norm(P.b)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dims", [
    (17, 17, 19), (24, 26, 7), (66, 71, 1),                        # padded rows, k and j
    (64, 65, 2), (48, 50, 5), (60, 61, 9), (5000, 1, 1), (900, 9, 1), (2100, 2, 1)])   # thin
@pytest.mark.parametrize("convect", [0, 0.02])   # weak: the refinement around the symmetric part converges
def test_padded_and_thin_grids_converge(engine, oracle, dims, precision, convect):
    """The solution in the caller's rows: its FP64 residual, formed on the
    host, with symmetric matrices and, by the residual of the seven arrays,
    non-symmetric ones."""
    P = problem(dims, convect, solids=0.1 if min(dims) > 2 else 0.0)   # no pockets on 1-D and 2-D grids
    x = np.zeros(P.N)
    with engine.Session(*dims, P.h) as s:
        s.upload_matrix(P.A)
        assert s.symmetric() == (convect == 0)
        E = engine.Engine(s)
        assert E.solve(x, P.b.copy(), tol=1e-9, precision=precision)
        assert relres(oracle, P, x) <= 1.0001e-9
        assert E.last.relres == pytest.approx(relres(oracle, P, x), rel=1e-3, abs=1e-13)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("convect", [0, 0.02])   # weak: the refinement around the symmetric part converges
@pytest.mark.parametrize("dims", [(17, 17, 19), (66, 71, 1)])
def test_refresh_of_padded_rows(engine, oracle, dims, convect, precision):
    """A changed matrix of the same shape, uploaded into the buffers that the
    hierarchy's padded copy was made from: the bits of a fresh session."""
    P, Q = problem(dims, convect), problem(dims, convect)
    for k in "cwesnbt":
        Q.A[k] = 3.0 * P.A[k]
    Q.A["c"] = Q.A["c"] + 0.01 * P.A["c"].max()
    with engine.Session(*dims, P.h) as s:
        s.upload_matrix(Q.A)
        ref = solve(engine, engine.Engine(s), Q, precision=precision)
    with engine.Session(*dims, P.h) as s:
        s.upload_matrix(P.A)
        E = engine.Engine(s)
        solve(engine, E, P, precision=precision)
        s.upload_matrix(Q.A)
        x = solve(engine, E, Q, precision=precision)
    assert np.array_equal(x, ref)
    assert relres(oracle, Q, x) <= 1.0001e-9


@pytest.mark.parametrize("dims", [(1, 1, 31), (3, 11, 1), (1, 1, 127), (43, 3, 1), (8, 9, 10), (10, 11, 10), (11, 12, 16),
                                  (15, 16, 17)])
def test_dense_inverse_of_the_whole_grid(engine, oracle, dims):
    """A grid that is its own coarsest level (31 to 4080 cells: block steps of
    32 pivots and column tiles of 128 with remainders, CTAs with one and with
    several column tiles): the dense inverse solves it in one FCG iteration,
    two where rounding leaves the first above the tolerance."""
    P = problem(dims, False, solids=0.0)
    x = np.zeros(P.N)
    with engine.Session(*dims, P.h) as s:
        s.upload_matrix(P.A)
        E = engine.Engine(s)
        assert E.solve(x, P.b.copy(), tol=1e-10, precision=engine.FP64, coarse_max=4096)
        assert s.levels(1) == [dims] and E.last.iterations <= 2
    assert relres(oracle, P, x) <= 1.0001e-10


def device_bytes(f):
    """Device memory that f() takes and keeps (allocations of the library)."""
    torch = pytest.importorskip("torch")
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    f()
    torch.cuda.synchronize()
    return free - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("dims,times", [((512, 512, 2), 1.5), ((512, 512, 5), 1.5), ((300000, 1, 1), 3.0),
                                        ((60000, 9, 1), 2.2)])
def test_thin_grids_are_not_padded(engine, dims, times):
    """Rows that whole vectors would lengthen by more than a seventh stay as
    they are: per cell, a thin grid takes the memory of one that needs no
    padding, times what its slower coarsening leaves on the levels below (an
    eighth to a half of a level's cells), where padding took 2.6, 1.8, 10 and
    2.5 times."""
    import torch

    def mem(d):
        n = d[0] * d[1] * d[2]
        rho = torch.ones(n, dtype=torch.float64, device="cuda")
        solid = torch.zeros(n, dtype=torch.uint8, device="cuda")
        b = torch.sin(torch.arange(n, dtype=torch.float64, device="cuda"))
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        with engine.Session(*d, 1.0) as s:
            s.assemble_pressure(rho, solid)
            E = engine.Engine(s)
            return device_bytes(lambda: E.solve(x, b, precision=engine.MIXED, max_sweeps=1, max_iter=2)) / n
    assert mem(dims) <= times * mem((512, 512, 4))

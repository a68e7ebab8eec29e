"""Calls that find too little device memory fail with an error and leave the
session usable: the same call after memory is free again gives the result of a
session that never failed."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def give_memory_back():
    yield
    import torch
    torch.cuda.empty_cache()   # torch keeps what it freed

DIMS = (160, 152, 161)   # 3.9 M cells: 31 MB an FP64 array


@pytest.mark.parametrize("kind", ["engine_fp64", "engine_mixed", "cg", "cg_ic2", "bicgs", "batch"])
def test_failed_allocation_leaves_the_session_usable(engine, kind):
    torch = pytest.importorskip("torch")
    n = DIMS[0] * DIMS[1] * DIMS[2]
    rho = torch.ones(n, dtype=torch.float64, device="cuda")
    rho[: n // 3] = 100.0
    solid = torch.zeros(n, dtype=torch.uint8, device="cuda")
    b = torch.sin(torch.arange(n, dtype=torch.float64, device="cuda"))
    x = torch.zeros(n, dtype=torch.float64, device="cuda")

    def session():
        s = engine.Session(*DIMS, 1.0 / 160)
        s.assemble_pressure(rho, solid)
        return s

    def solve(s):
        x.zero_()
        if kind.startswith("engine"):
            E = engine.Engine(s)
            E.solve(x, b, precision=engine.MIXED if kind == "engine_mixed" else engine.FP64, max_iter=3, max_sweeps=2)
        else:
            kr = engine.BiCGS(s) if kind == "bicgs" else engine.CG(s, prec="ic2" if kind == "cg_ic2" else "di")
            kr.solve(x, b, 1, 3, None, 1e-30, 1e-30)
        torch.cuda.synchronize()
        return x.clone()

    def batch(_):
        with engine.Batch(precision=engine.MIXED, slots=2) as B:
            i = B.add(DIMS, 1.0 / 160, rho=rho, solid=solid, b=b)
            B.set_x(i)
            B.solve([i], tol=1e-3)
            B.get_x(i, x)
        torch.cuda.synchronize()
        return x.clone()

    run = batch if kind == "batch" else solve
    with session() as s:
        ref = run(s)
    with session() as s:
        failed = 0
        for left in (64, 128, 192, 288, 400):   # MB: the call ends at one array or another
            torch.cuda.synchronize()
            torch.cuda.empty_cache()
            hold = torch.empty(torch.cuda.mem_get_info()[0] - (left << 20), dtype=torch.uint8, device="cuda")
            try:
                run(s)
            except engine.PbgError as e:
                assert "out of memory" in str(e)
                failed += 1
            del hold
        torch.cuda.empty_cache()   # torch keeps what it freed
        assert failed >= 1
        assert torch.equal(run(s), ref)


def test_gauss_seidel_without_room_for_its_sweep(engine):
    """The one-launch sweep's operands (72 bytes a cell, 281 MB here) do not
    fit: the solve goes plane by plane, with the same result."""
    torch = pytest.importorskip("torch")
    n = DIMS[0] * DIMS[1] * DIMS[2]
    rho = torch.ones(n, dtype=torch.float64, device="cuda")
    rho[: n // 3] = 100.0
    solid = torch.zeros(n, dtype=torch.uint8, device="cuda")
    b = torch.sin(torch.arange(n, dtype=torch.float64, device="cuda"))
    out, launches = [], []
    for left in (None, 200):
        with engine.Session(*DIMS, 1.0 / 160) as s:
            s.assemble_pressure(rho, solid)
            x = torch.zeros(n, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            torch.cuda.empty_cache()
            hold = None
            if left:
                hold = torch.empty(torch.cuda.mem_get_info()[0] - (left << 20), dtype=torch.uint8, device="cuda")
            before = engine.launch_count()
            engine.GaussSeidel(s).solve(x, b, 1, 2, None, 1e-30, 1e-30)
            launches.append(engine.launch_count() - before)
            out.append(x.cpu())
            del hold
    assert torch.equal(out[0], out[1])
    assert launches[0] < 20 < launches[1]

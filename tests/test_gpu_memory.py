"""Calls that find too little device memory fail with an error and leave the
session usable: the same call after memory is free again gives the result of a
session that never failed."""
import pytest

pytestmark = pytest.mark.gpu

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
        torch.cuda.empty_cache()
        assert failed >= 1
        assert torch.equal(run(s), ref)

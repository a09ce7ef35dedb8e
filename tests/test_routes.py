"""cuasr_b200_last_route names the kernel a call launched, not one its arguments suggest."""
import subprocess
import sys

import pytest

from cuasr_b200 import Arguments, DType, Layout, Op, Srgemm, SrgemmSplitKParallel, Status, device_status, srgemm_path

COL, ROW = Layout.COLUMN_MAJOR, Layout.ROW_MAJOR


def test_no_route_before_the_first_call():
    out = subprocess.run([sys.executable, "-c", "from cuasr_b200 import _lib; print(_lib.load().cuasr_b200_last_route())"],
                         capture_output=True, text=True, check=True).stdout
    assert out.strip() == "b'none'"


def run(op, m, n, k, workspace=False, offset=0, slices=1):
    """One product of zeros on `op`'s layouts (row, column, row); returns the route.  offset: elements in front of A."""
    import torch
    dt = torch.float64 if op.dtype == DType.F64 else torch.float32
    A, B, D = (torch.zeros(s, dtype=dt, device="cuda") for s in (m * k + offset, k * n, m * n))
    args = Arguments((m, n, k), (A.data_ptr() + offset * A.element_size(), k), (B, k), (None, n), (D, n), (), slices)
    need = op.get_workspace_size(args)
    if workspace and need == 0:
        need = op.get_optional_workspace_size(args)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda") if need else None
    assert op(args, ws) == Status.kSuccess
    assert device_status() == 0
    return op.last_route()


@pytest.mark.gpu
def test_routes(cuda_device):
    import torch
    minplus = Srgemm(Op.MINIMUM, Op.PLUS, DType.F32, ROW, COL, ROW)
    route = run(minplus, 256, 256, 256)
    assert route.startswith("product ") and "a=tma b=tma" in route and "tickets=0" in route, route
    assert "a=gather b=tma" in run(minplus, 256, 256, 256, offset=1)
    assert "a=copy+tma b=tma" in run(minplus, 256, 256, 256, workspace=True, offset=1)
    # a sum keeps the cutting that was asked for: the pieces meet through tickets in the workspace
    sums = SrgemmSplitKParallel(Op.PLUS, Op.MULTIPLIES, DType.F32, ROW, COL, ROW)
    route = run(sums, 256, 256, 4096, slices=8)
    assert "tile=128x128" in route and "pieces=8 tickets=1" in route, route
    assert run(Srgemm(Op.MINIMUM, Op.PLUS, DType.F64, ROW, COL, ROW), 4096, 2048, 2048).startswith("screened pieces=1 or product ")
    # fp64 minima below the size where the screen pays
    assert run(Srgemm(Op.MINIMUM, Op.PLUS, DType.F64, ROW, COL, ROW), 128, 128, 128).startswith("product ")
    n = 64
    A, D = torch.zeros(n * n, device="cuda"), torch.zeros(n * n, device="cuda")
    P = torch.zeros(n * n, dtype=torch.int32, device="cuda")
    assert srgemm_path(minplus, (n, n, n), (A, n), (A, n), (D, n), (P, n)) == Status.kSuccess
    assert minplus.last_route().startswith("path ")

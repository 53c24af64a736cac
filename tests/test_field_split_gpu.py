"""Point counts at which a field call is cut into pieces of segments and thickness
nodes: against the oracle at the parity bar (1e-12), and against the same call in a
captured graph, which evaluates in one piece."""
import numpy as np
import pytest

from conftest import gradient_band, rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-12


def make(ccoil, coils, points, seed=91):
    from ccoil_b200 import workloads
    rows = workloads.coil_rows_mixed(coils, seed=seed)
    return rows, workloads.coils_from_rows(rows, 5.0), workloads.points_cube(points, seed=seed + 1)


@pytest.mark.parametrize("coils,points", [(1, 1), (1, 37), (3, 129), (40, 5), (7, 1001)])
@pytest.mark.parametrize("field", [0, 1, 2, 3])
def test_pieces_match_oracle(ccoil, oracle, coils, points, field):
    rows, c, pts = make(ccoil, coils, points)
    plan = ccoil.CoilGroup(c, ccoil.PrecisionFactor(5.0)).plan(field)
    got = plan(pts)
    plan.close()
    e = rel_err(got, oracle.group_fields(rows, pts, field, pf=5.0))
    if field == 3:
        e = e[~gradient_band(rows, pts)]
    assert e.max(initial=0) < TOL, e.max()


@pytest.mark.parametrize("points", [1, 100, 4097, 60001])
@pytest.mark.parametrize("field", [1, 3])
def test_pieces_match_captured_call(ccoil, points, field):
    import torch
    _, c, pts = make(ccoil, 12, points)
    plan = ccoil.FieldPlan([k.struct() for k in c], field)
    x = torch.from_numpy(pts).cuda()
    eager = plan(x)
    out = torch.empty_like(eager)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        plan(x, out=out)
    for _ in range(2):
        out.fill_(float("nan"))
        g.replay()
        torch.cuda.synchronize()
        assert rel_err(out.cpu().numpy(), eager.cpu().numpy()).max() < TOL
    plan.close()


@pytest.mark.parametrize("mode", ["FP32_COMPENSATED", "FP32_REFINED"])
@pytest.mark.parametrize("points", [3, 700, 20011])
def test_pieces_in_fp32_modes(ccoil, mode, points):
    # the bars of test_fields32_gpu.py; points inside the windings included
    rows, c, pts = make(ccoil, 10, points)
    pts[::2] = 0.5 + 0.5 * pts[::2]
    for field in (0, 1, 3):
        got, ref = (ccoil.FieldPlan([k.struct() for k in c], field, ccoil.PrecisionMode[m])(pts)
                    for m in (mode, "FP64"))
        e = rel_err(got, ref)
        if field == 3:
            e = e[~gradient_band(rows, pts)]
        assert e.max() < 1e-5, (field, e.max())
        assert np.median(e) < 3e-7, (field, np.median(e))

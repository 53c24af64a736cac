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


@pytest.mark.parametrize("coils,points,lanes", [(24, 300, 32), (24, 1184, 32), (24, 1185, 16), (64, 2368, 16),
                                                (64, 2369, 8), (8, 18943, 8), (2, 20000, 8), (3, 40000, 4)])
def test_call_in_one_piece_shares_points_among_lanes(ccoil, coils, points, lanes):
    """A captured FP64 call, and one whose pieces' allocation fails, run in one piece:
    then only lanes per point fill the machine.  The lanes order a point's sums, so the
    automatic choice shows in the bits: those of the expected lane count."""
    import torch
    _, c, pts = make(ccoil, coils, points)
    plan = ccoil.FieldPlan([k.struct() for k in c], 1)
    x = torch.from_numpy(pts).cuda()

    def captured(n):
        out = torch.full((points, 3), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            plan(x, lanes=n, out=out)
        g.replay()
        torch.cuda.synchronize()
        return out

    auto, want = captured(0), captured(lanes)
    assert not torch.equal(captured(1), want)  # the bits do tell lane counts apart
    assert torch.equal(auto, want)
    assert ccoil.lib().ccoil_inject_allocation_failures(1) == 0
    try:
        failed = plan(x)
    finally:
        ccoil.lib().ccoil_inject_allocation_failures(0)
    assert torch.equal(failed, want)
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


def test_more_near_pairs_than_the_list_holds(ccoil):
    # the allocation-free entry point's list is far shorter than these points' pairs
    # (every point lies in the winding box of all 12 coils); the plan's holds them
    import ctypes
    import torch
    coils = [ccoil.Coil(0.1, 0.02, 0.05, 10 + i, 1.0 + i) for i in range(12)]
    g = np.random.default_rng(5)
    n = 40003
    r, phi = g.uniform(0.095, 0.125, n), g.uniform(0.0, 2.0 * np.pi, n)
    pts = np.stack([r * np.cos(phi), r * np.sin(phi), g.uniform(-0.03, 0.03, n)], axis=1)
    x = torch.from_numpy(pts).cuda()
    L = ccoil.lib()
    fn = L.ccoil_fields_fp32c_static
    fn.argtypes = [ctypes.POINTER(ccoil._lib.CoilStruct), ctypes.c_int, ctypes.c_void_p, ctypes.c_longlong,
                   ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
    structs = (ccoil._lib.CoilStruct * len(coils))(*[c.struct() for c in coils])
    for field, width in ((0, 3), (1, 3), (3, 9)):
        want = ccoil.FieldPlan(list(structs), field, ccoil.PrecisionMode.FP32_COMPENSATED)(x).cpu().numpy()
        out = torch.full((n, width), float("nan"), dtype=torch.float64, device="cuda")
        assert fn(structs, len(coils), ctypes.c_void_p(x.data_ptr()), n, field, ctypes.c_void_p(out.data_ptr()),
                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0, L.ccoil_last_error_message()
        assert rel_err(out.cpu().numpy(), want).max() < TOL, field


@pytest.mark.parametrize("count,n", [(32, 8193), (33, 7944), (77, 3405)])
def test_overflowing_list_over_groups_of_32_segments(ccoil, count, n):
    # just more pairs than the allocation-free entry point's list holds (2^18), over
    # segment counts around whole groups of 32; every second coil is far away
    import ctypes
    import torch
    coils = [ccoil.Coil(0.1, 0.02, 0.05, 10 + i, 1.0 + i, coordinate_position=(0.0, 0.0, 3.0 * (i % 2)))
             for i in range(2 * count)]
    g = np.random.default_rng(7)
    r, phi = g.uniform(0.095, 0.125, n), g.uniform(0.0, 2.0 * np.pi, n)
    x = torch.from_numpy(np.stack([r * np.cos(phi), r * np.sin(phi), g.uniform(-0.03, 0.03, n)], axis=1)).cuda()
    fn = ccoil.lib().ccoil_fields_fp32c_static
    fn.argtypes = [ctypes.POINTER(ccoil._lib.CoilStruct), ctypes.c_int, ctypes.c_void_p, ctypes.c_longlong,
                   ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
    structs = (ccoil._lib.CoilStruct * len(coils))(*[c.struct() for c in coils])
    want = ccoil.FieldPlan(list(structs), 1, ccoil.PrecisionMode.FP32_COMPENSATED)(x).cpu().numpy()
    out = torch.full((n, 3), float("nan"), dtype=torch.float64, device="cuda")
    assert fn(structs, len(coils), ctypes.c_void_p(x.data_ptr()), n, 1, ctypes.c_void_p(out.data_ptr()),
              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    assert rel_err(out.cpu().numpy(), want).max() < TOL


def test_batch_near_pairs_beyond_the_list_and_repeatable(ccoil):
    # one system whose points all lie in the winding boxes of 12 coils: 4.3 million
    # pairs over two fields, more than the batch's list; a second, shorter system
    coils = [ccoil.Coil(0.1, 0.02, 0.05, 10 + i, 1.0 + i) for i in range(12)]
    g = np.random.default_rng(6)

    def ring(n):
        r, phi = g.uniform(0.095, 0.125, n), g.uniform(0.0, 2.0 * np.pi, n)
        return np.stack([r * np.cos(phi), r * np.sin(phi), g.uniform(-0.03, 0.03, n)], axis=1)

    for systems in ([(coils, ring(180001)), (coils[:5], ring(77))], [(coils, ring(3001)), (coils[3:], ring(1))]):
        plan = ccoil.BatchPlan(systems, fields=("A", "B"), precision=ccoil.PrecisionMode.FP32_COMPENSATED)
        first = {f: v.clone() for f, v in plan.run().items()}
        again = plan.run()
        for f, field in (("A", 0), ("B", 1)):
            assert bool((first[f] == again[f]).all()), f
            for (c, pts), got in zip(systems, plan.split(first[f])):
                want = ccoil.FieldPlan([k.struct() for k in c], field, ccoil.PrecisionMode.FP32_COMPENSATED)(pts)
                assert rel_err(got.cpu().numpy(), want).max() < TOL, f
        plan.close()


def stack(ccoil, count):
    """RECTANGULAR coils 0.5 mm apart: a point on the winding lies in up to 48 boxes."""
    return [ccoil.Coil(0.1, 0.01, 0.004, 10 + i, 1.0, coordinate_position=(0.0, 0.0, 0.0005 * i))
            for i in range(count)]


def on_the_winding(n, height, seed=8):
    g = np.random.default_rng(seed)
    r, phi = g.uniform(0.092, 0.118, n), g.uniform(0.0, 2.0 * np.pi, n)
    return np.stack([r * np.cos(phi), r * np.sin(phi), g.uniform(0.0, height, n)], axis=1)


@pytest.mark.parametrize("count,points", [(1, 37), (2, 5), (9, 1), (70, 1), (70, 37), (70, 3001)])
@pytest.mark.parametrize("field", [0, 1, 3])
def test_points_in_many_near_boxes(ccoil, count, points, field):
    # runs of 1 to 48 pairs a point; every pair is FP64 (bars of test_fields32_gpu.py)
    import ctypes
    import torch
    coils, pts = stack(ccoil, count), on_the_winding(points, 0.0005 * count)
    structs = [c.struct() for c in coils]
    plan = ccoil.FieldPlan(structs, field, ccoil.PrecisionMode.FP32_COMPENSATED)
    got, again = plan(pts), plan(pts)
    want = ccoil.FieldPlan(structs, field)(pts)
    e = rel_err(got, want)
    assert np.array_equal(got, again)
    assert e.max() < 1e-5 and np.median(e) < 3e-7, (e.max(), np.median(e))
    # the allocation-free entry point, whose list is shorter: 137,000 pairs of 3,001 points
    x = torch.from_numpy(pts).cuda()
    out = torch.full((points, plan.width), float("nan"), dtype=torch.float64, device="cuda")
    fn = ccoil.lib().ccoil_fields_fp32c_static
    fn.argtypes = [ctypes.POINTER(ccoil._lib.CoilStruct), ctypes.c_int, ctypes.c_void_p, ctypes.c_longlong,
                   ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
    assert fn((ccoil._lib.CoilStruct * count)(*structs), count, x.data_ptr(), points, field, out.data_ptr(),
              torch.cuda.current_stream().cuda_stream) == 0
    assert rel_err(out.cpu().numpy(), got).max() < TOL
    if field != 3:
        batch = ccoil.BatchPlan([(coils, pts), (coils[:1], pts[:1])], fields=("A", "B", "G"),
                                precision=ccoil.PrecisionMode.FP32_COMPENSATED)
        res = batch.run()["AB"[field]][:points].cpu().numpy()
        batch.close()
        e = rel_err(res, want)
        assert e.max() < 1e-5 and np.median(e) < 3e-7, (e.max(), np.median(e))


def test_pairs_of_one_point_run_side_by_side(ccoil):
    """One point in 48 of 64 boxes against one in none: 1.1 times the time with a warp
    per pair, 10 times with one warp for all.  Bar 4."""
    import torch
    plan = ccoil.FieldPlan([c.struct() for c in stack(ccoil, 64)], 1, ccoil.PrecisionMode.FP32_COMPENSATED)

    def time(x, y, z):
        p = torch.tensor([[x, y, z]], dtype=torch.float64, device="cuda")
        best = float("inf")
        for _ in range(20):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            plan(p)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    far, near = time(0.0, 0.0, 0.016), time(0.105, 0.0, 0.016)
    plan.close()
    assert near < 4.0 * far, (near, far)


def test_batch_overflow_with_segments_shared_in_a_warp(ccoil):
    # 33 coils in one place: listed a warp per point.  3,900 and 4,100 points give 257,400
    # and 270,600 pairs over two fields, all listed; 4,800 points, above the bound for few
    # points, 316,800, more than the list's 2^18.  Every pair is FP64, so the plan's sums,
    # in the same order
    coils = [ccoil.Coil(0.1, 0.02, 0.05, 10 + i, 1.0 + i) for i in range(33)]
    g = np.random.default_rng(9)
    for n in (3900, 4100, 4800):
        r, phi = g.uniform(0.095, 0.125, n), g.uniform(0.0, 2.0 * np.pi, n)
        pts = np.stack([r * np.cos(phi), r * np.sin(phi), g.uniform(-0.03, 0.03, n)], axis=1)
        batch = ccoil.BatchPlan([(coils, pts)], fields=("A", "B"), precision=ccoil.PrecisionMode.FP32_COMPENSATED)
        got = batch.run()
        for f, field in (("A", 0), ("B", 1)):
            want = ccoil.FieldPlan([c.struct() for c in coils], field, ccoil.PrecisionMode.FP32_COMPENSATED)(pts)
            assert rel_err(got[f].cpu().numpy(), want).max() < TOL, (f, n)
        batch.close()


@pytest.mark.parametrize("mode", ["FP32_COMPENSATED", "FP32_REFINED"])
@pytest.mark.parametrize("field", [0, 1, 3])
@pytest.mark.parametrize("points", [37, 3001])
def test_captured_fp32_call_repeats(ccoil, mode, field, points):
    # the near-field list's counter is cleared by a kernel or a memset of the call: each
    # replay starts from an empty list.  The pieces that an eager call is cut into add in
    # another order (bar of test_pieces_match_captured_call; FP32_REFINED may pick another
    # pair at its threshold, as in test_pair_split_gpu.py: 1e-7)
    import torch
    plan = ccoil.FieldPlan([c.struct() for c in stack(ccoil, 40)], field, ccoil.PrecisionMode[mode])
    x = torch.from_numpy(on_the_winding(points, 0.02)).cuda()
    eager = plan(x).cpu().numpy()
    out = torch.empty((points, plan.width), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        plan(x, out=out)
    for _ in range(3):
        out.fill_(float("nan"))
        g.replay()
        torch.cuda.synchronize()
        assert rel_err(out.cpu().numpy(), eager).max() < (TOL if mode == "FP32_COMPENSATED" else 1e-7)
    plan.close()


def test_few_points_captured_after_many(ccoil):
    # 130 coils in one place: 9,000 points may list 1.17 million pairs, 12,000 points 2^20;
    # a call of 12,000 points has reserved enough for a captured one of 9,000.  Every pair is
    # FP64 and added in the same order, listed or not
    import torch
    coils = [ccoil.Coil(0.1, 0.0, 0.05, 10 + i, 1.0 + i) for i in range(130)]
    g = np.random.default_rng(10)
    r, phi = g.uniform(0.095, 0.105, 12000), g.uniform(0.0, 2.0 * np.pi, 12000)
    x = torch.from_numpy(np.stack([r * np.cos(phi), r * np.sin(phi), g.uniform(-0.03, 0.03, 12000)], axis=1)).cuda()
    plan = ccoil.FieldPlan([c.struct() for c in coils], 1, ccoil.PrecisionMode.FP32_COMPENSATED)
    whole = plan(x)
    out = torch.empty((9000, 3), dtype=torch.float64, device="cuda")
    y = x[:9000].contiguous()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan(y, out=out)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, whole[:9000])
    assert torch.equal(plan(y), out)
    plan.close()

"""The host side of one-shot calls: parameter rows to coils, one block of memory and
one copy per call (host arrays up to 64 KiB travel with the tables), poses as separate
arrays, and mutual-inductance gradients with poses on the GPU."""
import ctypes

import numpy as np
import pytest


def test_coils_from_params(ccoil):
    from ccoil_b200 import workloads
    L, lib = ccoil._lib, ccoil.lib()
    rows = workloads.coil_rows_mixed(9, seed=3)
    q = np.stack([rows[:, 0], rows[:, 1], rows[:, 2], rows[:, 3] * rows[:, 4], *rows[:, 6:11].T], axis=1).copy()
    precs = (L.PrecisionArgsStruct * 9)(*[L.PrecisionArgsStruct(1, 1, 1, 10 + i, 3, 2) for i in range(9)])
    got = (L.CoilStruct * 9)()
    dp = ctypes.POINTER(ctypes.c_double)
    assert lib.ccoil_coils_from_params(q.ctypes.data_as(dp), precs, 9, got) == 0
    for i in range(9):
        c = ccoil.Coil(q[i, 0], q[i, 1], q[i, 2], 1, q[i, 3], 0.0, ccoil.PrecisionFactor(5.0), 8, q[i, 4:7], q[i, 7],
                       q[i, 8])
        want = c.struct(ccoil.PrecisionArguments(1, 1, 1, 10 + i, 3, 2))
        assert bytes(got[i]) == bytes(want), i
    assert lib.ccoil_coils_from_params(None, precs, 1, got) == 1
    assert lib.ccoil_coils_from_params(q.ctypes.data_as(dp), precs, -1, got) == 1
    assert lib.ccoil_coils_from_params(None, None, 0, None) == 0
    q[4, 0] = -1.0
    assert lib.ccoil_coils_from_params(q.ctypes.data_as(dp), precs, 9, got) == 1


@pytest.mark.parametrize("shape,count", [((2, 8), 2), ((2, 10), 2), ((2, 9), 1), ((9,), 1), ((1, 2, 9), 1)])
def test_b_field_refuses_rows_and_precisions_of_the_wrong_count(ccoil, monkeypatch, shape, count):
    # before any native call: those read 9 values and one precision per coil
    import torch
    from ccoil_b200 import autograd

    def native():
        raise AssertionError("native call")

    monkeypatch.setattr(autograd, "lib", native)
    params = torch.full(shape, 0.1, dtype=torch.float64)
    precs = [ccoil.PrecisionArguments(1, 1, 1, 10, 3, 2)] * count
    with pytest.raises(ValueError):
        autograd.b_field(params, torch.zeros((4, 3), dtype=torch.float64), precs)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["FP64", "FP32_COMPENSATED", "FP32_REFINED"])
@pytest.mark.parametrize("points", [0, 1, 2730, 2731, 20000])
def test_one_shot_call_matches_plan(ccoil, mode, points):
    import torch
    from ccoil_b200 import workloads
    coils = workloads.coils_from_rows(workloads.coil_rows_mixed(5, seed=4), 4.0)
    pts = workloads.points_cube(points, seed=5)
    m = ccoil.PrecisionMode[mode]
    group = ccoil.CoilGroup(coils, ccoil.PrecisionFactor(4.0))
    for field, call in ((1, group.compute_all_B_field_vectors), (3, group.compute_all_B_gradient_matrices)):
        plan = group.plan(field, m)
        want = plan(pts)
        plan.close()
        # FP32_REFINED adds its FP64 values with atomics, in any order
        tol = 1e-13 if mode == "FP32_REFINED" else 0.0
        scale = np.abs(want).max(initial=1e-300)
        for x in (pts, torch.from_numpy(pts).cuda()):
            got = call(x, precision_mode=m)
            got = np.asarray(got.cpu() if hasattr(got, "cpu") else got).reshape(want.shape)
            assert np.max(np.abs(got - want), initial=0.0) <= tol * scale, (field, type(x))
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            x = torch.from_numpy(pts).cuda()
            got = call(x, precision_mode=m).reshape(want.shape)
        side.synchronize()
        assert np.max(np.abs(got.cpu().numpy() - want), initial=0.0) <= tol * scale


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 1638, 1639, 6000])
@pytest.mark.parametrize("quantity", [0, 1])
def test_separate_pose_arrays_match_packed(ccoil, n, quantity):
    from ccoil_b200 import coil as C, workloads
    prim, sec, pp, sp, py, pz, sy, sz = workloads.pair_config(n, seed=6)
    P, S = workloads.coils_from_rows(prim)[0], workloads.coils_from_rows(sec)[0]
    a, b = ccoil.Coil._pair_args(P, S, 1.0)
    args = ([P.struct(a)], S.struct(b), [b.to_struct()])
    packed = C._pair_arrangements(*args, C._poses(pp, py, pz), C._poses(sp, sy, sz), quantity)
    arrays = C._pair_arrangements(*args, C._PoseArrays(pp, py, pz), C._PoseArrays(sp, sy, sz), quantity)
    assert np.array_equal(packed[0], arrays[0]) and packed[1] == arrays[1]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("n", [1, 50])
def test_mutual_inductance_gradient_on_either_device(ccoil, dtype, n):
    """Poses on the CPU and on the GPU: the same kernel results, summed in another
    order (bar: 1e-12 of each gradient's scale, or FP32 rounding)."""
    import torch
    from ccoil_b200.autograd import mutual_inductance
    from ccoil_b200 import coil as C, workloads
    _, _, pp, sp, py, pz, sy, sz = workloads.pair_config(n, seed=8)
    values = ([0.1, 0.05, 0.1, 200.0], [0.05, 0.0, 0.2, 100.0], C._poses(pp, py, pz), C._poses(sp, sy, sz))
    got = {}
    for device in ("cpu", "cuda"):
        leaves = [torch.tensor(v, dtype=getattr(torch, dtype), device=device).requires_grad_() for v in values]
        m = mutual_inductance(*leaves, precision_factor=3.0)
        assert m.device.type == device and m.dtype == leaves[3].dtype
        (m * torch.linspace(0.5, 1.5, n, dtype=m.dtype, device=device)).sum().backward()
        got[device] = [m.detach().cpu().numpy()] + [v.grad.cpu().numpy() for v in leaves]
        assert all(v.grad.device.type == device and v.grad.dtype == v.dtype for v in leaves)
    tol = 1e-12 if dtype == "float64" else 1e-6
    for a, b in zip(got["cpu"], got["cuda"]):
        assert np.max(np.abs(a - b)) <= tol * np.abs(a).max()

"""Arrangement counts at which the pair kernels cut an arrangement into several
work units (node ranges, groups of primaries, lanes per secondary node): the same
arrangements in one large call, which takes one unit each, give the same values up
to the order of their FP64 sums (bar 1e-12 of the batch's scale), coaxial pairs
and their count included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12
COUNT = 45000  # above 8 waves of one unit per arrangement for every variant


def arrangements(n):
    from ccoil_b200 import workloads
    prim, sec, pp, sp, py, pz, sy, sz = workloads.pair_config(n, seed=77)
    pp[::3] = [0.01, -0.02, 0.03]
    sp[7::500] = [0.0, 0.0, 0.13]   # exactly coaxial with a primary at the origin
    pp[7::500] = 0.0
    sy[7::500] = 0.0
    return prim, sec, pp, sp, py, pz, sy, sz


@pytest.mark.parametrize("quantity", ["M", "FT"])
@pytest.mark.parametrize("mode", ["FP64", "FP32_COMPENSATED"])
@pytest.mark.parametrize("secondary", ["thin", "filament"])
def test_split_arrangements_match_whole(ccoil, quantity, mode, secondary):
    from ccoil_b200 import workloads
    prim, sec, pp, sp, py, pz, sy, sz = arrangements(COUNT)
    if secondary == "filament":
        sec[2] = 0.0
    P, S = workloads.coils_from_rows(prim)[0], workloads.coils_from_rows(sec)[0]
    call = (ccoil.Coil.compute_all_mutual_inductance_arrangements if quantity == "M"
            else ccoil.Coil.compute_all_force_torque_arrangements)
    m = ccoil.PrecisionMode[mode]

    def values(a, b):
        v = call(P, S, pp[a:b], sp[a:b], py[a:b], pz[a:b], sy[a:b], sz[a:b], ccoil.PrecisionFactor(2.0),
                 precision_mode=m)
        return v.reshape(b - a, -1)

    whole = values(0, COUNT)
    scale = np.abs(whole).max(axis=0)
    for a, b in ((7, 8), (0, 1), (5, 38), (0, 1000), (100, 4199), (0, 20000)):
        assert np.max(np.abs(values(a, b) - whole[a:b]) / scale) < TOL, (a, b)


@pytest.mark.parametrize("mode", ["FP64", "FP32_COMPENSATED"])
def test_split_groups_match_whole(ccoil, mode):
    from ccoil_b200 import workloads
    rows = workloads.coil_rows_mixed(5, seed=78)
    rows[0, 6:11] = 0.0  # a primary on the z axis: some pairs below are coaxial with it
    group = ccoil.CoilGroup(workloads.coils_from_rows(rows), ccoil.PrecisionFactor(2.0))
    _, sec, _, sp, _, _, sy, sz = arrangements(COUNT)
    S = workloads.coils_from_rows(sec)[0]
    m = ccoil.PrecisionMode[mode]

    def values(a, b):
        return group.compute_all_force_torque_arrangements(S, sp[a:b], sy[a:b], sz[a:b], ccoil.PrecisionFactor(2.0),
                                                           precision_mode=m)

    whole = values(0, COUNT)
    scale = np.abs(whole).max(axis=0)
    for a, b in ((7, 8), (0, 3), (400, 900), (0, 9000)):
        assert np.max(np.abs(values(a, b) - whole[a:b]) / scale) < TOL, (a, b)


@pytest.mark.parametrize("quantity", [2, 3])
def test_split_gradients_match_whole(ccoil, quantity):
    from ccoil_b200 import workloads
    prim, sec, pp, sp, py, pz, sy, sz = arrangements(COUNT)
    P, S = workloads.coils_from_rows(prim)[0], workloads.coils_from_rows(sec)[0]
    call = (ccoil.Coil.compute_all_mutual_inductance_gradient_arrangements if quantity == 2
            else ccoil.Coil.compute_all_mutual_inductance_parameter_gradient_arrangements)

    def values(a, b):
        return call(P, S, pp[a:b], sp[a:b], py[a:b], pz[a:b], sy[a:b], sz[a:b], ccoil.PrecisionFactor(1.0))

    whole = values(0, COUNT)
    scale = np.abs(whole).max(axis=0)
    for a, b in ((0, 1), (5, 38), (0, 1000), (100, 4199)):
        assert np.max(np.abs(values(a, b) - whole[a:b]) / scale) < TOL, (a, b)


@pytest.mark.parametrize("quantity", ["M", "FT"])
@pytest.mark.parametrize("secondary", ["thin", "filament"])
@pytest.mark.parametrize("fraction", [None, 0.0])
def test_refined_teams_match_whole(ccoil, quantity, secondary, fraction):
    """FP32_REFINED: 12, 4 or 1 warps per arrangement.  A node at the refinement
    threshold may fall on either side when the total is summed in another order: at
    most 0.1 of the total times the FP32 error of a node, 1e-6, so the bar is 1e-7 of
    the batch's scale; at fraction 0 every node is FP64 and it is 1e-12."""
    import ctypes
    from ccoil_b200 import workloads
    prim, sec, pp, sp, py, pz, sy, sz = arrangements(COUNT)
    if secondary == "filament":
        sec[2] = 0.0
    P, S = workloads.coils_from_rows(prim)[0], workloads.coils_from_rows(sec)[0]
    call = (ccoil.Coil.compute_all_mutual_inductance_arrangements if quantity == "M"
            else ccoil.Coil.compute_all_force_torque_arrangements)

    def values(a, b):
        v = call(P, S, pp[a:b], sp[a:b], py[a:b], pz[a:b], sy[a:b], sz[a:b], ccoil.PrecisionFactor(2.0),
                 precision_mode=ccoil.PrecisionMode.FP32_REFINED)
        return v.reshape(b - a, -1)

    L = ccoil.lib()
    L.ccoil_refine_fraction.restype = ctypes.c_double
    before = L.ccoil_refine_fraction()
    try:
        if fraction is not None:
            assert L.ccoil_set_refine_fraction(ctypes.c_double(fraction)) == 0
        whole = values(0, COUNT)
        scale = np.abs(whole).max(axis=0)
        for a, b in ((7, 8), (5, 38), (0, 444), (0, 445), (100, 5100), (0, 20000)):
            got = values(a, b)
            assert np.max(np.abs(got - whole[a:b]) / scale) < (1e-7 if fraction is None else TOL), (a, b)
            assert np.array_equal(got, values(a, b))
    finally:
        L.ccoil_set_refine_fraction(ctypes.c_double(before))

"""One primary's tables are staged in shared memory up to 48 KiB, beside what the
kernel itself keeps there: sizes at which both together pass 48 KiB."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

POSES = 31


def poses(n):
    """Secondary poses (n, 5) at least 0.25 m from the primary's centre (a coil of 0.1 m)."""
    g = np.random.default_rng(51)
    v = g.normal(size=(n, 3))
    v *= g.uniform(0.25, 0.5, (n, 1)) / np.linalg.norm(v, axis=1, keepdims=True)
    return np.column_stack([v, g.uniform(0.1, 3.0, n), g.uniform(0.0, 6.0, n)])


def arrangements(ccoil, quantity, mode, ring, n):
    """Values with a secondary ring of `ring` nodes (a multiple of 20): 32 bytes of
    table a node, under 1.7 KiB for the rest."""
    from ccoil_b200 import coil as C
    a = ccoil.PrecisionArguments(1, 1, 1, 20, 2, 1)
    b = ccoil.PrecisionArguments(20, 1, 1, ring // 20, 1, 2)
    P, S = ccoil.Coil(0.1, 0.02, 0.1, 100, 1.0), ccoil.Coil(0.05, 0.0, 0.05, 100, 1.0)
    v = C._pair_arrangements([P.struct(a)], S.struct(b), [b.to_struct()], np.zeros((n, 5)), poses(n), quantity,
                             ccoil.PrecisionMode[mode])[0].reshape(n, -1)
    # without dM/d(z angle of the primary): a turn about its own axis, zero by symmetry
    return np.delete(v, 5, axis=1) if quantity == 3 else v


@pytest.mark.parametrize("quantity,mode", [(0, "FP64"), (0, "FP32_COMPENSATED"), (0, "FP32_REFINED"), (1, "FP64"),
                                           (1, "FP32_COMPENSATED"), (1, "FP32_REFINED"), (2, "FP64"), (3, "FP64"),
                                           (3, "FP32_COMPENSATED")])
@pytest.mark.parametrize("n", [1, POSES, 445])
def test_failed_launch_is_an_error(ccoil, quantity, mode, n):
    """Right values or an error, never anything else.  The reference has a longer ring,
    whose tables are not staged: at this distance the ring integral converges long
    before (bar: 1e-11 of each column's scale; in the FP32 modes their error of a node)."""
    want = arrangements(ccoil, quantity, mode, 1600, n)
    scale = np.abs(arrangements(ccoil, quantity, mode, 1600, 445)).max(axis=0)
    for ring in (780, 1000, 1200, 1400, 1480):
        try:
            got = arrangements(ccoil, quantity, mode, ring, n)
        except ccoil.CCoilError:
            continue
        assert np.max(np.abs(got - want) / scale) < (1e-11 if mode == "FP64" else 1e-5), ring


@pytest.mark.parametrize("n", [1, 444, 445])
def test_failed_launch_is_an_error_beside_the_z_axis_pass(ccoil, n):
    # the public arrangement methods, whose calls end with the z-axis pass; bar: the
    # refined mode's error of a node (1e-6) against FP64
    P, S = ccoil.Coil(0.1, 0.0, 0.0, 100, 1.0), ccoil.Coil(0.05, 0.0, 0.0, 100, 1.0)
    s = poses(n)
    args = (np.zeros((n, 3)), s[:, :3], np.zeros(n), np.zeros(n), s[:, 3], s[:, 4], ccoil.PrecisionFactor(12.0))
    want = ccoil.Coil.compute_all_force_torque_arrangements(P, S, *args)
    try:
        got = ccoil.Coil.compute_all_force_torque_arrangements(P, S, *args,
                                                               precision_mode=ccoil.PrecisionMode.FP32_REFINED)
    except ccoil.CCoilError:
        return
    assert np.max(np.abs(got - want) / np.abs(want).max(axis=0)) < 1e-6


@pytest.mark.parametrize("quantity,mode", [(0, "FP64"), (0, "FP32_COMPENSATED"), (0, "FP32_REFINED"), (1, "FP64"),
                                           (1, "FP32_COMPENSATED"), (1, "FP32_REFINED"), (2, "FP64"), (3, "FP64"),
                                           (3, "FP32_COMPENSATED")])
@pytest.mark.parametrize("n", [1, 444, 445])
def test_tables_up_to_the_staging_limit(ccoil, quantity, mode, n):
    # the bars of test_failed_launch_is_an_error
    want = arrangements(ccoil, quantity, mode, 1600, n)
    scale = np.abs(arrangements(ccoil, quantity, mode, 1600, 445)).max(axis=0)
    for ring in (640, 780, 1000, 1200, 1400, 1480):
        got = arrangements(ccoil, quantity, mode, ring, n)
        assert np.max(np.abs(got - want) / scale) < (1e-11 if mode == "FP64" else 1e-5), ring


@pytest.mark.parametrize("n", [1, 444])
@pytest.mark.parametrize("shapes,pf", [(((0.0, 0.0), (0.0, 0.0)), 12.0), (((0.02, 0.05), (0.0, 0.0)), 15.0),
                                       (((0.0, 0.05), (0.02, 0.0)), 15.0)])
def test_refined_force_at_high_precision_factors(ccoil, shapes, pf, n):
    # filament-filament, rectangular-filament, thin-flat: 23 to 28 KB of tables beside
    # the 12-warp kernel's 27 KB; bar: the refined mode's error of a node against FP64
    (a, b), (c, d) = shapes
    P, S = ccoil.Coil(0.1, a, b, 100, 1.0), ccoil.Coil(0.05, c, d, 100, 1.0)
    s = poses(n)
    args = (np.zeros((n, 3)), s[:, :3], np.zeros(n), np.zeros(n), s[:, 3], s[:, 4], ccoil.PrecisionFactor(pf))
    want, got = (ccoil.Coil.compute_all_force_torque_arrangements(P, S, *args, precision_mode=ccoil.PrecisionMode[m])
                 for m in ("FP64", "FP32_REFINED"))
    assert np.max(np.abs(got - want) / np.abs(want).max(axis=0)) < 1e-6

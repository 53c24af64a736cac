"""FP64 integrands at the edges of the range in which they take their own roots
and quotients ([1e-36, 1e36] for squared distances; IEEE operations beyond):
geometries scaled across it, and points on a winding's own radius.  Bar: the
parity bar of test_fields_gpu.py, 1e-12 per point against the oracle."""
import numpy as np
import pytest

from conftest import gradient_band, rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-12


def coils_and_points(ccoil, scale, seed):
    from ccoil_b200 import workloads
    rows = workloads.coil_rows_mixed(8, seed=seed)
    rows[:, 0:3] *= scale
    rows[:, 6:9] *= scale
    pts = workloads.points_cube(97, seed=seed + 1) * scale
    return rows, workloads.coils_from_rows(rows, 4.0), pts


# squared distances span about 1e-4..10 times scale^2: inside the range, across
# its lower and upper ends, and outside it
@pytest.mark.parametrize("scale", [1.0, 1e-10, 3e-18, 1e-21, 1e10, 3e17, 1e21])
@pytest.mark.parametrize("field", [0, 1, 3])
def test_scaled_geometry_against_oracle(ccoil, oracle, scale, field):
    rows, coils, pts = coils_and_points(ccoil, scale, seed=31)
    group = ccoil.CoilGroup(coils, ccoil.PrecisionFactor(4.0))
    plan = group.plan(field)
    got = plan(pts)
    plan.close()
    e = rel_err(got, oracle.group_fields(rows, pts, field, pf=4.0))
    if field == 3:
        e = e[~gradient_band(rows, pts)]
    assert np.all(np.isfinite(got)) and e.max() < TOL, e.max()


@pytest.mark.parametrize("field", [0, 1])
@pytest.mark.parametrize("lanes", [1, 8])
def test_points_on_the_winding_radius(ccoil, oracle, field, lanes):
    # r equals the node radius: the smallest squared distance bound is exactly zero
    row = np.array([0.1, 0.0, 0.08, 40, 2.0, 50.0, 0.0, 0.0, 0.0, 0.0, 0.0])
    z = np.array([0.0, 0.02, -0.039, 0.04, 0.0401, -0.3])
    pts = np.stack([np.full_like(z, 0.1), np.zeros_like(z), z], axis=1)
    coil = ccoil.Coil(0.1, 0.0, 0.08, 40, 2.0)
    plan = ccoil.FieldPlan([coil.struct()], field)
    got = plan(pts, lanes=lanes)
    plan.close()
    e = rel_err(got, oracle.coil_fields(row, pts, field, pf=5.0))
    assert e.max() < TOL, e.max()


@pytest.mark.parametrize("scale", [1.0, 1e-10, 3e-18, 1e-21, 1e10, 3e17])
def test_adjoint_is_scale_invariant(ccoil, scale):
    """B falls as 1 / length: with every length scaled by s, dB/d(length) scales by
    s^-2 and dB/d(N I), dB/d(angle) by 1 / s.  The parameter gradient at the scaled
    geometry, inside, across and outside the range of the forms, against the
    unscaled one (bar 1e-11 of each parameter's scale: the forms differ by a few
    roundings per node, the points' coordinates by one)."""
    import torch
    from ccoil_b200 import autograd, workloads
    rows, pts = workloads.adjoint_config(coils=6, points=333, seed=41, types=(0, 1, 2, 3))
    q = np.stack([rows[:, 0], rows[:, 1], rows[:, 2], rows[:, 3] * rows[:, 4], *rows[:, 6:11].T], axis=1)
    v = np.random.default_rng(42).normal(size=pts.shape)

    def grad(s):
        p = q.copy()
        p[:, [0, 1, 2, 4, 5, 6]] *= s
        P = torch.tensor(p, requires_grad=True)
        B = autograd.b_field(P, torch.from_numpy(pts * s).cuda(), autograd.precisions_for(q))
        (B * torch.from_numpy(v).cuda()).sum().backward()
        g = P.grad.numpy() * s
        g[:, [0, 1, 2, 4, 5, 6]] *= s
        g[:, 1][q[:, 1] == 0.0] = 0.0  # a zero dimension is 1e-25 R at any scale
        g[:, 2][q[:, 2] == 0.0] = 0.0
        return g

    want = grad(1.0)
    assert np.max(np.abs(grad(scale) - want) / np.abs(want).max(axis=0)) < 1e-11


@pytest.mark.parametrize("points", [1, 31, 1025, 70001])
def test_adjoint_sums_over_points(ccoil, points):
    """The gradient over all points is the sum over two halves (bar 1e-12 of each
    parameter's scale: FP64 sums in another order)."""
    import torch
    from ccoil_b200 import autograd, workloads
    rows, pts = workloads.adjoint_config(coils=4, points=points, seed=43, types=(0, 2, 1, 3))
    q = np.stack([rows[:, 0], rows[:, 1], rows[:, 2], rows[:, 3] * rows[:, 4], *rows[:, 6:11].T], axis=1)
    precs = autograd.precisions_for(q, 3.0)

    def grad(x):
        P = torch.tensor(q, requires_grad=True)
        (autograd.b_field(P, torch.from_numpy(x).cuda(), precs) ** 2).sum().backward()
        return P.grad.numpy()

    whole, half = grad(pts), points // 2
    parts = grad(pts[:half]) + grad(pts[half:])
    assert np.max(np.abs(parts - whole) / np.abs(whole).max(axis=0)) < 1e-12


@pytest.mark.parametrize("shape,scale",
                         [(k, s) for k in ((0.02, 0.1), (0.0, 0.1), (0.03, 0.0))
                          for s in (1e10, 3e17, 1e21, 1e40, 1e76, 1e80, 1e120)
                          # the length nodes' 1 / distance^3 leaves FP64's range at 1e103
                          if not (k[1] == 0.0 and s == 1e120)])
@pytest.mark.parametrize("quantity", [2, 3])
def test_pair_gradient_is_scale_invariant(ccoil, scale, shape, quantity):
    """M grows as a length: with every length scaled by s, its derivatives by lengths stay
    and those by angles (and M) scale by s.  One pose lies inside the winding.  Bar 1e-11
    of each column's scale, as for the adjoint above."""
    from ccoil_b200 import coil as C
    g = np.random.default_rng(44)
    v = g.normal(size=(7, 3))
    v *= g.uniform(0.15, 0.4, (7, 1)) / np.linalg.norm(v, axis=1, keepdims=True)
    v[0] = [0.001, 0.002, 0.003]
    turns = g.uniform(0.1, 3.0, (7, 4))
    a, b = shape
    pa, sa = ccoil.Coil._pair_args(ccoil.Coil(0.1, a, b, 100, 1.0), ccoil.Coil(0.05, 0.0, 0.05, 100, 1.0), 3.0)

    def values(s):
        P, S = ccoil.Coil(0.1 * s, a * s, b * s, 100, 1.0), ccoil.Coil(0.05 * s, 0.0, 0.05 * s, 100, 1.0)
        out = C._pair_arrangements([P.struct(pa)], S.struct(sa), [sa.to_struct()],
                                   np.column_stack([np.zeros((7, 3)), turns[:, :2]]),
                                   np.column_stack([v * s, turns[:, 2:]]), quantity)[0].copy()
        if quantity == 3:
            out[:, [0, 4, 5, 12, 13]] /= s
            # a zero dimension is 1e-25 R at any scale
            out[:, [k for k, d in ((2, a), (3, b), (7, 0.0)) if d == 0.0]] = 0.0
        return out

    want = values(1.0)
    bar = 1e-11 * np.abs(want).max(axis=0)
    assert np.all(np.abs(values(scale) - want) <= bar)

"""What users of this framework have it do, as measurable cases.

Kinds of case:

  field          a coil's or a coil group's A, B, E or gradient at points: one call on host arrays
                 ("host"), one call on device tensors ("device"), or a kept FieldPlan ("plan")
  pairs          mutual inductance or force and torque of two coils over many arrangements
  batch          many independent coil systems through a kept BatchPlan
  adjoint        a step of coil optimisation: the group's B field, a loss, the gradient of every
                 coil parameter
  pair_gradient  the same for the mutual inductance of two coils over many arrangements

Coils, points and poses are those of the benchmark workloads (ccoil_b200/workloads.py): types mixed
evenly, R in [0.02, 0.3] m, sections up to 0.1 m, centres in a 1 m cube, any orientation.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "c-coil_b200"))

FP64, FP32C, FP32R = "FP64", "FP32_COMPENSATED", "FP32_REFINED"


def listed():
    return [
        # interactive use: one coil's field at a few probe positions, arrays in and out
        {"name": "coil_b_37_host", "kind": "field", "coils": 1, "field": "B", "points": 37, "mode": FP64,
         "call": "host", "pf": 5.0},
        # interactive use: one mutual inductance of two placed coils
        {"name": "pair_m_one", "kind": "pairs", "quantity": "M", "n": 1, "mode": FP64, "secondary": "thin",
         "pf": 5.0},
        # a magnet assembly's vector potential along a short probe line, arrays in and out
        {"name": "group_a_1001_host", "kind": "field", "coils": 24, "field": "A", "points": 1001, "mode": FP64,
         "call": "host", "pf": 5.0},
        # a field-gradient map of one coil from device-resident points
        {"name": "coil_g_65536", "kind": "field", "coils": 1, "field": "G", "points": 65536, "mode": FP64,
         "call": "device", "pf": 5.0},
        # the full field map of a large assembly through a kept plan, the default precision
        {"name": "group_b_524289", "kind": "field", "coils": 128, "field": "B", "points": 524289, "mode": FP64,
         "call": "plan", "pf": 5.0},
        # the same assembly in the fast precision mode, as a simulation calls it every step
        {"name": "group_b_fp32c_262144", "kind": "field", "coils": 128, "field": "B", "points": 262144,
         "mode": FP32C, "call": "plan", "pf": 5.0},
        # and in the mode that holds 1e-7 where the coils' fields cancel
        {"name": "group_a_fp32r_200003", "kind": "field", "coils": 128, "field": "A", "points": 200003,
         "mode": FP32R, "call": "plan", "pf": 5.0},
        # a parameter study of a moving pickup coil
        {"name": "pairs_m_4099", "kind": "pairs", "quantity": "M", "n": 4099, "mode": FP64, "secondary": "thin",
         "pf": 5.0},
        # force and torque maps for a dynamics table, the fast precision mode
        {"name": "pairs_ft_fp32c_65536", "kind": "pairs", "quantity": "FT", "n": 65536, "mode": FP32C,
         "secondary": "thin", "pf": 5.0},
        # a design sweep: uneven independent assemblies, B and gradient in one launch
        {"name": "batch_bg_40", "kind": "batch", "systems": 40, "fields": "BG", "mode": FP64, "pf": 5.0},
        # a gradient step of a shimming problem over all coil parameters
        {"name": "adjoint_64x4096", "kind": "adjoint", "coils": 64, "points": 4096, "dtype": "float64", "pf": 5.0},
        # a gradient step of a coupling-design problem
        {"name": "pair_gradient_1000", "kind": "pair_gradient", "n": 1000, "dtype": "float64", "pf": 5.0},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    while True:
        kind = rng.choice(["field"] * 5 + ["pairs"] * 3 + ["batch", "adjoint", "pair_gradient"])
        pf = rng.choice([3.0, 4.0, 5.0, 5.0, 5.0, 6.0])
        if kind == "field":
            c = {"kind": kind, "coils": _log_int(rng, 1, 128), "field": rng.choice("ABEGB"),
                 "points": _log_int(rng, 5, 524288), "mode": rng.choice([FP64, FP64, FP32C, FP32R]),
                 "call": rng.choice(["host", "device", "plan"]), "pf": pf}
        elif kind == "pairs":
            c = {"kind": kind, "quantity": rng.choice(["M", "FT"]), "n": _log_int(rng, 1, 65536),
                 "mode": rng.choice([FP64, FP64, FP32C, FP32R]),
                 "secondary": rng.choice(["thin", "flat", "filament"]), "pf": pf}
        elif kind == "batch":
            c = {"kind": kind, "systems": _log_int(rng, 3, 100), "fields": rng.choice(["BG", "B", "AB"]),
                 "mode": rng.choice([FP64, FP32C]), "pf": min(pf, 5.0)}
        elif kind == "adjoint":
            c = {"kind": kind, "coils": _log_int(rng, 2, 96), "points": _log_int(rng, 100, 20000),
                 "dtype": rng.choice(["float64", "float32"]), "pf": pf}
        else:
            c = {"kind": kind, "n": _log_int(rng, 1, 2000), "dtype": rng.choice(["float64", "float32"]),
                 "pf": min(pf, 5.0)}
        # a quarter of the largest listed case's work at most
        if work(c)["flops"] < 0.25 * work(listed()[4])["flops"]:
            return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _rows(count, seed, first=0):
    """Coil rows {R, a, b, N, I, f, x, y, z, y angle, z angle}, types cycling from `first`
    (0 RECTANGULAR, 1 THIN, 2 FLAT, 3 FILAMENT)."""
    g = np.random.default_rng([17, int(seed), int(count)])
    rows = np.zeros((count, 11))
    for i in range(count):
        t = (first + i) % 4
        a, b = g.uniform(0.005, 0.1, 2)
        rows[i] = [g.uniform(0.02, 0.3), 0.0 if t in (1, 3) else a, 0.0 if t in (2, 3) else b, g.integers(1, 501),
                   g.uniform(0.5, 5.0) * g.choice([-1.0, 1.0]), 50.0, *g.uniform(0.0, 1.0, 3),
                   math.acos(1.0 - 2.0 * g.uniform()), 2.0 * math.pi * g.uniform()]
    return rows


def _field_inputs(case, seed):
    n = case["points"]
    if case["coils"] == 1:
        # one RECTANGULAR coil on the z axis, points in the cylinder around it
        rows = np.array([[0.1, 0.1, 0.1, 100, 1.0, 50.0, 0.0, 0.0, 0.0, 0.0, 0.0]])
        g = np.random.default_rng([18, int(seed), n])
        r, phi = 0.5 * np.sqrt(g.uniform(size=n)), 2.0 * np.pi * g.uniform(size=n)
        pts = np.stack([r * np.cos(phi), r * np.sin(phi), g.uniform(-0.5, 0.5, n)], axis=1)
    else:
        rows = _rows(case["coils"], seed)
        pts = np.random.default_rng([19, int(seed), n]).uniform(-1.0, 1.0, (n, 3))
    return rows, pts


_PRIMARY = (0.1, 0.05, 0.1, 200)
_SECONDARY = {"thin": (0.05, 0.0, 0.2, 100), "flat": (0.05, 0.03, 0.0, 100), "filament": (0.05, 0.0, 0.0, 100)}


def _pose_inputs(n, seed):
    """Primary and secondary poses (n, 5): offsets in a 0.6 m cube, any orientation, one in twenty
    nearly coaxial and overlapping."""
    g = np.random.default_rng([20, int(seed), n])
    pp, sp = np.zeros((n, 5)), np.zeros((n, 5))
    sp[:, :3] = g.uniform(-0.3, 0.3, (n, 3))
    sp[:, 3] = np.arccos(1.0 - 2.0 * g.uniform(size=n))
    sp[:, 4] = 2.0 * np.pi * g.uniform(size=n)
    m = n // 20
    if m:
        i = g.choice(n, m, replace=False)
        sp[i, :2] = g.uniform(-2e-3, 2e-3, (m, 2))
        sp[i, 2] = g.uniform(-5e-3, 5e-3, m)
        sp[i, 3] = g.uniform(1e-5, 1e-3, m)
    return pp, sp


def _batch_inputs(case, seed):
    # sizes belong to the case (a sweep keeps its grids), values to the seed
    g = np.random.default_rng([21, case["systems"]])
    out = []
    for i in range(case["systems"]):
        coils = int(math.exp(g.uniform(0.0, math.log(64.0))))
        pts = int(math.exp(g.uniform(math.log(256.0), math.log(16384.0))))
        rows = _rows(coils, 1000 * (int(seed) % 1000003) + i, first=i)
        out.append((rows, np.random.default_rng([22, int(seed), i]).uniform(-1.0, 1.0, (pts, 3))))
    return out


def _adjoint_inputs(case, seed):
    # one RECTANGULAR coil of its own seed after the other
    rows = np.stack([_rows(1, 7919 * (int(seed) % 1000003) + i)[0] for i in range(case["coils"])])
    params = np.stack([rows[:, 0], rows[:, 1], rows[:, 2], rows[:, 3] * rows[:, 4], *rows[:, 6:11].T], axis=1)
    g = np.random.default_rng([23, int(seed), case["points"]])
    v = g.normal(size=(case["points"], 3))
    v *= 0.05 * np.cbrt(g.uniform(size=(len(v), 1))) / np.linalg.norm(v, axis=1, keepdims=True)
    return params, v


def prepare(case, seed):
    import ccoil_b200 as cc
    from ccoil_b200 import _lib, autograd
    kind, pf = case["kind"], cc.PrecisionFactor(case["pf"])

    def coils_of(rows):
        return [cc.Coil(r[0], r[1], r[2], int(r[3]), r[4], r[5], pf, 8, r[6:9], r[9], r[10]) for r in rows]

    if kind == "field":
        rows, pts = _field_inputs(case, seed)
        coils = coils_of(rows)
        mode = cc.PrecisionMode[case["mode"]]
        if case["call"] != "host":
            pts = torch.from_numpy(pts).cuda()
        owner = coils[0] if len(coils) == 1 else cc.CoilGroup(coils, pf)
        if case["call"] == "plan":
            field = {"A": _lib.FIELD_A, "B": _lib.FIELD_B, "E": _lib.FIELD_E, "G": _lib.FIELD_G}[case["field"]]
            call = cc.FieldPlan([c.struct() for c in coils], field, mode)
            return {"kind": kind, "run": lambda: call(pts)}
        call = {"A": owner.compute_all_A_potential_vectors, "B": owner.compute_all_B_field_vectors,
                "E": owner.compute_all_E_field_vectors, "G": owner.compute_all_B_gradient_matrices}[case["field"]]
        return {"kind": kind, "run": lambda: call(pts, precision_mode=mode)}
    if kind == "pairs":
        pp, sp = _pose_inputs(case["n"], seed)
        R, a, b, N = _PRIMARY
        prim = cc.Coil(R, a, b, N, 1.0)
        R, a, b, N = _SECONDARY[case["secondary"]]
        sec = cc.Coil(R, a, b, N, 1.0)
        mode = cc.PrecisionMode[case["mode"]]
        if case["n"] == 1 and case["mode"] == FP64:
            prim.set_position_and_orientation(pp[0, :3], pp[0, 3], pp[0, 4])
            sec.set_position_and_orientation(sp[0, :3], sp[0, 3], sp[0, 4])
            one = cc.Coil.compute_mutual_inductance if case["quantity"] == "M" else cc.Coil.compute_force_torque
            return {"kind": kind, "run": lambda: one(prim, sec, pf)}
        call = (cc.Coil.compute_all_mutual_inductance_arrangements if case["quantity"] == "M"
                else cc.Coil.compute_all_force_torque_arrangements)
        args = (pp[:, :3].copy(), sp[:, :3].copy(), pp[:, 3].copy(), pp[:, 4].copy(), sp[:, 3].copy(),
                sp[:, 4].copy())
        return {"kind": kind, "run": lambda: call(prim, sec, *args, pf, precision_mode=mode)}
    if kind == "batch":
        systems = [(coils_of(r), p) for r, p in _batch_inputs(case, seed)]
        plan = cc.BatchPlan(systems, fields=tuple(case["fields"]), precision=cc.PrecisionMode[case["mode"]])
        return {"kind": kind, "run": plan.run}
    dtype = getattr(torch, case["dtype"])
    if kind == "adjoint":
        params, pts = _adjoint_inputs(case, seed)
        precs = autograd.precisions_for(params, case["pf"])
        P = torch.from_numpy(params).to("cuda", dtype).requires_grad_()
        X = torch.from_numpy(pts).to("cuda", dtype)

        def step():
            P.grad = None
            B = autograd.b_field(P, X, precs)
            loss = ((B[:, 2] - 1e-3) ** 2 + B[:, 0] ** 2 + B[:, 1] ** 2).mean()
            loss.backward()
            return {"B": B.detach(), "grad": P.grad}
        return {"kind": kind, "run": step}
    pp, sp = _pose_inputs(case["n"], seed)
    leaves = [torch.tensor(v, dtype=dtype, device="cuda").requires_grad_()
              for v in (_PRIMARY, _SECONDARY["thin"], pp, sp)]
    precs = autograd.pair_precisions_for(_PRIMARY, _SECONDARY["thin"], case["pf"])
    weights = torch.linspace(0.5, 1.5, case["n"], dtype=dtype, device="cuda")

    def pair_step():
        for v in leaves:
            v.grad = None
        m = autograd.mutual_inductance(*leaves, precs)
        (m * weights).sum().backward()
        return {"M": m.detach(), "grads": [v.grad for v in leaves]}
    return {"kind": kind, "run": pair_step}


def run(state):
    return state["run"]()


# ---------------------------------------------------------------------------
# the same results from the definitions, in 64 bits
# ---------------------------------------------------------------------------
def _split(layer):
    blocks = (layer - 1) // 100 + 1
    return blocks, (layer // blocks + 1 if blocks > 1 else layer)


def _round(x):
    return int(math.floor(x + 0.5))


def _balance(total, parts):
    """The increments of each layer: in proportion to its measure, with the given product."""
    if len(parts) < 2:
        return {parts[0][0]: total}
    product = 1.0
    for _, m in parts:
        product *= m
    unit = (product / float(total)) ** (1.0 / float(len(parts)))
    return {i: _round(m / unit) for i, m in parts}


def _kind_of(R, a, b):
    """(thin thickness, thin length)"""
    return a / R < 1e-7, b / R < 1e-7


def _coil_nodes(R, a, b, pf):
    """[(blocks, increments) of the angle, the thickness, the length] of a coil at a PrecisionFactor."""
    thin_a, _ = _kind_of(R, a, b)
    k = 1.414213562
    m = [k * math.sqrt(math.pi * (R + 0.5 * a)), k * math.sqrt(a), k * math.sqrt(b)]
    parts = [(0, m[0])] + ([] if thin_a else [(1, m[1])])
    got = {0: 1, 1: 1, 2: 1}
    got.update(_balance(int(10.0 ** len(parts) * 2.0 ** (pf - 1.0)), parts))
    got[2] = _round(got[0] * m[2] / m[0]) or 1
    return [_split(got[i]) for i in range(3)]


def _pair_nodes(prim, sec, pf):
    """The same for a primary and a secondary coil that are integrated over each other."""
    k = 1.414213562
    (R, a, b, _), (S, c, d, _) = prim, sec
    m = [k * math.sqrt(math.pi * (R + 0.5 * a)), k * math.sqrt(a), k * math.sqrt(b),
         math.sqrt(2.0 * math.pi * (S + 0.5 * c)), math.sqrt(c), math.sqrt(d)]
    (pa, _), (sa, sb) = _kind_of(R, a, b), _kind_of(S, c, d)
    ids = [0] + ([] if pa else [1]) + [3] + ([] if sa else [4]) + ([] if sb else [5])
    got = {i: 1 for i in range(6)}
    got.update(_balance(int(10.0 ** len(ids) * 2.0 ** (pf - 1.0)), [(i, m[i]) for i in ids]))
    for i in range(1, 6):
        if got[i] == 1:
            got[i] = _round(got[0] * m[i] / m[0])
        got[i] = got[i] or 1
    layers = [_split(got[i]) for i in range(6)]
    return layers[:3], layers[3:]


def _unit_nodes(layer):
    """Composite Gauss-Legendre nodes on [0, 1] and their weights (summing to the block count)."""
    blocks, n = layer
    x, w = np.polynomial.legendre.leggauss(n)
    return (np.concatenate([(b + 0.5 + 0.5 * x) / blocks for b in range(blocks)]), np.tile(0.5 * w, blocks))


def _rotation(y, z):
    """Coil frame to global frame; y and z are tensors of one shape."""
    cy, sy, cz, sz = torch.cos(y), torch.sin(y), torch.cos(z), torch.sin(z)
    rows = [torch.stack([cz * cz * cy - sz * sz, -sz * cz * cy - sz * cz, cz * sy], -1),
            torch.stack([sz * cz * cy + sz * cz, cz * cz - sz * sz * cy, sz * sy], -1),
            torch.stack([-sy * cz, sy * sz, cy], -1)]
    return torch.stack(rows, -2)


def _ring_field(what, layers, R, a, b, r, z):
    """Fields of one ampere-turn in the coil's frame at (r, z), tensors of one shape: {A} for "A",
    {H, Z} for "B", {RPhi, RR, RZ, ZZ} for "G"; R, a and b are numbers or scalar tensors."""
    (phi, wphi), (u, wu), (v, wv) = (_unit_nodes(k) for k in layers)
    fast = not _kind_of(float(R), float(a), float(b))[1]
    c = torch.as_tensor(np.cos(np.pi * phi), device=r.device)
    # 2e-7 (pi / blocks) sum over half the turn; averages over the thickness and the length
    w = torch.as_tensor(wphi, device=r.device) * (2e-7 * math.pi / layers[0][0])
    r, z = r[..., None], z[..., None]
    out = None
    for vi, wi in [(0.5, 1.0)] if fast else list(zip(v, wv / wv.sum())):
        for uj, wj in zip(u, wu / wu.sum()):
            p = R + a * float(uj)
            scale = float(wi * wj)
            rho2 = (p - r) ** 2 + 2.0 * p * r * (1.0 - c)
            if fast:
                top, bot = z + 0.5 * b, z - 0.5 * b
                d1, d2 = rho2 + top * top, rho2 + bot * bot
                g1, g2 = 1.0 / torch.sqrt(d1), 1.0 / torch.sqrt(d2)
                if what == "A":
                    rho = torch.sqrt(rho2)
                    f = [p * c / b * (torch.asinh(top / rho) - torch.asinh(bot / rho))]
                elif what == "B":
                    f = [p * c / b * (g2 - g1), (p * p - p * r * c) / rho2 * (top * g1 - bot * g2) / b]
                else:
                    g13, g23 = g1 ** 3, g2 ** 3
                    t1, y = top * g13 - bot * g23, (top * g1 - bot * g2) / rho2
                    k = p * r * (1.0 - c * c) / rho2
                    f = [p * c / r * (g2 - g1) / b, p * c * (r - p * c) * (g13 - g23) / b,
                         p * (c * (t1 + y) - k * (2.0 * y + t1)) / b, (p * p - p * r * c) * (g13 - g23) / b]
            else:
                zl = z + b * float(vi - 0.5)
                d = rho2 + zl * zl
                g = 1.0 / torch.sqrt(d)
                g3 = g ** 3
                if what == "A":
                    f = [p * c * g]
                elif what == "B":
                    f = [p * c * zl * g3, (p * p - p * r * c) * g3]
                else:
                    g5 = g3 * g * g
                    f = [p * c * zl / r * g3, -3.0 * p * zl * (r - p * c) * c * g5,
                         p * (c * (2.0 * p * p + 2.0 * r * r - zl * zl - p * r * c) - 3.0 * p * r) * g5,
                         -3.0 * p * zl * (p - r * c) * g5]
            f = [scale * (x @ w) for x in f]
            out = f if out is None else [x + y for x, y in zip(out, f)]
    return out


def _cartesian(what, rows, pf, pts):
    """A group's field at points (n, 3) on the GPU."""
    field = {"E": "A"}.get(what, what)
    width = 9 if what == "G" else 3
    out = torch.zeros((len(pts), width), dtype=torch.float64, device=pts.device)
    for row in rows:
        R, a, b = (float(x) for x in row[:3])
        layers = _coil_nodes(R, a, b, pf)
        ang = torch.as_tensor(row[9:11], device=pts.device)
        T = _rotation(ang[0], ang[1])
        step = max(1, (1 << 25) // (layers[0][0] * layers[0][1]))
        for i in range(0, len(pts), step):
            q = (pts[i:i + step] - torch.as_tensor(row[6:9], device=pts.device)) @ T
            r = torch.hypot(q[:, 0], q[:, 1])
            c, s = q[:, 0] / r, q[:, 1] / r
            f = [x * float(row[3] * row[4]) for x in _ring_field(field, layers, R, a, b, r, q[:, 2])]
            if field == "A":
                k = 2.0 * math.pi * float(row[5]) if what == "E" else 1.0
                v = torch.stack([-k * f[0] * s, k * f[0] * c, 0.0 * s], 1) @ T.T
            elif field == "B":
                v = torch.stack([f[0] * c, f[0] * s, f[1]], 1) @ T.T
            else:
                o, rr, rz, zz = f
                m = torch.stack([rr * c * c + o * s * s, s * c * (rr - o), rz * c, s * c * (rr - o),
                                 rr * s * s + o * c * c, rz * s, rz * c, rz * s, zz], 1).reshape(-1, 3, 3)
                v = (T @ m).reshape(-1, 9)
            out[i:i + step] += v
    return out


def _pairs(quantity, prim, sec, layers, pp, sp):
    """(n,) mutual inductance or (n, 6) force and torque at poses (n, 5); prim and sec are
    {R, a, b, turns}, numbers or scalar tensors."""
    (R, a, b, N1), (S, c, d, N2) = prim, sec
    (va, wa), (vt, wt), (vl, wl) = (_unit_nodes(k) for k in layers[1])
    dev = sp.device
    phi = torch.as_tensor(2.0 * np.pi * va, device=dev)
    wn = torch.as_tensor((wl / wl.sum())[:, None, None] * (wt / wt.sum())[:, None] * (wa / wa.sum()), device=dev)
    ring = (S + c * torch.as_tensor(vt, device=dev))[:, None]                    # (thickness, 1)
    T1, T2 = _rotation(pp[:, 3], pp[:, 4]), _rotation(sp[:, 3], sp[:, 4])
    # ring basis {e1, e2, axis}: the axis is the third column of the rotation
    cy, sy, cz, sz = torch.cos(sp[:, 3]), torch.sin(sp[:, 3]), torch.cos(sp[:, 4]), torch.sin(sp[:, 4])
    e1 = torch.stack([cz * cy, sz * cy, -sy], -1)
    e2 = torch.stack([-sz, cz, 0.0 * sz], -1)
    ax = T2[:, :, 2]
    rad = (torch.cos(phi)[:, None] * e1[:, None, :] + torch.sin(phi)[:, None] * e2[:, None, :])   # (n, angle, 3)
    tan = (-torch.sin(phi)[:, None] * e1[:, None, :] + torch.cos(phi)[:, None] * e2[:, None, :])
    rel = ((d * torch.as_tensor(vl - 0.5, device=dev))[None, :, None, None, None] * ax[:, None, None, None, :] +
           ring[None, None, :, :, None] * rad[:, None, None, :, :])              # (n, length, thickness, angle, 3)
    q = torch.einsum("nltak,nkj->nltaj", rel + (sp[:, :3] - pp[:, :3])[:, None, None, None, :], T1)
    r = torch.sqrt(q[..., 0] ** 2 + q[..., 1] ** 2)
    co, si = q[..., 0] / r, q[..., 1] / r
    weight = wn[None] * (2.0 * math.pi * ring)[None, None] * N2
    if quantity == "M":
        f = _ring_field("A", layers[0], R, a, b, r, q[..., 2])[0] * N1
        A = torch.stack([-f * si, f * co, 0.0 * f], -1)
        A = torch.einsum("nltak,njk->nltaj", A, T1)
        return (weight * (A * tan[:, None, None]).sum(-1)).sum((1, 2, 3))
    H, Z = _ring_field("B", layers[0], R, a, b, r, q[..., 2])
    B = torch.stack([H * co, H * si, Z], -1) * N1
    B = torch.einsum("nltak,njk->nltaj", B, T1)
    dF = weight[..., None] * torch.cross(tan[:, None, None].expand_as(B), B, dim=-1)
    return torch.cat([dF.sum((1, 2, 3)), torch.cross(rel, dF, dim=-1).sum((1, 2, 3))], 1)


def exact(case, seed):
    kind, pf = case["kind"], case["pf"]
    if kind == "field":
        rows, pts = _field_inputs(case, seed)
        got = _cartesian(case["field"], rows, pf, torch.from_numpy(pts).cuda())
        return got.reshape(-1, 3, 3) if case["field"] == "G" and case["call"] != "plan" else got
    if kind == "batch":
        return {f: torch.cat([_cartesian(f, r, pf, torch.from_numpy(p).cuda()) for r, p in _batch_inputs(case, seed)])
                for f in case["fields"]}
    if kind == "pairs":
        prim, sec = _PRIMARY, _SECONDARY[case["secondary"]]
        layers = _pair_nodes(prim, sec, pf)
        pp, sp = (torch.from_numpy(v).cuda() for v in _pose_inputs(case["n"], seed))
        step = max(1, (1 << 25) // (_count(layers[1]) * layers[0][0][0] * layers[0][0][1]))
        got = torch.cat([_pairs(case["quantity"], prim, sec, layers, pp[i:i + step], sp[i:i + step])
                         for i in range(0, case["n"], step)])
        if case["n"] == 1 and case["mode"] == FP64:
            return float(got[0]) if case["quantity"] == "M" else (got[0, :3], got[0, 3:])
        return got
    dtype = getattr(torch, case["dtype"])
    if kind == "adjoint":
        params, pts = _adjoint_inputs(case, seed)
        P = torch.from_numpy(params).to(dtype).double().cuda()
        X = torch.from_numpy(pts).to(dtype).double().cuda()

        def coil(q, x, layers):
            T = _rotation(q[7], q[8])
            y = (x - q[4:7]) @ T
            r = torch.hypot(y[:, 0], y[:, 1])
            H, Z = _ring_field("B", layers, q[0], q[1], q[2], r, y[:, 2])
            return torch.stack([H * y[:, 0] / r, H * y[:, 1] / r, Z], 1) @ T.T * q[3]

        every = [_coil_nodes(*(float(v) for v in q[:3]), pf) for q in params]
        with torch.no_grad():
            B = sum(coil(q, X, k) for q, k in zip(P, every))
            up = 2.0 * torch.stack([B[:, 0], B[:, 1], B[:, 2] - 1e-3], 1) / len(X)
        grads = []
        for q, k in zip(P, every):
            q, g = q.clone().requires_grad_(), 0.0
            for i in range(0, len(X), 4096):
                g = g + torch.autograd.grad((coil(q, X[i:i + 4096], k) * up[i:i + 4096]).sum(), q)[0]
            grads.append(g)
        return {"B": B, "grad": torch.stack(grads)}
    layers = _pair_nodes(_PRIMARY, _SECONDARY["thin"], pf)
    pp, sp = _pose_inputs(case["n"], seed)
    leaves = [torch.tensor(v, dtype=dtype, device="cuda").double().requires_grad_()
              for v in (_PRIMARY, _SECONDARY["thin"])]
    poses = [torch.tensor(v, dtype=dtype, device="cuda").double().requires_grad_() for v in (pp, sp)]
    weights = torch.linspace(0.5, 1.5, case["n"], dtype=dtype, device="cuda").double()
    M = []
    for i in range(0, case["n"], 64):
        m = _pairs("M", leaves[0], leaves[1], layers, *(v[i:i + 64] for v in poses))
        (m * weights[i:i + 64]).sum().backward()
        M.append(m.detach())
    return {"M": torch.cat(M), "grads": [v.grad for v in leaves + poses]}


# ---------------------------------------------------------------------------
# the work of one pass
# ---------------------------------------------------------------------------
def _count(layers):
    return int(np.prod([b * n for b, n in layers]))


def _nodes(row, pf):
    R, a, b = (float(x) for x in row[:3])
    angle, thickness, length = _coil_nodes(R, a, b, pf)
    fast = not _kind_of(R, a, b)[1]
    return _count([angle, thickness] + ([] if fast else [length])), fast


# operations of one quadrature node (add, multiply, divide, root, logarithm one each):
# (analytic length integral, length nodes)
_OPS = {"A": (19, 7), "E": (19, 7), "B": (22, 13), "G": (61, 36)}


def _field_work(what, rows, pf, points):
    flops = sum(n * _OPS[what][0 if fast else 1] for n, fast in (_nodes(r, pf) for r in rows)) * points
    return {"bytes": 24.0 * points + (72.0 if what == "G" else 24.0) * points + 88.0 * len(rows),
            "flops": float(flops)}


def work(case):
    kind, pf = case["kind"], case["pf"]
    if kind == "field":
        rows, _ = _field_inputs(dict(case, points=1), 1)
        return _field_work(case["field"], rows, pf, case["points"])
    if kind == "batch":
        parts = [_field_work(f, r, pf, len(p)) for r, p in _batch_inputs(case, 1) for f in case["fields"]]
        return {k: sum(w[k] for w in parts) for k in ("bytes", "flops")}
    if kind == "adjoint":
        # forward, and the node's value with its derivatives by r', r and both slab faces
        params, _ = _adjoint_inputs(dict(case, points=1), 1)
        nodes = sum(_nodes(q, pf)[0] for q in params) * case["points"]
        return {"bytes": 72.0 * case["points"] + 144.0 * len(params), "flops": float(nodes * (22 + 60))}
    quantity = case.get("quantity", "M")
    prim, sec = _PRIMARY, _SECONDARY[case.get("secondary", "thin")]
    p, s = _pair_nodes(prim, sec, pf)
    nodes = _count(p[:2]) * _count(s) * case["n"]
    if kind == "pairs":
        return {"bytes": (80.0 + (8.0 if quantity == "M" else 48.0)) * case["n"],
                "flops": float(nodes * (_OPS["A"][0] if quantity == "M" else _OPS["B"][0]))}
    # the node's value with its derivatives by r', r, z and b
    return {"bytes": (80.0 + 8.0 + 80.0) * case["n"], "flops": float(nodes * 45)}

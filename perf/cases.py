"""The work a user of this library has it do, as cases that can be timed and compared.

The sizes are those of the package's own benchmark layouts (meshgen.py): the
single truncated cylinder in deep water, three cylinders with waterplane lids
over a flat bottom, the five-body array of about 6000 panels, the batch of
small cylinder groups and the request stream; beside them an irregular hull
(no symmetry and no two panels at one depth, as a mesh of a ship has) and the
wave-field map.  A case names the call (one frequency, a sweep, field points,
Green-function points, a group of requests), the form (plain: complex128
throughout; mixed: single-precision fill and LU with refinement), the layout
and the water.

    listed()             the cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  solver with its mesh, and the call's host arrays
    run(state)           one call of the package, and all it returns
    work(case)           bytes and operations the call cannot do without
    exact(case, seed)    the deep-water results in 64 bits by torch alone
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

GRAVITY, DENSITY = 9.80665, 1000.0


def _package():
    """The package directory's name has a hyphen: load it by path."""
    name = "hams_mrel_gb300"
    if name not in sys.modules:
        here = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hams-mrel_gb300")
        spec = importlib.util.spec_from_file_location(name, os.path.join(here, "__init__.py"),
                                                      submodule_search_locations=[here])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def _case(name, call, form, layout, **kw):
    c = {"name": name, "call": call, "form": form, "layout": layout, "bodies": 1, "az": 32, "vert": 8, "ring": 4,
         "lid": False, "depth": -1.0, "headings": 1, "freqs": 1, "slots": 1, "solver": 1, "points": 0}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: the wave field's Green function at a few hundred point pairs
        _case("points_deep", "points", "plain", "none", points=500),
        # one buoy, one frequency: what a design loop repeats thousands of times
        _case("plain_cylinder_384", "solve", "plain", "cylinders"),
        # three moored cylinders with irregular-frequency lids, 40 m of water, three headings
        _case("plain_lids_1536", "solve", "plain", "row", bodies=3, vert=12, lid=True, depth=40.0, headings=3),
        # a ship-like hull mesh in shallow water: no symmetry, no repeated depth, odd panel count
        _case("plain_hull_627", "solve", "plain", "hull", az=33, vert=13, ring=6, depth=25.0, headings=2),
        # the FP64 reference solution of the five-body array
        _case("plain_array_6048", "solve", "plain", "array", bodies=5, headings=8),
        # the array in the production form: one frequency alone (latency) with its potentials
        _case("mixed_array_6048", "solve", "mixed", "array", bodies=5, headings=8),
        # the array's frequency sweep, solves in flight side by side (throughput)
        _case("mixed_sweep_6048", "sweep", "mixed", "array", bodies=5, headings=8, freqs=16, slots=8),
        # the iterative solver on the array (Solver_type 2)
        _case("gmres_array_6048", "solve", "mixed", "array", bodies=5, headings=8, solver=2),
        # a small group of unequal cylinders, the batch's deep half: launches and latency
        _case("mixed_batch_deep", "sweep", "mixed", "cylinders", bodies=2, az=23, vert=11, ring=6, headings=3, freqs=16,
              slots=8),
        # the batch's finite-depth half: unequal cylinders in 150 m of water
        _case("mixed_batch_finite", "sweep", "mixed", "cylinders", bodies=2, az=31, vert=15, ring=8, depth=150.0,
              headings=2, freqs=4, slots=4),
        # a wave-field map: free-surface elevation around the array, every mode and heading
        _case("mixed_field_map", "field", "mixed", "array", bodies=5, headings=8, points=3992),
        # requests of different size and water served together
        _case("serve_requests", "serve", "mixed", "cylinders", bodies=6, az=24, vert=10, ring=5, headings=2, freqs=4,
              slots=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: the listed kinds over their ranges (300 to 6000 panels in deep water, to 2000 over a bottom)."""
    kind = rng.choice(["points", "plain_deep", "plain_finite", "plain_hull", "mixed_deep", "mixed_finite", "sweep",
                       "gmres", "field", "serve"])
    bodies = rng.randint(1, 4)
    heads = rng.randint(1, 8)
    depth = round(rng.uniform(30.0, 200.0), 2)

    def rows(total):  # azimuthal count, side and bottom rows of each body for a total panel count
        az = rng.randint(16, 48)
        n = max(4, int(round(total / bodies / az)))
        ring = max(1, int(round(n * rng.uniform(0.2, 0.5))))
        return {"bodies": bodies, "az": az, "vert": max(2, n - ring), "ring": ring, "headings": heads}

    if kind == "points":
        return _unnamed("points", "plain", "none", points=_log_int(rng, 100, 60000),
                        depth=-1.0 if rng.random() < 0.5 else depth)
    if kind == "plain_deep":
        return _unnamed("solve", "plain", "cylinders", **rows(_log_int(rng, 150, 5000)))
    if kind == "plain_finite":
        lid = rng.random() < 0.5
        return _unnamed("solve", "plain", rng.choice(["row", "cylinders"]), depth=depth if depth < 60.0 else 40.0,
                        lid=lid, **rows(_log_int(rng, 150, 1200)))
    if kind == "plain_hull":
        bodies = 1
        return _unnamed("solve", "plain", "hull", depth=-1.0 if rng.random() < 0.5 else round(rng.uniform(20, 60), 2),
                        **rows(_log_int(rng, 150, 700)))
    if kind == "mixed_deep":
        lid = rng.random() < 0.3
        return _unnamed("solve", "mixed", rng.choice(["cylinders", "hull"]), lid=lid, **rows(_log_int(rng, 300, 6000)))
    if kind == "mixed_finite":
        layout = rng.choice(["cylinders", "row", "hull"])
        return _unnamed("solve", "mixed", layout, depth=min(depth, 60.0) if layout == "hull" else depth,
                        lid=rng.random() < 0.3, **rows(_log_int(rng, 300, 1000)))
    if kind == "sweep":
        return _unnamed("sweep", rng.choice(["plain", "mixed", "mixed"]), "cylinders", freqs=rng.randint(2, 16),
                        slots=rng.randint(1, 8), **rows(_log_int(rng, 300, 1500)))
    if kind == "gmres":
        bodies = rng.randint(2, 4)
        return _unnamed("solve", rng.choice(["plain", "mixed"]), "cylinders", solver=2, **rows(_log_int(rng, 300, 3000)))
    if kind == "field":
        return _unnamed("field", rng.choice(["plain", "mixed"]), "cylinders", points=_log_int(rng, 50, 3000),
                        **rows(_log_int(rng, 300, 2500)))
    return _unnamed("serve", "mixed", "cylinders", freqs=rng.randint(1, 3), slots=rng.randint(3, 6),
                    bodies=rng.randint(2, 6), az=rng.randint(16, 24), vert=rng.randint(5, 10), ring=rng.randint(2, 5),
                    headings=rng.randint(1, 3))


def _unnamed(*a, **kw):
    c = _case("", *a, **kw)
    del c["name"]
    return c


# ---- inputs ---------------------------------------------------------------------------------------------------


def _mesh(case, rng, bodies=None):
    g = _package().meshgen
    nb = case["bodies"] if bodies is None else bodies
    if case["layout"] == "array":  # meshgen's five-body array, its 30 m grid perturbed by the seed
        return g.five_body_array(int(rng.integers(1 << 30)))
    made = []
    for k in range(nb):
        if case["layout"] == "row":  # equal bodies 15 m apart
            r, t, x, y = 3.0, 6.0, 15.0 * k, 0.0
        else:  # bodies of their own radius and draft
            r, t = rng.uniform(2.0, 8.0), rng.uniform(2.0, 10.0)
            x, y = 25.0 * k + rng.uniform(-3.0, 3.0), rng.uniform(-3.0, 3.0)
        b = g.cylinder(r, t, case["az"], case["vert"], case["ring"], cx=x, cy=y,
                       lid_rings=case["ring"] if case["lid"] else 0)
        if case["layout"] == "hull":  # every submerged node moved a little by itself
            d = b.nodes - np.array([x, y, 0.0])
            d *= 1.0 + rng.uniform(-0.02, 0.02, size=d.shape)
            b.nodes = np.where(b.nodes[:, 2:3] < 0.0, d + np.array([x, y, 0.0]), b.nodes)
        made.append(b)
    return g.combine(made)


def _waves(case, rng, nfreq=None, depth=None):
    """Wave state of the case's frequencies: v, wk, w1 arrays and the dispersion roots (None in deep water)."""
    n = case["freqs"] if nfreq is None else nfreq
    h = case["depth"] if depth is None else depth
    top = 2.0 if case["layout"] in ("none", "row", "hull") else 2.5
    w = np.sort(rng.uniform(0.2, top, size=n))
    props = [_package().hamsgpu.wave_properties(3, float(x), h) for x in w]
    roots = np.stack([p[3] for p in props]) if h > 0 else None
    return np.array([p[0] for p in props]), np.array([p[1] for p in props]), np.array([p[2] for p in props]), roots


def _headings(case):
    return np.linspace(0.0, 2.0 * math.pi, case["headings"], endpoint=False)


def _set_mesh(solver, mesh, lid):
    solver.set_mesh(mesh.nodes, mesh.ncon, mesh.ncn, mesh.xyz_p, mesh.ds, mesh.pnsz, mesh.dxyz_p, mesh.body_ranges,
                    mesh.lid_xyz_p if lid else None)


def _points(case, rng):
    """Source and field point pairs of the panels' ranges, from touching to tens of metres, and the near flags."""
    n = case["points"]
    r = np.exp(rng.uniform(math.log(0.05), math.log(80.0), size=n))
    r[::17] *= 1e-3  # near-vertical pairs
    a = rng.uniform(0.0, 2.0 * math.pi, size=n)
    q = np.column_stack([rng.uniform(-30, 30, n), rng.uniform(-30, 30, n), -rng.uniform(0.05, 10.0, n)])
    p = np.column_stack([q[:, 0] + r * np.cos(a), q[:, 1] + r * np.sin(a), -rng.uniform(0.05, 10.0, n)])
    return np.ascontiguousarray(np.hstack([q, p])), (r < 20.0).astype(np.int32)


def _map_points(case, mesh, rng):
    """Free-surface points around the bodies, none inside a body's waterline box."""
    lo, hi = mesh.xyz_p.min(axis=0) - 40.0, mesh.xyz_p.max(axis=0) + 40.0
    pts = np.zeros((0, 3))
    while len(pts) < case["points"]:
        p = rng.uniform(lo, hi, size=(2 * case["points"], 3))
        p[:, 2] = 0.0
        keep = np.ones(len(p), dtype=bool)
        for b0, b1 in mesh.body_ranges:
            q = mesh.xyz_p[b0 - 1:b1]
            blo, bhi = q.min(axis=0) - 1.0, q.max(axis=0) + 1.0
            keep &= ~((p[:, :2] > blo[:2]) & (p[:, :2] < bhi[:2])).all(axis=1)
        pts = np.vstack([pts, p[keep]])
    return np.ascontiguousarray(pts[:case["points"]])


def _requests(case, rng):
    """Requests of one to three bodies, every other one over a bottom."""
    out = []
    for k in range(case["bodies"]):
        mesh = _mesh(case, rng, bodies=1 + k % 3)
        depth = -1.0 if k % 2 == 0 else float(rng.uniform(30.0, 60.0))
        out.append((mesh, depth) + _waves(case, rng, depth=depth))
    return out


def prepare(case, seed):
    hg = _package().hamsgpu
    rng = np.random.default_rng([seed & 0xFFFFFFFF, 17])
    form = hg.HG_PREC_MIXED if case["form"] == "mixed" else hg.HG_PREC_FP64
    state = {"case": case, "betas": _headings(case)}
    if case["call"] == "serve":
        state["requests"] = _requests(case, rng)
        state["server"] = hg.Server(nslots=case["slots"], precision=form)
        return state
    s = state["solver"] = hg.Solver(precision=form, solver=case["solver"])
    state["waves"] = _waves(case, rng)
    v, wk, w1, wvn = state["waves"]
    first = (v[0], wk[0], w1[0], case["depth"], None if wvn is None else wvn[0])
    if case["call"] == "points":
        state["points"], state["flags"] = _points(case, rng)
        s.set_frequency(*first)
        return state
    mesh = state["mesh"] = _mesh(case, rng)
    _set_mesh(s, mesh, case["lid"])
    if case["call"] == "field":  # the map follows a solve
        state["points"] = _map_points(case, mesh, rng)
        s.solve_frequency(*first, state["betas"], want_potentials=False)
    state["first"] = first
    return state


def run(state):
    case, betas = state["case"], state["betas"]
    irsp = 1 if case["lid"] else 0
    if case["call"] == "serve":
        srv = state["server"]
        tickets = [srv.submit(mesh, depth, v, wk, w1, wvn, betas, irsp=irsp)
                   for mesh, depth, v, wk, w1, wvn in state["requests"]]
        got = [srv.wait(t)[:3] for t in tickets]
        return {"request%d" % k: {"added_mass": a, "damping": b, "excitation": f} for k, (a, b, f) in enumerate(got)}
    s = state["solver"]
    if case["call"] == "points":
        return s.green_points(state["points"], state["flags"])
    if case["call"] == "field":
        return s.field_points(state["points"], kind=s.FIELD_ELEVATION)
    if case["call"] == "sweep":
        v, wk, w1, wvn = state["waves"]
        a, b, f, _, _ = s.solve_sweep(v, wk, w1, case["depth"], wvn, betas, irsp=irsp, nslots=case["slots"])
        return {"added_mass": a, "damping": b, "excitation": f}
    a, b, f, x = s.solve_frequency(*state["first"], betas, irsp=irsp)
    return {"added_mass": a, "damping": b, "excitation": f, "potentials": x}


# ---- what a call cannot do without ------------------------------------------------------------------------------

PAIR_OPS = 590.0  # operations of one Green-function pair, deep water (oracle/opcount.py); over a bottom at least as many


def _panels(case, bodies):
    if case["layout"] == "array":
        return 6048, 0
    return bodies * case["az"] * (case["vert"] + case["ring"]), bodies * case["az"] * case["ring"] * int(case["lid"])


def _solve_work(case, bodies, freqs, potentials):
    n, nl = _panels(case, bodies)
    nd, nb = 6 * bodies, case["headings"]
    flops = PAIR_OPS * n * (n + nl) + 8.0 * n * (n + nl) * (nd + nb)  # fill, right-hand sides
    if case["solver"] == 2:
        flops += 4 * 8.0 * n * n * (nd + nb)  # a handful of products per column
    else:
        flops += 8.0 / 3.0 * n ** 3 + 8.0 * n * n * (nd + nb)
    if nl:
        flops += 8.0 * (n + nl) * n * (nd + nb) + 4.0 * (n + nl) * n * n  # the normal equations (Hermitian half)
    mesh = 8.0 * (24 * n + 3 * nl)
    out = 8.0 * (2 * nd * nd + 2 * nd * nb) + 16.0 * n * (nd + nb) * potentials
    return mesh + freqs * out, freqs * flops


def work(case):
    if case["call"] == "points":
        return {"bytes": case["points"] * (52.0 + 64.0), "flops": PAIR_OPS * case["points"]}
    if case["call"] == "serve":
        per = [_solve_work(case, 1 + k % 3, case["freqs"], 0) for k in range(case["bodies"])]
        return {"bytes": sum(p[0] for p in per), "flops": sum(p[1] for p in per)}
    if case["call"] == "field":
        n, cols, p = _panels(case, case["bodies"])[0], 6 * case["bodies"] + case["headings"], case["points"]
        return {"bytes": 24.0 * p + 192.0 * n + 16.0 * n * cols + 16.0 * p * cols,
                "flops": p * n * (PAIR_OPS + 16.0 * cols)}
    b, f = _solve_work(case, case["bodies"], case["freqs"], 1 if case["call"] == "solve" else 0)
    return {"bytes": b, "flops": f}


# ---- deep water in 64 bits by torch -------------------------------------------------------------------------------
# The collocation system written out from its definition (Newman's panel integrals, the Wu-Noblesse form of the
# deep-water Green function, the force integrals).  Over a bottom the reference's series are defined only to about
# 1e-7 (they extrapolate rounding), so those cases have no such value.


def exact(case, seed):
    if case["depth"] > 0 or case["solver"] == 2:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n = 0 if case["call"] == "points" else _panels(case, case["bodies"])[0]
    if dev == "cpu" and n > 1500:
        return None
    rng = np.random.default_rng([seed & 0xFFFFFFFF, 17])
    if case["call"] == "serve":
        out = {}
        for k, (mesh, depth, v, wk, w1, _) in enumerate(_requests(case, rng)):
            got = _solve_all(mesh, v, wk, w1, _headings(case), False, dev)[:3] if depth < 0 else (None, None, None)
            out["request%d" % k] = dict(zip(("added_mass", "damping", "excitation"), got))
        return out
    v, wk, w1, _ = _waves(case, rng)
    if case["call"] == "points":
        pts, flags = _points(case, rng)
        t = torch.tensor(pts, device=dev)
        near = torch.tensor(flags, device=dev) == 1
        return torch.stack(_green(t[:, :3].T, t[:, 3:].T, v[0], near), dim=1)
    mesh = _mesh(case, rng)
    if case["call"] == "field":
        pts = torch.tensor(_map_points(case, mesh, rng), device=dev)
        *_, x, w = _solve_all(mesh, v, wk, w1, _headings(case), False, dev, keep=True)
        a, s = _fill(_panel_frames(mesh, dev), pts, v[0], False)
        pot = (s @ w - a @ x) / (4.0 * math.pi)
        bt = torch.tensor(_headings(case), device=dev)
        nd = 6 * case["bodies"]
        phase = wk[0] * (pts[:, 0:1] * torch.cos(bt) + pts[:, 1:2] * torch.sin(bt))
        pot[:, nd:] += -GRAVITY / w1[0] * torch.exp(wk[0] * pts[:, 2:3]) * torch.exp(1j * phase)
        return 1j * w1[0] / GRAVITY * pot
    a, b, f, x = _solve_all(mesh, v, wk, w1, _headings(case), case["lid"], dev)
    if case["call"] == "sweep":
        return {"added_mass": a, "damping": b, "excitation": f}
    return {"added_mass": a[0], "damping": b[0], "excitation": f[0], "potentials": x}


def _horner(c, t):
    g = torch.full_like(t, c[-1])
    for k in reversed(c[:-1]):
        g = g * t + k
    return g


def _havelock(hh, vv):
    """Wave term of the deep-water Green function and its horizontal derivative (Wu et al. 2017), at v R and v (z + zeta)."""
    dd = torch.sqrt(hh * hh + vv * vv)
    al, be, rho = -vv / dd, hh / dd, dd / (1 + dd)
    ev, omr = torch.exp(vv), 1 - dd / (1 + dd)
    d3 = 1 + dd ** 3
    pa = _horner([1.21, -13.328, 215.896, -1763.96, 8418.94, -24314.21, 42002.57, -41592.9, 21859.0, -4838.6], rho)
    pb = _horner([0.938, 5.373, -67.92, 796.534, -4780.77, 17137.74, -36618.81, 44894.06, -29030.24, 7671.22], rho)
    pc = _horner([1.268, -9.747, 209.653, -1397.89, 5155.67, -9844.35, 9136.4, -3272.62], rho)
    pd = _horner([0.632, -40.97, 667.16, -6072.07, 31127.39, -96293.05, 181856.75, -205690.43, 128170.2, -33744.6], rho)
    da = _horner([2.948, -24.53, 249.69, -754.85, -1187.71, 16370.75, -48811.41, 68220.87, -46688.0, 12622.25], rho)
    db = _horner([1.11, 2.894, -76.765, 1565.35, -11336.19, 44270.15, -97014.11, 118879.26, -76209.82, 19923.28], rho)
    dc = _horner([14.19, -148.24, 847.8, -2318.58, 3168.35, -1590.27], rho)
    pp = (torch.log(0.5 * (dd - vv)) + 0.5772156649 - 2 * dd * dd) * ev + dd * dd - vv
    rr = (1 - be) * pa - be * pb - al * pc / (1 + 6 * al * rho * omr) + be * (1 - be) * pd
    l0 = 2 * pp / d3 + 2 * rho * omr ** 3 * rr
    # Bessel and Struve functions of order 0 and 1, below and above 3
    y = (hh / 3) ** 2
    j0 = _horner([0.999999999, -2.249999879, 1.265623060, -0.316394552, 0.044460948, -0.003954479, 0.000212950], y)
    j1 = hh * _horner([0.5, -0.562499992, 0.210937377, -0.039550040, 0.004447331, -0.000330547, 0.000015525], y)
    s0 = hh / 3 * _horner([1.909859164, -1.909855001, 0.687514637, -0.126164557, 0.013828813, -0.000876918], y)
    s1 = y * _horner([1.909859286, -1.145914713, 0.294656958, -0.042070508, 0.003785727, -0.000207183], y)
    big = hh > 3
    x = torch.where(big, hh, torch.full_like(hh, 4.0))
    z, i = 3 / x, 1 / torch.sqrt(x)
    y = z * z
    f0 = _horner([0.79788454, -0.00553897, 0.00099336, -0.00044346, 0.00020445, -0.00004959], y)
    t0 = x - math.pi / 4 + z * _horner([-0.04166592, 0.00239399, -0.00073984, 0.00031099, -0.00007605], y)
    f1 = _horner([0.79788459, 0.01662008, -0.00187002, 0.00068519, -0.00029440, 0.00006952], y)
    t1 = x - 0.75 * math.pi + z * _horner([0.12499895, -0.00605240, 0.00135825, -0.00049616, 0.00011531], y)
    h0 = 2 * _horner([0.99999906, 4.77228920, 3.85542044, 0.32303607], y) / (
        math.pi * x * _horner([1.0, 4.88331068, 4.28957333, 0.52120508], y)) + f0 * torch.sin(t0) * i
    h1 = 2 * _horner([1.00000004, 3.92205313, 2.64893033, 0.27450895], y) / (
        math.pi * _horner([1.0, 3.81095112, 2.26216956, 0.10885141], y)) + f1 * torch.sin(t1) * i
    j0, j1 = torch.where(big, f0 * torch.cos(t0) * i, j0), torch.where(big, f1 * torch.cos(t1) * i, j1)
    h0, h1 = torch.where(big, h0, s0), torch.where(big, h1, s1)
    tp = 2 * math.pi * ev
    ps = (be + hh) / (dd - vv) - 2 * be + 2 * ev * dd - hh
    qs = torch.exp(-dd) * (1 - be) * (1 + dd / d3)
    rr = be * da - (1 - al) * db + be * (1 - be) * rho * (1 - 2 * rho) * dc
    ls = 2 * ps / d3 - 4 * qs + 2 * rho * omr ** 3 * rr
    return torch.complex(l0 + tp * h0, -tp * j0), torch.complex(ls + tp * (2 / math.pi - h1), tp * j1)


def _green(q, p, v, near):
    """Deep-water Green function of sources q at fields p and its gradient; the Rankine term left out of near pairs."""
    dx, dy, zz, dz = q[0] - p[0], q[1] - p[1], p[2] + q[2], q[2] - p[2]
    rr = torch.sqrt(dx * dx + dy * dy)
    i1 = 1 / torch.sqrt(rr * rr + zz * zz)
    gf, gh = _havelock(v * rr, v * zz)
    far = rr > float(np.float32(1e-6))
    c = torch.where(far, -v * v / torch.where(far, rr, torch.ones_like(rr)), torch.zeros_like(rr))
    g = [-v * gf + i1, gh * c * dx - dx * i1 ** 3, gh * c * dy - dy * i1 ** 3, -v * v * gf + 2 * v * i1 - zz * i1 ** 3]
    i = torch.where(near, torch.zeros_like(rr), 1 / torch.sqrt(rr * rr + dz * dz).clamp_min(1e-300))
    return [g[0] + i, g[1] - dx * i ** 3, g[2] - dy * i ** 3, g[3] - dz * i ** 3]


def _panel_frames(mesh, dev):
    """Per panel: centroid, normal, area, near distance and the local frame of Newman's integrals (1986)."""
    tri = mesh.ncn == 3
    P = mesh.nodes[mesh.ncon - 1]
    v = P - P.mean(axis=1, keepdims=True)
    un = np.cross(v[:, 0], v[:, 1])
    ui = v[:, 0] / np.linalg.norm(v[:, 0], axis=1, keepdims=True)
    uk = un / np.linalg.norm(un, axis=1, keepdims=True)
    uj = np.cross(uk, ui)
    ks, et = np.einsum("nk,nck->nc", ui, v), np.einsum("nk,nck->nc", uj, v)
    po = P.mean(axis=1)
    a, b = P[:, 1] - P[:, 0], P[:, 2] - P[:, 0]  # triangles: origin at the foot of vertex 3 on edge 1-2
    alfa = ((a * b).sum(1) / (a * a).sum(1))[:, None]
    foot = P[:, 0] + alfa * a
    na, c = np.linalg.norm(a, axis=1, keepdims=True), P[:, 2] - foot
    nc = np.linalg.norm(c, axis=1, keepdims=True)
    zero = np.zeros(len(P))
    kt = np.stack([-np.copysign(1.0, alfa[:, 0]) * np.linalg.norm(P[:, 0] - foot, axis=1), zero,
                   np.linalg.norm(P[:, 1] - foot, axis=1), zero], axis=1)
    tt = np.stack([zero, nc[:, 0], zero, zero], axis=1)
    t1 = tri[:, None]
    with np.errstate(invalid="ignore", divide="ignore"):
        frame = [np.where(t1, x, y) for x, y in ((foot, po), (a / na, ui), (c / nc, uj), (np.cross(a / na, c / nc), uk),
                                                 (kt, ks), (tt, et))]
    arrays = [mesh.xyz_p, mesh.dxyz_p, mesh.ds, 50.0 * mesh.pnsz, tri] + frame
    return [torch.tensor(np.ascontiguousarray(x), device=dev) for x in arrays]


def _newman(fr, p):
    """Integral of 1/r over each panel at the fields p and its gradient (fields x panels)."""
    tri, po, ui, uj, uk, ks, et = fr[4:]
    d = p[:, None, :] - po[None]
    x, y, z = (d * ui).sum(2), (d * uj).sum(2), (d * uk).sum(2)
    del d
    nv = torch.where(tri, 3, 4)
    st, sx, sy, sz = (torch.zeros_like(x) for _ in range(4))
    for e in range(4):
        nx = torch.where(nv == e + 1, 0, min(e + 1, 3))
        k1, e1 = ks[:, e], et[:, e]
        k2, e2 = ks.gather(1, nx[:, None])[:, 0], et.gather(1, nx[:, None])[:, 0]
        dk, de = k2 - k1, e2 - e1
        l = torch.sqrt(dk * dk + de * de)
        use = (e < nv) & (tri | (l >= 1e-8))
        l = torch.where(use, l, torch.ones_like(l))
        r1 = torch.sqrt((k1 - x) ** 2 + (e1 - y) ** 2 + z * z)
        r2 = torch.sqrt((k2 - x) ** 2 + (e2 - y) ** 2 + z * z)
        b1, a1 = de * ((k1 - x) ** 2 + z * z) - dk * (k1 - x) * (e1 - y), r1 * z * dk
        b2, a2 = de * ((k2 - x) ** 2 + z * z) - dk * (k2 - x) * (e2 - y), r2 * z * dk
        off = use & (z.abs() >= 1e-6)
        sz += torch.where(off, torch.atan2(b1 * a2 - b2 * a1, a1 * a2 + b1 * b2), torch.zeros_like(z))
        s = r1 + r2
        ok = use & ((s - l).abs() >= 1e-6)
        lg = torch.where(ok, torch.log((s + l) / torch.where(ok, s - l, torch.ones_like(s))), torch.zeros_like(s))
        sx -= de / l * lg
        sy += dk / l * lg
        st += (de * (x - k1) - dk * (y - e1)) / l * lg
    sg = torch.where(tri, 1.0, -1.0)
    return [sg * (st - z * sz)] + [sg * (ui[:, k] * sx + uj[:, k] * sy + uk[:, k] * sz) for k in range(3)]


def _fill(fr, pts, v, diagonal):
    """Double- and single-layer matrices of the panels at the rows pts."""
    cen, nrm, area = fr[0], fr[1], fr[2]
    n = len(cen)
    A = torch.empty((len(pts), n), dtype=torch.complex128, device=pts.device)
    S = torch.empty_like(A)
    for i in range(0, len(pts), 1024):
        p = pts[i:i + 1024]
        near = torch.cdist(p, cen, compute_mode="donot_use_mm_for_euclid_dist") <= fr[3]
        g = _green(cen.T[:, None, :], p.T[:, :, None], v, near)
        nw = [torch.where(near, t, torch.zeros_like(t)) for t in _newman(fr, p)]
        S[i:i + 1024] = g[0] * area + nw[0]
        A[i:i + 1024] = sum((g[k + 1] * area + nw[k + 1]) * nrm[:, k] for k in range(3))
    if diagonal:
        A[torch.arange(n), torch.arange(n)] += 2 * math.pi
    return A, S


def _solve_all(mesh, v, wk, w1, betas, lid, dev, keep=False):
    """Added mass, damping, excitation of every frequency; with keep the last potentials and the source weights too."""
    fr = _panel_frames(mesh, dev)
    cen, nrm, area = fr[0], fr[1], fr[2]
    pts = torch.cat([cen, torch.tensor(mesh.lid_xyz_p, device=dev)]) if lid else cen
    n, nb = len(cen), len(mesh.body_ranges)
    nd = 6 * nb
    modes = torch.zeros((n, nd), dtype=torch.float64, device=dev)
    for b, (i0, i1) in enumerate(mesh.body_ranges):
        modes[i0 - 1:i1, 6 * b:6 * b + 6] = nrm[i0 - 1:i1]
    bt = torch.tensor(betas, device=dev)
    along = cen[:, 0:1] * torch.cos(bt) + cen[:, 1:2] * torch.sin(bt)
    out = []
    for f in range(len(v)):
        wave = torch.exp(wk[f] * cen[:, 2:3]) * torch.exp(1j * wk[f] * along)
        slope = torch.cos(bt) * nrm[:, 0:1] + torch.sin(bt) * nrm[:, 1:2]
        w = torch.cat([modes + 0j, w1[f] * wave * (1j * slope + nrm[:, 2:3])], dim=1)
        A, S = _fill(fr, pts, v[f], True)
        rhs = S @ w
        x = torch.linalg.solve(A.T @ A, A.T @ rhs) if lid else torch.linalg.solve(A, rhs)
        dif = x[:, nd:] - GRAVITY / w1[f] * wave
        t = (modes * area[:, None]).T.to(torch.complex128) @ x[:, :nd]
        e = (modes * area[:, None]).T.to(torch.complex128) @ dif
        out.append((DENSITY * t.real, DENSITY * w1[f] * t.imag, (1j * w1[f] * DENSITY * e).T))
    a, b, e = (torch.stack([o[k] for o in out]) for k in range(3))
    return (a, b, e, x, w) if keep else (a, b, e, x)

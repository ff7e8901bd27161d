"""The work that programs of this package have it do, as cases that can be timed.

A case names a body (or several), its mesh size, the water depth, the number of wave frequencies and headings,
the precision form and the entry point: `native.solve` / `native.solve_batch` (the batched entry) or
`native.Model` (the object model).  prepare() makes the inputs a program has in hand, run() is one call.
"""

import functools
import math

import numpy as np
import torch

from hydrobem_b200 import meshes
from hydrobem_b200 import native as nv

G, RHO = 9.80665, 1000.0

# One body's keys: shape and n1 n2 n3 (its mesh), depth (0: infinite), freqs, headings, kr0 kr1 (the range of the
# wave number times the body's length), sym (both mirror planes, the mesh a quarter), precision, api.
BASE = dict(shape="cylinder", n1=32, n2=8, n3=8, depth=0.0, freqs=10, headings=1, kr0=0.04, kr1=1.0, sym=False,
            precision="mixed", api="solve", bodies=1, points=0, angles=0, motions=False)


def listed():
    c = lambda name, **kw: dict(BASE, name=name, **kw)  # noqa: E731
    return [
        # a first look at a box hull: the smallest calls, all defaults (FP64), where latency counts
        c("box_first_look", shape="box", n1=6, n2=4, n3=3, freqs=3, precision="fp64"),
        # the 512-panel cylinder in deep water over ten periods, by the object model
        c("cylinder_512_model", api="model"),
        # an odd mesh with everything a seakeeping study asks for beside the coefficients: motions, elevations
        # at points, Kochin functions and the mean drift, FP64, finite depth
        c("hemisphere_study", shape="hemisphere", n1=15, n2=43, n3=0, depth=6.0, freqs=9, headings=3, precision="fp64",
          api="model", points=117, angles=104, motions=True),
        # radiation only (no headings), an odd mesh, FP64, finite depth, many frequencies
        c("hemisphere_radiation", shape="hemisphere", n1=19, n2=53, n3=0, depth=4.0, freqs=21, headings=0,
          precision="fp64"),
        # the benchmark workload: 4096 panels, depth 5 m, 40 periods, 4 headings
        c("cylinder_4096", n1=64, n2=32, n3=32, depth=5.0, freqs=40, headings=4, kr0=0.01, kr1=1.79),
        # the same body in the FP64 form, 8 of the periods
        c("cylinder_4096_fp64", n1=64, n2=32, n3=32, depth=5.0, freqs=8, headings=4, kr0=0.01, kr1=1.79,
          precision="fp64"),
        # a quarter mesh with both symmetry planes and the motions, by the object model
        c("quarter_motions", n1=16, n2=32, n3=32, depth=5.0, freqs=40, headings=4, kr0=0.01, kr1=1.79, sym=True,
          api="model", motions=True),
        # bodies of uneven panel counts in one batched call, 16 frequencies and 2 headings each
        c("uneven_batch", shape="uneven", n1=840, n2=4200, n3=0, freqs=16, headings=2, kr0=0.1, kr1=5.0, bodies=6),
        # small bodies in one batched call in the FP64 form
        c("small_batch_fp64", shape="uneven", n1=200, n2=1100, n3=0, freqs=6, headings=1, kr0=0.1, kr1=3.0, bodies=8,
          precision="fp64"),
        # three interacting cylinders, 18 modes: many right-hand sides, large matrices
        c("three_cylinders", shape="array", n1=64, n2=32, n3=32, freqs=4, headings=1, kr0=0.1, kr1=2.0),
        # the barge with its interior lid: the largest systems
        c("barge_lid", shape="barge", n1=64, n2=32, n3=75, freqs=5, headings=8, kr0=0.05, kr1=8.0, api="model"),
    ]


def draw(rng):
    """One more case of the ranges above, odd sizes among them."""
    lu = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    kind = rng.choice(["cylinder", "cylinder", "hemisphere", "box", "quarter", "uneven", "array"])
    fp64 = rng.random() < 0.4
    n = lu(80, 3000 if fp64 else 6000)
    c = dict(BASE, freqs=lu(1, 24), headings=rng.randint(0, 6), depth=rng.choice([0.0, 0.0, 3.5, 5.0, 12.0]),
             precision="fp64" if fp64 else "mixed", api=rng.choice(["solve", "model"]), kr0=0.02,
             kr1=round(rng.uniform(0.8, 2.0), 3))
    if kind in ("cylinder", "quarter"):
        p = max(3 if kind == "quarter" else 8, int(round(math.sqrt(n))) + rng.randint(-2, 2))
        z = max(2, n // (2 * p))
        c.update(n1=p, n2=z, n3=z + rng.randint(-1, 2), sym=kind == "quarter")
        if c["sym"]:  # the quarter of a body of n panels
            c["n1"] = max(3, p // 2)
            c["n2"] = max(2, z // 2)
            c["n3"] = max(2, c["n3"] // 2)
    elif kind == "hemisphere":
        p = max(8, int(round(math.sqrt(2 * n))) + rng.randint(-3, 3))
        c.update(shape="hemisphere", n1=max(3, n // p), n2=p, n3=0)
    elif kind == "box":
        q = max(2, int(round(math.sqrt(n / 10))))
        c.update(shape="box", n1=2 * q + rng.randint(0, 2), n2=q + 1, n3=q)
    elif kind == "uneven":
        c.update(shape="uneven", n1=max(80, n // 4), n2=max(160, n // 2), n3=0, bodies=rng.randint(2, 7), api="solve",
                 freqs=min(c["freqs"], 16))
    else:
        p = max(8, int(round(math.sqrt(n / 3))))
        c.update(shape="array", n1=p, n2=max(2, n // (6 * p)), n3=max(2, n // (6 * p)), api="solve")
    if c["shape"] in ("cylinder", "hemisphere", "box") and rng.random() < 0.3:
        c.update(motions=c["headings"] > 0, points=rng.choice([0, 33, 90]))
    return c


# ---------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=32)
def _mesh(shape, a, b, n, quarter=False):
    """The mesh of one body of unit size and the length its wave numbers refer to."""
    if shape == "cylinder":
        return meshes.cylinder(1.0, 1.0, a, b, n, quarter=quarter)
    if shape == "hemisphere":
        return meshes.hemisphere(1.0, a, b)
    if shape == "box":
        return meshes.box(1.0, 0.5, 0.5, n=(a, b, n))
    return meshes.barge((a, b, n))[0]


def _uneven_sizes(case):
    """The meshes of the batch's bodies: (shape, n1, n2, n3), fixed by the case."""
    rng = np.random.default_rng(case["n1"] * 7 + case["n2"] * 3 + case["bodies"])
    out = []
    for i in range(case["bodies"]):
        n = int(rng.uniform(case["n1"], case["n2"]))
        if i % 2:
            p = max(8, int(round(math.sqrt(2 * n) / 4)) * 4)
            out.append(("hemisphere", max(2, int(round(n / p))), p, 0))
        else:
            p = max(8, int(round(math.sqrt(n) / 4)) * 4)
            z = max(2, int(round(n / (2 * p))))
            out.append(("cylinder", p, z, z))
    return out


def _problems(case, seed):
    """The problems of the case as dicts of the keywords of native.Body."""
    rng = np.random.default_rng(seed)
    out = []
    for i in range(case["bodies"]):
        kw = {}
        if case["shape"] == "array":
            r, d = rng.uniform(0.95, 1.05), rng.uniform(0.9, 1.1)
            one = _mesh("cylinder", case["n1"], case["n2"], case["n3"]) * np.array([r, r, d])
            xs = (-4.0, 0.0, 4.0)
            v = np.concatenate([one + np.array([x, 0.0, 0.0]) for x in xs])
            kw.update(panel_body=np.repeat(np.arange(3, dtype=np.int32), len(one)),
                      rotation_centers=[[x, 0.0, 0.0] for x in xs])
            length = 1.0
        elif case["shape"] == "barge":
            v = _mesh("barge", case["n1"], case["n2"], case["n3"]) * np.array([rng.uniform(0.95, 1.05), 1.0,
                                                                             rng.uniform(0.9, 1.1)])
            kinds = np.zeros(len(v), np.int32)
            kinds[-case["n1"] * case["n2"]:] = 1
            kw.update(kinds=kinds)
            length = 80.0
        else:
            shape, a, b, n = _uneven_sizes(case)[i] if case["shape"] == "uneven" else (
                case["shape"], case["n1"], case["n2"], case["n3"])
            r = rng.uniform(0.5, 3.0) if case["shape"] == "uneven" else rng.uniform(0.95, 1.05)
            d = r * (rng.uniform(0.45, 0.55) if shape == "cylinder" else rng.uniform(0.9, 1.1))
            v = _mesh(shape, a, b, n, case["sym"]) * np.array([r, r, d])
            if case["sym"]:
                kw.update(symmetry=nv.SYM_BOTH)
            length = r
        f = case["freqs"]
        if case["shape"] in ("uneven", "barge"):  # wave numbers at random over the range
            k = np.sort(rng.uniform(case["kr0"], case["kr1"], f)) / length
            omegas = np.sqrt(k * G)
        else:  # periods evenly spaced
            t0, t1 = (2.0 * math.pi / math.sqrt(k / length * G) for k in (case["kr1"], case["kr0"]))
            omegas = 2.0 * math.pi / (np.linspace(t0, t1, f) * rng.uniform(0.99, 1.01))
        heads = (np.arange(case["headings"]) * (30.0 if case["headings"] < 7 else 22.5) + rng.uniform(0.0, 5.0))
        if case["motions"]:
            m = RHO * math.pi * r * r * d * 0.9
            g = [0.0, 0.0, -0.2 * d]
            kw.update(rigid={"mass": [m], "center_of_gravity": [g], "inertia_kind": [0], "inertia_origin": [g],
                             "inertia": [np.diag([0.3 * m * r * r, 0.3 * m * r * r, 0.5 * m * r * r])]})
        if case["points"]:
            p, q = rng.uniform(1.5, 6.0, case["points"]), rng.uniform(0.0, 2.0 * math.pi, case["points"])
            kw.update(points=np.stack([p * np.cos(q), p * np.sin(q), -0.5 * (np.arange(case["points"]) % 3)], 1))
        if case["angles"]:
            kw.update(kochin_angles=case["angles"])
        out.append(dict(vertices=v, omegas=omegas, headings_deg=heads, **kw))
    return out


def _model(case, p):
    """The object model of a problem, set up as a program sets it up."""
    m = nv.Model()
    m.reals("environment", "omegas", p["omegas"])
    if case["headings"]:
        m.reals("environment", "headings", p["headings_deg"])
    if case["depth"] > 0:
        m.real("environment", "depth", case["depth"])
    kinds = p.get("kinds")
    wet = p["vertices"] if kinds is None else p["vertices"][kinds == 0]
    m.add("meshes", "hull")
    m.reals("meshes/hull", "vertices", wet)
    m.add("bodies", "hull")
    m.text("bodies/hull", "mesh", "hull")
    if kinds is not None:  # the lid's panels, given as a mesh of their own
        m.add("meshes", "lid")
        m.reals("meshes/lid", "vertices", p["vertices"][kinds == 1])
        m.text("bodies/hull", "interior_surface", "mesh")
        m.text("bodies/hull", "interior_surface_mesh", "lid")
    if case["sym"]:
        m.text("meshes/hull", "symmetry", "xz_and_yz")
    if case["motions"]:
        r = p["rigid"]
        m.real("bodies/hull", "mass", r["mass"][0])
        m.reals("bodies/hull", "center_of_gravity", r["center_of_gravity"][0])
        m.reals("bodies/hull", "inertia_origin", r["inertia_origin"][0])
        i = r["inertia"][0]
        for q, name in enumerate(("Ixx", "Iyy", "Izz")):
            m.real("bodies/hull", name, i[q, q])
        m.boolean("options", "motion", True)
    if case["points"]:
        m.reals("options", "field_points", p["points"])
        m.boolean("options", "field_pressure", True)
    if case["angles"]:
        m.boolean("options", "drift_momentum_conservation", True)
        m.L.hb_set_int(m.m, m.obj("options"), b"drift_momentum_conservation_angles", case["angles"])
    m.text("options", "gpu_precision", case["precision"])
    return m


def prepare(case, seed):
    ps = _problems(case, seed)
    if case["api"] == "model":
        return dict(case=case, model=_model(case, ps[0]))
    return dict(case=case, problems=ps,
                options=dict(precision=nv.HBG_MIXED if case["precision"] == "mixed" else nv.HBG_FP64,
                             depth=case["depth"] if case["depth"] > 0 else math.inf))


def _quantities(case):
    """The quantities a program reads of the object model's results."""
    q = ["added_mass", "radiation_damping"]
    if case["headings"]:
        q += ["excitation_diffraction", "excitation_froude_krylov", "excitation_scattering", "excitation_haskind"]
    if case["motions"]:
        q += ["motion"]
    if case["points"]:
        q += ["field_points_pressure_radiation"] + (["field_points_pressure_incident", "field_points_pressure_diffraction"]
                                              if case["headings"] else [])
    if case["angles"]:
        q += ["drift_momentum_conservation"]
    return q


def run(state):
    case = state["case"]
    if case["api"] == "model":
        res = state["model"].solve()
        try:
            return {q: res.quantity(q) for q in _quantities(case)}
        finally:
            res.free()
    res = nv.solve_batch([nv.Body(**p) for p in state["problems"]], **state["options"])
    return [{k: v for k, v in r.items() if k not in ("hydrostatics", "kochin_angles")} for r in res]


def work(case):
    """The dense solves (8/3 M^3 real operations a system), the products with the right-hand sides and the pair
    kernels (about 100 operations an unordered pair); the bytes are the panels in and the results out."""
    flops = nbytes = 0.0
    for p in _problems(case, 0):
        n, f, h = len(p["vertices"]), case["freqs"], case["headings"]
        g = 4 if case["sym"] else 1
        d = 18 if case["shape"] == "array" else 6
        flops += f * g * (8.0 / 3.0 * n ** 3 + 24.0 * (d + h) * n ** 2 + 50.0 * n * n)
        nbytes += 96.0 * n + f * (16.0 * d * d + 64.0 * d * h) + 16.0 * f * case["points"] * (d + 3 * h)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------- the values in 64 bits
def _panels(v):
    """Centroids, normals, areas and the vertices in each panel's mid-plane (a triangle repeats its last one)."""
    c = v.mean(axis=1, keepdims=True)
    n = np.cross(v[:, 2] - v[:, 0], v[:, 3] - v[:, 1])
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    q = v - ((v - c) * n[:, None]).sum(-1, keepdims=True) * n[:, None]
    t = [0.5 * (np.cross(q[:, a] - q[:, 0], q[:, a + 1] - q[:, 0]) * n).sum(-1) for a in (1, 2)]
    area = t[0] + t[1]
    m = sum(t[a - 1][:, None] * (q[:, 0] + q[:, a] + q[:, a + 1]) / 3.0 for a in (1, 2))
    return m / area[:, None], n, area, q


def _wave_number(w, depth):
    """The root of k tanh(k h) = w^2 / g."""
    k = w * w / G
    for _ in range(100 if depth > 0 else 0):
        t = math.tanh(k * depth)
        k -= (k * t - w * w / G) / (t + k * depth * (1.0 - t * t))
    return k


def _incident(x, w, depth, heads):
    """The incident potential of unit amplitude at points x [P][3] and its vertical factor's log derivative: [H][P]."""
    k, b = _wave_number(w, depth), np.radians(heads)[:, None]
    z = x[:, 2]
    if depth > 0:
        e = np.exp(-k * (z + 2.0 * depth))
        zz, zd = (np.exp(k * z) + e) / (1.0 + math.exp(-2.0 * k * depth)), (np.exp(k * z) - e) / (np.exp(k * z) + e)
    else:
        zz, zd = np.exp(k * z), np.ones_like(z)
    return 1j * G / w * zz * np.exp(-1j * k * (x[:, 0] * np.cos(b) + x[:, 1] * np.sin(b))), k, k * zd


def _rankine(x, q, n, c):
    """The integrals of 1/r and its normal derivative at the source over every panel, [points][panels]."""
    w = torch.einsum("pjd,jd->pj", x[:, None] - c[None], n)
    a = q[None] - x[:, None, None]
    r = a.norm(dim=-1)
    om, s = torch.zeros_like(w), torch.zeros_like(w)
    for i in (1, 2):
        num = (a[..., 0, :] * torch.linalg.cross(a[..., i, :], a[..., i + 1, :])).sum(-1)
        dt = lambda e, f: (a[..., e, :] * a[..., f, :]).sum(-1)  # noqa: E731
        den = r[..., 0] * r[..., i] * r[..., i + 1] + dt(0, i) * r[..., i + 1] + dt(0, i + 1) * r[..., i] + dt(i, i + 1) * r[..., 0]
        om -= 2.0 * torch.atan2(num, den)
    om = torch.where(w.abs() < 1e-12, torch.zeros_like(om), om)
    for e in range(4):
        f = (e + 1) % 4
        edge = q[:, f] - q[:, e]
        ln = edge.norm(dim=-1)
        ok = ln > 1e-9
        em = torch.linalg.cross(edge, n) / ln.clamp(min=1e-9)[:, None]
        d = (a[..., e, :] * em[None]).sum(-1)
        g = r[..., e] * r[..., f] + (a[..., e, :] * a[..., f, :]).sum(-1)
        t = d * torch.log((r[..., e] + r[..., f] + ln) ** 2 / (2.0 * g.clamp(min=1e-300)))
        s += torch.where((ok & (d.abs() > 1e-13))[...] & (g > 0), t, torch.zeros_like(t))
    return s - w * om, om


def _log_part(xb, q, n, c, area):
    """The integrals of log(r - (z - z')) from the image points xb over every panel less one point's value each."""
    def terms(p, x):  # of points p against image points x
        d = p - x
        r = d.norm(dim=-1)
        den = r - d[..., 2]
        return den, r, d

    out = []
    rad = (q - c[:, None]).norm(dim=-1).max(dim=1).values
    for i in range(len(xb)):
        x = xb[i]
        near = (x - c).norm(dim=-1) < 4.0 * rad
        tot = torch.zeros(len(c), 2, dtype=torch.float64)
        for mask, cells, order in ((near, 8, 6), (~near, 1, 6)):
            if not bool(mask.any()):
                continue
            gx, gw = np.polynomial.legendre.leggauss(order)
            u = torch.tensor(np.concatenate([-1 + (2 * k + 1 + gx) / cells for k in range(cells)]))
            wu = torch.tensor(np.tile(gw, cells) / cells)
            U, V = torch.meshgrid(u, u, indexing="ij")
            W = wu[:, None] * wu[None]
            qq = q[mask]
            sh = [(1 - U) * (1 - V) / 4, (1 + U) * (1 - V) / 4, (1 + U) * (1 + V) / 4, (1 - U) * (1 + V) / 4]
            p = sum(s[None, ..., None] * qq[:, k][:, None, None] for k, s in enumerate(sh))
            xu = (1 - V)[None, ..., None] / 4 * (qq[:, 1] - qq[:, 0])[:, None, None] + (1 + V)[None, ..., None] / 4 * (qq[:, 2] - qq[:, 3])[:, None, None]
            xv = (1 - U)[None, ..., None] / 4 * (qq[:, 3] - qq[:, 0])[:, None, None] + (1 + U)[None, ..., None] / 4 * (qq[:, 2] - qq[:, 1])[:, None, None]
            jac = torch.linalg.cross(xu, xv).norm(dim=-1) * W
            den, r, d = terms(p, x)
            nn = n[mask][:, None, None]
            tot[mask, 0] = (jac * torch.log(den)).sum((-1, -2))
            tot[mask, 1] = (jac * (((d * nn).sum(-1) / r - nn[..., 2]) / den)).sum((-1, -2))
        den, r, d = terms(c, x)
        tot[:, 0] -= area * torch.log(den)
        tot[:, 1] -= area * ((d * n).sum(-1) / r - n[:, 2]) / den
        dist = r - d[:, 2]  # the correction's reach
        out.append(torch.where((dist * dist * 1e-4 < 0.6 * rad * rad)[:, None], tot, torch.zeros_like(tot)))
    return torch.stack(out)


def _wave(X, Y):
    """The deep-water wave term F, dF/dX (Havelock's form) and the Bessel functions J0, J1."""
    X = X.clamp(min=1e-7)
    th, wt = (torch.tensor(t) for t in np.polynomial.legendre.leggauss(48))
    th, wt = (th + 1) * math.pi / 4, wt / 2  # 2/pi times the weights of [0, pi/2]
    e, h0, h1 = torch.exp(-Y), torch.zeros_like(X), torch.zeros_like(X)
    i0, i1 = torch.zeros_like(X), torch.zeros_like(X)
    for t, w in zip(th, wt):
        ct = math.cos(t)
        h0 += w * torch.sin(X * ct)
        h1 += w * ct * torch.cos(X * ct)
    top = torch.asinh(Y / X)
    gx, gw = np.polynomial.legendre.leggauss(16)
    for part in range(4):
        for t, w in zip(gx, gw):
            s = top * ((part + 0.5 * (t + 1.0)) / 4.0)
            f = torch.exp(X * torch.sinh(s) - Y) * top * (w / 8.0)
            i0 += f
            i1 += f / torch.cosh(s) ** 2
    j0, j1 = torch.special.bessel_j0(X), torch.special.bessel_j1(X)
    F = -math.pi * e * (h0 + torch.special.bessel_y0(X)) - 2.0 * i0
    FX = -math.pi * e * (h1 - torch.special.bessel_y1(X)) + 2.0 * i1 / X
    return F, FX, e * j0, e * j1


def _deep_potentials(v, omegas, heads):
    """The radiation and scattering potentials on the panels of a body in deep water, [F][6 + H][N]."""
    c, n, area, q = (torch.tensor(a) for a in _panels(v))
    xb = c * torch.tensor([1.0, 1.0, -1.0])
    (s0, d0), (s1, d1) = _rankine(c, q, n, c), _rankine(xb, q, n, c)
    lg = _log_part(xb, q, n, c, area)
    dx, dy = c[:, None, 0] - c[None, :, 0], c[:, None, 1] - c[None, :, 1]
    R = torch.sqrt(dx * dx + dy * dy)
    a = torch.where(R > 0, (dx * n[None, :, 0] + dy * n[None, :, 1]) / R.clamp(min=1e-300), torch.zeros_like(R))
    Z = -(c[:, None, 2] + c[None, :, 2])
    modes = np.concatenate([n.numpy(), np.cross(c.numpy(), n.numpy())], 1).T
    out = []
    for w in omegas:
        K = w * w / G
        F, FX, ej0, ej1 = _wave(K * R, K * Z)
        FY = -F - 2.0 / (K * torch.sqrt(R * R + Z * Z))
        S = torch.complex(s0 + s1 + area * K * F - 2.0 * K * lg[..., 0], area * K * (-2.0 * math.pi) * ej0)
        D = torch.complex(d0 + d1 + area * (-K * K * FX * a - K * K * FY * n[:, 2]) - 2.0 * K * lg[..., 1],
                          area * 2.0 * math.pi * K * K * (-ej1 * a - ej0 * n[:, 2]))
        u = [modes.astype(complex)]
        if len(heads):
            pot, k, kz = _incident(c.numpy(), w, 0.0, heads)
            b = np.radians(heads)[:, None]
            nn = n.numpy()
            u.append(-pot * (-1j * k * (np.cos(b) * nn[:, 0] + np.sin(b) * nn[:, 1]) + kz * nn[:, 2]))
        rhs = -(S.numpy() @ np.concatenate(u).T)
        out.append(np.linalg.solve(2.0 * math.pi * np.eye(len(v)) - D.numpy(), rhs).T)
    return np.array(out)


def exact(case, seed):
    """The exciting force of the undisturbed wave and the incident elevation of every case; of one small body in
    deep water also the coefficients and forces of the whole solve."""
    ps, out = _problems(case, seed), []
    names = dict(A="added_mass", B="radiation_damping", X="excitation_diffraction", FK="excitation_froude_krylov",
                 SC="excitation_scattering", field_incident="field_points_pressure_incident")
    for p in ps:
        w, heads, v = p["omegas"], p["headings_deg"], p["vertices"]
        r = {}
        wet = v if p.get("kinds") is None else v[p["kinds"] == 0]
        if case["sym"]:
            wet = meshes.reflect_full(wet)
        c, n, area, _ = _panels(wet)
        body, cen = p.get("panel_body", np.zeros(len(wet), np.int32)), np.array(p.get("rotation_centers", [[0.0] * 3]))
        nb = len(cen)
        modes = np.zeros((6 * nb, len(wet)))
        for b in range(nb):
            on = body == b
            modes[6 * b:6 * b + 3, on] = n[on].T
            modes[6 * b + 3:6 * b + 6, on] = np.cross(c[on] - cen[b], n[on]).T
        if len(heads):
            pot = np.array([_incident(c, x, case["depth"], heads)[0] for x in w])
            r["FK"] = 1j * RHO * w[:, None, None] * np.einsum("fhj,dj->fhd", pot, modes * area)
            if case["points"]:
                r["field_incident"] = np.array([(-1j * x / G * _incident(p["points"], x, case["depth"], heads)[0]).T for x in w])
        if nb == 1 and case["depth"] == 0 and not case["sym"] and p.get("kinds") is None and len(wet) ** 2 * len(w) <= 3e6:
            phi = _deep_potentials(wet, w, heads)
            z = -RHO * np.einsum("dj,fkj->fdk", modes * area, phi[:, :6])
            r["A"], r["B"] = z.real, -w[:, None, None] * z.imag
            if len(heads):
                r["SC"] = 1j * RHO * w[:, None, None] * np.einsum("fhj,dj->fhd", phi[:, 6:], modes * area)
                r["X"] = r["FK"] + r["SC"]
        out.append(r)
    if case["api"] == "model":
        return {names[k]: np.ascontiguousarray(v) for k, v in out[0].items()} or None
    return out if any(out) else None

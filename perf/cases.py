"""The calls a user of this framework makes, as cases to time: boundary-element assembly and
solves on closed triangle meshes, the Laplace operators, many right-hand sides, batches of
meshes and ray queries, each through its public entry point.

``listed()`` gives the named cases, ``draw(rng)`` one more of the same ranges, ``prepare``
what a program has in hand before the call, ``run`` one pass of the call, ``work`` the bytes
and operations it cannot do without, ``exact`` the outputs in 64-bit arithmetic from plain
torch where that is affordable.

Meshes are icosphere levels (80 faces at level 1, 20480 at level 5) or latitude-longitude
spheres of any size, scaled to an ellipsoid and jittered along their radii by a seeded normal
of 1 % of the mean edge, as the many-incidence workload's ellipsoid is.
"""
import importlib
import math

import numpy as np
import torch

mf = importlib.import_module("mesh-ferrofluid_gb300")
ops = mf.mesh_MOM_3d
LAPLACE, MOM, LINEAR = int(mf.BEMType.LAPLACE), int(mf.BEMType.HELMHOLTZ_MOM), int(mf.OrderType.LINEAR)
DEV = "cuda"


# ---------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest assembly a program makes (a coarse shape in an optimisation loop): Z and
        # the excitation of one wave, 120 unknowns; launches and host work dominate
        {"name": "cfie_small", "kind": "cfie", "mesh": "ico", "level": 1, "a": 1.0, "b": 1.0, "c": 1.0, "k": 2.0,
         "gq": 4, "dtype": "f32", "waves": 1},
        # the many-incidence workload's system: ellipsoid, 7680 unknowns, 512 plane waves
        {"name": "cfie_ellipsoid_512_waves", "kind": "cfie", "mesh": "ico", "level": 4, "a": 1.0, "b": 0.7, "c": 0.5,
         "k": 6.0, "gq": 4, "dtype": "f32", "waves": 512},
        # the benchmark's headline: 30720 unknowns on the sphere at ka = 10
        {"name": "cfie_sphere_30720", "kind": "cfie", "mesh": "ico", "level": 5, "a": 1.0, "b": 1.0, "c": 1.0,
         "k": 10.0, "gq": 4, "dtype": "f32", "waves": 1},
        # the double-precision path on a mesh of odd size with a smaller rule
        {"name": "cfie_f64_ragged", "kind": "cfie", "mesh": "uv", "lat": 13, "lon": 29, "a": 1.0, "b": 0.8, "c": 0.9,
         "k": 3.0, "gq": 3, "dtype": "f64", "waves": 3},
        # the 7-point-rule EFIE at the large size
        {"name": "efie_sphere_30720", "kind": "efie", "mesh": "ico", "level": 5, "a": 1.0, "b": 1.0, "c": 1.0,
         "k": 10.0, "dtype": "f32", "waves": 1},
        # the demo's whole call: topology, solve_MOM (iterative) and the scattered field on a grid
        {"name": "solve_cfie_and_radiate", "kind": "solve_cfie", "mesh": "uv", "lat": 19, "lon": 37, "a": 1.0, "b": 0.9,
         "c": 0.8, "k": 4.0, "gq": 4, "points": 65000},
        # a whole preconditioned mixed-precision EFIE solve at 7680 unknowns, ka = 2
        {"name": "solve_efie_7680", "kind": "solve_efie", "mesh": "ico", "level": 4, "a": 1.0, "b": 1.0, "c": 1.0,
         "k": 2.0},
        # the product of one impedance matrix with 512 vectors, as each many-incidence step makes it
        {"name": "product_7680_by_512", "kind": "product", "n": 7680, "m": 512},
        # a batch of uneven star shapes, one wavenumber each: all matrices and excitations
        {"name": "batch_12_stars", "kind": "batch", "count": 12, "low": 2, "high": 4, "waves": 4},
        # the reference's Laplace rule, single and double layer, as its Dirichlet demo assembles them
        {"name": "laplace_ref_5120", "kind": "laplace_ref", "mesh": "ico", "level": 4, "a": 0.5, "b": 0.5, "c": 0.5,
         "gq": 2, "dtype": "f32"},
        # the accurate rule's three packed operators, as every mixed solve and pressure step needs them
        {"name": "laplace_sym_5120", "kind": "laplace_sym", "mesh": "ico", "level": 4, "a": 1.0, "b": 1.0, "c": 1.0,
         "dtype": "f32"},
        # a skydome of rays from 8 cameras over a terrain with spheres (the ray-query demo's image size)
        {"name": "rays_1048576", "kind": "rays", "cells": 512, "balls": 12, "cameras": 8, "theta": 256},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_mesh(rng, lo, hi):
    """A latitude-longitude sphere of about lo..hi faces (spread over the logarithm), often odd."""
    f = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    lon = max(5, int(round(math.sqrt(f) * rng.uniform(0.9, 1.3))))
    lat = max(3, int(round(f / (2 * lon))) + 1)
    return {"mesh": "uv", "lat": lat, "lon": lon, "a": round(rng.uniform(0.5, 1.0), 3),
            "b": round(rng.uniform(0.5, 1.0), 3), "c": round(rng.uniform(0.5, 1.0), 3)}


def draw(rng):
    kind = rng.choice(["cfie", "cfie", "cfie", "efie", "solve_cfie", "solve_efie", "product", "batch", "laplace_ref",
                       "laplace_sym", "rays"])
    if kind == "cfie":
        f64 = rng.random() < 0.25
        return {"kind": kind, **_draw_mesh(rng, 60, 900 if f64 else 16000), "k": round(rng.uniform(1.0, 10.0), 3),
                "gq": rng.choice([3, 4, 4]), "dtype": "f64" if f64 else "f32", "waves": _log_int(rng, 1, 64)}
    if kind == "efie":
        f64 = rng.random() < 0.25
        return {"kind": kind, **_draw_mesh(rng, 60, 2500 if f64 else 20000), "k": round(rng.uniform(1.0, 10.0), 3),
                "dtype": "f64" if f64 else "f32", "waves": _log_int(rng, 1, 64)}
    if kind == "solve_cfie":
        return {"kind": kind, **_draw_mesh(rng, 300, 4000), "k": round(rng.uniform(1.0, 6.0), 3), "gq": 4,
                "points": _log_int(rng, 1000, 260000)}
    if kind == "solve_efie":
        return {"kind": kind, "mesh": "ico", "level": rng.choice([3, 4]), "a": 1.0, "b": round(rng.uniform(0.9, 1.0), 3),
                "c": 1.0, "k": round(rng.uniform(1.0, 2.2), 3)}
    if kind == "product":
        return {"kind": kind, "n": 2 * _log_int(rng, 240, 3840), "m": _log_int(rng, 2, 512)}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 24), "low": rng.randint(1, 2), "high": 3,
                "waves": rng.randint(1, 4)}
    if kind == "laplace_ref":
        return {"kind": kind, **_draw_mesh(rng, 200, 6000), "gq": rng.choice([2, 2, 3]), "dtype": "f32"}
    if kind == "laplace_sym":
        return {"kind": kind, **_draw_mesh(rng, 200, 6000), "dtype": rng.choice(["f32", "f32", "f32", "f64"])
                if rng.random() < 0.5 else "f32"}
    return {"kind": kind, "cells": _log_int(rng, 16, 512), "balls": rng.randint(0, 12), "cameras": rng.randint(1, 8),
            "theta": _log_int(rng, 32, 256)}


# ---------------------------------------------------------------------------------------
# meshes
# ---------------------------------------------------------------------------------------
def _icosphere(level):
    """The refined icosahedron, vertices on the unit sphere, children of a face next to each other."""
    v, f = mf.meshes.icosphere(0)
    f = f.astype(np.int64)
    for _ in range(level):
        e = np.stack((f, np.roll(f, -1, 1)), -1)  # edges ab, bc, ca of each face
        key = e.min(-1) * v.shape[0] + e.max(-1)
        uniq, inv = np.unique(key.reshape(-1), return_inverse=True)
        mid = 0.5 * (v[uniq // v.shape[0]] + v[uniq % v.shape[0]])
        mid /= np.linalg.norm(mid, axis=1, keepdims=True)
        m = inv.reshape(-1, 3) + v.shape[0]
        v = np.concatenate((v, mid))
        f = np.stack((np.stack((f[:, 0], m[:, 0], m[:, 2]), 1), np.stack((f[:, 1], m[:, 1], m[:, 0]), 1),
                      np.stack((f[:, 2], m[:, 2], m[:, 1]), 1), m), 1).reshape(-1, 3)
    return v, f


def _uv_sphere(lat, lon):
    """Latitude-longitude sphere: lon (lat - 1) + 2 vertices, 2 lon (lat - 1) faces, seen from outside
    counter-clockwise."""
    th = np.pi * np.arange(1, lat) / lat
    ph = 2.0 * np.pi * np.arange(lon) / lon
    ring = np.stack((np.sin(th)[:, None] * np.cos(ph), np.sin(th)[:, None] * np.sin(ph),
                     np.cos(th)[:, None] + 0.0 * ph), -1).reshape(-1, 3)
    v = np.concatenate(([[0.0, 0.0, 1.0]], ring, [[0.0, 0.0, -1.0]]))
    j, j1 = np.arange(lon), (np.arange(lon) + 1) % lon
    f = [np.stack((0 * j, 1 + j, 1 + j1), 1)]
    for i in range(lat - 2):
        a, b = 1 + i * lon, 1 + (i + 1) * lon
        f.append(np.stack((np.stack((a + j, b + j, b + j1), 1), np.stack((a + j, b + j1, a + j1), 1)), 1).reshape(-1, 3))
    last = 1 + (lat - 2) * lon
    f.append(np.stack((last + j, 0 * j + v.shape[0] - 1, last + j1), 1))
    return v, np.concatenate(f)


def _mesh(case, seed):
    """(verts float64 [V, 3], faces int32 [F, 3]) as numpy."""
    v, f = _icosphere(case["level"]) if case["mesh"] == "ico" else _uv_sphere(case["lat"], case["lon"])
    h = np.linalg.norm(v[f[:, 0]] - v[f[:, 1]], axis=1).mean()
    v = v * (1.0 + 0.01 * h * np.random.default_rng(seed).standard_normal((v.shape[0], 1)))
    return v * np.array([case["a"], case["b"], case["c"]]), f.astype(np.int32)


def _star(level, rng):
    """A star-shaped surface r = 1 + a few smooth bumps up to 15 %."""
    v, f = _icosphere(level)
    r = np.ones(v.shape[0])
    for _ in range(6):
        d = rng.standard_normal(3)
        t = v @ (d / np.linalg.norm(d))
        r += rng.uniform(0.0, 0.15) * np.polynomial.legendre.legval(t, np.eye(5)[rng.integers(0, 5)])
    return v * r[:, None], f.astype(np.int32)


def _n_faces(case):
    return 20 * 4 ** case["level"] if case["mesh"] == "ico" else 2 * case["lon"] * (case["lat"] - 1)


def _waves(k, n, rng):
    """n plane waves of random direction and polarisation, unit amplitude, as [n, 9] float64."""
    d = rng.standard_normal((n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    e = np.cross(d, rng.standard_normal((n, 3)))
    e /= np.linalg.norm(e, axis=1, keepdims=True)
    return ops.plane_waves(k, d, e, device=DEV)


def _dtype(case):
    return torch.float64 if case.get("dtype") == "f64" else torch.float32


# ---------------------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------------------
def _on_device(case, seed):
    v, f = _mesh(case, seed)
    return torch.tensor(v, dtype=_dtype(case), device=DEV), torch.tensor(f, device=DEV)


def _batch_meshes(case, seed):
    rng = np.random.default_rng(seed)
    levels = [case["low"] + i % (case["high"] - case["low"] + 1) for i in range(case["count"])]
    return [_star(lv, rng) for lv in levels], [float(k) for k in rng.uniform(1.0, 8.0, case["count"])], rng


def _scene(case, seed):
    """A seeded height field and a few spheres above it; cameras above the terrain."""
    rng = np.random.default_rng(seed)
    n = case["cells"]
    g = np.linspace(-4.0, 4.0, n + 1)
    x, y = np.meshgrid(g, g, indexing="ij")
    z = 0.0 * x
    for _ in range(6):
        z += rng.uniform(0.05, 0.3) * np.sin(rng.uniform(0.5, 3.0) * x + rng.uniform(0.5, 3.0) * y + rng.uniform(0, 6))
    verts, faces = [np.stack((x, y, z), -1).reshape(-1, 3)], []
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    p = (i * (n + 1) + j).reshape(-1)
    faces.append(np.stack((np.stack((p, p + n + 1, p + n + 2), 1), np.stack((p, p + n + 2, p + 1), 1)), 1).reshape(-1, 3))
    top, bv, bf = verts[0].shape[0], *_icosphere(4)
    for _ in range(case["balls"]):
        c = np.array([*rng.uniform(-3.0, 3.0, 2), rng.uniform(1.5, 3.0)])
        verts.append(bv * rng.uniform(0.1, 0.4) + c)
        faces.append(bf + top)
        top += bv.shape[0]
    cams = np.stack((rng.uniform(-3.0, 3.0, case["cameras"]), rng.uniform(-3.0, 3.0, case["cameras"]),
                     rng.uniform(1.6, 2.4, case["cameras"])), 1)
    return np.concatenate(verts), np.concatenate(faces), cams


def prepare(case, seed):
    kind, rng = case["kind"], np.random.default_rng(seed + 1)
    s = {"case": case}
    if kind in ("cfie", "efie"):
        s["verts"], s["faces"] = _on_device(case, seed)
        edges, s["fei"], _ = mf.utils.get_edge_unique(s["verts"], s["faces"])
        s["n_edges"] = edges.shape[0]
        s["waves"] = _waves(case["k"], case["waves"], rng)
        s["solver"] = mf.MeshBEMSolver3d(case.get("gq", 4), LINEAR, MOM, case["k"], dtype=_dtype(case), device=DEV,
                                         rule="reference" if kind == "cfie" else "dunavant7")
    elif kind == "solve_cfie":
        s["verts"], s["faces"] = _on_device(case, seed)
        s["solver"] = mf.MeshBEMSolver3d(case["gq"], LINEAR, MOM, case["k"], dtype=torch.float32, device=DEV,
                                         solver="gmres", gmres_tol=1e-7)
        p = rng.uniform(-3.0, 3.0, (case["points"], 3))
        p *= np.maximum(1.0, 1.3 / np.linalg.norm(p, axis=1, keepdims=True))
        s["points"] = torch.tensor(p, dtype=torch.float32, device=DEV)
    elif kind == "solve_efie":
        s["verts"], s["faces"] = _on_device(case, seed)
        edges, s["fei"], _ = mf.utils.get_edge_unique(s["verts"], s["faces"])
        s["n_edges"] = edges.shape[0]
        s["areas"] = mf.utils.compute_face_areas(s["verts"], s["faces"]).contiguous()
        s["waves"] = _waves(case["k"], 1, rng)
    elif kind == "product":
        s["z"] = ops.split_tf32(_product_matrix(case, seed))
        s["x"] = _product_vectors(case, seed)
    elif kind == "batch":
        meshes, ks, rng = _batch_meshes(case, seed)
        s["batch"] = mf.batch.MeshBatch(meshes, ks, device=DEV, formulation="cfie_ref")
        s["waves"] = torch.stack([_waves(k, case["waves"], rng) for k in ks])
    elif kind == "laplace_ref":
        s["verts"], s["faces"] = _on_device(case, seed)
        s["areas"] = mf.utils.compute_face_areas(s["verts"], s["faces"]).contiguous()
        s["normals"] = mf.utils.compute_face_normals(s["verts"], s["faces"]).contiguous()
        s["relation"] = mf.utils.compute_panel_relation(s["faces"])
        kw = dict(gaussQR=case["gq"], order_type=LINEAR, BEM_type=LAPLACE, wavenumber=1.0, logger=None,
                  dtype=_dtype(case), device=DEV)
        s["V"], s["K"] = mf.SingleLayer3d(**kw), mf.DoubleLayer3d(**kw)
    elif kind == "laplace_sym":
        s["verts"], s["faces"] = _on_device(case, seed)
    else:
        v, f, cams = _scene(case, seed)
        s["app"] = mf.RayQueryApp(torch.tensor(v, dtype=torch.float32, device=DEV), torch.tensor(f, device=DEV))
        s["origins"] = torch.tensor(cams, dtype=torch.float32, device=DEV)
        d = mf.ray_query.SampleSkydomRays(2 * case["theta"] ** 2, device=DEV)[0]
        s["dirs"] = d[None].expand(case["cameras"], -1, -1).contiguous()
    return s


def _product_matrix(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    n = case["n"]
    z = torch.randn((n, n), generator=g, dtype=torch.complex64, device=DEV)
    return z / (1.0 + torch.arange(n, device=DEV).sub(torch.arange(n, device=DEV)[:, None]).abs())


def _product_vectors(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed + 1)
    return torch.randn((case["n"], case["m"]), generator=g, dtype=torch.complex64, device=DEV)


def run(s):
    kind = s["case"]["kind"]
    if kind in ("cfie", "efie"):
        z, rhs, areas = s["solver"].assemble_MOM(s["verts"], s["faces"], s["n_edges"], s["fei"], s["waves"])
        return {"Z": z, "rhs": rhs, "areas": areas}
    if kind == "solve_cfie":
        verts, faces = s["verts"], s["faces"]
        edges, fei, _ = mf.utils.get_edge_unique(verts, faces)
        js = s["solver"].solve_MOM(verts, faces, edges, fei)
        h = ops.radiate_H(s["points"], verts, mf.utils.compute_vert_areas(verts, faces), js[0], s["case"]["k"])
        return {"J": js, "H": h}
    if kind == "solve_efie":
        v, f, fei, n, k = s["verts"], s["faces"], s["fei"], s["n_edges"], s["case"]["k"]
        pairs = ops.near_pairs(f)
        z = ops.assemble_Z_rwg_sym(v, f, fei, n, k, pairs=pairs)
        rhs = ops.assemble_rhs_rwg_sym(v, f, fei, n, s["waves"])
        m = ops.spai_preconditioner(z, v, f, fei, n, pairs=pairs)
        x, _ = ops.pgmres(z, rhs, M=m, tol=1e-7, Z_half=ops.half_copy(z))
        return {"J": ops.interpolate_vert_js(v, f, fei, s["areas"], x.reshape(1, n))}
    if kind == "product":
        return {"Y": ops.multi_rhs_matmul(s["z"], s["x"])}
    if kind == "batch":
        z = s["batch"].assemble()
        return {"Z": z, "B": s["batch"].excitation(s["waves"])}
    if kind == "laplace_ref":
        out = {}
        for name, layer in (("V", s["V"]), ("K", s["K"])):
            getattr(layer, f"compute_{name}mat")(s["verts"], s["faces"], s["areas"], s["normals"], s["relation"])
            out[name] = getattr(layer, f"get_{name}mat_tight")(verts=s["verts"], faces=s["faces"])
        return out
    if kind == "laplace_sym":
        near = mf.layers.laplace_near_pairs(s["faces"], s["verts"].shape[0])
        return {name: mf.layers.laplace_sym_tight(s["verts"], s["faces"], op, near)
                for name, op in (("V", 1), ("K", 2), ("D", 3))}
    return {"hits": s["app"].QueryForNLOS(s["origins"], s["dirs"])}


# ---------------------------------------------------------------------------------------
# work: inputs read once, outputs written once; kernel evaluations of the rule at their
# algorithmic operation counts (CFIE 50, EFIE 30, Laplace single 15 / double 22, field 61)
# ---------------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "product":
        n, m = case["n"], case["m"]
        return {"bytes": 8.0 * n * n + 16.0 * n * m, "flops": 8.0 * n * n * m}
    if kind == "rays":
        f = 2 * case["cells"] ** 2 + 5120 * case["balls"]
        n = 2 * case["theta"] ** 2 * case["cameras"]
        return {"bytes": 28.0 * n + 36.0 * f, "flops": 40.0 * n * math.log2(f)}
    if kind == "batch":
        b = q = 0.0
        for i in range(case["count"]):
            f = 20.0 * 4 ** (case["low"] + i % (case["high"] - case["low"] + 1))
            b += 8 * (1.5 * f) ** 2 + 8 * case["waves"] * 1.5 * f
            q += 50.0 * 1296 * f * f
        return {"bytes": b, "flops": q}
    f = float(_n_faces(case))
    e, v, size = 1.5 * f, 0.5 * f + 2, 8 if case.get("dtype") == "f64" else 4
    if kind in ("cfie", "solve_cfie"):
        flops = 50.0 * 9 * case["gq"] ** 2 * (case["gq"] - 1) ** 2 * f * f
    elif kind in ("efie", "solve_efie"):
        flops = 30.0 * 49 * f * f
    if kind in ("cfie", "efie"):
        return {"bytes": 2 * size * e * e + 2 * size * e * case["waves"] + 36 * f, "flops": flops}
    if kind == "solve_cfie":  # Z is written once and read by about 40 products
        return {"bytes": 8 * e * e * 41 + 36 * case["points"], "flops": flops + 8 * 40 * e * e + 61 * v * case["points"]}
    if kind == "solve_efie":  # Z written and halved, then about 40 products on 4-byte entries
        return {"bytes": 8 * e * e * 3 + 4 * e * e * 40, "flops": flops + 8 * 40 * e * e}
    if kind == "laplace_ref":
        return {"bytes": 2 * size * v * v + 36 * f, "flops": (15.0 + 22.0) * case["gq"] ** 4 * f * f}
    return {"bytes": 3 * size * v * v + 36 * f, "flops": (15.0 + 22.0 + 15.0) * 49 * f * f}


# ---------------------------------------------------------------------------------------
# exact: plain torch in 64 bits
# ---------------------------------------------------------------------------------------
def _gauss(n, dtype):
    """Gauss-Legendre nodes and weights on [0, 1]; the tables pass through float32, the map to
    [0, 1] is done in the solver's type."""
    x, w = np.polynomial.legendre.leggauss(n)
    base = np.float64 if dtype == torch.float64 else np.float32
    x, w = x.astype(np.float32).astype(base), w.astype(np.float32).astype(base)
    return (((x + base(1)) / base(2)).astype(np.float64), (w / base(2)).astype(np.float64))


def _collapsed(n, dtype):
    """(r1, r2, w r1) of the collapsed rule on the triangle."""
    p, w = _gauss(n, dtype)
    r1 = np.repeat(p, n)
    return [torch.tensor(t, device=DEV) for t in (r1, np.tile(p, n) * r1, np.repeat(w, n) * np.tile(w, n) * r1)]


class _Geometry:
    """Face-edge data of a mesh in 64 bits: corners from the vertex opposite each local edge."""

    def __init__(self, verts, faces):
        self.v, self.f = verts.double(), faces.long()
        p = self.v[self.f]  # [F, 3, 3]
        cr = torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 1])
        self.area = 0.5 * cr.norm(dim=-1)
        self.normal = cr / (2.0 * self.area[:, None])
        self.c = torch.stack([p[:, [e, (e + 1) % 3, (e + 2) % 3]] for e in range(3)], 1).reshape(-1, 3, 3)
        ids = torch.stack([self.f[:, [(e + 1) % 3, (e + 2) % 3]] for e in range(3)], 1).reshape(-1, 2)
        side = (self.c[:, 2] - self.c[:, 1]).norm(dim=-1)
        self.scale = torch.where(ids[:, 0] < ids[:, 1], side, -side) / (2.0 * self.area.repeat_interleave(3))

    def points(self, rule):
        r1, r2, w = rule
        m = torch.stack((1.0 - r1, r1 - r2, r2), 1)  # [n, 3]
        return torch.einsum("nk,fkd->fnd", m, self.c), 2.0 * self.area.repeat_interleave(3)[:, None] * w[None]


def _edges(v, f):
    """The face-edge -> edge map, edges numbered by increasing (larger id, smaller id)."""
    f = f.long()
    e = torch.stack((f[:, [1, 2]], f[:, [2, 0]], f[:, [0, 1]]), 1).reshape(-1, 2)
    key = e.max(1)[0] * v.shape[0] + e.min(1)[0]
    uniq, inv = torch.unique(key, return_inverse=True)
    return inv, uniq.numel()


def _exact_cfie_z(verts, faces, gq, k, dtype):
    g = _Geometry(verts, faces)
    x, wx = g.points(_collapsed(gq, dtype))
    y, wy = g.points(_collapsed(gq - 1, dtype))
    n, (fei, ne) = g.c.shape[0], _edges(verts, faces)
    Z = torch.zeros((ne, ne), dtype=torch.complex128, device=DEV)
    rows = max(1, int(2.0e7 // (x.shape[1] * n * y.shape[1])))
    for r0 in range(0, n, rows):
        sl = slice(r0, min(n, r0 + rows))
        xs, a = x[sl], x[sl] - g.c[sl, None, 0]
        nr = g.normal.repeat_interleave(3, 0)[sl]
        an = torch.linalg.cross(a, nr[:, None, :].expand_as(a))
        d = xs[:, :, None, None, :] - y[None, None]  # [r, i, col, j, 3]
        R = d.norm(dim=-1)
        G = torch.polar(wy[None, None] / (4.0 * math.pi * R), -k * R)
        # h = G (1 + jkR) / R^2 times y.u with y from B0, u = (x - B0) x ((x - A0) x n)
        rho = y - g.c[:, None, 0]  # [col, j, 3]
        u = torch.linalg.cross(xs[:, :, None, :] - g.c[None, None, :, 0], an[:, :, None, :].expand(-1, -1, n, -1))
        yu = torch.einsum("cjd,ricd->ricj", rho, u)
        ay = torch.einsum("rid,cjd->ricj", a, rho)
        term = G * torch.complex(-yu / R ** 2, k * ay - 4.0 / k - yu * k / R)
        z = torch.einsum("ri,ricj->rc", wx[sl].to(term.dtype), term)
        same = torch.nonzero((torch.arange(n, device=DEV) // 3)[None, :] ==
                             (torch.arange(r0, r0 + z.shape[0], device=DEV) // 3)[:, None])
        rr, cc = same[:, 0], same[:, 1]
        s = (wx[sl][rr] * (a[rr] * (xs[rr] - g.c[cc, 0][:, None, :])).sum(-1)).sum(-1)
        z[rr, cc] += 0.5 * s
        z = z * g.scale[sl, None] * g.scale[None]
        t = torch.zeros((z.shape[0], ne), dtype=z.dtype, device=DEV).index_add_(1, fei, z)
        Z.index_add_(0, fei[sl], t)
    return Z


def _exact_cfie_rhs(verts, faces, gq, waves, dtype):
    g = _Geometry(verts, faces)
    x, w = g.points(_collapsed(gq, dtype))
    fv = g.scale[:, None, None] * (x - g.c[:, None, 0])
    n, (fei, ne) = g.normal.repeat_interleave(3, 0), _edges(verts, faces)
    out = torch.zeros((ne, waves.shape[0]), dtype=torch.complex128, device=DEV)
    for r in range(waves.shape[0]):
        kv, e, h = waves[r, 0:3], waves[r, 3:6], waves[r, 6:9]
        proj = (fv * (e + torch.linalg.cross(n, h.expand_as(n)))[:, None]).sum(-1)
        out[:, r].index_add_(0, fei, (torch.polar(w * proj, -(x @ kv))).sum(-1))
    return out


def _dunavant7():
    r = math.sqrt(15.0)
    b, w = [[1 / 3, 1 / 3, 1 / 3]], [0.225]
    for q, wt in (((6 - r) / 21, (155 - r) / 1200), ((6 + r) / 21, (155 + r) / 1200)):
        for i in range(3):
            row = [q, q, q]
            row[i] = 1.0 - 2.0 * q
            b.append(row)
            w.append(wt)
    return torch.tensor(b, dtype=torch.float64, device=DEV), torch.tensor(w, dtype=torch.float64, device=DEV)


def _exact_efie_rhs(verts, faces, waves):
    g, (b, w) = _Geometry(verts, faces), _dunavant7()
    x = torch.einsum("nk,fkd->fnd", b, g.c)
    fv = g.scale[:, None, None] * (x - g.c[:, None, 0])
    wt = g.area.repeat_interleave(3)[:, None] * w[None]
    fei, ne = _edges(verts, faces)
    out = torch.zeros((ne, waves.shape[0]), dtype=torch.complex128, device=DEV)
    for r in range(waves.shape[0]):
        out[:, r].index_add_(0, fei, torch.polar(wt * (fv @ waves[r, 3:6]), -(x @ waves[r, 0:3])).sum(-1))
    return out


def _exact_solve_cfie(case, seed):
    verts, faces = _on_device(case, seed)
    k = case["k"]
    Z = _exact_cfie_z(verts, faces, case["gq"], k, torch.float32)
    az, hd = math.pi / 6, math.pi / 6 - 0.5 * math.pi
    wave = torch.tensor([[k * math.cos(az), k * math.sin(az), 0, 0, 0, 1, math.cos(hd), math.sin(hd), 0]],
                        dtype=torch.float64, device=DEV)
    x = torch.linalg.solve(Z, _exact_cfie_rhs(verts, faces, case["gq"], wave, torch.float32))[:, 0]
    g, (fei, _) = _Geometry(verts, faces), _edges(verts, faces)
    J = torch.zeros((verts.shape[0], 3), dtype=torch.complex128, device=DEV)
    for e in range(3):
        for s in (1, 2):
            c = (g.scale[:, None] * (g.c[:, s] - g.c[:, 0])).reshape(-1, 3, 3)[:, e] * x[fei].reshape(-1, 3)[:, e, None]
            J.index_add_(0, g.f[:, (e + s) % 3], c)
    va = torch.zeros(verts.shape[0], dtype=torch.float64, device=DEV)
    va.index_add_(0, g.f.reshape(-1), (g.area / 3.0).repeat_interleave(3))
    p = prepare(case, seed)["points"].double()
    H = []
    for q in p.split(max(1, int(1.0e7 // verts.shape[0]))):
        # (1 + jkR) e^{jkR} / (4 pi R^3) (p - v), the phase sign of the reference's field helper
        d = q[:, None] - g.v[None]
        R = d.norm(dim=-1)
        G = torch.polar(1.0 / (4.0 * math.pi * R), k * R)
        f = (G * torch.complex(1.0 / R ** 2, k / R))[..., None] * d
        H.append((va[None, :, None] * torch.linalg.cross(J[None].expand_as(f), f)).sum(1))
    return {"J": J[None], "H": torch.cat(H)}


def _sauter_points(gq):
    """Per panel relation 0..3 the flattened rows (r1x, r2x, r1y, r2y, weight) of the reference's
    4-D rule: relative-coordinate maps of the collapsed rule taken twice."""
    p, w = (t.astype(np.float64) for t in _gauss(gq, torch.float32))
    r1, r2 = np.tile(p, gq), np.repeat(p, gq) * np.tile(p, gq)
    wt, q = np.repeat(w, gq) * np.tile(w, gq), gq * gq
    x, a = np.tile(r1, q), np.tile(r2, q)
    b, c = np.repeat(r1, q), np.repeat(r2, q)
    ww = np.repeat(wt, q) * np.tile(wt, q)
    ab, abc = a * b, a * b * c

    def edge(w0, w1, w2, w3):
        return w0, w3, w0 + w1, w2

    def face(z0, z1, z2, z3):
        return z0, z1, z0 - z2, z1 - z3

    w0, w1, w2, w3 = x, x * a, x * ab, x * abc
    maps = [
        [((x, a * x, b, b * c), x * b)],
        [((x, x * a, x * b, x * b * c), x ** 3 * b), ((x * b, x * b * c, x, x * a), x ** 3 * b)],
        [(edge(x, -x * ab, x * a * (1 - b), x * a * c), x ** 3 * a ** 2),
         (edge(x, -x * abc, x * ab * (1 - c), x * a), x ** 3 * a ** 2 * b),
         (edge(x * (1 - ab), x * ab, x * abc, x * a * (1 - b)), x ** 3 * a ** 2 * b),
         (edge(x * (1 - abc), x * abc, x * a, x * ab * (1 - c)), x ** 3 * a ** 2 * b),
         (edge(x * (1 - abc), x * abc, x * ab, x * a * (1 - b * c)), x ** 3 * a ** 2 * b)],
        [(face(w0, w0 - w1 + w2, w3, w2), x ** 3 * a ** 2 * b),
         (face(w0, w1 - w2 + w3, w2, w3), x ** 3 * a ** 2 * b),
         (face(w0 - w3, w1 - w3, -w3, w2 - w3), x ** 3 * a ** 2 * b)],
    ]
    rows = []
    for m in maps:
        rows.append(torch.tensor(np.concatenate([np.stack((*pts, jac * ww), 1) for pts, jac in m]), device=DEV))
    return rows


def _exact_laplace_ref(case, seed):
    verts, faces = _on_device(case, seed)
    g, nf, nv = _Geometry(verts, faces), faces.shape[0], verts.shape[0]
    rel = (g.f[:, None, :, None] == g.f[None, :, None, :]).flatten(2).sum(-1).clamp_max(3)
    p = g.v[g.f]
    out = {name: torch.zeros((nv, nv), dtype=torch.float64, device=DEV) for name in ("V", "K")}
    rules = _sauter_points(case["gq"])
    for r, rows in enumerate(rules):
        fy, fx = torch.nonzero(rel == r, as_tuple=True)
        X = torch.stack((1 - rows[:, 0], rows[:, 0] - rows[:, 1], rows[:, 1]), 1)
        Y = torch.stack((1 - rows[:, 2], rows[:, 2] - rows[:, 3], rows[:, 3]), 1)
        step = max(1, int(3.0e7 // rows.shape[0]))
        for a, b in zip(fy.split(step), fx.split(step)):
            d = torch.einsum("nk,pkd->pnd", X, p[b]) - torch.einsum("nk,pkd->pnd", Y, p[a])
            R = d.norm(dim=-1)
            jac = (4.0 * g.area[a] * g.area[b])[:, None] * rows[:, 4] / (4.0 * math.pi)
            for name, ker in (("V", 1.0 / R), ("K", torch.einsum("pnd,pd->pn", d, g.normal[a]) / R ** 3)):
                m = torch.einsum("pn,ni,nj->pij", ker * jac, Y, X)
                at = g.f[a][:, :, None] * nv + g.f[b][:, None, :]
                out[name].view(-1).index_add_(0, at.reshape(-1), m.reshape(-1))
    return out


def _triangle_potential(x, t):
    """Integrals over triangles t [n, 3, 3] of 1/R and (y - x_t)/R for points x [n, m, 3], x_t the
    projection of x on the triangle's plane (Wilton et al. 1984)."""
    cr = torch.linalg.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0])
    n = (cr / cr.norm(dim=-1, keepdim=True))[:, None]
    d = ((x - t[:, None, 0]) * n).sum(-1)
    proj = x - d[..., None] * n
    I0, I1 = torch.zeros_like(d), torch.zeros_like(x)
    for i in range(3):
        a, b = t[:, None, i], t[:, None, (i + 1) % 3]
        s = (b - a) / (b - a).norm(dim=-1, keepdim=True)
        m = torch.linalg.cross(s.expand_as(x), n.expand_as(x))
        P0 = ((a - proj) * m).sum(-1)
        lm, lp = ((a - proj) * s).sum(-1), ((b - proj) * s).sum(-1)
        Rm, Rp = (x - a).norm(dim=-1), (x - b).norm(dim=-1)
        R02 = P0 ** 2 + d ** 2
        up = lm + lp > 0
        f = torch.where(up, torch.log((Rp + lp) / (Rm + lm).clamp_min(1e-300)),
                        torch.log((Rm - lm).clamp_min(1e-300) / (Rp - lp).clamp_min(1e-300)))
        f = torch.where(R02 > 1e-28, f, torch.zeros_like(f))
        ad = d.abs()
        I0 += P0 * f - ad * (torch.atan2(P0 * lp, R02 + ad * Rp) - torch.atan2(P0 * lm, R02 + ad * Rm))
        I1 += 0.5 * (R02 * f + lp * Rp - lm * Rm)[..., None] * m
    return I0, I1, proj


def _exact_laplace_sym(case, seed):
    verts, faces = _on_device(case, seed)
    g, nf, nv = _Geometry(verts, faces), faces.shape[0], verts.shape[0]
    b, w = _dunavant7()
    p = g.v[g.f]
    x = torch.einsum("nk,fkd->fnd", b, p)
    near = (g.f[:, None, :, None] == g.f[None, :, None, :]).flatten(2).any(-1)
    V = torch.zeros((nv, nv), dtype=torch.float64, device=DEV)
    V0 = torch.zeros((nf, nf), dtype=torch.float64, device=DEV)
    hat = torch.stack([torch.linalg.cross(g.normal, p[:, (a + 2) % 3] - p[:, (a + 1) % 3]) for a in range(3)], 1)
    hat = hat / (2.0 * g.area[:, None, None])  # gradients of the corner functions

    def add(fy, fx, m):  # m [n, a, b] without the 1 / (4 pi)
        at = g.f[fy][:, :, None] * nv + g.f[fx][:, None, :]
        V.view(-1).index_add_(0, at.reshape(-1), m.reshape(-1) / (4.0 * math.pi))
        V0[fy, fx] = m.sum((1, 2)) / (4.0 * math.pi)

    fy, fx = torch.nonzero(~near, as_tuple=True)
    for i, j in zip(fy.split(500000), fx.split(500000)):
        ri = 1.0 / (x[i][:, :, None] - x[j][:, None]).norm(dim=-1)  # [n, y point, x point]
        add(i, j, torch.einsum("pst,sa,tb->pab", ri, w[:, None] * b, w[:, None] * b)
            * (g.area[i] * g.area[j])[:, None, None])
    fy, fx = torch.nonzero(near, as_tuple=True)
    I0, I1, proj = _triangle_potential(x[fx], p[fy])
    at0 = 1.0 / 3.0 + torch.einsum("pad,pnd->pna", hat[fy], proj - p[fy].mean(1)[:, None])
    inner = at0 * I0[..., None] + torch.einsum("pad,pnd->pna", hat[fy], I1)
    add(fy, fx, torch.einsum("pna,n,nb->pab", inner, w, b) * g.area[fx][:, None, None])
    curl = torch.stack([p[:, (a + 1) % 3] - p[:, (a + 2) % 3] for a in range(3)], 1) / (2.0 * g.area[:, None, None])
    D = torch.zeros((nv, nv), dtype=torch.float64, device=DEV)
    for d in range(3):
        C = torch.zeros((nv, nf), dtype=torch.float64, device=DEV)
        C.index_put_((g.f.reshape(-1), torch.arange(nf, device=DEV).repeat_interleave(3)), curl[:, :, d].reshape(-1),
                     accumulate=True)
        D += C @ V0 @ C.T
    return {"V": V, "K": None, "D": D}


def exact(case, seed):
    kind = case["kind"]
    if kind == "cfie":
        s, small = prepare(case, seed), _n_faces(case) <= 2000
        g = _Geometry(s["verts"], s["faces"])
        return {"Z": _exact_cfie_z(s["verts"], s["faces"], case["gq"], case["k"], _dtype(case)) if small else None,
                "rhs": _exact_cfie_rhs(s["verts"], s["faces"], case["gq"], s["waves"], _dtype(case)),
                "areas": g.area[:, None]}
    if kind == "efie":  # Z: the singular pairs' closed forms have no short restatement
        s = prepare(case, seed)
        return {"Z": None, "rhs": _exact_efie_rhs(s["verts"], s["faces"], s["waves"]),
                "areas": _Geometry(s["verts"], s["faces"]).area[:, None]}
    if kind == "solve_cfie":
        return _exact_solve_cfie(case, seed) if _n_faces(case) <= 2000 else None
    if kind == "product":
        return {"Y": _product_matrix(case, seed).to(torch.complex128) @ _product_vectors(case, seed).to(torch.complex128)}
    if kind == "batch":
        meshes, ks, rng = _batch_meshes(case, seed)
        total = sum(f.shape[0] ** 2 for _, f in meshes)
        z, rhs = [], []
        for (v, f), k in zip(meshes, ks):
            v, f = torch.tensor(v, dtype=torch.float32, device=DEV), torch.tensor(f, device=DEV)
            w = _waves(k, case["waves"], rng)
            rhs.append(_exact_cfie_rhs(v, f, 4, w, torch.float32))
            if total <= 4.0e6:  # even edge counts: the rows are not padded
                z.append(_exact_cfie_z(v, f, 4, k, torch.float32).reshape(-1))
        top = max(r.shape[0] for r in rhs)
        B = torch.cat([torch.cat((r, r.new_zeros((top - r.shape[0], r.shape[1])))) for r in rhs], 1)
        return {"Z": torch.cat(z) if z else None, "B": B}
    if kind == "laplace_ref":
        return _exact_laplace_ref(case, seed)
    if kind == "laplace_sym":
        return _exact_laplace_sym(case, seed)
    return None  # ray queries: found by search, not computed by a formula

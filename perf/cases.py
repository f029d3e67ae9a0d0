"""Workloads of the evaluator over the range of its use: what is prepared once, the call that a
frame repeats, the bytes and operations that call cannot do without, and its result in 64 bits.

A case names a kind and plain sizes:

* ``refine``: EvalStencils over a device table (GB300StencilTable), uniform refinement;
* ``raw``: EvalStencils over plain device arrays in Far's layout, as a client holding its own
  CudaStencilTable-shaped arrays calls it;
* ``limit``: EvalStencils over a limit table with derivative weights (P, du, dv or all six);
* ``patches``: device PatchMap lookup and EvalPatches at scattered limit locations;
* ``batch``: one frame of many uneven meshes through GB300StencilBatch's graph;
* ``tess``: Bfr-style tessellation of every face of a mesh and its limit points.

Stencil cages come from ``opensubdiv_gb300.shapes`` (seeded tori and cubes with split quads and
creases), patch tables from the reference's own small tables under ``tests/golden``, instanced
to the wanted size.  All data is float32, as everything the evaluator takes.
"""
from __future__ import annotations

import functools
import math
import os

import numpy as np
import torch

from opensubdiv_gb300 import shapes, workloads
from opensubdiv_gb300.bfr import MeshTessellation
from opensubdiv_gb300.evaluator import (BufferDescriptor, GB300Evaluator, GB300PatchTable,
                                        GB300StencilBatch, GB300StencilTable)
from opensubdiv_gb300.topology import UniformRefiner

GOLDEN = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests", "golden")
WEIGHTS = ("weights", "du_weights", "dv_weights", "duu_weights", "duv_weights", "dvv_weights")


# ---- the cases ---------------------------------------------------------------------------------

def listed():
    return [
        # a prop or a character part, refined every frame: the launch and the call count
        dict(name="refine_small", kind="refine", shape="torus", loop=False, nu=32, nv=16, level=2,
             length=3, stride=3, offset=0),
        # the unit cube of the plain method, level 4, positions only
        dict(name="refine_cube", kind="refine", shape="cube", loop=False, nu=8, nv=8, level=4,
             length=3, stride=3, offset=0),
        # a Loop character mesh of odd width: positions and a 2-wide channel, rows of 5 floats
        dict(name="refine_loop_5pv", kind="refine", shape="torus", loop=True, nu=123, nv=61,
             level=3, length=5, stride=5, offset=0),
        # the largest single mesh: 8 interleaved primvars, 8.6 M stencils
        dict(name="refine_torus_8pv", kind="refine", shape="torus", loop=False, nu=512, nv=256,
             level=3, length=8, stride=8, offset=0),
        # a client's own table arrays, wide rows
        dict(name="raw_cube_12pv", kind="raw", shape="cube", loop=False, nu=61, nv=61, level=3,
             length=12, stride=12, offset=0),
        # limit positions and tangents at scattered locations (normals of sampled points)
        dict(name="limit_uv_8pv", kind="limit", shape="torus", loop=False, nu=512, nv=256, level=3,
             points=1_000_000, length=8, stride=8, offset=0, outputs=3),
        # all six outputs for curvature at fewer locations, positions only
        dict(name="limit_second_xyz", kind="limit", shape="torus", loop=False, nu=128, nv=64,
             level=3, points=200_003, length=3, stride=3, offset=0, outputs=6),
        # scattered samples of a large adaptive Catmull-Clark mesh with Gregory end caps
        dict(name="patches_catmark", kind="patches", table="torus32x16_patches_L4", copies=234,
             points=4_000_000, length=3, stride=3, outputs=6),
        # the same of an adaptive Loop mesh
        dict(name="patches_loop", kind="patches", table="icosphere2_patches_L3", copies=96,
             points=4_000_000, length=3, stride=3, outputs=6),
        # a handful of queries (brush strokes, attachment points): position and tangents
        dict(name="patches_small", kind="patches", table="torus32x16_patches_L4", copies=1,
             points=10_000, length=3, stride=3, outputs=3),
        # a frame of a scene: uneven Catmull-Clark and Loop meshes, levels 1-4, 3-12 primvars
        dict(name="batch_scene", kind="batch", meshes=64, cv_min=500, cv_max=10_000),
        # a mesh of quads and triangles tessellated at per-edge rates, limit points and tangents
        dict(name="tess_edge_rates", kind="tess", table="bfr_torus16x8_e_f3", copies=500, length=3),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("refine", "refine", "raw", "limit", "limit", "patches", "patches", "batch",
                       "tess"))
    if kind in ("refine", "raw", "limit"):
        loop = rng.random() < 0.3
        level = rng.randint(1, 4)
        vertices = log(500, min(130_000, 8_000_000 // 4 ** level))  # of the cage
        if rng.random() < 0.5:
            nv = max(3, int(math.sqrt(vertices / 2)))
            c = dict(shape="torus", nu=max(3, vertices // nv), nv=nv)
        else:
            n = max(2, int(math.sqrt(vertices / 6)))
            c = dict(shape="cube", nu=n, nv=n)
        length = rng.choice((3, 3, 3, 4, 8, rng.randint(1, 16)))
        pad = rng.choice((0, 0, 0, rng.randint(1, 4)))  # the primvar inside a wider vertex
        c |= dict(kind=kind, loop=loop, level=level, length=length, stride=length + pad,
                  offset=rng.randint(0, pad))
        if kind == "limit":  # limit stencils of uniform refinement: Catmull-Clark cages
            c |= dict(loop=False, level=min(level, 3), points=log(1000, 1_000_000), outputs=rng.choice((3, 3, 6)))
            if c["outputs"] * length > 24:
                c["points"] = min(c["points"], 300_000)
        return c
    if kind == "patches":
        table = rng.choice(("torus32x16_patches_L4", "torus32x16_patches_L4",
                            "icosphere2_patches_L3"))
        length = rng.choice((3, 3, 3, 4, rng.randint(1, 8)))
        copies = log(1, 234)
        return dict(kind=kind, table=table, copies=copies, points=log(1000, 4_000_000 * 3 // max(3, length)),
                    length=length, stride=length + rng.choice((0, 0, rng.randint(1, 3))),
                    outputs=rng.choice((1, 3, 6)))
    if kind == "batch":
        return dict(kind=kind, meshes=log(8, 64), cv_min=500, cv_max=log(2000, 10_000))
    table = rng.choice(("bfr_torus16x8_e_f3", "bfr_icosphere1_u6_f3", "bfr_catmark_nonquads_u5_f3"))
    return dict(kind=kind, table=table, copies=log(1, 500), length=3)


# ---- inputs ------------------------------------------------------------------------------------

def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _cage(case):
    """The mesh of a case: one topology for every seed, whose values a frame moves."""
    scheme = shapes.LOOP if case["loop"] else shapes.CATMARK
    if case["shape"] == "cube":
        return shapes.cube(case["nu"], noise=0.01, seed=5, scheme=scheme)
    return shapes.torus(case["nu"], case["nv"], tri_fraction=0.05,
                        crease_fraction=0.0 if case["loop"] else 0.02, noise=0.002, seed=5,
                        scheme=scheme)


def _values(cage, case, seed):
    """The vertex buffer: moved positions and U[-1, 1] channels at the primvar's offset."""
    n, length = cage.num_vertices, case["length"]
    rng = np.random.default_rng(seed + 17)
    v = rng.uniform(-1, 1, (n, case["stride"])).astype(np.float32)
    k = min(3, length)
    xyz = cage.positions + rng.normal(0.0, 0.002, (n, 3))
    v[:, case["offset"]: case["offset"] + k] = xyz[:, :k]
    return v.ravel()


def _stencils(case, seed):
    """The cage, its vertex buffer and the host table in Far's layout."""
    cage = _cage(case)
    refiner = UniformRefiner(cage, case["level"])
    if case["kind"] != "limit":
        return cage, _values(cage, case, seed), refiner.stencil_table()
    face, u, v = shapes.uniform_locations(cage, case["points"], seed=seed + 5)
    table = refiner.limit_stencil_table(face, u, v)
    if case["outputs"] == 6:
        # the generator gives P, du, dv; second-derivative rows of the same supports, drawn so
        # that each row sums to zero as such rows do
        rng = np.random.default_rng(seed + 23)
        start = table["offsets"].astype(np.int64)
        for k in WEIGHTS[3:]:
            w = rng.normal(0.0, 4.0, len(table["indices"]))
            w -= np.repeat(np.add.reduceat(w, start) / table["sizes"], table["sizes"])
            table[k] = w.astype(np.float32)
    return cage, _values(cage, case, seed), table


def _golden(name):
    with np.load(os.path.join(GOLDEN, name + ".npz")) as z:
        return {k: z[k] for k in z.files}


def _patches(case, seed):
    """The instanced table and its source points, deformed differently in every copy."""
    z = _golden(case["table"])
    if "num_ptex" not in z:
        z["num_ptex"] = z["ptex_offsets"][-1]
    copies, length = case["copies"], case["length"]
    arrays, indices, params, _, ptex, tri = workloads.instanced_patch_table(z, copies)
    base = z["src"].reshape(-1, 3)
    rng = np.random.default_rng(seed)
    phase = rng.uniform(0, 2 * np.pi, (copies, 1, 3))
    xyz = base[None] + 0.02 * np.sin(3.0 * base[None] + phase)
    src = np.empty((copies * len(base), case.get("stride", length)), np.float32)
    src[:, :min(3, length)] = xyz.reshape(-1, 3)[:, :length]
    for k in range(3, src.shape[1]):
        src[:, k] = np.sin((1.0 + 0.3 * k) * xyz[..., k % 3] + phase[:, :, 0] * k).ravel()
    return z, arrays, indices, params, src.ravel(), ptex, tri


def _queries(case, ptex, tri, seed):
    rng = np.random.default_rng(seed + 3)
    n = case["points"]
    face = rng.integers(0, ptex, n).astype(np.int32)
    u, v = rng.random(n, np.float32), rng.random(n, np.float32)
    if tri:
        fold = u + v > 1.0
        u[fold], v[fold] = 1.0 - u[fold], 1.0 - v[fold]
    return face, u, v


def _scene(case, seed):
    """The meshes of a scene, the same for every seed, each at a moment of its own movement."""
    meshes = workloads.batch_population(case["meshes"], case["cv_min"], case["cv_max"])
    return [m | dict(src=workloads.deform(m["src"], m["phase"], seed)) for m in meshes]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("refine", "raw", "limit"):
        cage, values, table = _stencils(case, seed)
        length, n = case["length"], len(table["sizes"])
        s = dict(kind=kind, n=n, src=_cuda(values), dst_desc=BufferDescriptor(0, length, length),
                 src_desc=BufferDescriptor(case["offset"], length, case["stride"]),
                 out=[torch.zeros(n * length, device="cuda") for _ in range(case.get("outputs", 1))])
        if kind == "raw":
            s["arrays"] = [_cuda(table[k]) for k in ("sizes", "offsets", "indices", "weights")]
        else:
            s["table"] = GB300StencilTable.Create(
                table["sizes"], table["offsets"], table["indices"],
                *[table.get(k) for k in WEIGHTS])
        return s
    if kind == "patches":
        _, arrays, indices, params, src, ptex, tri = _patches(case, seed)
        face, u, v = _queries(case, ptex, tri, seed)
        n, length = case["points"], case["length"]
        return dict(kind=kind, n=n, table=GB300PatchTable.Create(arrays, indices, params, tri),
                    src=_cuda(src), face=_cuda(face), u=_cuda(u), v=_cuda(v),
                    src_desc=BufferDescriptor(0, length, case["stride"]),
                    dst_desc=BufferDescriptor(0, length, length),
                    coords=torch.zeros((n, 5), dtype=torch.int32, device="cuda"),
                    out=[torch.zeros(n * length, device="cuda") for _ in range(case["outputs"])])
    if kind == "batch":
        jobs, out = [], []
        for m in _scene(case, seed):
            t, d = m["table"], BufferDescriptor(0, m["length"], m["length"])
            out.append(torch.zeros(len(t["sizes"]) * m["length"], device="cuda"))
            jobs.append((GB300StencilTable.Create(t["sizes"], t["offsets"], t["indices"],
                                                  t["weights"]), _cuda(m["src"]), d, out[-1], d))
        return dict(kind=kind, jobs=jobs, batch=GB300StencilBatch(jobs), out=out)
    # tess
    z, arrays, indices, params, src, _, tri = _patches(case, seed)
    c = case["copies"]
    if len(z["rates"]) == len(z["verts_per_face"]):
        rates = dict(uniform_rate=int(z["rates"][0]))
    else:
        runs = np.concatenate([[0], np.tile(np.diff(z["rate_offsets"]), c)]).cumsum()
        rates = dict(rates=np.tile(z["rates"], c), rate_offsets=runs.astype(np.int32))
    mesh = MeshTessellation(int(z["regular_face_size"]), np.tile(z["verts_per_face"], c), **rates)
    n = mesh.num_coords
    return dict(kind=kind, mesh=mesh, table=GB300PatchTable.Create(arrays, indices, params, tri),
                src=_cuda(src), src_desc=BufferDescriptor(0, 3, 3),
                coords=torch.zeros((n, 2), device="cuda"),
                facets=torch.zeros((mesh.num_facets, 3), dtype=torch.int32, device="cuda"),
                patch_coords=torch.zeros((n, 5), dtype=torch.int32, device="cuda"),
                out=[torch.zeros((n, 3), device="cuda") for _ in range(3)])


# ---- one pass ----------------------------------------------------------------------------------

_EXTRA = ("du", "dv", "duu", "duv", "dvv")


def run(state):
    s, kind = state, state["kind"]
    if kind == "raw":
        GB300Evaluator.EvalStencils(s["src"], s["src_desc"], s["out"][0], s["dst_desc"],
                                    *s["arrays"], 0, s["n"])
        return s["out"]
    if kind == "batch":
        s["batch"].EvalGraph()
        return s["out"]
    if kind == "tess":
        s["mesh"].Count()  # rates follow the view: the inventory is taken every frame
        s["mesh"].Generate(s["coords"], s["facets"], table=s["table"],
                           patch_coords=s["patch_coords"])
        s["mesh"].Evaluate(s["src"], s["src_desc"], s["table"], s["patch_coords"],
                           outputs=s["out"])
        return dict(coords=s["coords"], facets=s["facets"], patch_coords=s["patch_coords"],
                    out=s["out"])
    d = s["dst_desc"]
    more = {}
    for name, buf in zip(_EXTRA, s["out"][1:]):
        more[name], more[name + "Desc"] = buf, d
    if kind == "patches":
        s["table"].FindPatches(s["n"], s["face"], s["u"], s["v"], s["coords"])
        GB300Evaluator.EvalPatchesTable(s["src"], s["src_desc"], s["out"][0], d, s["n"],
                                        s["coords"], s["table"], **more)
        return dict(coords=s["coords"], out=s["out"])
    GB300Evaluator.EvalStencilsTable(s["src"], s["src_desc"], s["out"][0], d, s["table"], **more)
    return s["out"]


# ---- what a pass cannot do without -------------------------------------------------------------

#: Operations of one point of all six outputs: (basis weights, per primvar element) -- the
#: tensor-product curves and their row and column sums, or the twelve quartics and six sums.
_POINT_FLOPS = {False: (70, 167), True: (762, 163)}


@functools.lru_cache(maxsize=64)
def _counts(key):
    case = dict(key)
    if case["kind"] == "batch":
        return [(len(m["table"]["sizes"]), len(m["table"]["indices"]), m["n_cv"], m["length"])
                for m in _scene(case, 0)]
    if case["kind"] in ("refine", "raw", "limit"):
        cage, _, t = _stencils(case, 0)
        return len(t["sizes"]), len(t["indices"]), cage.num_vertices
    z = _golden(case["table"])
    n = len(z["coords"]) * case["copies"] if case["kind"] == "tess" else case["points"]
    patches = len(z["params"]) * case["copies"]
    per = len(z["patch_indices"]) / len(z["params"])  # control points of a patch
    # patches that n uniform locations can touch, and the rows that those hold between them
    touched = min(patches, n)
    rows = min(len(z["src"]) // 3 * case["copies"], touched * per)
    return n, touched, per, rows, bool(z["triangular"]), z


def work(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if case["kind"] == "batch":
        c = _counts(key)
        return dict(bytes=sum(8 * n + 8 * e + 4 * w * (n + cv) for n, e, cv, w in c),
                    flops=sum(2 * e * w for _, e, _, w in c))
    if case["kind"] in ("refine", "raw", "limit"):
        n, entries, cv = _counts(key)
        k, w = case.get("outputs", 1), case["length"]
        return dict(bytes=8 * n + 4 * entries * (1 + k) + 4 * w * (k * n + cv),
                    flops=2 * entries * w * k)
    n, touched, per, rows, tri, z = _counts(key)
    k, w = case.get("outputs", 3), case["length"]
    basis, element = _POINT_FLOPS[tri]
    share = k / 6
    b = touched * (4 * per + 8) + 4 * w * (rows + k * n)
    if case["kind"] == "patches":
        b += (12 + 20) * n  # (face, u, v) read and the PatchCoord written
    else:
        b += (8 + 20) * n + 12 * len(z["facets"]) * case["copies"]
        b += 4 * (len(z["verts_per_face"]) + len(z["rates"])) * case["copies"]
    return dict(bytes=int(b), flops=int(n * (basis + element * w) * share))


# ---- the same in 64 bits -----------------------------------------------------------------------

def _apply64(table, weights, src):
    """sum_j w_j src[idx_j] for every stencil, entry j of all stencils at a time."""
    sizes, offsets = _cuda(table["sizes"]).long(), _cuda(table["offsets"]).long()
    idx, w = _cuda(table["indices"]).long(), _cuda(weights).double()
    order = torch.argsort(sizes, descending=True)
    sizes, offsets = sizes[order], offsets[order]
    acc = torch.zeros((len(sizes), src.shape[1]), dtype=torch.float64, device="cuda")
    counts = torch.bincount(sizes).flip(0).cumsum(0).flip(0).tolist()
    for j in range(len(counts) - 1):
        m = counts[j + 1]  # stencils of more than j entries
        for a in range(0, m, 1 << 21):
            e = offsets[a: min(a + (1 << 21), m)] + j
            acc[a: min(a + (1 << 21), m)] += w[e, None] * src[idx[e]]
    out = torch.empty_like(acc)
    out[order] = acc
    return out.reshape(-1)


_BSPLINE = np.array([[1, -3, 3, -1], [4, 0, -6, 3], [1, 3, 3, -3], [0, 0, 0, 1]]) / 6.0
_BEZIER = np.array([[1, -3, 3, -1], [0, 3, -6, 3], [0, 0, 3, -3], [0, 0, 0, 1]], float)
#: the twelve quartic box-spline polynomials x 12, over s^a t^b with a + b <= 4 in rising degree
_BOX = np.array([
    [1, -2, -4, 0, 6, 6, 2, 0, -6, -4, -1, -2, 0, 2, 1],
    [1, 2, -2, 0, -6, 0, -4, 0, 6, 2, 2, 4, 0, -2, -1],
    [0, 0, 0, 0, 0, 0, 2, 0, 0, 0, -1, -2, 0, 0, 0],
    [1, -4, -2, 6, 6, 0, -4, -6, 0, 2, 1, 2, 0, -2, -1],
    [6, 0, 0, -12, -12, -12, 8, 12, 12, 8, -1, -2, 0, -2, -1],
    [1, 4, 2, 6, 6, 0, -4, -6, -12, -4, -1, -2, 0, 4, 2],
    [0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 1, 2, 0, 0, 0],
    [1, -2, 2, 0, -6, 0, 2, 6, 0, -4, -1, -2, 0, 4, 2],
    [1, 2, 4, 0, 6, 6, -4, -12, -6, -4, 2, 4, 0, -2, -1],
    [0, 0, 0, 0, 0, 0, 2, 6, 6, 2, -1, -2, 0, -2, -1],
    [0, 0, 0, 0, 0, 0, 0, 0, 0, 2, 0, 0, 0, -2, -1],
    [0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 2, 1]]) / 12.0
_POWERS = [(d - b, b) for d in range(5) for b in range(d + 1)]
_ORDERS = [(0, 0), (1, 0), (0, 1), (2, 0), (1, 1), (0, 2)]


def _bezier_triangle():
    """The fifteen quartic Bernstein polynomials u^i v^j (1 - u - v)^k over the same monomials."""
    rows = []
    for j in range(5):
        for i in range(5 - j):
            k = 4 - i - j
            row = np.zeros(15)
            scale = math.factorial(4) // (math.factorial(i) * math.factorial(j) * math.factorial(k))
            for p in range(k + 1):
                for q in range(k + 1 - p):
                    c = (-1) ** (p + q) * math.factorial(k) // (
                        math.factorial(p) * math.factorial(q) * math.factorial(k - p - q))
                    row[_POWERS.index((i + p, j + q))] += scale * c
            rows.append(row)
    return np.array(rows)


def _falling(n, k):
    return math.prod(range(n - k + 1, n + 1))


def _curve(coef, t, order):
    """[points, 4] weights of a cubic curve's derivative."""
    p = torch.stack([_falling(k, order) * t ** (k - order) if k >= order else torch.zeros_like(t)
                     for k in range(4)], 1)
    return p @ torch.from_numpy(coef.T.copy()).cuda()


def _surface(coef, s, t, ds, dt):
    """[points, rows of coef] weights of a quartic triangle's derivative."""
    p = torch.stack([_falling(a, ds) * _falling(b, dt) * s ** (a - ds) * t ** (b - dt)
                     if a >= ds and b >= dt else torch.zeros_like(s) for a, b in _POWERS], 1)
    return p @ torch.from_numpy(coef.T.copy()).cuda()


def _ratio(a, b):
    z = b <= 0
    return torch.where(z, torch.zeros_like(a), a / torch.where(z, torch.ones_like(b), b))


def _fold(w, bits, first, last):
    """Boundary patches: the absent end point of a curve is 2 p - q of its neighbours."""
    for bit, a, b, c in ((first, 0, 1, 2), (last, 3, 2, 1)):
        x = torch.where(bits & bit != 0, w[:, a], torch.zeros_like(w[:, a]))
        w[:, a] -= x
        w[:, b] += 2 * x
        w[:, c] -= x
    return w


#: the 4 x 4 Bezier grid of a Gregory patch: points, and pairs that a rational weight blends
_GREGORY = [[0, 1, 7, 5], [2, (3, 0), (8, 1), 6], [16, (18, 3), (13, 2), 12], [15, 17, 11, 10]]
_GREGORY_TRI = [0, 1, 15, 7, 5, 2, (3, 0), (8, 1), 6, 17, (13, 2), 16, 11, 12, 10]


def _weights64(kind, bits, s, t):
    """Per derivative the weights [points, control points] of one basis."""
    n = len(s)
    if kind in (6, 9):
        coef = _BSPLINE if kind == 6 else _BEZIER
        ws = [_curve(coef, s, k) for k in range(3)]
        wt = [_curve(coef, t, k) for k in range(3)]
        if kind == 6:
            ws = [_fold(w, bits, 8, 2) for w in ws]
            wt = [_fold(w, bits, 1, 4) for w in wt]
        sc, tc = 1 - s, 1 - t
        blend = [_ratio(s, s + t), _ratio(t, sc + t), _ratio(sc, sc + tc), _ratio(tc, s + tc)]
    elif kind == 10:
        w = 1 - s - t
        blend = [torch.where(b > 0, _ratio(a, b), torch.ones_like(a))
                 for a, b in ((s, s + t), (t, t + w), (w, w + s))]
        other = [_ratio(a, b) for a, b in ((t, s + t), (w, t + w), (s, w + s))]
    out = []
    for ds, dt in _ORDERS:
        if kind == 6:
            w = (wt[dt][:, :, None] * ws[ds][:, None, :]).reshape(n, 16)
        elif kind == 9:
            w = torch.zeros((n, 20), dtype=torch.float64, device="cuda")
            for r in range(4):
                for c in range(4):
                    cell, at = wt[dt][:, r] * ws[ds][:, c], _GREGORY[r][c]
                    if isinstance(at, int):
                        w[:, at] += cell
                    else:
                        w[:, at[0]] += cell * blend[at[1]]
                        w[:, at[0] + 1] += cell * (1 - blend[at[1]])
        elif kind == 5:
            w = _surface(_BOX, s, t, ds, dt)
        else:
            b = _surface(_bezier_triangle(), s, t, ds, dt)
            w = torch.zeros((n, 18), dtype=torch.float64, device="cuda")
            for m, at in enumerate(_GREGORY_TRI):
                if isinstance(at, int):
                    w[:, at] += b[:, m]
                else:
                    w[:, at[0]] += b[:, m] * blend[at[1]]
                    w[:, at[0] + 1] += b[:, m] * other[at[1]]
        out.append(w)
    return out


def _quadrants(tri, u, v, levels):
    """The path of (u, v) through the quadtree, as base-4 digits, after 0 .. levels steps."""
    path, paths = torch.zeros_like(u, dtype=torch.int64), []
    rot = torch.zeros_like(u, dtype=torch.bool)
    median = 0.5
    u, v = u.clone(), v.clone()
    for _ in range(levels + 1):
        paths.append(path)
        m = torch.full_like(u, median)
        z = torch.zeros_like(u)
        if not tri:
            a, b = u >= m, v >= m
            u, v = u - torch.where(a, m, z), v - torch.where(b, m, z)
            q = a.long() + 2 * b.long()
        else:
            # upright: right, top, centre (which turns the triangle), else left; turned: mirrored
            a = torch.where(rot, u < m, u >= m)
            b = ~a & torch.where(rot, v < m, v >= m)
            both = ~a & ~b & rot
            u2 = u - torch.where((~rot & a) | (rot & b) | both, m, z)
            v2 = v - torch.where((~rot & b) | (rot & a) | both, m, z)
            c = ~a & ~b & torch.where(rot, u2 + v2 < m, u2 + v2 >= m)
            u, v = u2, v2
            q = torch.where(a, 1, torch.where(b, 2, torch.where(c, 3, 0)))
            rot = rot ^ c
        path = path * 4 + q
        median /= 2
    return paths


def _patches64(arrays, indices, params, src, tri, face, u, v, outputs):
    """Every location's patch and its limit values: list of [points, length] in 64 bits."""
    par = _cuda(params).long()
    f, p1 = par[:, 0] & 0xFFFFFFF, par[:, 1]
    depth, root = p1 & 15, (p1 >> 4) & 1
    pu, pv = (p1 >> 22) & 1023, (p1 >> 12) & 1023
    steps = depth - root
    levels = int(steps.max())
    if tri:  # an inner point of the patch tells its way down
        side = (1 << steps).double()
        turned = pu + pv >= (1 << depth)
        iu = torch.where(turned, (1 << depth) - pu - 0.25, pu + 0.25) / side
        iv = torch.where(turned, (1 << depth) - pv - 0.25, pv + 0.25) / side
    else:
        side = (1 << steps).double()
        iu, iv = (pu + 0.5) / side, (pv + 0.5) / side
    way = torch.stack(_quadrants(tri, iu, iv, levels))
    way = way.gather(0, steps[None])[0]
    key, at = torch.sort((f << 24) + (steps << 20) + way)
    arr, idx, src = np.asarray(arrays), _cuda(indices), src.double()
    first = torch.from_numpy(arr[:, 5].copy()).cuda()
    n = len(face)
    out = [torch.zeros((n, src.shape[1]), dtype=torch.float64, device="cuda") for _ in range(outputs)]
    for lo in range(0, n, 1 << 18):
        part = slice(lo, min(lo + (1 << 18), n))
        fc, s, t = face[part].long(), u[part].double(), v[part].double()
        patch = torch.full_like(fc, -1)
        for k, w in enumerate(_quadrants(tri, s, t, levels)):
            want = (fc << 24) + (k << 20) + w
            j = torch.searchsorted(key, want).clamp(max=len(key) - 1)
            patch = torch.where((key[j] == want) & (patch < 0), at[j], patch)
        a = torch.bucketize(patch, first, right=True) - 1
        regular = (p1[patch] >> 5) & 1
        kind = torch.where(regular == 1, torch.from_numpy(arr[:, 0].copy()).cuda()[a],
                           torch.from_numpy(arr[:, 1].copy()).cuda()[a])
        side = (1 << steps[patch]).double()
        qu, qv, d = pu[patch], pv[patch], depth[patch]
        turned = ((qu + qv) >= (1 << d)) & torch.full_like(qu, tri, dtype=torch.bool)
        ps = torch.where(turned, ((1 << d) - qu) - s * side, s * side - qu)
        pt = torch.where(turned, ((1 << d) - qv) - t * side, t * side - qv)
        d1 = torch.where(turned, -1.0, 1.0).double() * (1 << d)
        d2 = torch.where(turned, -1.0, 1.0).double() * d1 * d1
        for ki in torch.unique(kind).tolist():
            for ai in torch.unique(a[kind == ki]).tolist():
                sel = torch.nonzero((kind == ki) & (a == ai))[:, 0]
                h = patch[sel]
                cvs = {6: 16, 9: 20, 5: 12, 10: 18}[ki]
                rows = int(arr[ai, 3]) + int(arr[ai, 4]) * (h - int(arr[ai, 5]))
                x = src[idx[rows[:, None] + torch.arange(cvs, device="cuda")].long()]
                w = _weights64(ki, (p1[h] >> 7) & 31, ps[sel], pt[sel])
                for o in range(outputs):
                    scale = 1.0 if o == 0 else (d1 if o < 3 else d2)[sel, None]
                    out[o][part.start + sel] = scale * (w[o][:, :, None] * x).sum(1)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("refine", "raw", "limit"):
        _, values, table = _stencils(case, seed)
        src = _cuda(values).double().reshape(-1, case["stride"])
        src = src[:, case["offset"]: case["offset"] + case["length"]].contiguous()
        return [_apply64(table, table[k], src) for k in WEIGHTS[:case.get("outputs", 1)]]
    if kind == "batch":
        return [_apply64(m["table"], m["table"]["weights"],
                         _cuda(m["src"]).double().reshape(-1, m["length"]))
                for m in _scene(case, seed)]
    z, arrays, indices, params, src, ptex, tri = _patches(case, seed)
    if kind == "patches":
        at = [_cuda(x) for x in _queries(case, ptex, tri, seed)]
        rows = _cuda(src).reshape(-1, case["stride"])[:, :case["length"]]
        out = _patches64(arrays, indices, params, rows, tri, *at, case["outputs"])
        return dict(coords=None, out=[x.reshape(-1) for x in out])
    # tess: the reference's own coords of these faces, and its limit locations
    c = case["copies"]
    step = np.repeat(np.arange(c, dtype=np.int32) * int(z["num_ptex"]), len(z["q_face"]))
    out = _patches64(arrays, indices, params, _cuda(src).reshape(-1, 3), tri,
                     _cuda(np.tile(z["q_face"], c) + step), _cuda(np.tile(z["q_s"], c)),
                     _cuda(np.tile(z["q_t"], c)), 3)
    return dict(coords=_cuda(np.tile(z["coords"], (c, 1))).double(), facets=None,
                patch_coords=None, out=out)

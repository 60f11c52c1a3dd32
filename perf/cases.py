"""The performance cases of the framework: what a user of it runs, through its
public entry points, from the smallest mesh to the largest.

    listed()             the cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what the user's program holds before the call
    run(state)           one pass; its outputs whole
    work(case)           the bytes one pass cannot do without
    exact(case, seed)    smoothed fields in 64 bits (all other outputs are
                         whole numbers, which have one right value)

Meshes are the generators of tetragpu_gb300/meshgen.py (Kuhn cube grids with a
seeded share of the cubes centre-coned, vertex ids permuted, slots shuffled),
made on the GPU because they are made often.
"""
from __future__ import annotations

import ctypes as C
import itertools
import math

import numpy as np
import torch

import tetragpu_gb300 as tg

ALL = "TE EV ET TF FV FE FT EF VT TT FF EE VV"
REFERENCE_SUBSETS = ("VV", "TE EV TF FV", "EV ET EE", "FV FE FT FF", "TF TT VT")


def listed():
    return [
        # the smallest meshes of a batch or a request stream, one at a time:
        # launches, allocations and host round trips are the time
        dict(name="all_7", what="all", nx=7, ny=7, nz=7, cone=0.1, permute=True, dtype="f32"),
        # the small configuration: 16^3 cubes, every relation and the classes
        dict(name="all_16", what="all", nx=16, ny=16, nz=16, cone=0.0, permute=True, dtype="f32"),
        # an ordinary mesh with odd sides, ids as the generator gave them, a
        # float64 field
        dict(name="all_ragged_f64", what="all", nx=41, ny=23, nz=17, cone=0.13, permute=False,
             dtype="f64"),
        # the irregular configuration: 64^3, 20% of the cubes coned
        dict(name="all_64_coned", what="all", nx=64, ny=64, nz=64, cone=0.2, permute=True,
             dtype="f32"),
        # the large configuration: 12.6M tets
        dict(name="all_128", what="all", nx=128, ny=128, nz=128, cone=0.0, permute=True,
             dtype="f32"),
        # the batched configuration: 512 uneven meshes as one
        dict(name="batch_512", what="batch", meshes=512, lo=2000, hi=400000, dtype="f32"),
        # critical points from cells alone (the reference's critPoints driver:
        # VV, then the classes), nothing else extracted
        dict(name="critical_50", what="critical", nx=51, ny=47, nz=53, cone=0.05, permute=True,
             dtype="f32"),
        # the relations the reference's own driver builds most: cell, edge and
        # face numbering
        dict(name="subset_96", what="subset", relations="TE EV TF FV", nx=96, ny=96, nz=96,
             cone=0.0, permute=True),
        # a new field on a mesh that is resident (30% of the request stream)
        dict(name="field_128", what="field", nx=128, ny=128, nz=128, cone=0.0, permute=True,
             dtype="f32"),
        # a consumer of the resident VV: ten smoothing steps of a vertex field
        dict(name="smooth_64", what="smooth", nx=64, ny=64, nz=64, cone=0.2, permute=True,
             iterations=10),
        # the vertex-sharing form of TT (TV x TV transposed), and VT
        dict(name="tt_vertex_40", what="tt_vertex", nx=40, ny=40, nz=40, cone=0.1, permute=True),
        # a burst of requests from host memory to the server: new meshes with
        # a field, and new fields on them; classes back in host memory
        dict(name="serve_24", what="serve", requests=24, median=50000, dtype="f32"),
    ]


def _sides(rng, lo, hi):
    """Grid sides of a Kuhn mesh of lo..hi tets (log-uniform), not always a cube."""
    cubes = math.exp(rng.uniform(math.log(lo), math.log(hi))) / 6.0
    a, b = math.exp(rng.uniform(-0.5, 0.5)), math.exp(rng.uniform(-0.5, 0.5))
    side = cubes ** (1.0 / 3.0)
    nx, ny = max(1, round(side * a)), max(1, round(side * b))
    return dict(nx=nx, ny=ny, nz=max(1, int(cubes / (nx * ny))))


def draw(rng):
    what = rng.choice(["all", "all", "all", "batch", "critical", "subset", "field", "smooth",
                       "tt_vertex", "serve"])
    dtype = rng.choice(["f32", "f32", "f64"])
    if what == "batch":
        hi = int(math.exp(rng.uniform(math.log(1e4), math.log(4e5))))
        return dict(what=what, meshes=int(math.exp(rng.uniform(math.log(4), math.log(200)))),
                    lo=2000, hi=hi, dtype=dtype)
    if what == "serve":
        return dict(what=what, requests=rng.randrange(2, 25), median=rng.randrange(3000, 60000),
                    dtype=dtype)
    # a coned cube counts twice: leave room for it below the largest case
    most = {"all": 9e6, "critical": 6e6, "subset": 6e6, "field": 9e6, "smooth": 9e6,
            "tt_vertex": 4e5}[what]
    case = dict(what=what, **_sides(rng, 2000, most), cone=round(rng.choice([0.0, rng.uniform(0, 0.3)]), 3),
                permute=what in ("subset", "tt_vertex") or rng.random() < 0.7)
    if what == "subset":
        case["relations"] = rng.choice(REFERENCE_SUBSETS)
    elif what == "smooth":
        case["iterations"] = rng.randrange(1, 13)
    elif what != "tt_vertex":
        case["dtype"] = dtype
    return case


# ---------------------------------------------------------------------------
# meshes and fields
# ---------------------------------------------------------------------------
def _kuhn_tets():
    out = []
    for p in itertools.permutations(range(3)):
        v, path = [0, 0, 0], [(0, 0, 0)]
        for a in p:
            v[a] = 1
            path.append(tuple(v))
        out.append(path)
    return np.array(out, dtype=np.int64)          # [6, 4, 3]


def _cone_triangles():
    tris = []
    for a in range(3):
        b, c = [x for x in range(3) if x != a]
        for t in (0, 1):
            base = [0, 0, 0]
            base[a] = t
            eb, ec, top = list(base), list(base), list(base)
            eb[b] = ec[c] = top[b] = top[c] = 1
            tris += [[base, eb, top], [base, ec, top]]
    return np.array(tris, dtype=np.int64)         # [12, 3, 3]


def _mesh(nx, ny, nz, cone, permute, gen):
    """(TV int32 [T, 4], vertex coordinates float64 [V, 3]) on the GPU."""
    dev = "cuda"
    gx, gy, gz = nx + 1, ny + 1, nz + 1
    n_grid, n_cubes = gx * gy * gz, nx * ny * nz
    n_coned = int(round(cone * n_cubes))
    q = torch.arange(n_cubes, device=dev)
    i, j, k = q % nx, (q // nx) % ny, q // (nx * ny)
    base = i + gx * (j + gy * k)
    step = np.array([1, gx, gx * gy])
    tets = torch.from_numpy((_kuhn_tets() * step).sum(-1)).to(dev)        # [6, 4]
    tris = torch.from_numpy((_cone_triangles() * step).sum(-1)).to(dev)   # [12, 3]
    if n_coned:
        coned = torch.zeros(n_cubes, dtype=torch.bool, device=dev)
        # the same cubes for every seed, so that all outputs keep their sizes
        picked = torch.randperm(n_cubes, generator=_generator(1), device=dev)[:n_coned].sort().values
        coned[picked] = True
        first = torch.where(coned, 12, 6).cumsum(0)
        tv = torch.empty((int(first[-1]), 4), dtype=torch.int64, device=dev)
        first = first - torch.where(coned, 12, 6)
        plain = ~coned
        at = first[plain][:, None] + torch.arange(6, device=dev)
        tv[at.reshape(-1)] = (base[plain][:, None, None] + tets).reshape(-1, 4)
        at = first[picked][:, None] + torch.arange(12, device=dev)
        centre = (n_grid + torch.arange(n_coned, device=dev))[:, None, None].expand(-1, 12, 1)
        tv[at.reshape(-1)] = torch.cat([centre, base[picked][:, None, None] + tris], 2).reshape(-1, 4)
    else:
        tv = (base[:, None, None] + tets).reshape(-1, 4)
    g = torch.arange(n_grid, device=dev)
    xyz = torch.stack([(g % gx) / nx, (g // gx % gy) / ny, (g // (gx * gy)) / nz], 1).double()
    if n_coned:
        mid = torch.stack([(i[picked] + 0.5) / nx, (j[picked] + 0.5) / ny, (k[picked] + 0.5) / nz], 1)
        xyz = torch.cat([xyz, mid.double()])
    if permute:
        perm = torch.randperm(xyz.shape[0], generator=gen, device=dev)
        tv = perm[tv]
        moved = torch.empty_like(xyz)
        moved[perm] = xyz
        xyz = moved
    # the slots of every tet shuffled
    order = torch.rand(tv.shape, generator=gen, device=dev).argsort(1)
    return tv.gather(1, order).int().contiguous(), xyz


def _field(xyz, gen, dtype):
    """Sine product for the large meshes, a mixture of Gaussians for the
    others, plus noise."""
    n = xyz.shape[0]
    rand = lambda *s: torch.rand(*s, generator=gen, device="cuda", dtype=torch.float64)  # noqa: E731
    if n > 1_000_000:
        a = rand(3) * (8 * math.pi) + 4 * math.pi
        f = torch.sin(xyz * a).prod(1)
        noise = 1e-4
    else:
        f = torch.zeros(n, dtype=torch.float64, device="cuda")
        centre, sigma, amp = rand(32, 3), rand(32) * 0.18 + 0.02, rand(32) * 2 - 1
        for c, s, a in zip(centre, sigma, amp):
            f += a * torch.exp(-((xyz - c) ** 2).sum(1) / (2 * s * s))
        noise = 1e-3
    f += noise * torch.randn(n, generator=gen, device="cuda", dtype=torch.float64)
    return f.float() if dtype == "f32" else f


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _batch_sides(case):
    """The meshes' grid sides and coned shares: the same for every seed, so
    that a pass is the same amount of work."""
    rng = np.random.default_rng(case["meshes"])
    out = []
    for _ in range(case["meshes"]):
        tets = math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))
        n = max(1, round((tets / 6) ** (1 / 3)))
        out.append((n, n, max(1, round(tets / (6 * n * n))), round(float(rng.uniform(0, 0.3)), 3)))
    return out


def _serve_sides(case):
    rng = np.random.default_rng(case["requests"])
    new = max(1, round(0.7 * case["requests"]))
    out = []
    for _ in range(new):
        tets = min(float(np.exp(rng.normal(math.log(case["median"]), 1.0))), 1e6)
        n = max(1, round((tets / 6) ** (1 / 3)))
        out.append((n, n, max(1, round(tets / (6 * n * n))), 0.1))
    return out


_FIELD_TYPE = {"f32": tg.FIELD_F32, "f64": tg.FIELD_F64}


def prepare(case, seed):
    gen, what = _generator(seed), case["what"]
    st = dict(case=case)
    if what == "batch":
        parts = [_mesh(*s, True, gen) for s in _batch_sides(case)]
        st["n_cells"] = np.array([tv.shape[0] for tv, _ in parts], dtype=np.int64)
        st["n_verts"] = np.array([x.shape[0] for _, x in parts], dtype=np.int64)
        st["tv"] = torch.cat([tv for tv, _ in parts])
        st["field"] = torch.cat([_field(x, gen, case["dtype"]) for _, x in parts])
    elif what == "serve":
        st["meshes"], st["fields"] = [], []
        for s in _serve_sides(case):
            tv, xyz = _mesh(*s, True, gen)
            st["meshes"].append((tv.cpu().numpy(), xyz.shape[0],
                                 _field(xyz, gen, case["dtype"]).cpu().numpy()))
        for i in range(case["requests"] - len(st["meshes"])):
            at = (i * 7) % len(st["meshes"])
            f = torch.randn(st["meshes"][at][1], generator=gen, device="cuda", dtype=torch.float64)
            st["fields"].append((at, f.cpu().numpy().astype(
                np.float32 if case["dtype"] == "f32" else np.float64)))
        st["server"] = tg.Server()
    else:
        st["tv"], xyz = _mesh(case["nx"], case["ny"], case["nz"], case["cone"], case["permute"], gen)
        st["n_verts"] = xyz.shape[0]
        if what in ("all", "critical", "field"):
            st["field"] = _field(xyz, gen, case["dtype"])
        if what == "smooth":
            st["field"] = _field(xyz, gen, "f32")
        if what in ("field", "smooth"):
            # the mesh a server or an application keeps resident
            m = tg.Mesh(st["tv"].data_ptr(), st["n_verts"], st["tv"].shape[0], on_device=True)
            m.extract(["VV"], tg.OPT_LINK_ADJACENCY if what == "field" else 0)
            st["mesh"] = m
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
class _DeviceArray:
    """A relation's device array for torch, keeping its mesh alive."""

    def __init__(self, ptr, shape, typestr, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False),
                                         "version": 2}


def _tensor(ptr, shape, typestr, owner):
    if not ptr or 0 in shape:
        return torch.empty(shape, device="cuda", dtype=torch.int64 if typestr == "<i8" else torch.int32)
    return torch.as_tensor(_DeviceArray(ptr, shape, typestr, owner), device="cuda")


def _relations(mesh, names):
    """The mesh's resident relations as device tensors (no copies)."""
    out = {}
    for name in names:
        d = mesh.device_relation(name)
        if d["width"]:
            out[name] = _tensor(d["entries"], (d["rows"], d["width"]), "<i4", mesh)
        else:
            out[name + "_offsets"] = _tensor(d["offsets"], (d["rows"] + 1,), "<i8", mesh)
            out[name] = _tensor(d["entries"], (d["n_entries"],), "<i4", mesh)
    return out


class _BatchHandle:
    """A batch and its union mesh through the C interface, with the
    device_relation of tg.Mesh."""

    def __init__(self, st):
        lib = tg.load()
        self.h = C.c_void_p()
        n = len(st["n_cells"])
        _check(lib.tg_batch_create(st["tv"].data_ptr(), st["n_cells"].ctypes.data,
                                   st["n_verts"].ctypes.data, n, 1, None, C.byref(self.h)))
        self.u = C.c_void_p(lib.tg_batch_union(self.h))

    def device_relation(self, name):
        off, ent = C.c_void_p(), C.c_void_p()
        rows, n, width = C.c_int64(), C.c_int64(), C.c_int32()
        _check(tg.load().tg_get_relation(self.u, tg.REL[name], C.byref(off), C.byref(ent),
                                         C.byref(rows), C.byref(n), C.byref(width)))
        return {"offsets": off.value, "entries": ent.value, "rows": rows.value,
                "n_entries": n.value, "width": width.value}

    def __del__(self):
        if self.h:
            tg.load().tg_batch_destroy(self.h)


def _check(rc):
    if rc:
        raise RuntimeError(tg.load().tg_last_error_string().decode())


def run(st):
    case = st["case"]
    what = case["what"]
    if what == "serve":
        return _serve(st)
    if what == "batch":
        b, lib = _BatchHandle(st), tg.load()
        _check(lib.tg_batch_extract(b.h, tg.ALL_RELATIONS, tg.OPT_LINK_ADJACENCY, None))
        classes = torch.empty((int(st["n_verts"].sum()), 3), dtype=torch.int32, device="cuda")
        _check(lib.tg_batch_critical_points(b.h, st["field"].data_ptr(), _FIELD_TYPE[case["dtype"]],
                                            1, classes.data_ptr(), 1, None))
        out = _relations(b, ALL.split())
        out["classes"] = classes
        return out
    if what == "field":
        classes = torch.empty((st["n_verts"], 3), dtype=torch.int32, device="cuda")
        st["mesh"].critical_points(st["field"].data_ptr(), on_device=True,
                                   out_ptr=classes.data_ptr(), field_type=_FIELD_TYPE[case["dtype"]])
        return classes
    if what == "smooth":
        out, scratch = torch.empty_like(st["field"]), torch.empty_like(st["field"])
        st["mesh"].smooth_field(st["field"].data_ptr(), out.data_ptr(), case["iterations"],
                                scratch.data_ptr())
        return out
    m = tg.Mesh(st["tv"].data_ptr(), st["n_verts"], st["tv"].shape[0], on_device=True)
    if what == "subset":
        m.extract(case["relations"].split())
        return _relations(m, case["relations"].split())
    if what == "tt_vertex":
        m.extract(["TT", "VT"], tg.OPT_TT_VERTEX_SHARING)
        return _relations(m, ["TT", "VT"])
    if what == "all":
        m.extract(tg.ALL_RELATIONS, tg.OPT_LINK_ADJACENCY)
    classes = torch.empty((st["n_verts"], 3), dtype=torch.int32, device="cuda")
    m.critical_points(st["field"].data_ptr(), on_device=True, out_ptr=classes.data_ptr(),
                      field_type=_FIELD_TYPE[case["dtype"]])
    out = _relations(m, ALL.split()) if what == "all" else {}
    out["classes"] = classes
    return out


def _serve(st):
    server = st["server"]
    sent = [server.submit_mesh(tv, n_verts, field) for tv, n_verts, field in st["meshes"]]
    asked = [rid for rid, _ in sent]
    asked += [server.submit_field(sent[at][1], field) for at, field in st["fields"]]
    classes = [server.wait(rid)[0].view(np.int32) for rid in asked]
    for _, mesh_id in sent:
        server.release(mesh_id)
    return classes


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _counts(nx, ny, nz, cone):
    """Vertices, edges, faces, cells and boundary faces of a grid mesh."""
    cubes = nx * ny * nz
    coned = int(round(cone * cubes))
    v = (nx + 1) * (ny + 1) * (nz + 1) + coned
    t = 6 * (cubes + coned)
    b = 4 * (nx * ny + ny * nz + nx * nz)
    f = (4 * t + b) // 2
    return v, v + f - t - 1, f, t, b


def _relation_bytes(names, v, e, f, t, b):
    """Bytes written: int32 entries, int64 offsets.  EE counts the pairs of
    edges at a vertex as if every vertex had the mean degree."""
    ee = int((2 * e) ** 2 / v) - 2 * e
    size = {"TE": 24 * t, "EV": 8 * e, "ET": 24 * t + 8 * e, "TF": 16 * t, "FV": 12 * f, "FE": 12 * f,
            "FT": 8 * f, "EF": 12 * f + 8 * e, "VT": 16 * t + 8 * v, "TT": 4 * (4 * t - b) + 8 * t,
            "FF": 12 * (2 * f - b) + 8 * f, "EE": 4 * ee + 8 * e, "VV": 8 * e + 8 * v}
    return sum(size[n] for n in names)


def work(case):
    what = case["what"]
    width = 8 if case.get("dtype") == "f64" else 4
    if what in ("batch", "serve"):
        sides = _batch_sides(case) if what == "batch" else _serve_sides(case)
        total = 0
        for s in sides:
            v, e, f, t, b = _counts(*s)
            total += 16 * t + (width + 12) * v + _relation_bytes(ALL.split(), v, e, f, t, b)
        return {"bytes": total, "flops": 0}
    v, e, f, t, b = _counts(case["nx"], case["ny"], case["nz"], case["cone"])
    if what == "field":      # the field, VV and the link masks once; the classes
        return {"bytes": (width + 12 + 8) * v + 2 * e * (4 + 8), "flops": 0}
    if what == "smooth":     # VV and the field read once, the smoothed field written
        return {"bytes": 16 * v + 8 * e, "flops": case["iterations"] * 2 * e}
    if what == "tt_vertex":  # cells sharing a vertex, by inclusion and exclusion over mean stars
        n = (4 * t) ** 2 / v - (6 * t) ** 2 / e + (4 * t) ** 2 / f - 2 * t
        return {"bytes": int(16 * t + 4 * n + 8 * t) + _relation_bytes(["VT"], v, e, f, t, b), "flops": 0}
    names = {"all": ALL, "critical": "", "subset": case.get("relations", "")}[what].split()
    total = 16 * t + _relation_bytes(names, v, e, f, t, b)
    if what != "subset":
        total += (width + 12) * v
    return {"bytes": total, "flops": 0}


def exact(case, seed):
    if case["what"] != "smooth":
        return None
    gen = _generator(seed)
    tv, xyz = _mesh(case["nx"], case["ny"], case["nz"], case["cone"], case["permute"], gen)
    f = _field(xyz, gen, "f32").double()
    n = f.shape[0]
    pairs = torch.cat([tv[:, list(p)] for p in itertools.combinations(range(4), 2)]).long()
    keys = torch.unique(pairs.min(1).values * n + pairs.max(1).values)
    a, b = keys // n, keys % n
    one = torch.ones_like(a, dtype=torch.float64)
    count = torch.ones(n, dtype=torch.float64, device="cuda").index_add(0, a, one).index_add(0, b, one)
    for _ in range(case["iterations"]):
        f = f.index_add(0, a, f[b]).index_add(0, b, f[a]) / count
    return f

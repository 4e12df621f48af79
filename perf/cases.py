"""Performance cases of the element broadphase: what a contact code asks of it, from a few hundred elements to
17 million, through the public entry points (distbvh_b200.Context and the C ABI).

listed() names the cases, draw() gives others of the same ranges, prepare() makes the inputs and handles that a
program holds before the call, run() is one pass, work() the bytes and operations it cannot do without, exact() the
floating-point results in plain torch.

Every pass ends with its pair list in ascending order, in a buffer that the program keeps (-1 past the pairs): the
library returns pairs in no particular order, and a contact code that wants the same forces from the same step orders
them before it sums over them.

The kinds:

  step      two objects: set_elements, build both (rebuild, or refit of last step's trees), broadphase
  self      one object: set_elements, build, self-collision, with global ids
  batch     many two-body scenes in one call, rebuilt each step
  bodies    a time step of moving bodies: every pair of bodies in one refit batch
  sweep     sort-and-sweep candidates of two patch-sized built objects
  patches   build, Morton clustering into patches, patch boxes, and the pairs grouped by patch pair
"""
import ctypes
import math

import numpy as np
import torch

import distbvh_b200 as bvhg
from distbvh_b200 import meshes

PRECISION = {"fp64": bvhg.PLAIN_FP64, "fp32": bvhg.FILTER_FP32}


def listed():
    return [
        # The smallest calls: two 8x8x8 blocks of hexahedra (a unit test's grid, one patch of a decomposed mesh) from
        # host arrays and back, through the plain Python calls; 26-DOP, the reference's default.
        {"name": "grids_host", "kind": "step", "scene": "hexes", "size": 8, "k": 26, "precision": "fp64", "eps": 0.0,
         "mode": "rebuild", "mem": "host"},
        # Small contact surfaces: two plates of 10,000 triangles each, a gap closed by the inflation.
        {"name": "two_plates", "kind": "step", "scene": "plates", "size": 100, "k": 18, "precision": "fp64",
         "eps": 0.005, "mode": "rebuild", "mem": "device"},
        # A deforming solid against itself: 200,003 tetrahedra with global ids.
        {"name": "self_tets", "kind": "self", "size": 200003, "verts": 4, "k": 18, "precision": "fp64", "eps": 0.001},
        # The headline scene: a sphere of 5,242,880 triangles pressed into a plate of 4,194,304.
        {"name": "sphere_plate", "kind": "step", "scene": "sphere_plate", "size": 512, "k": 18, "precision": "fp64",
         "eps": 0.0, "mode": "rebuild", "mem": "device"},
        # The same contact at a quarter of the elements, with the FP32 filter and FP64 recheck.
        {"name": "sphere_plate_filter", "kind": "step", "scene": "sphere_plate", "size": 256, "k": 18,
         "precision": "fp32", "eps": 0.0, "mode": "rebuild", "mem": "device"},
        # A time step that keeps the trees' topology and refits them to the moved vertices.
        {"name": "sphere_plate_refit", "kind": "step", "scene": "sphere_plate", "size": 512, "k": 18,
         "precision": "fp64", "eps": 0.0, "mode": "refit", "mem": "device"},
        # Dense contact, every element touching its neighbours: 16.8M tetrahedra in two interleaved objects.
        {"name": "tets_fp64", "kind": "step", "scene": "tets", "size": 256, "k": 26, "precision": "fp64", "eps": 0.0,
         "mode": "rebuild", "mem": "device"},
        # Dense contact through the FP32 filter, at an odd size.
        {"name": "tets_filter", "kind": "step", "scene": "tets", "size": 161, "k": 18, "precision": "fp32",
         "eps": 0.0, "mode": "rebuild", "mem": "device"},
        # 512 independent two-body scenes of very uneven sizes, about 19M triangles in all.
        {"name": "batch_scenes", "kind": "batch", "scenes": 512, "lo": 1000, "hi": 200000, "k": 18,
         "precision": "fp64"},
        # One step of 32 tumbling bodies of 262,144 triangles, 496 body pairs.
        {"name": "bodies_refit", "kind": "bodies", "bodies": 32, "size": 512, "k": 18, "precision": "fp32"},
        # Candidates between two patch-sized soups by sorting along an axis.
        {"name": "sweep", "kind": "sweep", "size": 262144, "k": 18},
        # A patch-decomposed contact step, as a narrowphase per patch pair wants it.
        {"name": "patches", "kind": "patches", "size": 128, "patches": 64, "k": 26},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "self", "batch", "bodies", "sweep", "patches"])
    precision = rng.choice(["fp64", "fp64", "fp32"])
    k = rng.choice([6, 18, 18, 26])
    if kind == "step":
        scene = rng.choice(["hexes", "plates", "sphere_plate", "tets"])
        case = {"kind": kind, "scene": scene, "k": k, "precision": precision, "eps": 0.0,
                "mode": rng.choice(["rebuild", "rebuild", "refit"]), "mem": "device"}
        if scene == "hexes":
            case.update(size=_log(rng, 4, 40), mem=rng.choice(["host", "device"]))
        elif scene == "plates":
            case.update(size=_log(rng, 24, 400), eps=rng.choice([0.003, 0.004, 0.005]))
        elif scene == "sphere_plate":
            case.update(size=_log(rng, 24, 500))
        else:
            case.update(size=_log(rng, 20, 200), k=rng.choice([18, 26]))
        return case
    if kind == "self":
        return {"kind": kind, "size": _log(rng, 1000, 500000), "verts": rng.choice([3, 4, 8]), "k": k,
                "precision": precision, "eps": rng.choice([0.0, 0.001])}
    if kind == "batch":
        return {"kind": kind, "scenes": _log(rng, 16, 500), "lo": 1000, "hi": _log(rng, 4000, 200000), "k": 18,
                "precision": precision}
    if kind == "bodies":
        return {"kind": kind, "bodies": rng.randint(4, 32), "size": 2 * _log(rng, 24, 250), "k": 18,
                "precision": precision}
    if kind == "sweep":
        return {"kind": kind, "size": _log(rng, 4000, 250000), "k": k}
    return {"kind": kind, "size": _log(rng, 16, 250), "patches": _log(rng, 4, 1000), "k": k}


# ---- geometry, on the GPU, from the seed ------------------------------------------------------------------------

DEV = "cuda"
F64 = torch.float64


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=F64)


def _rotation(g):
    q = torch.randn(4, generator=g, device=DEV, dtype=F64)
    w, x, y, z = (q / q.norm()).tolist()
    return torch.tensor([[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
                         [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
                         [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]], dtype=F64, device=DEV)


def _unit(v):
    return v / (v * v).sum(-1, keepdim=True).sqrt()


def _sphere(f):
    """Unit sphere of 20 f^2 triangles: each face of an icosahedron cut into f0 x f0 (f0 the odd part of f), then
    subdivided in four while f allows; meshes.icosphere(level) for f = 2^level."""
    t = torch.from_numpy(meshes.icosphere(0)).to(DEV)
    levels = 0
    while f % 2 == 0:
        f //= 2
        levels += 1
    if f > 1:
        a, b, c = t[:, None, 0], t[:, None, 1], t[:, None, 2]

        def p(i, j):
            return a + (b - a) * (i / f)[None, :, None] + (c - a) * (j / f)[None, :, None]

        i, j = (x.reshape(-1) for x in torch.meshgrid(torch.arange(f, device=DEV, dtype=F64),
                                                      torch.arange(f, device=DEV, dtype=F64), indexing="ij"))
        up, down = i + j < f, i + j < f - 1
        iu, ju, iw, jw = i[up], j[up], i[down], j[down]
        t = torch.cat([torch.stack([p(iu, ju), p(iu + 1, ju), p(iu, ju + 1)], dim=2),
                       torch.stack([p(iw + 1, jw), p(iw + 1, jw + 1), p(iw, jw + 1)], dim=2)], dim=1)
        t = _unit(t.reshape(-1, 3, 3))
    for _ in range(levels):
        a, b, c = t[:, 0], t[:, 1], t[:, 2]
        ab, bc, ca = _unit(a + b), _unit(b + c), _unit(c + a)
        t = torch.stack([torch.stack([a, ab, ca], 1), torch.stack([ab, b, bc], 1), torch.stack([ca, bc, c], 1),
                         torch.stack([ab, bc, ca], 1)], dim=1).reshape(-1, 3, 3)
    return t


def _plate(nx, ny, x0, x1, y0, y1, z):
    """nx * ny quads of two triangles; z: (ny + 1, nx + 1)."""
    v = torch.empty(ny + 1, nx + 1, 3, dtype=F64, device=DEV)
    v[..., 0] = x0 + (x1 - x0) * torch.arange(nx + 1, device=DEV, dtype=F64)[None, :] / nx
    v[..., 1] = y0 + (y1 - y0) * torch.arange(ny + 1, device=DEV, dtype=F64)[:, None] / ny
    v[..., 2] = z
    v00, v10, v11, v01 = v[:-1, :-1], v[:-1, 1:], v[1:, 1:], v[1:, :-1]
    return torch.stack([torch.stack([v00, v10, v11], 2), torch.stack([v00, v11, v01], 2)], 2).reshape(-1, 3, 3)


def _hexes(n, g):
    """n^3 hexahedra of a unit block, every corner moved by up to 0.3 cells."""
    i = torch.arange(n, device=DEV, dtype=F64)
    k, j, i = torch.meshgrid(i, i, i, indexing="ij")
    base = torch.stack([i, j, k], -1).reshape(-1, 1, 3)
    corner = torch.tensor([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]],
                          dtype=F64, device=DEV)
    return (base + corner + 0.6 * (_rand(g, n ** 3, 8, 3) - 0.5)) / n


def _tets(m, g):
    """Jittered, log-normally scaled tetrahedra, one per cell of an m^3 lattice (meshes.tet_lattice), as the two
    colours of a checkerboard."""
    h = 1.0 / m
    idx = torch.arange(m ** 3, device=DEV)
    i, j, k = idx % m, (idx // m) % m, idx // (m * m)
    corner = torch.tensor([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], dtype=F64, device=DEV)
    t = (torch.stack([i, j, k], 1).to(F64)[:, None, :] + corner) * h
    t += (2.0 * _rand(g, m ** 3, 4, 3) - 1.0) * (0.3 * h)
    c = t.mean(1, keepdim=True)
    t -= c
    t *= torch.exp(0.4 * torch.randn(m ** 3, generator=g, device=DEV, dtype=F64))[:, None, None]
    t += c
    even = ((i + j + k) & 1) == 0
    return t[even].contiguous(), t[~even].contiguous()


def _soup(n, verts, size, g):
    """n elements: a centre in the unit cube, every vertex within +-size of it."""
    return _rand(g, n, 1, 3) + (2.0 * _rand(g, n, verts, 3) - 1.0) * size


def _scene(case, g):
    """The two objects of a "step" or "patches" case."""
    n, scene = case["size"], case.get("scene", "sphere_plate")
    if scene == "hexes":
        shift = (0.2 + 0.6 * _rand(g, 3)) / n
        return _hexes(n, g), _hexes(n, g) + shift
    if scene == "plates":
        # n x n / 2 quads of 0.01 x 0.02, the upper plate's vertices 0.002 to 0.006 above the lower one's
        m = n // 2
        gap = 0.004 + 0.002 * (2.0 * _rand(g, m + 1, n + 1) - 1.0)
        return _plate(n, m, 0.0, 0.01 * n, 0.0, 0.02 * m, 0.0), _plate(n, m, 0.0, 0.01 * n, 0.0, 0.02 * m, gap)
    if scene == "tets":
        return _tets(n, g)
    # a sphere of radius 0.5, turned at random, pressed 0.01 into a plate (4 n x 2 n quads)
    s = 0.5 * (_sphere(n) @ _rotation(g).T)
    at = torch.cat([0.2 * (_rand(g, 2) - 0.5), torch.tensor([0.49], dtype=F64, device=DEV)])
    return (s + at).contiguous(), _plate(4 * n, 2 * n, -1.0, 1.0, -0.5, 0.5, 0.0)


def _moved(x, g):
    """The next step's vertices: a small rigid motion and a smaller deformation."""
    d = 2e-4 * (2.0 * _rand(g, 3) - 1.0)
    return x + d + 1e-4 * torch.sin(7.0 * x.flip(-1))


# ---- passes -------------------------------------------------------------------------------------------------------

def _context(case, **more):
    stream = torch.cuda.Stream()
    ctx = bvhg.Context(k=case["k"], precision=PRECISION[case.get("precision", "fp64")], epsilon=case.get("eps", 0.0),
                       stream=stream.cuda_stream, **more)
    return stream, ctx


def _capacity(case, elements):
    """Room for the pairs of a pass, as a program keeps it between steps: more than the scene can give."""
    per = {"hexes": 10, "plates": 16, "tets": 3, "sphere_plate": 1}.get(case.get("scene"))
    per = per or {"self": 6, "batch": 2, "bodies": 1, "sweep": 1, "patches": 1}[case["kind"]]
    return 4096 + per * elements


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    stream, ctx = _context(case)
    s = {"case": case, "stream": stream, "ctx": ctx}
    if kind in ("step", "patches"):
        a, b = _scene(case, g)
        s["a"], s["b"] = ctx.object(), ctx.object()
        if case.get("mode") == "refit":
            # last step's trees exist; the vertices have moved since, in the same buffers
            for o, x in ((s["a"], a), (s["b"], b)):
                torch.cuda.synchronize()
                ctx.set_elements(o, x)
                ctx.build(o)
                ctx.synchronize()
                x.copy_(_moved(x, g))
        if case.get("mem") == "host":
            a, b = a.cpu().numpy(), b.cpu().numpy()
        s["xa"], s["xb"] = a, b
        elements = a.shape[0] + b.shape[0]
    elif kind == "self":
        n = case["size"]
        s["xa"] = _soup(n, case["verts"], 0.5 * n ** (-1.0 / 3.0), g)
        s["gid"] = torch.randperm(4 * n, generator=g, device=DEV)[:n].contiguous()
        s["a"] = ctx.object()
        elements = n
    elif kind == "batch":
        n = case["scenes"]
        u = (np.arange(n) + np.random.default_rng(seed).uniform(0.0, 1.0, n)) / n
        counts = np.exp(np.log(case["lo"]) + u * (np.log(case["hi"]) - np.log(case["lo"]))).astype(np.int64)
        np.random.default_rng(seed + 1).shuffle(counts)
        s["x"], ia, ib = [], [], []
        for c in counts.tolist():
            na = max(1, c // 2)
            size = 0.75 * c ** (-1.0 / 3.0)
            a, b = _soup(na, 3, size, g), _soup(max(1, c - na), 3, size, g) + (_rand(g, 3) - 0.5)
            for x, ids in ((a, ia), (b, ib)):
                o = ctx.object()
                ctx.set_elements(o, x)
                s["x"].append(x)
                ids.append(o)
        s["ia"], s["ib"] = np.array(ia, dtype=np.int32), np.array(ib, dtype=np.int32)
        elements = int(1.3 * n * (case["hi"] - case["lo"]) / np.log(case["hi"] / case["lo"])) + case["hi"]
    elif kind == "bodies":
        n, nu = case["bodies"], case["size"]
        base = torch.from_numpy(meshes.torus(nu, nu // 2)).to(DEV)
        s["x"], objs = [], []
        for i in range(n):
            centre = torch.tensor([1.2 * (i % 4), 1.2 * ((i // 4) % 4), 0.9 * (i // 16)], dtype=F64, device=DEV)
            s["x"].append((base @ _rotation(g).T + centre).contiguous())
            objs.append(ctx.object())
        torch.cuda.synchronize()
        for o, x in zip(objs, s["x"]):
            ctx.set_elements(o, x)
            ctx.build(o)
        ctx.synchronize()
        for x in s["x"]:
            x.copy_(_moved(x, g))
        pairs = [(i, j) for i in range(n) for j in range(i + 1, n)]
        s["ia"] = np.array([objs[i] for i, _ in pairs], dtype=np.int32)
        s["ib"] = np.array([objs[j] for _, j in pairs], dtype=np.int32)
        elements = n * base.shape[0]
    elif kind == "sweep":
        n = case["size"]
        size = 0.004 * (262144 / n) ** (1.0 / 3.0)
        s["xa"], s["xb"] = _soup(n, 3, size, g), _soup(n, 3, size, g)
        s["a"], s["b"] = ctx.object(), ctx.object()
        torch.cuda.synchronize()
        for o, x in ((s["a"], s["xa"]), (s["b"], s["xb"])):
            ctx.set_elements(o, x)
            ctx.build(o)
        ctx.synchronize()
        elements = 2 * n
    else:
        raise ValueError(kind)
    if "ia" in s:
        s["counts"] = np.zeros(len(s["ia"]), dtype=np.uint64)
    cap = _capacity(case, elements)
    if case.get("mem") == "host":
        s["pairs"] = np.full(cap, -1, dtype=np.int64)
    else:
        s["out"] = torch.empty((cap, 2), dtype=torch.int64, device=DEV)
        s["pairs"] = torch.full((cap,), -1, dtype=torch.int64, device=DEV)
        s["place"] = torch.empty(cap, dtype=torch.int64, device=DEV)
    if kind == "patches":
        p, d = case["patches"], case["k"] // 2
        s["cut"] = [(torch.empty(p + 1, dtype=torch.int64, device=DEV),
                     torch.empty(x.shape[0], dtype=torch.int32, device=DEV),
                     torch.empty((p, d, 2), dtype=F64, device=DEV)) for x in (s["xa"], s["xb"])]
        s["groups"] = torch.full((min(p * p, 1 << 18), 4), -1, dtype=torch.int32, device=DEV)
    torch.cuda.synchronize()
    return s


def _ok(status):
    if status != bvhg.OK:
        raise RuntimeError(f"status {status}")


def _ordered(s, keys):
    """The pairs' keys in ascending order, in the program's buffer."""
    n = keys.shape[0]
    torch.sort(keys, out=(s["pairs"][:n], s["place"][:n]))
    return {"count": n, "pairs": s["pairs"]}


def _keys(out, n):
    """Pairs (a, b) as a << 32 | b."""
    return out[:n, 0] * (1 << 32) + out[:n, 1]


def _batch(s, mode):
    ctx, out, counts = s["ctx"], s["out"], s["counts"]
    _ok(ctx.batch_broadphase_raw(s["ia"].ctypes.data, s["ib"].ctypes.data, len(s["ia"]), mode, out.data_ptr(),
                                 out.shape[0], counts.ctypes.data, bvhg.MEM_DEVICE))
    n = int(counts.sum())
    per_scene = torch.from_numpy(counts.astype(np.int64)).to(DEV, non_blocking=True)
    scene = torch.repeat_interleave(per_scene, output_size=n)
    # scene, element of a, element of b: scenes hold fewer than 2^20 elements per object and number fewer than 2^20
    keys = (scene * (1 << 40)) + out[:n, 0] * (1 << 20) + out[:n, 1]
    return {"scenes": counts.astype(np.int64), **_ordered(s, keys)}


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    mode = bvhg.REFIT if case.get("mode") == "refit" else bvhg.REBUILD
    with torch.cuda.stream(s["stream"]):
        if kind == "step" and case["mem"] == "host":
            for o, x in ((s["a"], s["xa"]), (s["b"], s["xb"])):
                ctx.set_elements(o, x)
                ctx.build(o, mode)
            pairs = ctx.broadphase(s["a"], s["b"])
            n = pairs.shape[0]
            s["pairs"][:n] = np.sort((pairs[:, 0] * np.uint64(1 << 32) + pairs[:, 1]).astype(np.int64))
            return {"count": n, "pairs": s["pairs"]}
        if kind == "step":
            ctx.set_elements(s["a"], s["xa"])
            ctx.set_elements(s["b"], s["xb"])
            ctx.build(s["a"], mode)
            ctx.build(s["b"], mode)
            st, n = ctx.broadphase_raw(s["a"], s["b"], s["out"].data_ptr(), s["out"].shape[0], bvhg.MEM_DEVICE)
            _ok(st)
            return _ordered(s, _keys(s["out"], n))
        if kind == "self":
            ctx.set_elements(s["a"], s["xa"], gid=s["gid"])
            ctx.build(s["a"])
            n = ctypes.c_uint64()
            _ok(bvhg.lib.bvhg_self_collision(ctx._h, s["a"], s["out"].data_ptr(), s["out"].shape[0], ctypes.byref(n),
                                             bvhg.MEM_DEVICE))
            return _ordered(s, _keys(s["out"], n.value))
        if kind == "batch":
            return _batch(s, bvhg.REBUILD)
        if kind == "bodies":
            return _batch(s, bvhg.REFIT)
        if kind == "sweep":
            st, n, axis = ctx.sort_and_sweep_raw(s["a"], s["b"], -1, s["out"].data_ptr(), s["out"].shape[0],
                                                 bvhg.MEM_DEVICE)
            _ok(st)
            return {"axis": axis, **_ordered(s, _keys(s["out"], n))}
        # patches
        p, ids = case["patches"], (s["a"], s["b"])
        ctx.set_elements(s["a"], s["xa"])
        ctx.set_elements(s["b"], s["xb"])
        ctx.build(s["a"])
        ctx.build(s["b"])
        for o, (bounds, order, boxes) in zip(ids, s["cut"]):
            _ok(bvhg.lib.bvhg_cluster(ctx._h, o, p, bounds.data_ptr(), order.data_ptr(), bvhg.MEM_DEVICE))
            _ok(bvhg.lib.bvhg_patch_kdops(ctx._h, o, boxes.data_ptr(), bvhg.MEM_DEVICE))
        ng, n = ctypes.c_uint64(), ctypes.c_uint64()
        pairs = s["out"].view(torch.int32)
        _ok(bvhg.lib.bvhg_patch_pairs(ctx._h, s["a"], s["b"], s["groups"].data_ptr(), s["groups"].shape[0],
                                      ctypes.byref(ng), pairs.data_ptr(), s["out"].shape[0], ctypes.byref(n),
                                      bvhg.MEM_DEVICE))
        groups = s["groups"][:ng.value]
        flat = pairs.reshape(-1, 2)[:n.value].to(torch.int64)
        group = torch.repeat_interleave(groups[:, 3].to(torch.int64), output_size=n.value)
        # group, place in the patch of a, place in the patch of b: patches hold fewer than 2^22 elements
        keys = group * (1 << 44) + flat[:, 0] * (1 << 22) + flat[:, 1]
        return {"groups": s["groups"], "a": list(s["cut"][0]), "b": list(s["cut"][1]), **_ordered(s, keys)}


# ---- what a pass cannot do without --------------------------------------------------------------------------------

def work(case):
    """Each vertex read once and each pair written once (16 bytes), from the pairs per element that the scenes give;
    the projections of every vertex onto the K/2 normals."""
    kind, k = case["kind"], case["k"]
    verts, per = 3, 0.0
    if kind == "batch":
        span = math.log(case["hi"] / case["lo"])
        n = case["scenes"] * (case["hi"] - case["lo"]) / span
        per = 0.15
    elif kind == "bodies":
        n, per = case["bodies"] * case["size"] * case["size"], 0.005
    elif kind == "self":
        n, verts, per = case["size"], case["verts"], 1.0
    elif kind == "sweep":
        n, per = 2 * case["size"], 0.03
    elif case.get("scene") == "hexes":
        n, verts, per = 2 * case["size"] ** 3, 8, 5.0
    elif case.get("scene") == "plates":
        n, per = 2 * case["size"] * 2 * (case["size"] // 2), 3.0
    elif case.get("scene") == "tets":
        n, verts, per = case["size"] ** 3, 4, 2.2
    else:
        n, per = 36 * case["size"] ** 2, 0.001
    size = n * (verts * 24.0 + 16.0 * per)
    if kind == "self":
        size += 8.0 * n
    if kind == "patches":
        size += 4.0 * n + 2.0 * case["patches"] * k * 8.0
    return {"bytes": size, "flops": n * verts * (k // 2) * 5.0}


# ---- the floating-point results in plain torch --------------------------------------------------------------------

_R2, _R3 = 0.7071067811865475, 0.5773502691896258


def _normals(k):
    axes = [(1, 0, 0), (0, 1, 0), (0, 0, 1)]
    corners = [(_R3, _R3, _R3), (_R3, -_R3, _R3), (_R3, _R3, -_R3), (_R3, -_R3, -_R3)]
    edges = [(_R2, _R2, 0), (_R2, 0, _R2), (0, _R2, _R2), (_R2, -_R2, 0), (_R2, 0, -_R2), (0, _R2, -_R2)]
    return axes if k == 6 else axes + edges if k == 18 else axes + corners + edges


def _slabs(x, k):
    """(n, K/2, 2) minima and maxima of the projections of every element's vertices."""
    out = []
    for nx, ny, nz in _normals(k):
        p = (x[..., 0] * nx + x[..., 1] * ny) + x[..., 2] * nz
        out.append(torch.stack([p.amin(1), p.amax(1)], -1))
    return torch.stack(out, 1)


def _patch_boxes(x, k, patches):
    """The boxes of the Morton clustering: elements by the 30-bit Morton hash of their centroids (stable), cut where
    neighbouring hashes split highest."""
    n = x.shape[0]
    slabs = _slabs(x, k)
    centre = torch.zeros(n, 3, dtype=F64, device=x.device)
    for v in range(x.shape[1]):
        centre = centre + x[:, v]
    centre = centre / x.shape[1]
    lo, hi = slabs[:, :3, 0].amin(0), slabs[:, :3, 1].amax(0)
    q = (centre - lo) * (1.0 / (hi - lo)) * 2097152.0
    q = torch.nan_to_num(q, nan=0.0).to(torch.int64) & 0x1FFFFF
    h = torch.zeros(n, dtype=torch.int64, device=x.device)
    for bit in range(10):  # the top 10 of the 21 bits per axis, and x's place lowest
        for c in range(3):
            h |= ((q[:, c] >> (11 + bit)) & 1) << (3 * bit + c)
    h, order = torch.sort(h, stable=True)
    split = h[1:] ^ h[:-1]
    depth = torch.where(split > 0, 31 - torch.log2(split.clamp(min=1).to(F64)).floor().to(torch.int64), 32)
    take = min(patches - 1, n - 1)
    cuts = torch.sort(torch.sort(depth, stable=True)[1][:take])[0]
    bounds = [0] + cuts.tolist() + [n - 1] * (patches - 1 - take) + [n]
    s = slabs[order]
    out = torch.empty(patches, k // 2, 2, dtype=F64, device=x.device)
    for p in range(patches):
        part = s[bounds[p]:bounds[p + 1]]
        if part.shape[0]:
            out[p, :, 0], out[p, :, 1] = part[..., 0].amin(0), part[..., 1].amax(0)
        else:
            out[p, :, 0], out[p, :, 1] = math.inf, -math.inf
    return out


def exact(case, seed):
    """The patch boxes; every other output is whole numbers."""
    if case["kind"] != "patches":
        return None
    a, b = _scene(case, _gen(seed))
    return {"groups": None, "count": None, "pairs": None, "a": [None, None, _patch_boxes(a, case["k"], case["patches"])],
            "b": [None, None, _patch_boxes(b, case["k"], case["patches"])]}

"""The work that programs have this library do, as cases that can be timed and
compared: every extractor over seeded scenes of the kinds that the tests and
the benchmark use, a caller's own field, the chunk batch, and the surrogate's
training step and inference.

A case is a dict of plain values; ``kind`` picks the entry point.  One
library context serves every state, as it does in a program that meshes one
source after the other.
"""
import math

import numpy as np
import torch

from isosurface_gb300 import (CentralDifference, Context, Difference, Program, RectangularPrism, Sphere, Torus,
                              Translate, Union, scenes, unit_to_cube)
from isosurface_gb300.api import Batch
from isosurface_gb300.surrogate import Surrogate

_context = None


def _ctx():
    global _context
    if _context is None:
        _context = Context(0)
    return _context


def listed():
    return [
        # the smallest call: a preview mesh of one primitive, delivered to page-locked host buffers, as the
        # binding's IndexedVertices sink takes it
        {"name": "mc_sphere_65", "kind": "mc", "scene": "sphere", "size": 65, "normals": False, "to": "host"},
        # the examples' torus with central-difference normals at the reference benchmark's grid
        # (IndexedInterleavedNormals), for a program that exports it
        {"name": "mc_torus_128_normals", "kind": "mc", "scene": "torus", "size": 128, "normals": True, "to": "host"},
        # an ordinary CSG model at a preview resolution, for a program that draws it on the same device
        {"name": "mc_csg_257", "kind": "mc", "scene": "csg", "size": 257, "normals": False, "to": "device"},
        # the headline workload: 512 x 512 x 513 cells over a hard union of 64 spheres
        {"name": "mc_union_513", "kind": "mc", "scene": "union", "count": 64, "size": 513, "normals": False,
         "to": "device"},
        # the expensive source: a smooth union of thousands of spheres, at half of its full resolution
        {"name": "mc_smooth_257", "kind": "mc", "scene": "smooth", "count": 4096, "size": 257, "normals": False,
         "to": "device"},
        # a scan or simulation already on the device: a dense field with odd rows, not a source
        {"name": "mc_field_401", "kind": "field", "size": 401, "layers": 301, "pitch": 401, "features": 20},
        # sharp-feature meshing of the CSG model, features placed by the QEF
        {"name": "dc_csg_257", "kind": "dc", "scene": "csg", "size": 257, "placer": 0},
        # the adaptive extractor at the depth of the same grid
        {"name": "lhmc_csg_8", "kind": "lhmc", "scene": "csg", "depth": 8},
        # the viewer's largest grid of the sharp-feature extractor over the Directed metric
        {"name": "emc_solid_128", "kind": "emc", "size": 128},
        # a terrain-like world of many small uneven chunks, one call
        {"name": "chunks_1024", "kind": "chunks", "count": 1024},
        # one training step's forward and backward of the surrogate network at its batch size
        {"name": "train_65536", "kind": "train", "points": 65536},
        # the surrogate network at scattered points of the caller
        {"name": "infer_250001", "kind": "infer", "points": 250001},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mc", "mc", "mc", "mc", "field", "dc", "lhmc", "emc", "chunks", "train", "infer"])
    if kind == "mc":
        scene = rng.choice(["sphere", "torus", "csg", "union", "smooth"])
        case = {"kind": kind, "scene": scene, "size": _log_int(rng, 17, 256 if scene == "smooth" else 513),
                "normals": scene != "smooth" and rng.random() < 0.3}
        case["to"] = "host" if case["size"] < 150 else "device"
        if scene == "union":
            case["count"] = _log_int(rng, 4, 250)
        if scene == "smooth":
            case["count"] = _log_int(rng, 32, 4096)
        return case
    if kind == "field":
        n = _log_int(rng, 40, 420)
        return {"kind": kind, "size": n, "layers": rng.randint(max(2, n // 2), n + 1), "pitch": n + rng.choice([0, 0, 1, 7]),
                "features": rng.randint(6, 24)}
    if kind == "dc":
        return {"kind": kind, "scene": rng.choice(["csg", "torus"]), "size": _log_int(rng, 40, 257),
                "placer": rng.choice([0, 0, 1])}
    if kind == "lhmc":
        return {"kind": kind, "scene": rng.choice(["csg", "torus"]), "depth": rng.randint(5, 8)}
    if kind == "emc":
        return {"kind": kind, "size": _log_int(rng, 24, 160)}
    if kind == "chunks":
        return {"kind": kind, "count": _log_int(rng, 16, 1024)}
    if kind == "train":
        return {"kind": kind, "points": _log_int(rng, 1000, 65536)}
    return {"kind": "infer", "points": _log_int(rng, 1, 250001)}


# ---------------------------------------------------------------- inputs ----
def _source(case, seed):
    rng = np.random.default_rng([seed, 77])
    scene = case["scene"]
    if scene == "sphere":
        return unit_to_cube(Sphere(float(rng.uniform(0.70, 0.80))))
    if scene == "torus":
        torus = Torus(float(rng.uniform(0.23, 0.27)), float(rng.uniform(0.09, 0.11)))
        src = Translate(torus, tuple(float(v) for v in rng.uniform(0.48, 0.52, 3)))
        return CentralDifference(src) if case["kind"] == "mc" else src
    if scene == "csg":
        return scenes.csg(seed)
    if scene == "union":
        return scenes.sphere_union(seed, case["count"])
    return scenes.smooth_spheres(seed, case["count"])


def _solid(seed):
    """Box-cornered ball and ring: the Directed metric has no rotation, so the parts are only moved."""
    rng = np.random.default_rng([seed, 78])

    def moved(part):
        return Translate(part, tuple(float(v) for v in rng.uniform(-0.08, 0.08, 3)))

    half = tuple(float(v) for v in rng.uniform(0.57, 0.63, 3))
    ball, ring = Sphere(float(rng.uniform(0.68, 0.72))), Torus(float(rng.uniform(0.48, 0.52)), 0.15)
    return unit_to_cube(Union(Difference(moved(ball), moved(RectangularPrism(half))), moved(ring)))


def _dense_field(case, seed):
    """A smooth random field on the device, (layers, size, pitch) with the row's tail unused: trilinear
    interpolation of random values, some `features` of them along an axis."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, nz, k = case["size"], case["layers"], case["features"]
    coarse = torch.randn((1, 1, max(2, k * nz // n), k, k), generator=g, device="cuda")
    fine = torch.nn.functional.interpolate(coarse, size=(nz, n, n), mode="trilinear", align_corners=True)[0, 0]
    field = torch.ones((nz, n, case["pitch"]), device="cuda")
    field[:, :, :n] = fine
    return field


def _net_inputs(case, seed):
    rng = np.random.default_rng([seed, 79])
    points = rng.uniform(-1.0, 1.0, (case["points"], 3)).astype(np.float32)
    spheres = scenes.random_spheres(seed, 64, 0.9, (0.05, 0.25))
    # signed distance to the union, as a data set labels its points
    targets = np.full(case["points"], np.inf, np.float32)
    for cx, cy, cz, r in spheres:
        d = np.sqrt(((points - np.array([cx, cy, cz], np.float32)) ** 2).sum(1)) - r
        np.minimum(targets, d, out=targets)
    return points, targets


def prepare(case, seed):
    ctx = _ctx()
    kind = case["kind"]
    state = {"case": case, "ctx": ctx}
    if kind in ("mc", "dc", "lhmc", "emc"):
        state["program"] = Program(ctx, _solid(seed) if kind == "emc" else _source(case, seed))
    if kind in ("mc", "dc", "lhmc", "emc", "field", "chunks"):
        # the program's own vertex and index buffers, with room to spare
        room = int(1.5 * _vertices(case)) + 8192
        floats = 6 if case.get("normals") else 3
        to = {"device": "cuda"} if _on_device(case) else {"pin_memory": True}
        state["vertices"] = torch.zeros((room, floats), dtype=torch.float32, **to)
        state["indices"] = torch.zeros((2 * room, 3), dtype=torch.int32, **to)
        if not _on_device(case):
            state["arrays"] = state["vertices"].numpy(), state["indices"].numpy().view(np.uint32)
    if kind == "field":
        state["field"] = _dense_field(case, seed)
        torch.cuda.synchronize()
    elif kind == "chunks":
        state["batch"] = Batch(ctx, scenes.chunks(seed, case["count"]))  # 16^3 to 64^3 cells, 1-16 primitives each
        state["batch"].run()  # sizes the batch's buffers, as a program's first frame does
    elif kind in ("train", "infer"):
        state["net"] = Surrogate(ctx, seed=seed)
        state["points"], state["targets"] = _net_inputs(case, seed)
    return state


# ------------------------------------------------------------------ runs ----
class _DeviceArray:
    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _on_device(case):
    return case["kind"] in ("field", "chunks") or case.get("to") == "device"


def _mesh(state, info):
    """The mesh of the last extraction in the program's own buffers (the context's are the next call's)."""
    ctx, vertices, indices = state["ctx"], state["vertices"], state["indices"]
    nv, nt = info.num_vertices, info.num_triangles
    if not _on_device(state["case"]):
        ctx.download(info, out=state["arrays"])
    elif nt:
        v, i, _, _ = ctx.device_mesh()
        vertices[:nv].copy_(torch.as_tensor(_DeviceArray(v, (nv, vertices.shape[1]), "<f4"), device="cuda"))
        indices[:nt].copy_(torch.as_tensor(_DeviceArray(i, (nt, 3), "<i4"), device="cuda"))
    return {"vertices": vertices, "indices": indices, "count": nv, "triangles": nt}


def run(state):
    case, ctx, kind = state["case"], state["ctx"], state["case"]["kind"]
    if kind == "mc":
        if case["to"] == "host":
            info = ctx.mc_extract_host(state["program"], case["size"], state["vertices"], state["indices"],
                                       normals=case["normals"])
            return {"vertices": state["vertices"], "indices": state["indices"], "count": info.num_vertices,
                    "triangles": info.num_triangles}
        return _mesh(state, ctx.mc_extract(state["program"], case["size"], normals=case["normals"]))
    if kind == "field":
        n = case["size"]
        return _mesh(state, ctx.mc_extract_field(state["field"].data_ptr(), n, n, case["layers"], case["pitch"]))
    if kind == "dc":
        return _mesh(state, ctx.dc_extract(state["program"], case["size"], case["placer"]))
    if kind == "lhmc":
        return _mesh(state, ctx.lhmc_extract(state["program"], case["depth"]))
    if kind == "emc":
        info, flips = ctx.emc_extract(state["program"], case["size"])
        return dict(_mesh(state, info), flips=flips)
    if kind == "chunks":
        info = state["batch"].run()
        return dict(_mesh(state, info), extents=state["batch"].extents().astype(np.int64))
    if kind == "train":
        loss, grad = state["net"].loss_grad(state["points"], state["targets"])
        return {"loss": float(loss), "grad": grad}
    return {"values": state["net"].forward(state["points"], bf16=True)}


# ------------------------------------------------------------------ work ----
def _area(case):
    """Surface area of the scene in the unit sample frame (expected, for the seeded ones)."""
    scene = case.get("scene", "solid")
    if scene == "sphere":
        return math.pi * 0.75 ** 2
    if scene == "torus":
        return 4.0 * math.pi ** 2 * 0.25 * 0.1
    if scene in ("csg", "solid"):
        return 3.0
    # spheres of radius U[a, b] with centres in a cube: areas times the share that no other sphere covers
    a, b, side = (0.05, 0.25, 1.6) if scene == "union" else (0.01, 0.08, 1.8)
    r2, r3 = (b ** 3 - a ** 3) / (3 * (b - a)), (b ** 4 - a ** 4) / (4 * (b - a))
    bare = math.exp(-case["count"] * 4.0 / 3.0 * math.pi * r3 / side ** 3)
    return case["count"] * math.pi * r2 * bare


def _vertices(case):
    """Lattice edges that a surface of this area crosses: 1.5 per cell face of area, on average."""
    if case["kind"] == "field":
        return 1.4 * case["features"] * case["size"] * case["layers"]  # about one sheet for each random value
    if case["kind"] == "chunks":
        # half 16^3, 35 % 32^3, 15 % 64^3 cells, a surface of about 1.9 faces of the chunk
        return case["count"] * 1.5 * 1.9 * (0.5 * 16 ** 2 + 0.35 * 32 ** 2 + 0.15 * 64 ** 2)
    cells = 2 ** case["depth"] if case["kind"] == "lhmc" else case["size"] - 1
    return 1.5 * _area(case) * cells * cells


def work(case):
    kind = case["kind"]
    if kind in ("train", "infer"):
        n, weights = case["points"], 96 * 256 + 5 * 256 * 256 + 256
        if kind == "infer":
            return {"bytes": 16 * n + 2 * weights, "flops": 2 * n * weights}
        return {"bytes": 16 * n + 8 * weights, "flops": 6 * n * weights - 2 * n * 96 * 256}
    # a mesh: 12 bytes a vertex (24 with normals), two triangles of 12 bytes for each; the source's value at both
    # ends of each crossed edge, and for the feature extractors its normals
    vertices = _vertices(case)
    each = 48 if case.get("normals") else 36
    flops = {"csg": 110, "solid": 110}.get(case.get("scene", "solid"), 22)
    if kind in ("dc", "emc"):
        flops *= 8
    read = 4 * case["size"] ** 2 * case["layers"] if kind == "field" else 0
    return {"bytes": read + each * vertices, "flops": 2 * flops * vertices}


# ----------------------------------------------------------------- exact ----
def _weights(seed):
    """The surrogate's initial parameters in 64 bits: uniform in +-sqrt(6 / (fan_in + fan_out)) from SplitMix64 of the
    seed and the parameter's place, biases zero (rounded to 32 bits, as the network holds them)."""
    def splitmix(z):
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))

    layers, at = [], 0
    for fin, fout in [(96, 256)] + [(256, 256)] * 5 + [(256, 1)]:
        a = np.sqrt(np.float32(6.0) / np.float32(fin + fout))
        with np.errstate(over="ignore"):
            h = splitmix(np.uint64(seed) * np.uint64(1000003) + np.arange(at, at + fin * fout, dtype=np.uint64))
        u = (h >> np.uint64(40)).astype(np.float32) * np.float32(1.0 / 16777216.0)
        w = (a * (np.float32(2.0) * u - np.float32(1.0))).astype(np.float64).reshape(fout, fin)
        layers.append((torch.from_numpy(w).cuda(), torch.zeros(fout, dtype=torch.float64, device="cuda")))
        at += fin * fout + fout
    return layers


def _features(x):
    w = math.pi * 2.0 ** (7.0 * torch.arange(16, dtype=torch.float64, device=x.device) / 15.0)
    arg = x[:, :, None] * w  # (n, 3, 16)
    return torch.stack([torch.sin(arg), torch.cos(arg)], 3).reshape(len(x), 96)


def _net(layers, x):
    h = _features(x)
    for w, b in layers[:-1]:
        h = torch.nn.functional.softplus(h @ w.T + b, beta=100.0, threshold=1e9)
    w, b = layers[-1]
    return (h @ w.T + b)[:, 0]


def exact(case, seed):
    """Meshes have no plain counterpart in their vertex order; the network's numbers do."""
    if case["kind"] not in ("train", "infer"):
        return None
    points, targets = _net_inputs(case, seed)
    layers = _weights(seed)
    x, t = torch.from_numpy(points).cuda().double(), torch.from_numpy(targets).cuda().double()
    if case["kind"] == "infer":
        with torch.no_grad():
            parts = [_net(layers, x[i:i + 65536]) for i in range(0, len(x), 65536)]
        return {"values": torch.cat(parts).cpu().numpy()}
    for w, b in layers:
        w.requires_grad_(True)
        b.requires_grad_(True)
    d, total = 0.1, 0.0
    for i in range(0, len(x), 16384):
        y, ti = _net(layers, x[i:i + 16384]), t[i:i + 16384]
        # L1 inside the band |t| < d, one-sided where the target saturates
        e = torch.where(ti >= d, torch.clamp(y - d, max=0.0), torch.where(ti <= -d, torch.clamp(y + d, min=0.0), y - ti))
        loss = e.abs().sum() / len(x)
        loss.backward()
        total += float(loss)
    grad = torch.cat([p.grad.reshape(-1) for pair in layers for p in pair])
    return {"loss": total, "grad": grad.cpu().numpy()}

"""Performance cases of the mesh -> volume -> mesh path on one GPU.

Every case is one pass of a user's program through the public entry points
(`baby_shark_gb300`'s classes, or the C ABI of `include/baby_shark_gb300.h`
where the mesh already lies in device memory or the result goes to a buffer
that the program keeps).  Meshes are the shapes of this repository's workloads
(displaced tori, noisy icospheres, icospheres with holes), generated on the
GPU from the seed.  Kinds:

  remesh   mesh arrays on the host -> volume -> CornerTable tables
  convert  mesh in device memory -> signed volume exported to pinned memory
  batch    several uneven meshes in one conversion
  boolean  two volumes -> union / subtraction / intersection, exported
  offset   a volume grown or shrunk, exported
  contour  a volume -> triangle soup in pinned memory
  points   a mesh's winding numbers at arbitrary points
  learned  a network trained on winding numbers, and its predictions

Results go to buffers of a fixed capacity, zero past the result's end, with
the sizes beside them.
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

import baby_shark_gb300 as bs
from baby_shark_gb300 import _native as N

# Most band voxels, triangles and query points of a drawn case (the largest listed sizes).
MAX_BAND, MAX_TRI, MAX_POINTS = 3.5e7, 1_048_576, 1_500_000


def listed():
    return [
        # a preview of a coarse part while a slider moves: the smallest call, launches and waits only
        dict(name="convert_tiny", kind="convert", shape="icosphere", subdiv=2, noise=0.0, voxel=0.05, band=1,
             tree="reference"),
        # the repository's plain remesh workload, through the Python classes
        dict(name="remesh_dc", kind="remesh", shape="icosphere", subdiv=4, noise=0.05, voxel=0.02, band=3,
             method="FeaturePreserving"),
        # VoxelRemesher as it comes: marching cubes, band 0, a scanned part of ordinary size
        dict(name="remesh_mc", kind="remesh", shape="icosphere", subdiv=6, noise=0.002, voxel=0.008, band=0,
             method="Manifold"),
        # one operand of the boolean workload: the library's largest usual conversion
        dict(name="convert_torus", kind="convert", shape="torus", nu=1024, nv=512, noise=0.02, voxel=0.002, band=3,
             tree="reference"),
        # a scan with holes (triangle soup), signs as the reference's tree gives them
        dict(name="convert_soup", kind="convert", shape="soup", subdiv=8, noise=0.1, voxel=0.003, band=3,
             tree="reference"),
        # the same kind of scan with the library's faster tree
        dict(name="convert_soup_fast", kind="convert", shape="soup", subdiv=8, noise=0.1, voxel=0.003, band=2,
             tree="fast"),
        # a folder of parts of uneven size in one call
        dict(name="batch_uneven", kind="batch", meshes=15, tri_max=60000, res_max=200, band=3),
        # the boolean workload's subtraction
        dict(name="subtract", kind="boolean", op="subtract", nu=700, nv=350, voxel=0.003, band=3),
        # the boolean workload's offset
        dict(name="offset_grow", kind="offset", nu=512, nv=256, voxel=0.004, distance=0.01, band=3),
        # the surface of a finished model, for display or printing
        dict(name="contour_dc", kind="contour", mesher="dc", nu=700, nv=350, voxel=0.003, band=3),
        # inside / outside of sampled points (training data, point-cloud filters)
        dict(name="points_fast", kind="points", subdiv=5, points=1_500_000, tree="fast", order=2),
        # the learned far field's training and evaluation on one model
        dict(name="learned", kind="learned", samples=131072, batch=8192, epochs=2, points=1_000_000),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _torus_grid(rng, most):
    nv = int(_log(rng, 12, math.sqrt(most / 4)))
    return max(8, int(nv * rng.uniform(1.4, 2.2))), nv


def _voxel(rng, area, extent, band, most=MAX_BAND):
    """A voxel size that makes the grid 40 to 1200 voxels long, within the band-voxel limit."""
    h = extent / _log(rng, 40, 1200)
    return float(np.float32(max(h, math.sqrt(area * (2 * band + 6) / most))))


def draw(rng):
    kind = rng.choice(["remesh", "convert", "convert", "convert", "batch", "boolean", "offset", "contour", "points",
                       "learned"])
    if kind in ("remesh", "convert"):
        band = rng.choice([0, 1, 2, 3, 3, 4])
        case = dict(kind=kind, band=band)
        shape = rng.choice(["icosphere", "torus", "soup"] if kind == "convert" else ["icosphere", "torus"])
        case["shape"] = shape
        most = MAX_BAND if kind == "convert" else 3.0e6
        if shape == "torus":
            case["nu"], case["nv"] = _torus_grid(rng, MAX_TRI if kind == "convert" else 2e5)
            case["noise"] = rng.uniform(0.0, 0.02)
            case["voxel"] = _voxel(rng, 11.8, 2.6, band, most)
        else:
            case["subdiv"] = rng.randint(2, 6 if kind == "remesh" else 7)
            # noise below the edge length keeps the surface a scan, not a hedgehog
            case["noise"] = rng.uniform(0.0, 0.1) if shape == "soup" else rng.uniform(0.0, 0.3) / 2 ** case["subdiv"]
            case["voxel"] = _voxel(rng, 12.6, 2.0, band, most)
        if kind == "convert":
            case["tree"] = rng.choice(["reference", "reference", "fast"])
        else:
            case["method"] = rng.choice(["FeaturePreserving", "Manifold"])
            if case["method"] == "FeaturePreserving":
                case["band"] = max(band, 2)  # its gradients need both neighbours of a crossing edge
        return case
    if kind == "batch":
        return dict(kind=kind, meshes=rng.randint(2, 12), tri_max=int(_log(rng, 2000, 50000)),
                    res_max=int(_log(rng, 70, 180)), band=rng.choice([1, 2, 3]))
    if kind in ("boolean", "offset", "contour"):
        nu, nv = _torus_grid(rng, 4e5)
        band = rng.choice([2, 3])
        case = dict(kind=kind, nu=nu, nv=nv, band=band, voxel=_voxel(rng, 11.8, 2.6, band, 1.0e7))
        if kind == "boolean":
            case["op"] = rng.choice(["union", "subtract", "intersect"])
        elif kind == "offset":
            case["distance"] = rng.choice([-1, 1]) * case["voxel"] * rng.uniform(0.5, 3.0)
        else:
            case["mesher"] = rng.choice(["dc", "dc", "qef", "mc"])
        return case
    if kind == "points":
        tree = rng.choice(["fast", "reference"])
        return dict(kind=kind, subdiv=rng.randint(2, 5), tree=tree, order=rng.choice([2, 3]) if tree == "fast" else 2,
                    points=int(_log(rng, 1000, MAX_POINTS)))
    batch = 128 * rng.randint(8, 64)
    return dict(kind=kind, samples=batch * rng.randint(2, 16), batch=batch, epochs=rng.randint(1, 3),
                points=int(_log(rng, 1000, 1_000_000)))


# ---------------------------------------------------------------- meshes ----
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 2654435761 % (1 << 31))
    return g


@functools.lru_cache(maxsize=None)
def _icosphere(subdiv):
    """Unit icosphere (vertices float64, outward faces int64) on the GPU."""
    t = (1.0 + 5.0 ** 0.5) / 2.0
    v = torch.tensor([[-1, t, 0], [1, t, 0], [-1, -t, 0], [1, -t, 0], [0, -1, t], [0, 1, t], [0, -1, -t], [0, 1, -t],
                      [t, 0, -1], [t, 0, 1], [-t, 0, -1], [-t, 0, 1]], dtype=torch.float64, device="cuda")
    f = torch.tensor([[0, 11, 5], [0, 5, 1], [0, 1, 7], [0, 7, 10], [0, 10, 11], [1, 5, 9], [5, 11, 4], [11, 10, 2],
                      [10, 7, 6], [7, 1, 8], [3, 9, 4], [3, 4, 2], [3, 2, 6], [3, 6, 8], [3, 8, 9], [4, 9, 5],
                      [2, 4, 11], [6, 2, 10], [8, 6, 7], [9, 8, 1]], device="cuda")
    v = v / v.norm(dim=1, keepdim=True)
    for _ in range(subdiv):
        e = torch.cat([f[:, [0, 1]], f[:, [1, 2]], f[:, [2, 0]]]).sort(dim=1).values
        key, inv = torch.unique(e[:, 0] * len(v) + e[:, 1], return_inverse=True)
        mid = v[key // len(v)] + v[key % len(v)]
        m01, m12, m20 = (inv + len(v)).split(len(f))
        v = torch.cat([v, mid / mid.norm(dim=1, keepdim=True)])
        f = torch.cat([torch.stack([f[:, 0], m01, m20], 1), torch.stack([f[:, 1], m12, m01], 1),
                       torch.stack([f[:, 2], m20, m12], 1), torch.stack([m01, m12, m20], 1)])
    return v, f


def _lattice_noise(p, gen):
    """Smooth gradient noise in about [-1, 1]: random gradients on a hashed lattice, quintic fade."""
    grad = torch.randn(4096, 3, generator=gen, device="cuda", dtype=torch.float64)
    grad = grad / grad.norm(dim=1, keepdim=True)
    i = p.floor().long()
    u = p - i
    w = u * u * u * (u * (u * 6 - 15) + 10)
    out = torch.zeros(len(p), device="cuda", dtype=torch.float64)
    for k in range(8):
        d = torch.tensor([k >> 2, (k >> 1) & 1, k & 1], device="cuda")
        c = i + d
        h = (c[:, 0] * 73856093 ^ c[:, 1] * 19349663 ^ c[:, 2] * 83492791) & 4095
        out += torch.where(d.bool(), w, 1 - w).prod(dim=1) * ((u - d) * grad[h]).sum(dim=1)
    return out


def _torus(nu, nv, noise, gen, second=False):
    """Displaced torus (R 1, r 0.3); the second operand is turned 90 degrees about x and shifted 0.5 in x."""
    u = torch.arange(nu, device="cuda", dtype=torch.float64)[:, None] * (2 * math.pi / nu)
    w = torch.arange(nv, device="cuda", dtype=torch.float64)[None, :] * (2 * math.pi / nv)
    n = torch.stack([torch.cos(w) * torch.cos(u), torch.cos(w) * torch.sin(u), (torch.sin(w) + 0 * u)], -1)
    ring = torch.stack([torch.cos(u) + 0 * w, torch.sin(u) + 0 * w, 0 * u + 0 * w], -1)
    n, ring = n.reshape(-1, 3), ring.reshape(-1, 3)
    p = ring + 0.3 * n
    p = p + (noise * _lattice_noise(4.0 * p, gen))[:, None] * n
    if second:
        p = torch.stack([p[:, 0] + 0.5, -p[:, 2], p[:, 1]], 1)
    i = torch.arange(nu, device="cuda")[:, None]
    j = torch.arange(nv, device="cuda")[None, :]
    a, b = i * nv + j, (i + 1) % nu * nv + j
    c, d = (i + 1) % nu * nv + (j + 1) % nv, i * nv + (j + 1) % nv
    f = torch.cat([torch.stack([a, b, c], -1).reshape(-1, 3), torch.stack([a, c, d], -1).reshape(-1, 3)])
    return p.float().contiguous(), f


def _mesh(case, gen):
    """(vertices float32, faces int32) on the GPU."""
    if case["shape"] == "torus":
        v, f = _torus(case["nu"], case["nv"], case["noise"], gen)
        return v, f.int().contiguous()
    v, f = _icosphere(case["subdiv"])
    if case["shape"] == "icosphere":
        r = 1.0 + case["noise"] * (2 * torch.rand(len(v), generator=gen, device="cuda", dtype=torch.float64) - 1)
        # a rotation of its own for every seed: no two of them share voxels
        return (v * r[:, None] @ _rotation(gen)).float().contiguous(), f.int().contiguous()
    disp = sum(0.5 ** k * _lattice_noise(2.0 ** k * 2.0 * v + 31.0 * k, gen) for k in range(4))
    v = v * (1.0 + case["noise"] * disp / disp.abs().max())[:, None]
    keep = torch.rand(len(f), generator=gen, device="cuda") >= 0.1  # 10 % of the faces missing
    return (v @ _rotation(gen)).float().contiguous(), f[keep].int().contiguous()


def _rotation(gen):
    q, r = torch.linalg.qr(torch.randn(3, 3, generator=gen, device="cuda", dtype=torch.float64))
    q = q * torch.sign(torch.diagonal(r))
    return q * torch.sign(torch.linalg.det(q))  # a proper rotation keeps the faces outward


def _batch_sizes(case):
    """Triangles and grid resolution of each mesh of a batch, spread over their ranges."""
    n = case["meshes"]
    for k in range(n):
        x, y = (k + 0.5) / n, (k * 7 % n + 0.5) / n
        yield k, 1000 * (case["tri_max"] / 1000) ** x, 64 * (case["res_max"] / 64) ** y


def _batch(case, gen):
    out = []
    for k, tri, res in _batch_sizes(case):
        noise = float(0.01 + 0.04 * torch.rand(1, generator=gen, device="cuda"))
        if k % 2:
            nv = max(8, int(math.sqrt(tri / 4)))
            v, f = _torus(2 * nv, nv, noise, gen)
        else:
            sub = int(min(max(round(math.log(tri / 20) / math.log(4)), 3), 6))
            v, f = _mesh(dict(shape="icosphere", subdiv=sub, noise=noise), gen)
        extent = float((v.max(dim=0).values - v.min(dim=0).values).max())
        out.append((v, f.int().contiguous(), float(np.float32(extent / res))))
    return out


# ----------------------------------------------------------- entry points ----
_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = bs.Context(0)
    return _ctx


def _params(voxel, band, tree, order=2):
    p = N.M2VParams()
    N.load().bs_m2v_params_default(C.byref(p))
    p.voxel_size, p.band_width, p.wn_order, p.wn_tree = voxel, band, order, 0 if tree == "reference" else 1
    return p


def _convert(ctx, v, f, params):
    out = C.c_void_p()
    N.check(N.load().bs_mesh_to_volume_device(ctx.h, v.data_ptr(), len(v), f.data_ptr(), len(f), C.byref(params),
                                              C.byref(out)), ctx.h)
    return bs.Volume(out, ctx)


class _Leaves:
    """Pinned buffers for the leaves (and active tiles) of exported volumes."""

    def __init__(self, leaves, tiles=0, volumes=1):
        self.origins = torch.zeros((leaves, 3), dtype=torch.int32).pin_memory()
        self.values = torch.zeros((leaves, 512), dtype=torch.float32).pin_memory()
        self.masks = torch.zeros((leaves, 16), dtype=torch.int32).pin_memory()
        self.tiles = [torch.zeros((tiles, 3), dtype=torch.int32).pin_memory(),
                      torch.zeros(tiles, dtype=torch.int32).pin_memory(),
                      torch.zeros(tiles, dtype=torch.float32).pin_memory()] if tiles else []
        self.counts = np.zeros((volumes, 2), np.int64)

    def put(self, vol, k=0):
        c = vol.counts()
        at, n = int(self.counts[:k, 0].sum()), c["leaves"]
        assert at + n <= len(self.values) and (not self.tiles or c["tiles"] <= len(self.tiles[1])), c
        N.check(N.load().bs_volume_export(vol.ctx.h, vol.h, self.origins[at:].data_ptr(), self.values[at:].data_ptr(),
                                          self.masks[at:].data_ptr()), vol.ctx.h)
        if self.tiles and c["tiles"]:
            N.check(N.load().bs_volume_export_tiles(vol.ctx.h, vol.h, *(t.data_ptr() for t in self.tiles)), vol.ctx.h)
        self.counts[k] = n, c["tiles"]

    def outputs(self):
        return [self.counts, self.origins, self.values, self.masks, *self.tiles]


class _Table:
    """Buffers for a corner table."""

    def __init__(self, faces, vertices):
        self.out = [np.zeros((vertices, 3), np.float32), np.zeros(vertices, np.uint8), np.zeros(vertices, np.int32),
                    np.zeros(3 * faces, np.int32), np.zeros(3 * faces, np.int32)]

    def put(self, table):
        c = table.counts()
        assert c["corners"] <= len(self.out[3]) and c["vertex_slots"] <= len(self.out[0]), c
        N.check(N.load().bs_corner_table_export(table.h, *(x.ctypes.data for x in self.out)))
        return [np.array([c["faces"], c["vertices"], c["vertex_slots"]], np.int64), *self.out]


def _rough(case):
    """How much larger than the smooth shape a noisy one's surface may be."""
    if case.get("shape") == "icosphere":
        return 1.0 + 2.0 * case["noise"] * 2 ** case["subdiv"]
    return 1.3


def _volume(ctx, case, gen, second=False):
    v, f = _torus(case["nu"], case["nv"], 0.02, gen, second)
    f = f.int().contiguous()
    torch.cuda.synchronize()
    return _convert(ctx, v, f, _params(case["voxel"], case["band"], "fast"))


def prepare(case, seed):
    ctx, gen, kind = _context(), _gen(seed), case["kind"]
    s = dict(case=case, ctx=ctx)
    if kind == "remesh":
        v, f = _mesh(case, gen)
        most = int(5 * _rough(case) * 12.6 / case["voxel"] ** 2) + 4096
        s["table"] = _Table(2 * most, most)
        s["mesh"] = (v.cpu().numpy(), f.cpu().numpy().astype(np.uint32))
        s["remesher"] = (bs.VoxelRemesher(ctx).with_voxel_size(case["voxel"]).with_narrow_band_width(case["band"])
                         .with_meshing_method(case["method"]))
    elif kind == "convert":
        s["v"], s["f"] = _mesh(case, gen)
        s["leaves"] = _Leaves(_leaves(_rough(case) * 12.6, case["voxel"], case["band"]))
        s["params"] = _params(case["voxel"], case["band"], case["tree"])
    elif kind == "batch":
        meshes = _batch(case, gen)
        s["v"], s["f"] = torch.cat([m[0] for m in meshes]), torch.cat([m[1] for m in meshes])
        s["nv"] = np.array([len(m[0]) for m in meshes], np.uint64)
        s["nt"] = np.array([len(m[1]) for m in meshes], np.uint64)
        s["leaves"] = _Leaves(_batch_leaves(case, 4.0), volumes=len(meshes))
        s["params"] = (N.M2VParams * len(meshes))(*[_params(m[2], case["band"], "reference") for m in meshes])
    elif kind == "boolean":
        s["a"], s["b"] = _volume(ctx, case, gen), _volume(ctx, case, gen, True)
        s["leaves"] = _Leaves(_leaves(2.6 * 11.8, case["voxel"], case["band"]),
                              int(3.0 / (8 * case["voxel"]) ** 3) + 64)
    elif kind == "offset":
        s["volume"] = _volume(ctx, case, gen)
        s["leaves"] = _Leaves(_leaves(1.3 * 11.8, case["voxel"], 4 + abs(case["distance"]) / case["voxel"]))
    elif kind == "contour":
        s["volume"] = _volume(ctx, case, gen)
        s["soup"] = torch.zeros((int(6 * 11.8 / case["voxel"] ** 2) + 4096, 3, 3), dtype=torch.float32).pin_memory()
    elif kind == "points":
        v, f, s["points"] = _points_inputs(case, gen)
        s["tree"] = bs.WindingNumbers.from_mesh((v.cpu().numpy(), f.cpu().numpy()), order=case["order"], ctx=ctx,
                                                tree=case["tree"])
    else:
        s.update(_learned_inputs(case, gen))
    torch.cuda.synchronize()
    return s


def run(state):
    case, ctx, L = state["case"], state["ctx"], N.load()
    kind = case["kind"]
    if kind == "remesh":
        return state["table"].put(state["remesher"].remesh(state["mesh"]))
    if kind == "convert":
        state["leaves"].put(_convert(ctx, state["v"], state["f"], state["params"]))
        return state["leaves"].outputs()
    if kind == "batch":
        n = len(state["nv"])
        out = (C.c_void_p * n)()
        N.check(L.bs_mesh_to_volume_batch_device(ctx.h, n, state["v"].data_ptr(), state["nv"].ctypes.data,
                                                 state["f"].data_ptr(), state["nt"].ctypes.data, state["params"], out),
                ctx.h)
        for k in range(n):
            state["leaves"].put(bs.Volume(C.c_void_p(out[k]), ctx), k)
        return state["leaves"].outputs()
    if kind == "boolean":  # booleans consume their operands: the program keeps its own
        state["leaves"].put(getattr(state["a"].clone(), case["op"])(state["b"].clone()))
        return state["leaves"].outputs()
    if kind == "offset":
        state["leaves"].put(state["volume"].clone().offset(case["distance"]))
        return state["leaves"].outputs()
    if kind == "contour":
        vol = state["volume"].clone()  # a volume keeps its last extraction
        fn = {"dc": L.bs_dual_contour, "qef": L.bs_dual_contour_qef, "mc": L.bs_marching_cubes}[case["mesher"]]
        n = C.c_uint64()
        N.check(fn(ctx.h, vol.h, case["voxel"], state["soup"].data_ptr(), len(state["soup"]), C.byref(n)), ctx.h)
        assert n.value <= len(state["soup"]), n.value
        return [n.value, state["soup"]]
    if kind == "points":
        p = state["points"]
        out = torch.empty(len(p), dtype=torch.float32, device="cuda")
        N.check(L.bs_winding_numbers_approximate(ctx.h, state["tree"].h, p.data_ptr(), len(p), 2.0, out.data_ptr()),
                ctx.h)
        return out
    net = C.c_void_p()
    params, loss = np.empty(len(state["params"]), np.float32), np.empty(case["epochs"], np.float32)
    N.check(L.bs_mlp_create(ctx.h, state["centre"].ctypes.data, state["scale"], state["freq"].ctypes.data,
                            state["params"].ctypes.data, C.byref(net)), ctx.h)
    try:
        N.check(L.bs_mlp_train(ctx.h, net, state["samples"].data_ptr(), state["targets"].data_ptr(),
                               len(state["samples"]), case["batch"], case["epochs"], 3e-3, 1e-4, loss.ctypes.data),
                ctx.h)
        N.check(L.bs_mlp_get_params(ctx.h, net, params.ctypes.data), ctx.h)
        out = torch.empty(len(state["points"]), dtype=torch.float32, device="cuda")
        N.check(L.bs_mlp_predict(ctx.h, net, state["points"].data_ptr(), len(out), out.data_ptr()), ctx.h)
    finally:
        L.bs_mlp_free(net)
    return [params, loss, out]


def _points_inputs(case, gen):
    """A mesh with holes and query points uniform in its box padded by 10 %."""
    v, f = _mesh(dict(shape="soup", subdiv=case["subdiv"], noise=0.1), gen)
    lo, hi = v.min(dim=0).values, v.max(dim=0).values
    p = lo - 0.1 * (hi - lo) + 1.2 * (hi - lo) * torch.rand(case["points"], 3, generator=gen, device="cuda")
    return v, f, p.contiguous()


def _learned_inputs(case, gen):
    """Samples with inside / outside targets of a noisy ball, and a fresh network's parameters."""
    def ball(n):
        p = 2.4 * torch.rand(n, 3, generator=gen, device="cuda") - 1.2
        r = 1.0 + 0.1 * torch.sin(5 * p[:, 0]) * torch.cos(4 * p[:, 1])
        return p.contiguous(), torch.sigmoid(40 * (r - p.norm(dim=1))).contiguous()

    samples, targets = ball(case["samples"])
    rng = np.random.default_rng(int(torch.randint(1 << 30, (1,), generator=gen, device="cuda")))
    dirs = rng.normal(size=(32, 3))
    freq = dirs / np.linalg.norm(dirs, axis=1, keepdims=True) * np.exp(np.linspace(0.0, np.log(16.0), 32))[:, None]
    params = np.zeros(N.load().bs_mlp_num_params(), np.float32)
    lim = math.sqrt(6.0 / 128.0)
    params[0:4096] = rng.uniform(-lim, lim, 4096)
    params[4160:8256] = rng.uniform(-lim, lim, 4096)
    params[8320:8384] = rng.uniform(-0.1, 0.1, 64)
    params[8384] = float(targets.mean())
    return dict(samples=samples, targets=targets, points=ball(case["points"])[0], params=params,
                freq=np.ascontiguousarray(freq, np.float32), centre=np.zeros(3, np.float32), scale=0.75)


# ------------------------------------------------------------------- work ----
def _band(area, h, band):
    """Band voxels of a surface: the pieces' boxes reach band voxels and about three more on either side."""
    return area * (2 * band + 6) / h ** 2


def _leaves(area, h, band):
    """Leaves that a band fills, most of the outer ones in part."""
    return int(1.2 * area * (2 * band + 14) / h ** 2 / 512) + 200


def _volume_bytes(area, h, band):
    return _leaves(area, h, band) * 2124  # values, mask and origin


def _batch_leaves(case, rough):
    return sum(_leaves(rough * 12.6, (2.6 if k % 2 else 2.0) / res, case["band"]) for k, _, res in _batch_sizes(case))


def work(case):
    """Each input read and each output written once; one closest point (84 FLOP) per band voxel, one solid angle
    (60 FLOP) per query point, the network's products."""
    kind = case["kind"]
    if kind in ("remesh", "convert"):
        if case["shape"] == "torus":
            tri, area = 2 * case["nu"] * case["nv"], 11.8
        else:
            tri, area = 20 * 4 ** case["subdiv"], 12.6
        mesh = 18 * tri  # half a vertex of 12 bytes and 12 bytes of indices
        band = _band(area, case["voxel"], case["band"])
        if kind == "remesh":  # two triangles a surface voxel: 3 corners of 8 bytes, half a vertex of 17 bytes
            return dict(bytes=mesh + 2 * area / case["voxel"] ** 2 * (24 + 9), flops=84 * band)
        return dict(bytes=mesh + _volume_bytes(area, case["voxel"], case["band"]), flops=84 * band)
    if kind == "batch":
        b = fl = 0.0
        for k, tri, res in _batch_sizes(case):
            area, h = (11.8, 2.6 / res) if k % 2 else (12.6, 2.0 / res)
            b += 18 * tri + _volume_bytes(area, h, case["band"])
            fl += 84 * _band(area, h, case["band"])
        return dict(bytes=b, flops=fl)
    if kind in ("boolean", "offset", "contour"):
        vol = _volume_bytes(11.8, case["voxel"], case["band"])
        if kind == "boolean":
            return dict(bytes=4 * vol, flops=0)
        if kind == "offset":
            return dict(bytes=2 * vol, flops=0)
        return dict(bytes=vol + 2 * 11.8 / case["voxel"] ** 2 * 36, flops=0)
    if kind == "points":
        return dict(bytes=16 * case["points"] + 16 * 20 * 4 ** case["subdiv"], flops=60 * case["points"])
    steps = case["samples"] // case["batch"] * case["batch"] * case["epochs"]
    return dict(bytes=16 * (steps + case["points"]), flops=2 * 8256 * (3 * steps + case["points"]))


# ------------------------------------------------------------------ exact ----
def exact(case, seed):
    """The outputs in 64 bits: band distances and signs of small conversions, winding numbers by direct summation, the
    trained network.  Tables, soups and swept volumes have no value that does not follow the path's own steps."""
    gen = _gen(seed)
    if case["kind"] == "convert":
        tri = 2 * case["nu"] * case["nv"] if case["shape"] == "torus" else 20 * 4 ** case["subdiv"]
        if _band(12.6, case["voxel"], case["band"]) * max(tri, 2000) > 5e9:
            return None
        v, f = _mesh(case, gen)
        leaves = _exact_volume(v, f.long(), case["voxel"], case["band"])
        values = torch.zeros((_leaves(_rough(case) * 12.6, case["voxel"], case["band"]), 512), dtype=torch.float64)
        values[:len(leaves)] = leaves.cpu()
        return [None, None, values, None]
    if case["kind"] == "points" and case["points"] * 18 * 4 ** case["subdiv"] < 3.5e10:
        v, f, p = _points_inputs(case, gen)
        return _exact_winding(v.double()[f.long()], p.double())
    if case["kind"] == "learned":
        return _exact_learned(case, _learned_inputs(case, gen))
    return None


def _exact_winding(tri, p):
    out = torch.empty(len(p), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 26) // len(tri))
    for k in range(0, len(p), step):
        q = p[k:k + step]
        # corner by corner in components, so that no (points, triangles, 3) array is made
        d = [[tri[None, :, c, x] - q[:, None, x] for x in range(3)] for c in range(3)]
        n = [(e[0] * e[0] + e[1] * e[1] + e[2] * e[2]).sqrt_() for e in d]
        (a, b, c), (la, lb, lc) = d, n
        num = (a[0] * (b[1] * c[2] - b[2] * c[1]) + a[1] * (b[2] * c[0] - b[0] * c[2])
               + a[2] * (b[0] * c[1] - b[1] * c[0]))

        def dot(x, y):
            return x[0] * y[0] + x[1] * y[1] + x[2] * y[2]

        den = la * lb * lc + dot(a, b) * lc + dot(a, c) * lb + dot(b, c) * la
        out[k:k + step] = torch.atan2(num, den).sum(dim=1) / (2 * math.pi)
    return out


def _subdivided(t, h):
    """Triangles (n, 3, 3) cut into floor(longest side / h)^2 pieces each (one below 2)."""
    side = torch.stack([t[:, 1] - t[:, 0], t[:, 2] - t[:, 0], t[:, 2] - t[:, 1]]).norm(dim=2).max(dim=0).values
    n = (side / h).floor().long().clamp_min(1)
    out = [t[n < 2]]
    for m in torch.unique(n[n >= 2]).tolist():
        p = t[n == m]
        s1, s2 = ((p[:, 1] - p[:, 0]) / m)[:, None], ((p[:, 2] - p[:, 1]) / m)[:, None]
        at = lambda r, k: p[:, :1] + r * s1 + k * s2  # noqa: E731
        for r in range(m):
            for k in range(r + 1):
                out.append(torch.cat([at(r, k), at(r + 1, k), at(r + 1, k + 1)], 1))
                if k < r:
                    out.append(torch.cat([at(r, k), at(r + 1, k + 1), at(r, k + 1)], 1))
    return torch.cat(out)


def _distance(p, a, b, c):
    """Point-triangle distance: the plane's inside case, else the nearest of the three sides."""
    def side(u, v):
        e = v - u
        x = ((p - u) * e).sum(1) / (e * e).sum(1)
        return (u + x.clamp(0, 1)[:, None] * e - p).norm(dim=1)

    n = torch.linalg.cross(b - a, c - a)
    inside = torch.ones(len(p), dtype=torch.bool, device="cuda")
    for u, v in ((a, b), (b, c), (c, a)):
        inside &= (torch.linalg.cross(v - u, p - u) * n).sum(1) >= 0
    plane = ((p - a) * n).sum(1).abs() / n.norm(dim=1)
    return torch.where(inside, plane, torch.minimum(torch.minimum(side(a, b), side(b, c)), side(c, a)))


def _exact_volume(v, f, h, band):
    """Values (leaves, 512) of the narrow-band volume: for every grid point the distance to the nearest piece whose
    widened box holds it, negative where the winding number reaches 0.2, 0 where no box does."""
    h32 = torch.tensor(h, dtype=torch.float32, device="cuda")
    t = _subdivided(v.double()[f], float(h32))
    inv = torch.ones((), device="cuda") / h32
    lo = (t.min(dim=1).values.float() * inv).floor().long() - band
    hi = (t.max(dim=1).values.float() * inv).ceil().long() + band
    flat = ((hi == lo).any(dim=1))[:, None].long()
    lo, hi = lo - flat, hi + flat
    base = torch.div(lo.min(dim=0).values, 8, rounding_mode="floor") * 8
    dims = torch.div(hi.max(dim=0).values - base, 8, rounding_mode="floor") * 8 + 8
    grid = torch.full((int(dims.prod()),), math.inf, dtype=torch.float64, device="cuda")
    size = hi - lo + 1
    count = size.prod(dim=1)
    ends = count.cumsum(0)
    start = 0
    while start < len(t):
        stop = max(start + 1, int(torch.searchsorted(ends, ends[start] - count[start] + (1 << 22))))
        k = torch.repeat_interleave(torch.arange(start, stop, device="cuda"), count[start:stop])
        j = torch.arange(len(k), device="cuda") - (ends[k] - count[k] - (ends[start] - count[start]))
        s = size[k]
        g = lo[k] + torch.stack([j // (s[:, 1] * s[:, 2]), j // s[:, 2] % s[:, 1], j % s[:, 2]], 1)
        p = (g.float() * h32).double()
        at = ((g - base) * torch.stack([dims[1] * dims[2], dims[2], dims[2] * 0 + 1])).sum(1)
        grid.scatter_reduce_(0, at, _distance(p, t[k, 0], t[k, 1], t[k, 2]), "amin")
        start = stop
    act = torch.nonzero(torch.isfinite(grid)).squeeze(1)
    g = base + torch.stack([act // (dims[1] * dims[2]), act // dims[2] % dims[1], act % dims[2]], 1)
    wn = _exact_winding(v.double()[f], (g.float() * h32).double())
    grid[act] = torch.where(wn < 0.2, grid[act], -grid[act])
    d = (dims // 8).tolist()
    leaves = grid.reshape(d[0], 8, d[1], 8, d[2], 8).permute(0, 2, 4, 1, 3, 5).reshape(-1, 512)
    leaves = leaves[torch.isfinite(leaves).any(dim=1)]
    return torch.where(torch.isfinite(leaves), leaves, torch.zeros_like(leaves))


def _exact_learned(case, s):
    freq = torch.from_numpy(s["freq"]).cuda().double()
    theta = torch.from_numpy(s["params"]).cuda().double().requires_grad_(True)

    def predict(points):
        x = points.double() * s["scale"] @ freq.T * math.pi
        z = torch.cat([torch.sin(x), torch.cos(x)], 1)
        z = torch.nn.functional.silu(z @ theta[0:4096].reshape(64, 64) + theta[4096:4160])
        z = torch.nn.functional.silu(z @ theta[4160:8256].reshape(64, 64) + theta[8256:8320])
        return z @ theta[8320:8384] + theta[8384]

    opt = torch.optim.Adam([theta], lr=3e-3)
    per, batch = case["samples"] // case["batch"], case["batch"]
    loss = torch.zeros(case["epochs"], dtype=torch.float64, device="cuda")
    for k in range(per * case["epochs"]):
        opt.param_groups[0]["lr"] = 1e-4 + 0.5 * (3e-3 - 1e-4) * (1 + math.cos(math.pi * k / (per * case["epochs"])))
        at = slice(k % per * batch, (k % per + 1) * batch)
        opt.zero_grad()
        e = (predict(s["samples"][at]) - s["targets"][at].double()).square().mean()
        e.backward()
        opt.step()
        loss[k // per] += e.detach() / per
    with torch.no_grad():
        return [theta.detach(), loss, torch.cat([predict(q) for q in s["points"].split(1 << 18)])]

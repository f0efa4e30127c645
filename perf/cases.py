"""The work that programs have this library do, as a list of timed cases.

Each case is one pass through the public entry points: spectral (RSB),
coordinate (RCB) and inertial (RIB) partitioning from host or device arrays,
gencon's vertex numbering, the batched Fiedler solve, the partition report and
one training step of the warm-start network.  The meshes are seeded and made
on the GPU, so that preparing a case costs little beside running it:

  box    structured hexes (nx, ny, nz) or quads (nx, ny) on the unit box, the
         interior vertices jittered by +-jitter h (0: an exact box mesh, whose
         centroids share coordinates, as generators of box meshes write them)
  pipe   hex annular cylinder (around, across, along), jittered
  annulus  quads around a circle, a seeded sinusoidal radial perturbation

with the elements in lattice order, from a seeded first element on, or
shuffled (meshes of unstructured generators have no spatial order).
"""
import ctypes
import math
import os

import numpy as np
import torch

import parrsb_gb300 as P
from parrsb_gb300 import warm

QUAD = ((0, 0), (1, 0), (1, 1), (0, 1))
HEX = ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))

# The library's two working methods.  "default": FP64 vectors, the reference's
# start vector and stopping rule.  "mixed": FP32 vectors on exact integer
# weights, the geometric start, restarts until the residual is below rsb_tol
# (the benchmark's method).  A program sets them in its environment.
METHODS = {"default": {},
           "mixed": {"PARRSB_GPU_FP32": "1", "PARRSB_GPU_RESID_STOP": "1", "PARRSB_GPU_START": "2"}}


def listed():
    return [
        # The first mesh of a user, a test or a coupling code that partitions
        # small patches: 16^3 hexes to 8 ranks from host arrays.
        {"name": "rsb-hex-small", "kind": "rsb", "api": "host", "mesh": "box", "dims": "16x16x16",
         "jitter": 0.1, "order": "lattice", "nparts": 8, "method": "default"},
        # A workstation-size unstructured mesh, odd sizes, no spatial order,
        # to an odd number of ranks; the program prints the partition report.
        {"name": "rsb-hex-ragged-report", "kind": "rsb", "api": "host", "mesh": "box",
         "dims": "61x37x29", "jitter": 0.1, "order": "shuffled", "nparts": 45,
         "method": "default", "report": True},
        # A production pipe mesh in the library's default precision.
        {"name": "rsb-pipe", "kind": "rsb", "api": "device", "mesh": "pipe", "dims": "128x64x128",
         "jitter": 0.05, "order": "lattice", "nparts": 256, "method": "default"},
        # The largest: 8.4M hexes to 1024 ranks, the benchmark's workload.
        {"name": "rsb-hex-large", "kind": "rsb", "api": "device", "mesh": "box",
         "dims": "256x256x128", "jitter": 0.1, "order": "lattice", "nparts": 1024,
         "method": "mixed"},
        # A 2D multi-material box mesh: tagged partitioning, disconnected
        # parts repaired, exact coordinates (ties).
        {"name": "rsb-quad-tagged", "kind": "tagged", "dims": "301x203", "jitter": 0.0,
         "ntags": 3, "nparts": 24, "repair": 1},
        # RCB inside a fixed-memory solver loop: a small patch, no allocation.
        {"name": "rcb-patch", "kind": "noalloc", "mesh": "box", "dims": "13x15x17", "jitter": 0.1,
         "order": "lattice", "nparts": 6},
        # Fast partition of the large mesh by coordinates.
        {"name": "rcb-hex-large", "kind": "geom", "partitioner": 1, "mesh": "box",
         "dims": "256x256x128", "jitter": 0.1, "order": "lattice", "nparts": 1024},
        # Inertial bisection of the 2D annulus.
        {"name": "rib-annulus", "kind": "geom", "partitioner": 2, "mesh": "annulus",
         "dims": "512x512", "jitter": 0.0, "order": "lattice", "nparts": 1024},
        # Connectivity of a mesh file that holds corner coordinates only.
        {"name": "gencon-hex", "kind": "gencon", "api": "device", "dims": "128x128x64",
         "jitter": 0.1, "order": "lattice", "periodic": False},
        # The same for a small 2D periodic mesh from host arrays.
        {"name": "gencon-quad-periodic", "kind": "gencon", "api": "host", "dims": "173x97",
         "jitter": 0.1, "order": "lattice", "periodic": True},
        # Fiedler vectors of many uneven pieces at once (the batched solve).
        {"name": "fiedler-pieces", "kind": "fiedler", "count": 256, "smin": 200, "smax": 20000,
         "shapes": 1, "delete": 0.05, "method": "mixed"},
        # One training step of the warm-start network: forward, loss, backward.
        {"name": "warm-train-step", "kind": "warm", "count": 24, "smin": 1000, "smax": 64000,
         "shapes": 2},
    ]


def _log(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def _sides(rng, n, d, aspect):
    """d side lengths of about n elements, at least 2, uneven up to `aspect`."""
    a = [aspect ** rng.random() for _ in range(d)]
    s = (n / math.prod(a)) ** (1.0 / d)
    return [max(2, int(round(x * s))) for x in a]


def _text(dims):
    return "x".join(str(int(x)) for x in dims)


def draw(rng):
    kind = rng.choice(["rsb", "rsb", "rsb", "tagged", "noalloc", "geom", "geom", "gencon",
                       "gencon", "fiedler", "warm"])
    order = rng.choice(["lattice", "shuffled"])
    if kind == "rsb":
        method = rng.choice(["default", "mixed"])
        d = _sides(rng, _log(rng, 1000, 200000 if method == "default" else 4000000), 3, 3.0)
        n = math.prod(d)
        mesh = rng.choice(["box", "box", "pipe"])
        if mesh == "pipe":
            d = [max(8, d[0]), d[1], d[2]]
        return {"kind": "rsb", "api": rng.choice(["host", "device"]), "mesh": mesh,
                "dims": _text(d), "jitter": rng.choice([0.05, 0.1]), "order": order,
                "nparts": int(max(2, min(1024, _log(rng, 2, n / 400.0)))), "method": method,
                "report": n < 300000 and rng.random() < 0.5}
    if kind == "tagged":
        ntags = rng.randint(2, 4)
        d = _sides(rng, _log(rng, 2000, 120000), 2, 2.0)
        return {"kind": "tagged", "dims": _text(d), "jitter": rng.choice([0.0, 0.1]),
                "ntags": ntags, "nparts": ntags * rng.randint(2, 12), "repair": rng.randint(0, 1)}
    if kind == "noalloc":
        d = _sides(rng, _log(rng, 100, 7000), rng.choice([2, 3]), 2.0)
        return {"kind": "noalloc", "mesh": "box", "dims": _text(d),
                "jitter": rng.choice([0.0, 0.1]), "order": order, "nparts": rng.randint(2, 64)}
    if kind == "geom":
        part = rng.choice([1, 1, 2])
        dim = rng.choice([2, 3])
        d = _sides(rng, _log(rng, 1000, 6000000 if part == 1 else 400000), dim, 3.0)
        mesh = rng.choice(["box", "annulus" if dim == 2 else "pipe"])
        if mesh != "box":
            d[0] = max(8, d[0])
        return {"kind": "geom", "partitioner": part, "mesh": mesh, "dims": _text(d),
                "jitter": rng.choice([0.0, 0.1]), "order": order,
                "nparts": int(_log(rng, 2, min(1024, math.prod(d) / 50.0)))}
    if kind == "gencon":
        dim = rng.choice([2, 3])
        api = rng.choice(["host", "device"])
        d = _sides(rng, _log(rng, 500, 900000 if api == "device" else 150000), dim, 2.0)
        return {"kind": "gencon", "api": api, "dims": _text(d),
                "jitter": rng.choice([0.0, 0.1]), "order": order,
                "periodic": api == "host" and rng.random() < 0.5}
    if kind == "fiedler":
        return {"kind": "fiedler", "count": int(_log(rng, 4, 256)), "smin": 200,
                "smax": int(_log(rng, 1000, 20000)), "shapes": rng.randint(1, 10 ** 6),
                "delete": rng.choice([0.02, 0.05]), "method": rng.choice(["default", "mixed"])}
    return {"kind": "warm", "count": rng.randint(2, 24), "smin": 1000,
            "smax": int(_log(rng, 4000, 64000)), "shapes": rng.randint(1, 10 ** 6)}


# ---------------------------------------------------------------------------
# Meshes
# ---------------------------------------------------------------------------
def _dims(text):
    return [int(x) for x in text.split("x")]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFFFFFF)


def _lattice(dims):
    """Element lattice corners (nel, nv, ndim), the first index fastest."""
    r = [torch.arange(n, device="cuda") for n in reversed(dims)]
    base = torch.stack([x.reshape(-1) for x in reversed(torch.meshgrid(*r, indexing="ij"))], 1)
    off = torch.tensor(QUAD if len(dims) == 2 else HEX, device="cuda")
    return base[:, None, :] + off[None]


def _vertex(c, dims, wrap=False):
    nx = dims[0] if wrap else dims[0] + 1
    i = c[..., 0] % nx if wrap else c[..., 0]
    v = i + nx * c[..., 1]
    if len(dims) == 3:
        v = v + nx * (dims[1] + 1) * c[..., 2]
    return v


def _jittered(c, dims, jitter, gen, wrap=False):
    """Lattice coordinates (float64) of every corner, interior vertices moved
    by +-jitter of a lattice step; every copy of a vertex moves alike."""
    nx = dims[0] if wrap else dims[0] + 1
    nvert = nx * math.prod(n + 1 for n in dims[1:])
    x = c.to(torch.float64)
    if wrap:
        x[..., 0] = x[..., 0] % nx
    if jitter:
        v = _vertex(c, dims, wrap)
        inside = torch.ones(v.shape, dtype=torch.bool, device="cuda")
        for d, n in enumerate(dims):
            if d > 0 or not wrap:
                inside &= (c[..., d] > 0) & (c[..., d] < n)
        for d in range(len(dims)):
            j = torch.rand(nvert, dtype=torch.float64, device="cuda", generator=gen) * 2.0 - 1.0
            x[..., d] += torch.where(inside, j[v] * jitter, torch.zeros_like(x[..., d]))
    return x


def _mesh(kind, dims, jitter, order, seed, need_vtx=True):
    """(vtx (nel, nv) int64 or None, xyz (nel, nv, ndim) float64, the lattice
    index of every element) on the GPU."""
    gen = _generator(seed)
    c = _lattice(dims)
    wrap = kind != "box"
    vtx = _vertex(c, dims, wrap) + 1 if need_vtx else None
    if kind == "annulus":  # r in [1, 2], a perturbation that vanishes on both circles
        a = torch.rand(2, dtype=torch.float64, device="cuda", generator=gen)
        mode = torch.floor(3.0 + 6.0 * a[0])
        x = c.to(torch.float64)
        th = (x[..., 0] % dims[0]) * (2.0 * math.pi / dims[0])
        s = x[..., 1] / dims[1]
        r = 1.0 + s + 0.02 * torch.sin(mode * th + 2.0 * math.pi * a[1]) * torch.sin(math.pi * s)
        xyz = torch.stack([r * torch.cos(th), r * torch.sin(th)], -1)
    else:
        x = _jittered(c, dims, jitter, gen, wrap)
        if kind == "pipe":
            th = x[..., 0] * (2.0 * math.pi / dims[0])
            r = 1.0 + x[..., 1] / dims[1]
            xyz = torch.stack([r * torch.cos(th), r * torch.sin(th), x[..., 2] * (4.0 / dims[2])],
                              -1)
        else:
            xyz = x / torch.tensor(dims, dtype=torch.float64, device="cuda")
    n = len(xyz)
    if order == "shuffled":
        at = torch.randperm(n, device="cuda", generator=gen)
    else:
        at = (torch.arange(n, device="cuda") +
              torch.randint(n, (1,), device="cuda", generator=gen)) % n
    return (None if vtx is None else vtx[at].contiguous()), xyz[at].contiguous(), at


def _shapes(case, aspect):
    """Side lengths of the case's pieces (the same for every seed of a case)."""
    rng = np.random.Generator(np.random.PCG64(case["shapes"]))
    out = []
    for _ in range(case["count"]):
        n = math.exp(rng.uniform(math.log(case["smin"]), math.log(case["smax"])))
        a = np.exp(rng.uniform(0.0, math.log(aspect), 3))
        a = np.sort(a)[::-1]
        a[0] = max(a[0], 1.3 * a[1])  # a longest side: a separated Fiedler value
        d = np.maximum(2, np.round(a * (n / np.prod(a)) ** (1.0 / 3.0))).astype(int)
        out.append([int(x) for x in d[rng.permutation(3)]])
    return out


def _pieces(shapes, seed, jitter, delete=0.0):
    """Disjoint jittered boxes of unit-size elements, concatenated: (vtx, xyz,
    group) on the GPU, a fraction `delete` of the elements missing."""
    vs, xs, gs, off = [], [], [], 0
    gen = _generator(seed)
    for g, d in enumerate(shapes):
        c = _lattice(d)
        v = _vertex(c, d) + 1 + off
        x = _jittered(c, d, jitter, gen) / float(max(d))
        off += math.prod(n + 1 for n in d)
        if delete:
            n = len(v) - int(delete * len(v))  # as many for every seed
            keep = torch.randperm(len(v), device="cuda", generator=gen)[:n].sort().values
            v, x = v[keep], x[keep]
        vs.append(v)
        xs.append(x)
        gs.append(torch.full((len(v),), g, dtype=torch.int32, device="cuda"))
    return torch.cat(vs).contiguous(), torch.cat(xs).contiguous(), torch.cat(gs)


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def _use(method):
    """The method's settings in this process's environment (and no messages)."""
    os.environ.setdefault("PARRSB_VERBOSE_LEVEL", "0")
    want = METHODS[method]
    for k in METHODS["mixed"]:
        if os.environ.get(k) != want.get(k):
            if k in want:
                os.environ[k] = want[k]
            else:
                del os.environ[k]


def _ptr(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def prepare(case, seed):
    P.library()
    kind = case["kind"]
    s = {"kind": kind, "method": case.get("method", "default"), "case": case}
    if kind == "rsb":
        vtx, xyz, _ = _mesh(case["mesh"], _dims(case["dims"]), case["jitter"], case["order"], seed)
        if case["api"] == "host":
            s["vtx"], s["xyz"] = vtx.cpu().numpy(), xyz.cpu().numpy()
        else:
            s["vtx"], s["xyz"] = vtx, xyz
            s["part"] = torch.empty(len(vtx), dtype=torch.int32, device="cuda")
    elif kind == "tagged":
        dims = _dims(case["dims"])
        vtx, xyz, at = _mesh("box", dims, case["jitter"], "lattice", seed)
        # materials in vertical strips, their order from the seed
        col = at % dims[0]
        strip = (col * case["ntags"]) // dims[0]
        names = torch.randperm(case["ntags"], device="cuda", generator=_generator(seed + 1))
        s["vtx"], s["xyz"] = vtx.cpu().numpy(), xyz.cpu().numpy()
        s["tag"] = (names[strip] * 7 + 1).to(torch.int32).cpu().numpy()
    elif kind in ("noalloc", "geom"):
        _, s["xyz"], _ = _mesh(case["mesh"], _dims(case["dims"]), case["jitter"], case["order"],
                               seed, need_vtx=False)
        s["part"] = torch.empty(len(s["xyz"]), dtype=torch.int32, device="cuda")
        if kind == "noalloc":  # the set-up call that the entry point asks for
            P.library().parrsb_part_mesh_rcb_noalloc(None, None, 0, s["xyz"].shape[1], 1, None)
    elif kind == "gencon":
        dims = _dims(case["dims"])
        _, xyz, at = _mesh("box", dims, case["jitter"], case["order"], seed, need_vtx=False)
        if case["api"] == "host":
            s["xyz"] = xyz.cpu().numpy()
            # the two x sides are one face: (element, face, partner, face), 1-based
            where = torch.argsort(at).cpu().numpy() + 1
            lo, hi = where[::dims[0]], where[dims[0] - 1::dims[0]]
            s["periodic"] = (np.stack([lo, np.full_like(lo, 4), hi, np.full_like(lo, 2)], 1)
                             if case["periodic"] else None)
        else:
            s["xyz"] = xyz
            s["ids"] = torch.empty(xyz.shape[:2], dtype=torch.int64, device="cuda")
    elif kind == "fiedler":
        vtx, _, grp = _pieces(_shapes(case, 3.0), seed, 0.1, case["delete"])
        s["vtx"], s["grp"] = vtx.cpu().numpy(), grp.cpu().numpy()
    else:
        shapes = _shapes(case, 4.0)
        vtx, xyz, grp = _pieces(shapes, seed, 0.1)
        s["batch"] = warm.Batch(vtx.cpu().numpy(), xyz.cpu().numpy(), grp.cpu().numpy(),
                                len(shapes))
        s["label"] = _warm_label(shapes)
        s["params"] = _warm_params(seed)
        s["grad"] = torch.empty_like(s["params"])
    torch.cuda.synchronize()
    return s


def run(state):
    kind, case = state["kind"], state["case"]
    _use(state["method"])
    if kind == "rsb":
        if case["api"] == "host":
            part = P.part_mesh(state["vtx"], state["xyz"], case["nparts"])
        else:
            part = _part_device(state, 0, state["vtx"])
        if case.get("report"):
            vtx = state["vtx"] if case["api"] == "host" else state["vtx"].cpu().numpy()
            here = part if case["api"] == "host" else part.cpu().numpy()
            return [part, P.part_quality(here, vtx, case["nparts"])]
        return part
    if kind == "tagged":
        return P.part_mesh(state["vtx"], state["xyz"], case["nparts"], tag=state["tag"], tagged=1,
                           repair=case["repair"])
    if kind == "noalloc":
        xyz, part = state["xyz"], state["part"]
        rc = P.library().parrsb_part_mesh_rcb_noalloc(
            _ptr(part), _ptr(xyz), xyz.shape[0], xyz.shape[1], case["nparts"],
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != P.OK:
            raise P.ParrsbError(rc, "parrsb_part_mesh_rcb_noalloc")
        return part
    if kind == "geom":
        return _part_device(state, case["partitioner"], None)
    if kind == "gencon":
        if case["api"] == "host":
            return P.conn_mesh(state["xyz"], state["xyz"].shape[2], 0.2, state["periodic"])
        xyz, ids = state["xyz"], state["ids"]
        rc = P.library().parrsb_conn_mesh_device(_ptr(ids), _ptr(xyz), xyz.shape[0], xyz.shape[2],
                                                 0.2)
        if rc != P.OK:
            raise P.ParrsbError(rc, "parrsb_conn_mesh_device")
        return ids
    if kind == "fiedler":
        return list(P.fiedler_groups(state["vtx"], state["grp"], case["count"]))
    loss, pred = state["batch"].step(state["params"], state["label"], state["grad"],
                                     want_pred=True)
    return [loss, pred, state["grad"]]


def _part_device(state, partitioner, vtx):
    xyz, part = state["xyz"], state["part"]
    o = P.ParrsbOptions.make(partitioner=partitioner, verbose_level=0)
    rc = P.library().parrsb_part_mesh_device(_ptr(part), _ptr(vtx), _ptr(xyz), xyz.shape[0],
                                             xyz.shape[1], ctypes.byref(o),
                                             state["case"]["nparts"])
    if rc != P.OK:
        raise P.ParrsbError(rc, "parrsb_part_mesh_device")
    return part


def work(case):
    """Inputs read once and outputs written once.  The iterations of the
    spectral cases are not counted: how many there are is the method's."""
    kind = case["kind"]
    if kind in ("fiedler", "warm"):
        shapes = _shapes(case, 3.0 if kind == "fiedler" else 4.0)
        n = sum(math.prod(d) for d in shapes)
        if kind == "fiedler":  # ids and groups in, the vectors out
            n *= 1.0 - case["delete"]
            return {"bytes": n * (64 + 4 + 8), "flops": 0}
        # features, graph (26 neighbours), label, prediction; forward and
        # backward products of the three layers
        mac = n * (16 * 64 + 2 * 128 * 64)
        return {"bytes": n * (32 + 26 * 4 + 8 + 4), "flops": 2 * 3 * mac}
    dims = _dims(case["dims"])
    n, nd = math.prod(dims), len(dims)
    nv = 2 ** nd
    xyz, vtx = 8 * nv * nd, 8 * nv
    if kind == "gencon":
        return {"bytes": n * (xyz + vtx), "flops": n * nv * nd * 3 * nd}
    if kind in ("geom", "noalloc"):
        return {"bytes": n * (xyz + 4), "flops": n * nv * nd}
    return {"bytes": n * (xyz + vtx + 4 + (vtx + 4 if case.get("report") else 0)),
            "flops": n * nv * nd}


# ---------------------------------------------------------------------------
# 64-bit values.  Partitions and vertex ids are whole numbers.  A Fiedler
# vector is an iterate stopped at a tolerance and the report belongs to the
# partition, so neither has a value of its own.  The training step has one.
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] != "warm":
        return None
    return _warm_exact(case, seed)


HID = 64


def _warm_label(shapes):
    """The Fiedler vector of every piece: a half cosine along its longest
    side (the pieces have one), unit norm."""
    out = []
    for d in shapes:
        ax = max(range(3), key=lambda a: d[a])
        i = _lattice(d)[:, 0, ax].to(torch.float64)
        y = torch.cos(math.pi * (i + 0.5) / d[ax])
        out.append(y / y.norm())
    return torch.cat(out).contiguous()


def _warm_params(seed):
    """Network parameters early in training (He-scaled layers)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    parts = []
    for k in (16, 128, 128):
        parts += [rng.normal(0.0, math.sqrt(2.0 / k), k * HID), rng.normal(0.0, 0.02, HID)]
    parts += [rng.normal(0.0, 0.02, HID), rng.normal(0.0, 0.02, 1)]
    return torch.from_numpy(np.concatenate(parts).astype(np.float32)).cuda()


def _warm_exact(case, seed):
    shapes = _shapes(case, 4.0)
    _, xyz, grp = _pieces(shapes, seed, 0.1)
    label = _warm_label(shapes)
    p = _warm_params(seed).to(torch.float64)
    sizes, o = [16 * HID, HID, 128 * HID, HID, 128 * HID, HID, HID, 1], 0
    leaves = []
    for n in sizes:
        leaves.append(p[o:o + n].clone().requires_grad_(True))
        o += n
    W1, b1, W2, b2, W3, b3, wo, bo = leaves
    W1, W2, W3 = W1.view(16, HID), W2.view(128, HID), W3.view(128, HID)
    cent = xyz.mean(1)
    total, preds, o = 0.0, [], 0
    for d in shapes:
        n = math.prod(d)
        c, f = cent[o:o + n], label[o:o + n]
        o += n
        # centroids on the lattice (z, y, x), and the sums over the 26
        # neighbours (4 shared vertices across a face, 2 an edge, 1 a corner)
        grid = c.view(d[2], d[1], d[0], 3)

        def neighbours(h):
            g = h.reshape(d[2], d[1], d[0], -1)
            s = torch.zeros_like(g)
            for dz in (-1, 0, 1):
                for dy in (-1, 0, 1):
                    for dx in (-1, 0, 1):
                        k = abs(dx) + abs(dy) + abs(dz)
                        if k == 0:
                            continue
                        to, fr = [], []
                        for m, sh in ((d[2], dz), (d[1], dy), (d[0], dx)):
                            to.append(slice(max(0, -sh), m - max(0, sh)))
                            fr.append(slice(max(0, sh), m - max(0, -sh)))
                        add = torch.zeros_like(g)
                        add[tuple(to)] = g[tuple(fr)] * float(2 ** (3 - k))
                        s = s + add
            return s.reshape(n, -1)

        deg = neighbours(torch.ones(n, 1, dtype=torch.float64, device="cuda"))
        # element spacings: root mean square centroid difference over faces
        sq, cnt = torch.zeros(3, dtype=torch.float64, device="cuda"), 0
        for a in range(3):
            q = (grid.narrow(a, 1, grid.shape[a] - 1) -
                 grid.narrow(a, 0, grid.shape[a] - 1)).reshape(-1, 3)
            sq, cnt = sq + (q * q).sum(0), cnt + len(q)
        x = c / torch.sqrt(sq / cnt)
        x = x - x.mean(0)
        lam, V = torch.linalg.eigh(x.T @ x)
        lam, R = lam.flip(0), V.T.flip(0)
        if lam[0] - lam[1] <= 0.05 * lam[0]:  # no principal axis: the longest edge first
            ext = c.max(0).values - c.min(0).values
            ax = int(torch.argmax(ext))
            R = torch.eye(3, dtype=torch.float64, device="cuda")[
                [ax] + [a for a in range(3) if a != ax]]
            lam = (x[:, ax] ** 2).sum()[None]
        big = R.gather(1, R.abs().argmax(1, keepdim=True))
        R = torch.where(big < 0, -R, R)
        x = (x @ R.T) / torch.sqrt(3.0 * lam[0] / n)
        guess = -torch.sin(math.pi * x[:, :1] / 2.0)
        h = torch.cat([x, deg / 56.0, guess, torch.zeros_like(x)], 1)
        for W, b in ((W1, b1), (W2, b2), (W3, b3)):
            h = torch.relu(torch.cat([h, neighbours(h) / deg], 1) @ W + b)
        y = h @ wo + bo + guess[:, 0]
        yc, fc = y - y.mean(), f - f.mean()
        loss = (1.0 - (yc @ fc) ** 2 / ((yc @ yc) * (fc @ fc))) / len(shapes)
        loss.backward()
        total += float(loss)
        preds.append(y.detach())
    return [total, torch.cat(preds), torch.cat([q.grad for q in leaves])]

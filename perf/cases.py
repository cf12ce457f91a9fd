"""The work a user of isoext_gb300 has it do, as measurable cases.

Each case is one pass through the public entry points on inputs that are on
the GPU (or, for the served stream, one burst of requests to a server that is
up).  Dense grids run from a few thousand points, where the call's latency
counts, to 512^3; sparse grids from a 128^3 to a 1024^3 lattice.  The fields are
the repository's own workloads: a sphere, unions of spheres and boxes, the seeded
CSG with sharp edges, a sphere with random Fourier features, the smooth union
of 64 spheres in 8^3 bricks, and the mixed stream of MC and DC requests.

A case fixes the geometry (``geometry``); the seed fixes the field that has it
as its level set: the values' distances from the level are scaled by a smooth
positive factor, as in a learned field that is a distance only roughly.  So every
seed gives other values and other vertices, on the same crossed edges.
"""

from __future__ import annotations

import math

import numpy as np
import torch

BRICK = 8
# About the surface area of each field in units of (half the box's edge)^2, from
# which work() takes the sizes of the meshes.
AREA = {"sphere": 8.0, "union": 4.0, "csg": 4.5, "fourier": 4.7, "smoothmin": 12.6}


def listed():
    def dense(name, kind, shape, field, level=0.0, method="nagae", half=1.0):
        return {"name": name, "kind": kind, "nx": shape[0], "ny": shape[1], "nz": shape[2], "field": field,
                "level": level, "method": method, "half": half, "geometry": 1}

    return [
        # a preview or a unit test: the call's latency is everything
        dense("mc_32_union", "mc", (32, 32, 32), "union"),
        dense("dc_odd_41x57x48", "dc", (41, 57, 48), "union"),
        # the ordinary grid: 128^3, the reference's example workload
        dense("mc_128_sphere", "mc", (128, 128, 128), "sphere"),
        # an anisotropic ragged volume, a level off zero, the other table, a
        # box that is not [-1, 1]^3
        dense("mc_ragged_201x334x143_lorensen", "mc", (201, 334, 143), "fourier", 0.05, "lorensen", 1.7),
        # CAD-like shape with sharp edges, the reason for dual contouring
        dense("dc_256_csg", "dc", (256, 256, 256), "csg"),
        # the documented two-step flow: the crossings with their normals first
        # (users read or replace them), then dual contouring of them
        dense("dc_two_step_192_sphere", "its", (192, 192, 192), "sphere"),
        # the benchmark's volume
        dense("mc_512_sphere", "mc", (512, 512, 512), "sphere"),
        dense("dc_512_sphere", "dc", (512, 512, 512), "sphere"),
        # sparse grids: a small one through dual contouring, the 1024^3 band
        dense("sparse_dc_200_smoothmin", "sparse_dc", (200, 200, 200), "smoothmin"),
        dense("sparse_mc_1024_smoothmin", "sparse_mc", (1024, 1024, 1024), "smoothmin"),
        # one optimisation step's extraction, forward and backward, MC and DC
        {"name": "grad_8x256_fourier", "kind": "grad", "n": 256, "batch": 8, "field": "fourier", "geometry": 1},
        # a burst of mixed requests to the server
        {"name": "serve_burst_24", "kind": "serve", "requests": 24, "most": 256, "geometry": 1},
    ]


def draw(rng):
    kind = rng.choice(["mc", "mc", "mc", "dc", "dc", "its", "sparse_mc", "sparse_dc", "grad", "serve"])
    geometry = rng.randint(2, 999)
    if kind == "grad":
        return {"kind": kind, "geometry": geometry, "n": round(math.exp(rng.uniform(math.log(32), math.log(256)))),
                "batch": rng.randint(1, 8), "field": "fourier"}
    if kind == "serve":
        return {"kind": kind, "geometry": geometry, "requests": rng.randint(4, 24), "most": rng.choice([96, 128, 192, 256])}
    case = {"kind": kind, "geometry": geometry, "level": round(rng.choice([0.0, rng.uniform(-0.05, 0.05)]), 3),
            "method": rng.choice(["nagae", "lorensen"]) if kind in ("mc", "sparse_mc") else "nagae",
            "half": rng.choice([1.0, round(rng.uniform(0.5, 4.0), 2)])}
    if kind in ("sparse_mc", "sparse_dc"):
        n = round(math.exp(rng.uniform(math.log(128), math.log(1024 if kind == "sparse_mc" else 400))))
        case.update(nx=n, ny=max(100, n - rng.randint(0, 24)), nz=max(100, n - rng.randint(0, 24)), field="smoothmin")
    else:
        n = math.exp(rng.uniform(math.log(24), math.log(460)))
        nx, ny, nz = (max(16, min(512, round(n * math.exp(rng.uniform(-0.35, 0.35))))) for _ in range(3))
        case.update(nx=nx, ny=ny, nz=nz, field=rng.choice(["sphere", "union", "csg", "fourier"]))
    return case


# ---------------------------------------------------------------------------
# inputs

def _axes(shape, half, dtype=torch.float32, dev="cuda"):
    """Grid coordinates along each axis of the box [-half, half]^3."""
    out = []
    for n in shape:
        f = torch.arange(n, dtype=dtype, device=dev) / torch.full((1,), n - 1, dtype=dtype, device=dev)
        out.append(-half + f * (2.0 * half))
    return out


def _factor(seed, half):
    """The smooth positive factor of a seed's field."""
    g = np.random.default_rng([seed, 22])
    w, phi = (g.normal(0.0, 1.0, 3) / half).tolist(), float(g.uniform(0.0, 2 * np.pi))
    return lambda x, y, z: 1.0 + 0.05 * torch.sin(x * w[0] + y * w[1] + z * w[2] + phi)


def _field(name, geometry, half):
    """The named field of points given as three tensors that broadcast together."""
    g = np.random.default_rng([geometry, 20])

    def norm(x, y, z):
        return torch.sqrt(x * x + y * y + z * z)

    def box(x, y, z, h):
        qx, qy, qz = x.abs() - h[0], y.abs() - h[1], z.abs() - h[2]
        m = torch.maximum(qx, torch.maximum(qy, qz))
        return norm(qx.clamp(min=0), qy.clamp(min=0), qz.clamp(min=0)) + m.clamp(max=0)

    if name == "sphere":
        c, r = g.uniform(-0.05, 0.05, 3).tolist(), float(g.uniform(0.79, 0.81))
        unit = lambda x, y, z: norm(x - c[0], y - c[1], z - c[2]) - r  # noqa: E731
    elif name == "union":
        c, s, kind = g.uniform(-0.5, 0.5, (8, 3)).tolist(), g.uniform(0.15, 0.35, 8).tolist(), g.integers(0, 2, 8)

        def unit(x, y, z):
            d = None
            for k in range(8):
                p = (x - c[k][0], y - c[k][1], z - c[k][2])
                q = norm(*p) - s[k] if kind[k] == 0 else box(*p, (s[k], 0.8 * s[k], 0.6 * s[k]))
                d = q if d is None else torch.minimum(d, q)
            return d
    elif name == "csg":
        h, rs = g.uniform(0.3, 0.6, 3).tolist(), float(g.uniform(0.2, 0.4))
        big, small = float(g.uniform(0.3, 0.5)), float(g.uniform(0.05, 0.15))
        cb, cs, ct = (g.uniform(-0.3, 0.3, 3).tolist() for _ in range(3))

        def unit(x, y, z):
            d = torch.maximum(box(x - cb[0], y - cb[1], z - cb[2], h), rs - norm(x - cs[0], y - cs[1], z - cs[2]))
            tx, ty, tz = x - ct[0], y - ct[1], z - ct[2]
            ring = torch.sqrt(tx * tx + ty * ty) - big
            return torch.minimum(d, torch.sqrt(ring * ring + tz * tz) - small)
    elif name == "fourier":
        w, a = g.normal(0.0, 3.0, (32, 3)).tolist(), g.normal(0.0, 0.02, 32).tolist()
        phi = g.uniform(0.0, 2 * np.pi, 32).tolist()

        def unit(x, y, z):
            d = norm(x, y, z) - 0.6
            for k in range(32):
                d += a[k] * torch.sin(x * w[k][0] + y * w[k][1] + z * w[k][2] + phi[k])
            return d
    else:
        c, r = g.uniform(-0.7, 0.7, (64, 3)).tolist(), g.uniform(0.05, 0.25, 64).tolist()

        def unit(x, y, z):
            s = None
            for k in range(64):
                e = torch.exp((r[k] - norm(x - c[k][0], y - c[k][1], z - c[k][2])) / 0.05)
                s = e if s is None else s.add_(e)
            return -0.05 * torch.log(s)
    return lambda x, y, z: unit(x / half, y / half, z / half) * half


def _shape(case):
    return (case["nx"], case["ny"], case["nz"])


def _dense_values(case, seed):
    shape = _shape(case)
    x, y, z = _axes(shape, case["half"])
    at = (x[:, None, None], y[None, :, None], z[None, None, :])
    v = _field(case["field"], case["geometry"], case["half"])(*at)
    return _scaled(v, case, seed, at).contiguous()


def _scaled(v, case, seed, at):
    """level + (v - level) * factor.  A grid point nearer to the surface than 32
    bits tell from it is on it, and no other is nearer than 1e-4 of a cell: which
    vertices meet on a grid point, and so the mesh's size, is the same for every
    seed's field."""
    d = v - case["level"]
    h = 2.0 * case["half"] / (max(_shape(case)) - 1)
    d = torch.where(d.abs() < 1.5e-8 * case["half"], 0.0,
                    torch.where(d < 0, d.clamp(max=-1e-4 * h), d.clamp(min=1e-4 * h)))
    return case["level"] + d * _factor(seed, case["half"])(*at)


def _sparse_cells(case, seed):
    """Cells (ascending ids) and their 8 values: the bricks of BRICK^3 cells that
    have a lattice point within 2 h of the surface."""
    shape, dev, B = _shape(case), "cuda", BRICK
    ax = _axes(shape, case["half"])
    f = _field("smoothmin", case["geometry"], case["half"])
    nc = [n - 1 for n in shape]
    h = 2.0 * case["half"] / min(nc)
    nb = [(n + B - 1) // B for n in nc]
    bricks = torch.cartesian_prod(*(torch.arange(n, device=dev) for n in nb))
    mid = [ax[k][(bricks[:, k] * B + B // 2).clamp(max=nc[k])] for k in range(3)]
    near = 2.0 * h + 0.5 * B * h * 3 ** 0.5 + h
    bricks = bricks[(f(*mid) - case["level"]).abs() <= near]
    o = torch.arange(B + 1, device=dev)
    ids, vals = [], []
    for s in range(0, len(bricks), 8192):
        b = bricks[s:s + 8192]
        p = [ax[k][(b[:, k, None] * B + o).clamp(max=nc[k])] for k in range(3)]
        at = (p[0][:, :, None, None], p[1][:, None, :, None], p[2][:, None, None, :])
        v = f(*at)
        keep = (v - case["level"]).abs().amin(dim=(1, 2, 3)) < 2.0 * h
        b, v = b[keep], _scaled(v, case, seed, at)[keep]
        c = [b[:, k, None] * B + o[:B] for k in range(3)]
        i = (c[0][:, :, None, None] * nc[1] + c[1][:, None, :, None]) * nc[2] + c[2][:, None, None, :]
        ok = ((c[0] < nc[0])[:, :, None, None] & (c[1] < nc[1])[:, None, :, None] & (c[2] < nc[2])[:, None, None, :])
        cv = torch.stack([v[:, j >> 2:(j >> 2) + B, (j >> 1) & 1:((j >> 1) & 1) + B, j & 1:(j & 1) + B]
                          for j in range(8)], -1)
        ids.append(i[ok].int())
        vals.append(cv[ok])
    ids, order = torch.sort(torch.cat(ids))
    return ids, torch.cat(vals)[order].contiguous()


def _requests(case, seed):
    """A burst of the mixed stream: grid edge over the stream's sizes, 70 % MC,
    unions of 1..16 spheres and boxes; the seed swaps x and y in half of them."""
    g, turn = np.random.default_rng([case["geometry"], 21]), np.random.default_rng([seed, 23])
    sizes = [n for n in (64, 96, 128, 192, 256) if n <= case["most"]]
    out = []
    for _ in range(case["requests"]):
        k = int(g.integers(1, 17))
        prims = np.zeros((k, 7), np.float32)
        prims[:, 0] = g.integers(0, 2, k)
        prims[:, 1:4] = g.uniform(-0.5, 0.5, (k, 3))
        size = g.uniform(0.05, 0.4, (k, 1))
        prims[:, 4:7] = np.where(prims[:, :1] == 0, size, size * g.uniform(0.5, 1.0, (k, 3)))
        if turn.random() < 0.5:
            prims[:, [1, 2]] = prims[:, [2, 1]]
            box = prims[:, 0] == 1
            prims[np.ix_(box, [4, 5])] = prims[np.ix_(box, [5, 4])]
        out.append(("mc" if g.random() < 0.7 else "dc", int(g.choice(sizes)), prims))
    return out


_server = None


def _the_server():
    """The program's one server, up and warm for the stream's sizes."""
    global _server
    if _server is None:
        from isoext_gb300 import serve

        _server = serve.NativeServer(slots=8, budget_bytes=40 << 30, warm_sizes=(64, 96, 128, 192, 256), tune=False)
    return _server


def _grad_case(case, i):
    """Grid i of the batch as a dense case."""
    return {"nx": case["n"], "ny": case["n"], "nz": case["n"], "half": 1.0, "level": 0.0, "field": case["field"],
            "geometry": 1000 * case["geometry"] + i}


def prepare(case, seed):
    import isoext_gb300 as iso

    kind = case["kind"]
    state = {"case": case}
    if kind == "serve":
        from isoext_gb300 import serve

        state["server"] = _the_server()
        state["requests"] = [serve.Request(k, n, p, rid=i) for i, (k, n, p) in enumerate(_requests(case, seed))]
    elif kind == "grad":
        state["values"] = [_dense_values(_grad_case(case, i), seed).requires_grad_(True) for i in range(case["batch"])]
    else:
        box = ([-case["half"]] * 3, [case["half"]] * 3)
        if kind in ("sparse_mc", "sparse_dc"):
            grid = iso.SparseGrid(_shape(case), *box)
            ids, vals = _sparse_cells(case, seed)
            grid.add_cells(ids)
            grid.set_values(vals)
        else:
            grid = iso.UniformGrid(_shape(case), *box)
            grid.set_values(_dense_values(case, seed))
        state["grid"] = grid
    return state


def run(state):
    import isoext_gb300 as iso

    case = state["case"]
    kind = case["kind"]
    if kind in ("mc", "sparse_mc"):
        return iso.marching_cubes(state["grid"], level=case["level"], method=case["method"])
    if kind in ("dc", "sparse_dc"):
        return iso.dual_contouring(state["grid"], level=case["level"])
    if kind == "its":
        its = iso.get_intersection(state["grid"], level=case["level"], compute_normals=True)
        v, f = iso.dual_contouring(state["grid"], level=case["level"], intersection=its)
        return v, f, its.get_points(), its.get_normals()
    if kind == "grad":
        from isoext_gb300 import diff

        xs = state["values"]
        for x in xs:
            x.grad = None
        meshes = diff.marching_cubes_batch(xs) + diff.dual_contouring_batch(xs)
        loss = ((torch.cat([v for v, _ in meshes]).norm(dim=-1) - 1.0) ** 2).mean()
        loss.backward()
        return {"loss": loss.detach(), "grad": [x.grad for x in xs], "vertices": [v.detach() for v, _ in meshes],
                "faces": [f for _, f in meshes]}
    waiting = [state["server"].submit(r) for r in state["requests"]]
    meshes = [w.result() for w in waiting]
    return [(m.vertices, m.faces) for m in meshes]


# ---------------------------------------------------------------------------
# the least work of a pass

def _mesh_bytes(area, h2):
    v = 1.5 * area / h2  # crossed edges, and about as many active cells; two faces each
    return v, 12.0 * v + 24.0 * v


def work(case):
    kind = case["kind"]
    if kind == "serve":
        # every grid is evaluated in place; its mesh leaves the device
        nbytes = flops = 0.0
        for k, n, prims in _requests(case, 0):
            _, out = _mesh_bytes(2.5, (2.0 / (n - 1)) ** 2)
            nbytes += 8.0 * n ** 3 + out
            flops += 12.0 * len(prims) * n ** 3
        return {"bytes": nbytes, "flops": flops}
    if kind == "grad":
        n, b = case["n"], case["batch"]
        v, out = _mesh_bytes(AREA[case["field"]], (2.0 / (n - 1)) ** 2)
        # values read by both forwards at once, meshes written, vertex gradients
        # read, the grid gradient written
        return {"bytes": b * (8.0 * n ** 3 + 2 * (out + 12.0 * v)), "flops": b * v * 4000.0}
    shape = _shape(case)
    v, out = _mesh_bytes(AREA[case["field"]] * (0.97 if case["level"] else 1.0),
                         4.0 / (sum((n - 1) ** 2 for n in shape) / 3.0))
    flops = 1500.0 * v if kind in ("dc", "its", "sparse_dc") else 12.0 * v
    if kind == "its":
        out += 2 * 12.0 * 4.0 * v  # points and normals of about four crossings per cell
    if kind in ("sparse_mc", "sparse_dc"):
        # about 11.5 kept cells per vertex at 8^3 bricks within 2 h
        return {"bytes": 36.0 * 11.5 * v + out, "flops": flops}
    return {"bytes": 4.0 * shape[0] * shape[1] * shape[2] + out, "flops": flops}


# ---------------------------------------------------------------------------
# the results in 64 bits

# Corner j = 4 dx + 2 dy + dz; the 12 edges of a cell as corner pairs.
EDGES = ((0, 1), (1, 3), (2, 3), (0, 2), (4, 5), (5, 7), (6, 7), (4, 6), (0, 4), (1, 5), (3, 7), (2, 6))
CA = [a for a, _ in EDGES]
CB = [b for _, b in EDGES]


def _off(k):
    """Offsets (x, y, z) of the given corners."""
    k = torch.as_tensor(k, device="cuda")
    return torch.stack([k >> 2, (k >> 1) & 1, k & 1], -1)


def _below(v, level):
    return (v - torch.tensor(level, dtype=torch.float32, device=v.device)) < 0


def _first_of(keys):
    """Positions of the first occurrence of each key, ascending."""
    k, order = torch.sort(keys, stable=True)
    new = torch.ones_like(k, dtype=torch.bool)
    new[1:] = k[1:] != k[:-1]
    return torch.sort(order[new]).values


def _coords32(shape, half):
    """Grid coordinates as 32-bit arithmetic with fused multiply-adds gives them."""
    size, lo = float(np.float32(half) + np.float32(half)), float(np.float32(-half))
    out = []
    for n in shape:
        f = torch.arange(n, dtype=torch.float32, device="cuda") / torch.full((1,), n - 1.0, device="cuda")
        out.append((f.double() * size + lo).float())
    return out


def _weld_keys(v32, level, index, point_ids, edge_keys, case, shape):
    """A key per vertex under which the positions that are equal in 32 bits meet:
    its edge, or the grid point at its end that it rounds to.  v32, index,
    point_ids: the two ends' values, grid indices and point ids."""
    ax = _coords32(shape, case["half"])
    a, b = (torch.stack([ax[k][i[:, k]] for k in range(3)], -1) for i in index)
    t = ((torch.tensor(level, dtype=torch.float32, device=a.device) - v32[0]) / (v32[1] - v32[0]))[:, None]
    pos = ((1 - t).double() * a.double() + (t * b).double()).float()
    key = edge_keys.clone()
    for e, p in zip((a, b), point_ids):
        on = (pos == e).all(-1)
        key[on] = -1 - p[on]
    return key


def _exact_mc(v, case):
    """MC vertices [V, 3] of dense values v in edge order."""
    nx, ny, nz = v.shape
    ax = _axes(v.shape, case["half"], torch.float64)
    s = _below(v, case["level"])
    nw = (nz + 31) // 32
    parts = []
    for axis in range(3):
        a = s.narrow(axis, 0, v.shape[axis] - 1)
        b = s.narrow(axis, 1, v.shape[axis] - 1)
        i = (a != b).nonzero()
        order = (((i[:, 0] * ny + i[:, 1]) * nw + (i[:, 2] >> 5)) * 3 + axis) * 32 + (i[:, 2] & 31)
        j = i.clone()
        j[:, axis] += 1
        parts.append((order, i, j))
    order, i, j = (torch.cat(p) for p in zip(*parts))
    at = torch.argsort(order)
    order, i, j = order[at], i[at], j[at]
    pa = torch.stack([ax[k][i[:, k]] for k in range(3)], -1)
    pb = torch.stack([ax[k][j[:, k]] for k in range(3)], -1)
    pid = [(c[:, 0] * ny + c[:, 1]) * nz + c[:, 2] for c in (i, j)]
    v32 = [v.reshape(-1)[p] for p in pid]
    va, vb = (u.double() for u in v32)
    t = ((case["level"] - va) / (vb - va))[:, None]
    pos = (1 - t) * pa + t * pb
    return pos[_first_of(_weld_keys(v32, case["level"], (i, j), pid, order, case, v.shape))]


def _cells_of(v, level):
    """Active cells [A, 3] of dense values in id order."""
    s = _below(v, level)
    nx, ny, nz = v.shape
    some = torch.zeros((nx - 1, ny - 1, nz - 1), dtype=torch.bool, device=v.device)
    every = torch.ones_like(some)
    for k in range(8):
        c = s[k >> 2:nx - 1 + (k >> 2), (k >> 1) & 1:ny - 1 + ((k >> 1) & 1), k & 1:nz - 1 + (k & 1)]
        some |= c
        every &= c
    return (some & ~every).nonzero()


def _corner_values(v, cells):
    i = cells[:, None, :] + _off(range(8))
    return v.reshape(-1)[(i[..., 0] * v.shape[1] + i[..., 1]) * v.shape[2] + i[..., 2]]


def _crossings(cv32, cv, cells, case, shape):
    """Crossed edges [A, 12] of the cells and their points [A, 12, 3]."""
    ax = _axes(shape, case["half"], torch.float64)
    s = _below(cv32, case["level"])
    hit = s[:, CA] != s[:, CB]
    va, vb = cv[:, CA], cv[:, CB]
    t = torch.where(hit, (case["level"] - va) / torch.where(hit, vb - va, 1.0), 0.5)[..., None]
    ia, ib = cells[:, None, :] + _off(CA), cells[:, None, :] + _off(CB)
    pa = torch.stack([ax[k][ia[..., k]] for k in range(3)], -1)
    pb = torch.stack([ax[k][ib[..., k]] for k in range(3)], -1)
    return hit, (1 - t) * pa + t * pb, ia, ib


def _normals(cv, lo, hi, p):
    """Central differences of each cell's trilinear interpolant at its points."""
    size = (hi - lo)[:, None, :]
    t = ((p - lo[:, None, :]) / size).clamp(0.01, 0.99)

    def at(u):
        x, y, z = (u[..., k, None] for k in range(3))
        c = cv[:, None, :]
        c = c[..., 0::2] * (1 - z) + c[..., 1::2] * z
        c = c[..., 0::2] * (1 - y) + c[..., 1::2] * y
        return (c[..., 0::2] * (1 - x) + c[..., 1::2] * x)[..., 0]

    g = []
    for k in range(3):
        up, dn = t.clone(), t.clone()
        up[..., k] = (t[..., k] + 0.02).clamp(max=0.99)
        dn[..., k] = (t[..., k] - 0.02).clamp(min=0.01)
        g.append((at(up) - at(dn)) / ((up[..., k] - dn[..., k]) * size[..., k]))
    g = torch.stack(g, -1)
    return g / g.norm(dim=-1, keepdim=True).clamp(min=1e-30)


def _exact_dc(cv32, cv, cells, case, shape):
    """Dual vertices of the cells that faces use, welded, in cell order; and the
    crossings' points and normals."""
    ax = _axes(shape, case["half"], torch.float64)
    lo = torch.stack([ax[k][cells[:, k]] for k in range(3)], -1)
    hi = torch.stack([ax[k][cells[:, k] + 1] for k in range(3)], -1)
    hit, p, ia, _ = _crossings(cv32, cv, cells, case, shape)
    n = _normals(cv, lo, hi, p)
    w = hit.double()[..., None]
    nw = n * w
    m = torch.einsum("aei,aej->aij", nw, n) + 0.01 * torch.eye(3, dtype=torch.float64, device=cv.device)
    r = (nw * (n * p).sum(-1, keepdim=True)).sum(1) + 0.01 * (p * w).sum(1) / w.sum(1)
    x = torch.linalg.solve(m, r[..., None])[..., 0]
    x = torch.maximum(torch.minimum(x, hi), lo)
    # an edge has its quad when all four of its cells lie in the grid
    along = (_off(CB) - _off(CA)).bool()
    top = torch.tensor(shape, device=cv.device) - 2
    whole = (along | ((ia >= 1) & (ia <= top))).all(-1)
    used = (hit & whole).any(-1)
    xs = x[used]
    key = torch.unique(xs.detach().float(), dim=0, return_inverse=True)[1]
    return xs[_first_of(key)], p[hit], n[hit]


def _lattice_cells(ids, shape):
    nc1, nc2 = shape[1] - 1, shape[2] - 1
    i = ids.long()
    return torch.stack([i // (nc1 * nc2), (i // nc2) % nc1, i % nc2], -1)


def _exact_mesh(kind, v, case):
    if kind == "mc":
        return _exact_mc(v, case)
    cells = _cells_of(v, case["level"])
    cv = _corner_values(v, cells)
    return _exact_dc(cv, cv.double(), cells, case, v.shape)


def exact(case, seed):
    kind = case["kind"]
    if kind == "mc":
        return _exact_mesh("mc", _dense_values(case, seed), case), None
    if kind in ("dc", "its"):
        v, p, n = _exact_mesh("dc", _dense_values(case, seed), case)
        return (v, None, p, n) if kind == "its" else (v, None)
    if kind in ("sparse_mc", "sparse_dc"):
        ids, vals = _sparse_cells(case, seed)
        s = _below(vals, case["level"])
        crossed = s.any(-1) & ~s.all(-1)
        cells, cv = _lattice_cells(ids[crossed], _shape(case)), vals[crossed]
        del ids, vals, s
        if kind == "sparse_dc":
            return None  # which cells faces use depends on which are in the grid
        hit, pos, ia, ib = _crossings(cv, cv.double(), cells, case, _shape(case))
        ny, nz = case["ny"], case["nz"]
        pid = [((c[..., 0] * ny + c[..., 1]) * nz + c[..., 2])[hit] for c in (ia, ib)]
        axis = torch.tensor([2, 1, 2, 1, 2, 1, 2, 1, 0, 0, 0, 0], device="cuda").expand(len(cells), 12)[hit]
        keys = _weld_keys((cv[:, CA][hit], cv[:, CB][hit]), case["level"], (ia[hit], ib[hit]), pid, 3 * pid[0] + axis,
                          case, _shape(case))
        return pos[hit][_first_of(keys)], None
    if kind == "grad":
        return _exact_grad(case, seed)
    box = {"half": 1.0, "level": 0.0}
    out = []
    for k, n, prims in _requests(case, seed):
        v = _union_values(n, prims)
        r = _exact_mesh(k, v, box)
        out.append((r if k == "mc" else r[0], None))
    return out


def _union_values(n, prims):
    """Values of a request's union, each operation rounded to 32 bits on its own."""
    x, y, z = _axes((n, n, n), 1.0)
    d = None
    for p in torch.from_numpy(prims):
        q = [a - c for a, c in zip((x[:, None, None], y[None, :, None], z[None, None, :]), p[1:4].tolist())]
        if p[0] == 0:
            k = torch.sqrt((q[0] * q[0] + q[1] * q[1]) + q[2] * q[2]) - p[4].item()
        else:
            q = [a.abs() - h for a, h in zip(q, p[4:7].tolist())]
            o = [a.clamp(min=0) for a in q]
            k = torch.sqrt((o[0] * o[0] + o[1] * o[1]) + o[2] * o[2]) + \
                torch.maximum(q[0], torch.maximum(q[1], q[2])).clamp(max=0)
        d = k if d is None else torch.minimum(d, k)
    return d.contiguous()


def _exact_grad(case, seed):
    xs = [_dense_values(_grad_case(case, i), seed) for i in range(case["batch"])]
    one = _grad_case(case, 0)  # its box and level are the whole batch's
    parts = []  # per grid: the values that its meshes depend on, and the vertices
    for v in xs:
        cells = _cells_of(v, 0.0)
        if not len(cells):
            return None
        at = (cells[:, None, :] + _off(range(8)))
        at = (at[..., 0] * v.shape[1] + at[..., 1]) * v.shape[2] + at[..., 2]
        ids, inv = torch.unique(at, return_inverse=True)
        u = v.reshape(-1)[ids].double().requires_grad_(True)
        cv = u[inv]
        dc = _exact_dc(cv.detach().float(), cv, cells, one, v.shape)[0]
        # MC vertices through the cells' own low edges is the whole set, in edge order
        pos = _exact_mc(v, one)
        parts.append((ids, u, cv, cells, dc, pos))
    total = sum(len(p[4]) + len(p[5]) for p in parts)
    loss = 0.0
    grads = []
    for v, (ids, u, cv, cells, dc, pos) in zip(xs, parts):
        # each crossed edge's vertex once: the edge counted in one of its cells
        hit, q, ia, _ = _crossings(cv.detach().float(), cv, cells, one, v.shape)
        pid = ((ia[..., 0] * v.shape[1] + ia[..., 1]) * v.shape[2] + ia[..., 2])[hit]
        axis = torch.tensor([2, 1, 2, 1, 2, 1, 2, 1, 0, 0, 0, 0], device="cuda").expand(len(cells), 12)[hit]
        mc = q[hit][_first_of(3 * pid + axis)]
        part = (((mc.norm(dim=-1) - 1) ** 2).sum() + ((dc.norm(dim=-1) - 1) ** 2).sum()) / total
        (gu,) = torch.autograd.grad(part, u)
        g = torch.zeros(v.numel(), dtype=torch.float64, device="cuda")
        g[ids] = gu
        grads.append(g.reshape(v.shape))
        loss = loss + part.detach()
    vertices = [p[5] for p in parts] + [p[4].detach() for p in parts]
    return {"loss": loss, "grad": grads, "vertices": vertices, "faces": [None] * len(vertices)}

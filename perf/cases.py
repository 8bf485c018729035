"""The framework's work as its users have it done, one case per kind and size:
tortuosity solves (one volume from host memory, several directions of a
device-resident volume, batches, a serving stream), connected components and
reactive areas.  Volumes are seeded random packings of overlapping solid
spheres or ellipsoids (255 = solid, 0 = pore), painted on the GPU.

listed() names the cases, draw() makes further ones of the same ranges,
prepare() builds what a program holds before the call, run() is the call,
work() what it cannot do without, exact() its outputs in 64 bits from plain
torch."""
import math

import numpy as np
import torch

import fast_gb300 as ft
from fast_gb300 import alpha, ccl
from fast_gb300.serve import TauServer

_DIRS = (ft.Dir.X_POS, ft.Dir.X_NEG, ft.Dir.Y_POS, ft.Dir.Y_NEG, ft.Dir.Z_POS, ft.Dir.Z_NEG)
_D = (1.0, float(np.float32(0.001)))  # pore and solid diffusivity


def listed():
    return [
        # One small volume from host memory in double precision, field
        # included: a probe of a sub-volume, bound by launches and latency.
        {"name": "host_f64_cg_small", "kind": "host", "nx": 28, "ny": 24, "nz": 20, "radius": 3.0, "solid": 0.5,
         "solver": "cg", "precision": "f64", "dir": 0, "tol": 1e-6, "field": True},
        # The drop-in call at its usual size: `fast tau` with its defaults.
        {"name": "host_f64_cg_64", "kind": "host", "nx": 64, "ny": 64, "nz": 64, "radius": 5.0, "solid": 0.6,
         "solver": "cg", "precision": "f64", "dir": 0, "tol": 1e-6, "field": False},
        # The API's defaults (BiCGSTAB, X_NEG, double) on an odd-sized volume.
        {"name": "host_f64_bicgstab_odd", "kind": "host", "nx": 97, "ny": 83, "nz": 110, "radius": 6.0, "solid": 0.55,
         "solver": "bicgstab", "precision": "f64", "dir": 1, "tol": 1e-6, "field": False},
        # `fast slice`: every sub-volume of a grid in three directions, single
        # precision, one batched call from host memory.
        {"name": "slice_f32_batch", "kind": "slice", "count": 12, "edge": 48, "radius": 4.0, "solid": 0.55,
         "tol": 1e-5},
        # Three directions of one packed volume as right-hand sides sharing
        # the phase field, mixed precision, mask on the device.
        {"name": "mixed_bicgstab_256_xyz", "kind": "dirs", "nx": 256, "ny": 256, "nz": 256, "radius": 12.0,
         "aspect": 0.35, "solid": 0.55, "solver": "bicgstab", "ndirs": 3, "tol": 1e-7},
        # A large sample in one direction, mixed-precision CG, ragged sizes.
        {"name": "mixed_cg_large", "kind": "dirs", "nx": 450, "ny": 391, "nz": 420, "radius": 10.0, "aspect": 1.0,
         "solid": 0.65, "solver": "cg", "ndirs": 1, "tol": 1e-6},
        # Uneven volumes in one batched mixed-precision launch.
        {"name": "mixed_cg_batch", "kind": "batch", "count": 24, "lo": 64, "hi": 192, "tol": 1e-6},
        # A burst of requests of mixed size, direction and solver served by
        # continuous batching, masks in host memory.
        {"name": "serve_burst", "kind": "serve", "count": 24, "lo": 32, "hi": 160, "tol": 1e-6},
        # Reachability pre-pass of a large volume resident on the device.
        {"name": "ccl_device_large", "kind": "ccl", "nx": 768, "ny": 700, "nz": 720, "radius": 10.0, "solid": 0.65,
         "host": False},
        # The same from host memory at the size of one sub-volume.
        {"name": "ccl_host_odd", "kind": "ccl", "nx": 101, "ny": 90, "nz": 77, "radius": 5.0, "solid": 0.6,
         "host": True},
        # `fast alpha` on a device-resident volume: labelling and the area
        # reachable from every face.
        {"name": "alpha_tensor_512", "kind": "alpha", "nx": 512, "ny": 512, "nz": 512, "radius": 10.0, "solid": 0.65,
         "host": False},
        # Area and porosity of one mid-sized volume from host memory, as
        # `fast slice` reports them for each sub-volume.
        {"name": "area_porosity_host", "kind": "alpha", "nx": 200, "ny": 181, "nz": 190, "radius": 6.0, "solid": 0.5,
         "host": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "host", "slice", "dirs", "dirs", "batch", "serve", "ccl", "ccl", "alpha", "alpha"])
    solid, radius = round(rng.uniform(0.4, 0.7), 3), round(rng.uniform(3.0, 10.0), 2)
    if kind == "host":
        c = {"nx": _log(rng, 16, 112), "ny": _log(rng, 16, 112), "nz": _log(rng, 16, 112),
             "radius": min(radius, 6.0), "solid": solid, "solver": rng.choice(["cg", "cg", "bicgstab"]),
             "precision": "f64", "dir": rng.randrange(6), "tol": 1e-6, "field": False}
    elif kind == "slice":
        c = {"count": rng.randint(4, 20), "edge": _log(rng, 24, 64), "radius": min(radius, 5.0), "solid": solid,
             "tol": 1e-5}
    elif kind == "dirs":
        # up to about the listed 256^3 x 3 or the one-direction large volume
        nd = rng.randint(1, 3)
        hi = 256 if nd > 1 else 384
        c = {"nx": _log(rng, 40, hi), "ny": _log(rng, 40, hi), "nz": _log(rng, 40, hi), "radius": radius,
             "aspect": round(rng.uniform(0.35, 1.0), 2), "solid": solid, "solver": "cg" if hi > 256 else
             rng.choice(["cg", "bicgstab"]), "ndirs": nd, "tol": rng.choice([1e-6, 1e-7])}
    elif kind in ("batch", "serve"):
        c = {"count": rng.randint(6, 24), "lo": 32 if kind == "serve" else 48, "hi": _log(rng, 80, 160), "tol": 1e-6}
    elif kind == "ccl":
        host = rng.random() < 0.4
        hi = 200 if host else 700
        c = {"nx": _log(rng, 40, hi), "ny": _log(rng, 40, hi), "nz": _log(rng, 40, hi), "radius": radius,
             "solid": solid, "host": host}
    else:
        host = rng.random() < 0.5
        hi = 200 if host else 512
        c = {"nx": _log(rng, 40, hi), "ny": _log(rng, 40, hi), "nz": _log(rng, 40, hi), "radius": radius,
             "solid": solid, "host": host}
    c["kind"] = kind
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _packing(nx, ny, nz, radius, aspect, solid, seed):
    """uint8 [nz, ny, nx] on the GPU: ellipsoids with semi-axes (radius,
    radius * aspect, radius * aspect), uniform centres and rotations, as many
    as give `solid` for overlapping bodies."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    vol = torch.zeros(nz * ny * nx, dtype=torch.uint8, device="cuda")
    body = 4.0 / 3.0 * math.pi * radius ** 3 * aspect ** 2
    # centres fall up to one radius outside, so the faces see whole bodies
    ext = torch.tensor([nx, ny, nz], device="cuda", dtype=torch.float32)
    room = (nx + 2 * radius) * (ny + 2 * radius) * (nz + 2 * radius)
    n = max(1, int(round(-math.log(1.0 - solid) * room / body)))
    centre = torch.rand(n, 3, generator=gen, device="cuda") * (ext + 2 * radius) - radius
    axis = torch.nn.functional.normalize(torch.randn(n, 3, generator=gen, device="cuda"), dim=1)
    reach = int(math.ceil(radius)) + 1
    o = torch.arange(-reach, reach + 1, device="cuda")
    oz, oy, ox = torch.meshgrid(o, o, o, indexing="ij")
    off = torch.stack([ox, oy, oz], -1).reshape(-1, 3)
    step = max(1, (1 << 24) // off.shape[0])
    for a in range(0, n, step):
        c, u = centre[a:a + step], axis[a:a + step]
        base = c.floor().long()
        p = base[:, None, :] + off[None]
        d = p.float() + 0.5 - c[:, None, :]
        along = (d * u[:, None, :]).sum(-1)
        inside = along ** 2 + (d.square().sum(-1) - along ** 2) / (aspect * aspect) <= radius * radius
        inside &= (p >= 0).all(-1) & (p < ext.long()).all(-1)
        vol[((p[..., 2] * ny + p[..., 1]) * nx + p[..., 0])[inside]] = 255
    return vol.view(nz, ny, nx)


def _mixture(case):
    """The sizes, packings, directions and solvers of a batch or a stream:
    part of the case, the same for every seed."""
    rng = np.random.RandomState(case["count"] * 1000 + case["hi"])
    out = []
    for _ in range(case["count"]):
        if case["kind"] == "serve":
            e = int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))))
            dims = (e, e, e)
        else:
            dims = tuple(int(v) for v in rng.randint(case["lo"], case["hi"] + 1, 3))
        out.append({"dims": dims, "radius": float(rng.uniform(3, 8)), "aspect": float(rng.choice([1.0, 0.5])),
                    "solid": float(rng.uniform(0.4, 0.7)), "dir": _DIRS[int(rng.randint(6))],
                    "cg": bool(rng.randint(2))})
    return out


def _volumes(case, seed):
    """The masks of a case, on the GPU, each with its directions."""
    k = case["kind"]
    if k in ("batch", "serve"):
        return [(_packing(*m["dims"], m["radius"], m["aspect"], m["solid"], seed * 1000 + i), [m["dir"]])
                for i, m in enumerate(_mixture(case))]
    if k == "slice":
        e = case["edge"]
        return [(_packing(e, e, e, case["radius"], 1.0, case["solid"], seed * 1000 + i), list(_DIRS[0::2]))
                for i in range(case["count"])]
    dirs = list(_DIRS[0::2])[:case["ndirs"]] if k == "dirs" else [_DIRS[case.get("dir", 0)]]
    return [(_packing(case["nx"], case["ny"], case["nz"], case["radius"], case.get("aspect", 1.0), case["solid"], seed),
             dirs)]


def prepare(case, seed):
    vols = _volumes(case, seed)
    k = case["kind"]
    state = {"case": case}
    if k in ("host", "slice", "serve") or case.get("host"):
        vols = [(m.cpu().numpy(), d) for m, d in vols]
    state["vols"] = vols
    solver = ft.DSOLVER_CG if case.get("solver", "cg") == "cg" else ft.DSOLVER_BICGSTAB
    if k == "host":
        state["params"] = ft.TortuosityParams(dir=_DIRS[case["dir"]], tolerance=case["tol"],
                                              precision=ft.Precision.F64)
        state["field"] = np.zeros(vols[0][0].shape, dtype=np.float64) if case["field"] else None
    elif k == "slice":
        state["params"] = ft.TortuosityParams(tolerance=case["tol"], precision=ft.Precision.F32)
    elif k in ("dirs", "batch"):
        state["params"] = ft.TortuosityParams(tolerance=case["tol"], precision=ft.Precision.MIXED)
    elif k == "serve":
        state["server"] = TauServer(tolerance=case["tol"], hbm_budget=32 << 30)
        state["solvers"] = [ft.DSOLVER_CG if m["cg"] else ft.DSOLVER_BICGSTAB for m in _mixture(case)]
    elif k == "ccl" and not case["host"]:
        state["labels"] = torch.zeros(vols[0][0].shape, dtype=torch.int32, device="cuda")
    state["solver"] = solver
    torch.cuda.synchronize()
    return state


# ---------------------------------------------------------------------------
# The calls
# ---------------------------------------------------------------------------
def _table(c, mask):
    """The face rows by label in a table whose width depends on the volume's
    size alone (volumes of one size differ in their number of labels)."""
    out = np.zeros((7, math.prod(mask.shape) // 64 + 2), dtype=np.uint8)
    out[:, :c.num_labels] = c.boundary_label_mask
    return out


def run(state):
    case, vols = state["case"], state["vols"]
    k = case["kind"]
    if k == "host":
        tau = ft.get_tortuosity(vols[0][0], state["params"], state["solver"], concentration_output=state["field"])
        return {"tau": tau} if state["field"] is None else {"tau": tau, "field": state["field"]}
    if k == "slice":
        return [r.tau for r in ft.solve_batch([(m, d) for m, dirs in vols for d in dirs], state["params"],
                                              state["solver"])]
    if k == "dirs":
        m, dirs = vols[0]
        return [r.tau for r in ft.solve_directions_device(m.data_ptr(), tuple(m.shape), dirs, state["params"],
                                                          state["solver"])]
    if k == "batch":
        return [r.tau for r in ft.solve_batch_device([(m.data_ptr(), tuple(m.shape), d[0]) for m, d in vols],
                                                     state["params"], state["solver"])]
    if k == "serve":
        srv = state["server"]
        for (m, d), solver in zip(vols, state["solvers"]):
            srv.submit(m, d[0], solver)
        return [c.result.tau for c in sorted(srv.drain(), key=lambda c: c.ticket)]
    m = vols[0][0]
    if k == "ccl" and case["host"]:
        c = ccl.get_volume_ccl(m)
        return {"labels": c.labels.view(np.int32), "num_labels": c.num_labels, "faces": _table(c, m)}
    if k == "ccl":
        c = ccl.get_volume_ccl_device(m.data_ptr(), tuple(m.shape), state["labels"].data_ptr())
        return {"labels": state["labels"], "num_labels": c.num_labels, "faces": _table(c, m)}
    if case["host"]:
        return {"area": alpha.get_reactive_area_density(m), "porosity": ft.get_porosity(m)}
    tensor, area = alpha.get_reactive_area_density_tensor_device(m.data_ptr(), tuple(m.shape))
    return {"tensor": tensor, "area": area}


def work(case):
    """Bytes and operations of one pass.  A Jacobi-preconditioned solve takes
    about 40 sqrt(n) matrix products at n voxels across; each reads and
    writes the iterate, residual and direction once (25 B per voxel in 32
    bits, 49 in 64) and does about 30 operations per voxel."""
    k = case["kind"]

    def solve(dims, rhs, size):
        n = dims[0] * dims[1] * dims[2]
        products = 40.0 * math.sqrt(max(dims))
        return n * rhs * products * (6 * size + 1), n * rhs * products * 30.0

    if k in ("batch", "serve"):
        parts = [solve(m["dims"], 1, 4) for m in _mixture(case)]
    elif k == "slice":
        parts = [solve((case["edge"],) * 3, 3, 4)] * case["count"]
    elif k in ("host", "dirs"):
        parts = [solve((case["nx"], case["ny"], case["nz"]), case.get("ndirs", 1), 8 if k == "host" else 4)]
    else:
        n = case["nx"] * case["ny"] * case["nz"]
        parts = [(5.0 * n, 2.0 * n)] if k == "ccl" else [(1.0 * n, (8.0 if case["host"] else 56.0) * n)]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


# ---------------------------------------------------------------------------
# The same in 64 bits from plain torch
# ---------------------------------------------------------------------------
def _solve64(mask, d, tol=1e-11, limit=20000):
    """(tau, field) of the variable-coefficient 7-point diffusion problem:
    arithmetic-mean faces, 1 and 0 on the two faces normal to the direction at
    half a cell's distance, zero flux on the others."""
    axis, positive = 2 - int(d) // 2, int(d) % 2 == 0
    cell = torch.where(mask == 0, _D[0], _D[1]).to(torch.float64)
    face = [0.5 * (cell.narrow(a, 0, cell.shape[a] - 1) + cell.narrow(a, 1, cell.shape[a] - 1)) for a in range(3)]
    diag, rhs = torch.zeros_like(cell), torch.zeros_like(cell)
    for a in range(3):
        n = cell.shape[a]
        diag.narrow(a, 0, n - 1).add_(face[a])
        diag.narrow(a, 1, n - 1).add_(face[a])
    n = cell.shape[axis]
    for end in (0, n - 1):
        diag.select(axis, end).add_(2 * cell.select(axis, end))
    begin = 0 if positive else n - 1
    rhs.select(axis, begin).add_(2 * cell.select(axis, begin))

    def product(p, q):
        torch.mul(diag, p, out=q)
        for a in range(3):
            m = p.shape[a] - 1
            q.narrow(a, 0, m).addcmul_(face[a], p.narrow(a, 1, m), value=-1)
            q.narrow(a, 1, m).addcmul_(face[a], p.narrow(a, 0, m), value=-1)

    inv = 1.0 / diag
    ramp = (torch.arange(n, device=mask.device, dtype=torch.float64) + 0.5) / n
    shape = [1, 1, 1]
    shape[axis] = n
    x = ((1 - ramp) if positive else ramp).view(shape).expand_as(cell).clone()
    q = torch.empty_like(x)
    product(x, q)
    r = rhs - q
    z = inv * r
    p = z.clone()
    rz, stop = torch.sum(r * z), tol * tol * float(rhs.square().sum())
    for it in range(limit):
        product(p, q)
        step = rz / torch.sum(p * q)
        x.addcmul_(p, step)
        r.addcmul_(q, -step)
        if it % 25 == 0 and float(r.square().sum()) <= stop:
            break
        torch.mul(inv, r, out=z)
        new = torch.sum(r * z)
        p.mul_(new / rz).add_(z)
        rz = new
    ahead = torch.zeros_like(x)  # the neighbour one step along; 0 behind the far face
    src, dst = ((1, 0) if positive else (0, 1))
    ahead.narrow(axis, dst, n - 1).copy_(x.narrow(axis, src, n - 1))
    flux = cell * (x - ahead)
    flux.select(axis, n - 1 if positive else 0).mul_(2)
    pores = float((mask == 0).sum())
    return pores / mask.numel() * (mask.numel() / n) / float(flux.sum()), x


_A, _B = (0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3), (1, 2, 3, 0, 5, 6, 7, 4, 4, 5, 6, 7)  # a cell's edges
_CORNER = ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))
_FACES = ((0, 1, 2, 3), (4, 5, 6, 7), (0, 1, 5, 4), (3, 2, 6, 7), (0, 3, 7, 4), (1, 2, 6, 5))


def _triangles(pattern):
    """Triangles (edge triples) of a corner pattern: each face's cut edges are
    paired, with the two corners below kept apart on an ambiguous face; the
    loops are fanned from their smallest edge."""
    links = {}
    for f in _FACES:
        edges = [next(e for e in range(12) if {_A[e], _B[e]} == {f[q], f[(q + 1) % 4]}) for q in range(4)]
        below = [pattern >> c & 1 for c in f]
        cut = [edges[q] for q in range(4) if below[q] != below[(q + 1) % 4]]
        pairs = [cut] if len(cut) == 2 else []
        if len(cut) == 4:
            first = 3 if below[0] else 0
            pairs = [[edges[first], edges[(first + 1) % 4]], [edges[(first + 2) % 4], edges[(first + 3) % 4]]]
        for a, b in pairs:
            links.setdefault(a, []).append(b)
            links.setdefault(b, []).append(a)
    seen, out = set(), []
    for e in sorted(links):
        if e in seen:
            continue
        loop, last, at = [e], e, min(links[e])
        while at != e:
            loop.append(at)
            last, at = at, links[at][1] if links[at][0] == last else links[at][0]
        seen.update(loop)
        out += [(loop[0], loop[q], loop[q + 1]) for q in range(1, len(loop) - 1)]
    return out


def _area64(field, iso=0.5):
    """Marching-cubes area of a boolean volume [z, y, x]: corner values are
    the means of the 2x2x2 voxels around them, axis a scaled by 1/n_a."""
    nz, ny, nx = field.shape
    v = torch.nn.functional.pad(field[None, None].to(torch.float16), (1,) * 6, mode="replicate")[0, 0].to(torch.uint8)
    corner = sum(v[c:c + nz + 1, b:b + ny + 1, a:a + nx + 1] for a in (0, 1) for b in (0, 1) for c in (0, 1))
    pattern = torch.zeros((nz, ny, nx), dtype=torch.uint8, device=field.device)
    for c, (a, b, d) in enumerate(_CORNER):
        pattern |= (corner[d:d + nz, b:b + ny, a:a + nx] < 8 * iso).to(torch.uint8) << c
    pattern, flat = pattern.reshape(-1), corner.reshape(-1)
    cell = torch.nonzero((pattern != 0) & (pattern != 255)).squeeze(1)
    of = pattern[cell]
    order = torch.argsort(of, stable=True)
    cell, of = cell[order], of[order]
    counts = torch.bincount(of.long(), minlength=256).tolist()
    size = torch.tensor([1.0 / nx, 1.0 / ny, 1.0 / nz], dtype=torch.float64, device=field.device)
    offset = torch.tensor(_CORNER, dtype=torch.float64, device=field.device) * size
    total, at = 0.0, 0
    for cs, m in enumerate(counts):
        mine = cell[at:at + m]
        at += m
        if not m:
            continue
        x, y, z = mine % nx, mine // nx % ny, mine // (nx * ny)
        f = [flat[((z + d) * (ny + 1) + y + b) * (nx + 1) + x + a].double() / 8 for a, b, d in _CORNER]
        cut = {}
        for tri in _triangles(cs):
            for e in tri:
                if e not in cut:
                    t = (iso - f[_A[e]]) / (f[_B[e]] - f[_A[e]])
                    cut[e] = offset[_A[e]] + t[:, None] * (offset[_B[e]] - offset[_A[e]])
            a, b, c = (cut[e] for e in tri)
            total += float(torch.linalg.cross(b - a, c - a).norm(dim=1).sum()) / 2
    return total


def _reached(pore, d):
    """The pore voxels connected to face d (Dir order: the positive face of an
    axis is its last plane)."""
    axis = 2 - d // 2
    got = torch.zeros_like(pore)
    end = pore.shape[axis] - 1 if d % 2 == 0 else 0
    got.select(axis, end).copy_(pore.select(axis, end))
    count = -1
    while True:
        for _ in range(24):
            for a in range(3):
                n = pore.shape[a] - 1
                got.narrow(a, 1, n).logical_or_(got.narrow(a, 0, n).clone())
                got.narrow(a, 0, n).logical_or_(got.narrow(a, 1, n).clone())
                got &= pore
        now = int(got.sum())
        if now == count:
            return got
        count = now


def exact(case, seed):
    k = case["kind"]
    if k == "ccl":
        return None  # whole numbers
    if k == "dirs" and case["nx"] * case["ny"] * case["nz"] * case["ndirs"] > 55e6:
        return None  # half a minute and more
    vols = _volumes(case, seed)
    if k == "host":
        tau, field = _solve64(vols[0][0], vols[0][1][0])
        return {"tau": tau, "field": field} if case["field"] else {"tau": tau}
    if k != "alpha":
        return [_solve64(m, d)[0] for m, dirs in vols for d in dirs]
    mask = vols[0][0]
    pore = mask == 0
    if case["host"]:
        return {"area": _area64(~pore), "porosity": float(pore.sum()) / pore.numel()}
    return {"tensor": [_area64(_reached(pore, d)) for d in range(6)], "area": _area64(~pore)}

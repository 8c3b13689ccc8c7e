"""Performance cases of porerad_b200: the work its users have it do, through its public entry points.

Each case makes a seeded voxel microstructure of one of the four benchmark archetypes (FI isotropic
fibers, FA fibers along z, OF open-cell foam, TL perforated layers) in plain torch, keeps what a
program would keep between calls (phase array, count tables, operator), and makes one pass of one of
these workflows:

counts     build_surface_patches and the host pass of first_hit_counts (pr_first_hit_counts_host) into a
           program's own pinned arrays: the reference-facing tracing call.
sets       a whole device-resident case: two seeded ray sets, their pool, the three balanced
           operators and the mixed-precision channels of each.
sweep      many small geometries in shared launches: batched counts, batched operators, channels.
arrays     the plain drop-in path from host edge lists: pool_counts, ExchangeOperator, channels.
fields     repeated solves on a resident operator, as an outer iteration over temperature fields.
power      net patch power and its derivative from host vectors (the Newton solver's evaluations).
products   the five sparse products from host vectors, one after the other.
coupled    conduction assembly and solve, then the strictly coupled Newton-Krylov solve.
statistics radiative properties and penetration of one microstructure (multi-bounce rays).
morphology all scalar and directional descriptors of one microstructure.

``exact`` restates tracing, balancing, radiosity and the coupled solve in plain binary64 torch.
"""

from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

SIGMA = 5.670374419e-8
K_SOLID, K_GAS = 0.20, 0.026
H_M = 0.01  # slab thickness: 1 cm, as in the benchmark configurations


def listed():
    return [
        # the small plain configuration: a 64^3 fiber slab at 64 rays per patch, where launches and latency count
        dict(name="counts fibers 64", kind="counts", arch="FI", nx=64, ny=64, nz=64, phi=0.10, rays=64),
        # the headline configuration: a 128^3 foam at 1000 rays per patch, one full ray set to NumPy arrays
        dict(name="counts foam 128", kind="counts", arch="OF", nx=128, ny=128, nz=128, phi=0.10, rays=1000),
        # a non-cubic box with odd sides and an odd ray count (cropped scans, repeats along the axis)
        dict(name="counts layers odd", kind="counts", arch="TL", nx=151, ny=77, nz=93, phi=0.17, rays=333),
        # one prescribed-field case of the foam end to end on the device, two ray sets of 500 rays
        dict(name="sets foam 128", kind="sets", arch="OF", nx=128, ny=128, nz=128, phi=0.10, rays=500, eps=0.6),
        # a parameter sweep: all four archetypes at several solid fractions in shared launches
        dict(name="sweep 12 at 64", kind="sweep", arch="all", nx=64, ny=64, nz=64, phi=0.10, rays=125, eps=0.6, count=12),
        # the drop-in NumPy path between tracing and channels, fibers along z with rays along x
        dict(name="arrays fibers 96", kind="arrays", arch="FA", nx=96, ny=96, nz=96, phi=0.10, rays=500, eps=0.9),
        # repeated solves at perturbed fields on a resident layer operator larger than the L2
        dict(name="fields layers 160", kind="fields", arch="TL", nx=160, ny=160, nz=160, phi=0.10, rays=500, eps=0.6, count=4),
        # a small operator's radiosity and derivative from host vectors
        dict(name="power foam 48", kind="power", arch="OF", nx=48, ny=48, nz=48, phi=0.12, rays=200, eps=0.5),
        # single products of a small operator: the smallest calls
        dict(name="products fibers 40", kind="products", arch="FI", nx=40, ny=40, nz=40, phi=0.10, rays=64),
        # a strictly coupled solve at the size of the stored core cases' lower resolution
        dict(name="coupled foam 64", kind="coupled", arch="OF", nx=64, ny=64, nz=64, phi=0.10, rays=500, eps=0.6),
        # the ray statistics of one identification at the archived ray counts
        dict(name="statistics fibers 128", kind="statistics", arch="FI", nx=128, ny=128, nz=128, phi=0.10, rays=200000, eps=0.8),
        # the descriptors of one stored-size microstructure
        dict(name="morphology foam 128", kind="morphology", arch="OF", nx=128, ny=128, nz=128, phi=0.10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["counts", "counts", "counts", "sets", "sets", "sweep", "arrays", "fields", "power", "products",
                       "coupled", "statistics", "morphology"])
    arch = rng.choice(["OF", "FI", "FA", "TL"])
    phi = round(rng.uniform(0.05, 0.20), 3)
    eps = round(rng.uniform(0.3, 0.95), 3)
    lo, hi = {"counts": (20, 160), "sets": (24, 128), "sweep": (24, 72), "arrays": (24, 96), "fields": (32, 150),
              "power": (24, 80), "products": (20, 80), "coupled": (24, 64), "statistics": (48, 128),
              "morphology": (128, 170)}[kind]
    nx, ny, nz = (_log_int(rng, lo, hi) for _ in range(3))
    case = dict(kind=kind, arch=arch, nx=nx, ny=ny, nz=nz, phi=phi)
    if kind == "morphology":
        return case
    if kind == "statistics":
        return dict(case, rays=_log_int(rng, 20000, 200000), eps=eps)
    most = {"counts": 2.2e8, "sets": 9e7, "sweep": 8e6, "arrays": 4e7, "fields": 2e8, "power": 2e7, "products": 2e7,
            "coupled": 1.5e7}[kind]
    rays = min(_log_int(rng, 16 if kind == "counts" else 64, 1000), int(most / _patches(case)))
    case["rays"] = rays
    if kind == "sweep":
        case.update(arch="all", count=rng.randint(3, 12))
    if kind == "fields":
        case["count"] = rng.randint(1, 4)
    if kind not in ("counts", "products"):
        case["eps"] = eps
    return case


def _patches(case):
    """About how many surface patches a case's microstructure has."""

    per = {"FI": 1.35, "FA": 1.25, "OF": 1.1, "TL": 0.65, "all": 1.1}[case["arch"]]
    return per * case["phi"] * case["nx"] * case["ny"] * case["nz"] + 2.0 * (1 - case["phi"]) * case["ny"] * case["nz"]


def work(case):
    """Inputs read once and outputs written once; per ray about 60 operations to make it and 9 per visited
    cell (about half a box side of cells); 2 operations per matrix entry and sparse product."""

    kind, cells = case["kind"], case["nx"] * case["ny"] * case["nz"]
    P = _patches(case)
    cells_per_ray = 0.35 * (cells ** (1 / 3))
    rays = P * case.get("rays", 0)
    pairs = 0.55 * rays
    traced = rays * (60 + 9 * cells_per_ray)
    if kind == "counts":
        return {"bytes": cells + 16 * pairs, "flops": traced}
    if kind == "sets":  # two sets, three operators (4-byte entries, about 45 products each)
        return {"bytes": cells + 3 * 45 * 4 * 1.5 * pairs, "flops": 2 * traced + 3 * 45 * 2 * 1.5 * pairs}
    if kind == "sweep":
        n = case["count"]
        return {"bytes": n * (cells + 45 * 4 * 3 * pairs), "flops": n * (2 * traced + 45 * 2 * 3 * pairs)}
    if kind == "arrays":  # two edge lists in, their pool out and in again
        return {"bytes": 2 * 16 * pairs + 2 * 16 * 1.8 * pairs + 45 * 4 * 2 * pairs, "flops": 45 * 2 * 2 * pairs}
    if kind == "fields":
        return {"bytes": case["count"] * (8 * cells + 20 * 4 * 1.6 * pairs), "flops": case["count"] * 20 * 2 * 1.6 * pairs}
    if kind == "power":
        return {"bytes": 60 * 4 * 1.6 * pairs + 10 * 8 * P, "flops": 60 * 2 * 1.6 * pairs}
    if kind == "products":
        return {"bytes": 3 * 4 * 1.6 * pairs + 2 * 8 * pairs + 10 * 8 * P, "flops": 5 * 2 * 1.6 * pairs}
    if kind == "coupled":  # about 600 stencil products and 250 sparse products
        return {"bytes": 600 * 48 * cells + 250 * 4 * 1.6 * pairs, "flops": 600 * 20 * cells + 250 * 2 * 1.6 * pairs}
    if kind == "statistics":  # two seeds, three bounces a ray or so
        return {"bytes": cells, "flops": 4 * case["rays"] * 3 * (60 + 9 * cells_per_ray)}
    return {"bytes": cells + 8.0 * 3 * case["nx"], "flops": 40.0 * cells}


# ---------------------------------------------------------------- microstructures (plain torch)


def _ball(radius):
    r = int(math.ceil(radius))
    g = np.arange(-r, r + 1)
    dx, dy, dz = np.meshgrid(g, g, g, indexing="ij")
    keep = dx * dx + dy * dy + dz * dz <= radius * radius
    return np.stack((dx[keep], dy[keep], dz[keep]), axis=1)


def _fibers(shape, phi, rng, aligned):
    """Periodic cylinders of radius 2 (random axes, or along z) until the solid fraction reaches phi."""

    nx, ny, nz = shape
    box = torch.tensor(shape, device="cuda")
    solid = torch.zeros(nx * ny * nz, dtype=torch.uint8, device="cuda")
    ball = torch.from_numpy(_ball(2.0)).cuda()
    length = float(nz) if aligned else 1.5 * max(shape)
    t = np.arange(-length / 2, length / 2 + 0.25, 0.25)
    target = phi * solid.numel()
    while int(solid.sum()) < target:
        p = rng.random(3) * shape
        d = np.array([0.0, 0.0, 1.0]) if aligned else rng.standard_normal(3)
        pts = np.rint(p + t[:, None] * (d / np.linalg.norm(d))).astype(np.int64)
        c = (torch.from_numpy(pts).cuda()[:, None, :] + ball).reshape(-1, 3) % box
        solid[(c[:, 0] * ny + c[:, 1]) * nz + c[:, 2]] = 1
    return solid.reshape(shape)


def _foam(shape, phi, rng):
    """Struts where a cell's first and third nearest of 64 periodic seed points are nearly equally far."""

    pts = torch.from_numpy(rng.random((64, 3)) * shape).float().cuda()
    field = torch.empty(shape, device="cuda")
    axes = [torch.arange(n, device="cuda") + 0.5 for n in shape]

    def gap(a):  # squared minimum-image distance along one axis, (n, 64)
        d = (axes[a][:, None] - pts[None, :, a]).abs()
        return torch.minimum(d, shape[a] - d) ** 2

    gx, gy, gz = gap(0), gap(1), gap(2)
    for i in range(shape[0]):
        d3 = torch.topk((gx[i] + gy[:, None, :]) + gz[None, :, :], 3, dim=-1, largest=False).values.sqrt()
        field[i] = d3[..., 2] - d3[..., 0]
    k = max(1, int(phi * field.numel()))
    return (field <= field.flatten().kthvalue(k).values).to(torch.uint8)


def _layers(shape, phi, rng):
    """Sheets of 4 cells normal to z, perforated by holes of 8 cells until the solid fraction is down to phi."""

    nx, ny, nz = shape
    m = max(1, int(math.ceil(phi * nz / 4)))
    start = int(rng.integers(0, nz))
    z0 = [(start + (s * nz) // m) % nz for s in range(m)]
    solid = torch.zeros(shape, dtype=torch.uint8, device="cuda")
    for z in z0:
        for k in range(4):
            solid[:, :, (z + k) % nz] = 1
    g = np.arange(-4, 5)
    dx, dy = np.meshgrid(g, g, indexing="ij")
    keep = dx * dx + dy * dy <= 16
    disk = np.stack((dx[keep], dy[keep]), axis=1)
    target = phi * solid.numel()
    holes = max(8, nx * ny // 400)
    while int(solid.sum()) > target:
        for _ in range(holes):
            z, c = z0[int(rng.integers(0, m))], rng.integers(0, (nx, ny))
            xy = torch.from_numpy((c + disk) % (nx, ny)).cuda()
            for k in range(4):
                solid[xy[:, 0], xy[:, 1], (z + k) % nz] = 0
    return solid


def _microstructure(arch, shape, phi, rng):
    if arch == "OF":
        return _foam(shape, phi, rng)
    if arch == "TL":
        return _layers(shape, phi, rng)
    return _fibers(shape, phi, rng, arch == "FA")


def _shape(case):
    return case["nx"], case["ny"], case["nz"]


def _rng(seed, what):
    return np.random.default_rng([int(seed), what])


def _ray_seeds(seed, n):
    return [int(s) for s in np.random.default_rng([int(seed), 7]).integers(1, 2**62, n)]


def _phases(case, seed):
    """The case's microstructures, uint8 host arrays of 1 (solid) and 0.  Tracing and everything after it
    keeps one microstructure per case, so that its patches do not change with the seed; the seed then
    gives the rays and the vectors."""

    fixed = case["kind"] not in ("statistics", "morphology")
    rng = _rng(1000 * case["nx"] + 10 * case["ny"] + case["nz"] if fixed else seed, 1)
    if case["arch"] != "all":
        return [_microstructure(case["arch"], _shape(case), case["phi"], rng).cpu().numpy()]
    fracs = (0.05, 0.10, 0.20)
    return [_microstructure(("OF", "FI", "FA", "TL")[k % 4], _shape(case), fracs[(k // 4) % 3], rng).cpu().numpy()
            for k in range(case["count"])]


def _area(patches, ph):
    return np.full(patches.n_patches, (H_M / ph.shape[0]) ** 2)


def _fields(case, seed, device="cuda"):
    """Linear fields from 710 to 690 K along x with 5 K of noise per cell."""

    g = torch.Generator(device=device).manual_seed(int(seed) + 3)
    nx, ny, nz = _shape(case)
    line = 710.0 - (torch.arange(nx, dtype=torch.float64, device=device) + 0.5) * 20.0 / nx
    return [line[:, None, None] + 5.0 * torch.randn((nx, ny, nz), generator=g, dtype=torch.float64, device=device)
            for _ in range(case["count"])]


def _vectors(case, seed, P):
    rng = _rng(seed, 5)
    return dict(T=700.0 + 40.0 * (rng.random(P) - 0.5), dT=rng.standard_normal(P),
                eps=np.clip(case.get("eps", 0.6) + 0.1 * (rng.random(P) - 0.5), 0.05, 1.0), x=rng.random(P) + 0.5)


# ---------------------------------------------------------------- what a program has in hand


def prepare(case, seed):
    from porerad_b200 import exchange, view_factors as vf

    kind = case["kind"]
    phases = _phases(case, seed)
    s = {"case": case, "phases": phases, "seeds": _ray_seeds(seed, 2 * max(1, case.get("count", 1)))}
    if kind == "counts":
        n = vf.build_surface_patches(phases[0], H_M).n_patches
        # room for one pair per ray; the full sets of a foam have about 0.6
        room = int(n * case["rays"] * (0.75 if case["arch"] == "OF" and case["rays"] >= 800 else 1.0))
        s["list"] = [torch.zeros(room, dtype=t, pin_memory=True).numpy() for t in (torch.int32, torch.int32, torch.int64)]
    if kind == "arrays":
        p = vf.build_surface_patches(phases[0], H_M)
        s["patches"], s["area"] = p, _area(p, phases[0])
        s["tables"] = [vf.first_hit_counts(p, case["rays"], q) for q in s["seeds"][:2]]
    if kind in ("fields", "power", "products", "coupled"):
        p = vf.build_surface_patches(phases[0], H_M)
        table = vf.first_hit_counts_pooled(p, case["rays"], s["seeds"][:1])
        area = _area(p, phases[0])
        op = exchange.ExchangeOperator(table, None, None, np.full(p.n_patches, case["rays"], np.int64), area)
        table.close()
        s.update(patches=p, area=area, op=op)
        if kind == "fields":
            s["T"] = _fields(case, seed)
        if kind in ("power", "products"):
            s.update(_vectors(case, seed, p.n_patches))
        if kind == "coupled":
            s["k"] = np.where(phases[0] == 1, K_SOLID, K_GAS)
    return s


def _channels(ch):
    return [ch.q_h, ch.q_c, ch.q_i, ch.coarse_source]


def run(s):
    from porerad_b200 import (_lib, conduction, coupled, descriptors, exchange, penetration, properties,
                              view_factors as vf)

    case = s["case"]
    kind, rays = case["kind"], case.get("rays")
    ph = s["phases"][0]
    if kind == "counts":
        p = vf.build_surface_patches(ph, H_M)
        o, r, c = s["list"]
        seed = _lib.seeds_struct([_lib.pcg64_state(s["seeds"][0])])
        n = ctypes.c_int64()
        _lib.check(_lib.load().pr_first_hit_counts_host(p.device().handle, rays, ctypes.addressof(seed), 1, None,
                                                        o.ctypes.data, r.ctypes.data, c.ctypes.data, o.size,
                                                        ctypes.byref(n)))
        return [o, r, c, int(n.value)]
    if kind == "sets":
        p = vf.build_surface_patches(ph, H_M)
        a, b = (vf.first_hit_counts_pooled(p, rays, [q]) for q in s["seeds"][:2])
        tables = [(a, rays), (b, rays), (a.merge(b), 2 * rays)]
        out = []
        for table, r in tables:
            op = exchange.ExchangeOperator(table, None, None, np.full(p.n_patches, r, np.int64), _area(p, ph))
            ch = coupled.prescribed_field_channels(op, p, 700.0, 100.0, case["eps"], precision="mixed")
            out.append([op.nnz, op.nnz_symmetric, op.scale, *_channels(ch)])
            op.close()
            table.close()
        return out
    if kind == "sweep":
        ps = [vf.build_surface_patches(x, H_M) for x in s["phases"]]
        n = len(ps)
        tables = vf.first_hit_counts_batch(ps, rays, [s["seeds"][2 * k:2 * k + 2] for k in range(n)])
        ops = exchange.ExchangeOperator.from_tables(tables, [np.full(p.n_patches, 2 * rays, np.int64) for p in ps],
                                                    [_area(p, x) for p, x in zip(ps, s["phases"])])
        out = []
        for p, op in zip(ps, ops):
            ch = coupled.prescribed_field_channels(op, p, 700.0, 100.0, case["eps"], precision="mixed")
            out.append([op.scale, np.array([ch.q_h, ch.q_c, ch.q_i]), ch.coarse_source])
        for x in ops + tables:
            x.close()
        return out
    if kind == "arrays":
        p = s["patches"]
        o, r, c = vf.pool_counts(s["tables"], p.n_patches)
        op = exchange.ExchangeOperator(o, r, c, np.full(p.n_patches, 2 * rays, np.int64), s["area"])
        ch = coupled.prescribed_field_channels(op, p, 650.0, 20.0, case["eps"])
        out = [op.nnz, op.nnz_symmetric, op.scale, *_channels(ch)]
        op.close()
        return out
    if kind == "fields":
        return [_channels(coupled.cell_field_channels(s["op"], s["patches"], T, 710.0, 690.0, case["eps"],
                                                      reference_temperature_K=700.0, precision="mixed"))
                for T in s["T"]]
    if kind == "power":
        op = s["op"]
        a = exchange.net_patch_power(op, s["T"], s["eps"], s["area"], relative_tolerance=1e-13,
                                     reference_temperature_K=700.0)
        b = exchange.net_patch_power(op, s["T"], s["eps"], s["area"], relative_tolerance=1e-13)
        j = exchange.net_patch_power_jvp(op, s["T"], s["dT"], s["eps"], s["area"], relative_tolerance=1e-12)
        return [a.emitted_power_W, a.absorbed_power_W, a.net_power_W, b.emitted_power_W, b.absorbed_power_W, j]
    if kind == "products":
        op, x = s["op"], s["x"]
        return [op.matvec(x), op.rmatvec(x), op.symmetric_matvec(x), op.raw_matvec(x), op.raw_rmatvec(x)]
    if kind == "coupled":
        system = conduction.assemble_conduction(s["k"], H_M)
        T0 = conduction.solve_conduction(system, 750.0, 650.0)
        r = coupled.solve_coupled(system, s["op"], s["patches"], 750.0, 650.0, case["eps"], T0)
        m = coupled.wall_flux_metrics(system, s["patches"], r, 750.0, 650.0)
        system.close()
        return [T0, r.temperature_K, r.state.cell_net_power_W, r.state.patch_net_power_W,
                [m[k] for k in ("q_total_hot_W_m2", "q_total_cold_W_m2", "q_rad_hot_W_m2", "radiative_fraction_hot",
                                "k_eff_apparent_W_mK")], bool(r.converged)]
    if kind == "statistics":
        a = properties.identify_properties(ph, "x", case["eps"], n_rays=rays)
        b = penetration.penetration_response(ph, "x", case["eps"], n_rays=rays)
        return [a, b]
    scalar, rows = descriptors.all_descriptors(ph)
    return [scalar, [{k: r[k] for k in ("lineal_path", "chord_counts", "pore_chord_cells_mean", "pore_chord_cells_std",
                                        "pore_chord_cells_q95", "all_pore_line_count", "interface_face_count_axis",
                                        "interface_normal_fraction_axis", "lineal_integral_cells")} for r in rows]]


# ---------------------------------------------------------------- binary64 restatement in plain torch


def _patch_table(ph):
    """Patch table in the reference's order: wall patches by (j, k), hot before cold, then the solid-pore faces by
    (cell, face) with faces +x, -x, +y, -y, +z, -z; patches only where the wall cell is pore."""

    s = torch.from_numpy(ph).cuda() == 1
    nx, ny, nz = s.shape
    wall = torch.stack((~s[0], ~s[-1]), dim=-1).reshape(-1).nonzero()[:, 0]
    wsite, wc = wall // 2, wall % 2
    wj, wk = wsite // nz, wsite % nz
    m = torch.zeros((nx, ny, nz, 6), dtype=torch.bool, device="cuda")
    m[:-1, ..., 0] = s[:-1] & ~s[1:]
    m[1:, ..., 1] = s[1:] & ~s[:-1]
    for f, axis, sh in ((2, 1, -1), (3, 1, 1), (4, 2, -1), (5, 2, 1)):
        m[..., f] = s & ~torch.roll(s, sh, axis)
    at = m.reshape(-1).nonzero()[:, 0]
    cell, face = at // 6, at % 6
    inset = 1.0e-9
    o = torch.stack((cell // (ny * nz), (cell // nz) % ny, cell % nz), dim=1).double() + 0.5
    sign = 1.0 - 2.0 * (face % 2).double()
    rows = torch.arange(face.numel(), device="cuda")
    o[rows, face // 2] += sign * (0.5 + inset)
    o[:, 1] = torch.remainder(o[:, 1], ny)
    o[:, 2] = torch.remainder(o[:, 2], nz)
    wo = torch.stack((torch.where(wc == 0, inset, nx - inset), wj + 0.5, wk + 0.5), dim=1).double()
    nw = wall.numel()
    P = nw + face.numel()
    table = torch.full((6 * nx * ny * nz + 2 * ny * nz,), -1, dtype=torch.int64, device="cuda")
    table[at] = torch.arange(nw, P, device="cuda")
    table[6 * nx * ny * nz + wc * ny * nz + wsite] = torch.arange(nw, device="cuda")
    return dict(solid=s, P=P, origin=torch.cat((wo, o)), axis=torch.cat((torch.zeros_like(wc), face // 2)),
                sign=torch.cat((1.0 - 2.0 * wc.double(), sign)), cls=torch.cat((wc, torch.full_like(face, 2))),
                cell=torch.cat((torch.zeros_like(wc), cell)), table=table)


def _trace(pt, p0, p1, R, u):
    """First patch hit by the rays of patches [p0, p1), u the four uniforms of each ray."""

    s = pt["solid"]
    nx, ny, nz = s.shape
    solid = s.reshape(-1)
    ax = pt["axis"][p0:p1].repeat_interleave(R)
    sign = pt["sign"][p0:p1].repeat_interleave(R)
    o = pt["origin"][p0:p1].repeat_interleave(R, dim=0).clone()
    n = ax.numel()
    rows = torch.arange(n, device="cuda")
    first = torch.tensor([1, 0, 0], device="cuda")[ax]
    second = torch.tensor([2, 2, 1], device="cuda")[ax]
    o[rows, first] += u[:, 0].clamp(1e-12, 1 - 1e-12) - 0.5
    o[rows, second] += u[:, 1].clamp(1e-12, 1 - 1e-12) - 0.5
    o[:, 1] = torch.remainder(o[:, 1], ny)
    o[:, 2] = torch.remainder(o[:, 2], nz)
    radius, phi = torch.sqrt(u[:, 2]), (2.0 * math.pi) * u[:, 3]
    d = torch.empty((n, 3), dtype=torch.float64, device="cuda")
    d[rows, ax] = sign * torch.sqrt(1.0 - u[:, 2])
    d[rows, first] = radius * torch.cos(phi)
    d[rows, second] = sign * (radius * torch.sin(phi))
    d = d / torch.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2])[:, None]
    cell = torch.floor(o) - ((d < 0) & ((o - torch.round(o)).abs() <= 1e-12)).double()
    step = torch.sign(d).long()
    tmax = torch.where(d > 0, (cell + 1.0 - o) / d, (cell - o) / d)
    tdel = torch.where(d > 0, 1.0 / d, -1.0 / d)
    zero = d == 0
    tmax[zero] = 1e300
    tdel[zero] = 1e300
    c = cell.long()
    c[:, 1] %= ny
    c[:, 2] %= nz
    out = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    face = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    t = torch.zeros(n, dtype=torch.float64, device="cuda")
    live = rows
    size = torch.tensor([1 << 40, ny, nz], device="cuda")
    for it in range(1 << 20):
        x = c[:, 0]
        wall = (x < 0) | (x >= nx)
        flat = (x.clamp(0, nx - 1) * ny + c[:, 1]) * nz + c[:, 2]
        hit = ~wall & solid[flat]
        done = wall | hit
        if it % 4 == 3 or live.numel() < 1024:
            w = wall.nonzero()[:, 0]
            q = live[w]
            site = torch.remainder(torch.floor(o[q, 1] + d[q, 1] * t[w]).long(), ny) * nz + torch.remainder(
                torch.floor(o[q, 2] + d[q, 2] * t[w]).long(), nz)
            out[q] = pt["table"][6 * nx * ny * nz + (x[w] >= nx).long() * ny * nz + site]
            h = hit.nonzero()[:, 0]
            out[live[h]] = pt["table"][flat[h] * 6 + face[h]]
            keep = (~done).nonzero()[:, 0]
            if keep.numel() == 0:
                return out
            live, c, tmax, tdel, step, face, t = (v[keep] for v in (live, c, tmax, tdel, step, face, t))
            go = torch.ones((keep.numel(), 1), dtype=torch.bool, device="cuda")
        else:
            go = ~done[:, None]
        tn = tmax.min(dim=1, keepdim=True).values
        cross = (tmax - tn <= 1e-12) & go
        a = cross.int().argmax(dim=1)  # the first crossed axis names the face
        f = 2 * a + (step.gather(1, a[:, None])[:, 0] > 0)
        face = torch.where(go[:, 0], f, face)
        t = torch.where(go[:, 0], tn[:, 0], t)
        c = c + step * cross
        c = torch.where(c == size, 0, torch.where((c < 0) & (size < (1 << 40)), size - 1, c))
        tmax = torch.where(cross, tmax + tdel, tmax)
    raise RuntimeError("rays did not end")


def _counts(pt, R, seed):
    """Sorted (origin P + receiver) keys and counts of one seeded ray set."""

    P = pt["P"]
    gen = np.random.Generator(np.random.PCG64(int(seed)))
    keys, cnts = [], []
    per = max(1, 3_000_000 // R)
    for p0 in range(0, P, per):
        p1 = min(P, p0 + per)
        u = torch.from_numpy(gen.random(((p1 - p0) * R, 4))).cuda()
        r = _trace(pt, p0, p1, R, u)
        k, c = torch.unique(torch.arange(p0, p1, device="cuda").repeat_interleave(R) * P + r, return_counts=True)
        keys.append(k)
        cnts.append(c)
    return torch.cat(keys), torch.cat(cnts)


def _pool(tables):
    k, inv = torch.unique(torch.cat([t[0] for t in tables]), return_inverse=True)
    return k, torch.zeros(k.numel(), dtype=torch.int64, device="cuda").scatter_add_(0, inv, torch.cat([t[1] for t in tables]))


class _Operator:
    def __init__(self, pt, table, rays, area, balance=True):
        k, c = table
        P = pt["P"]
        self.P, self.A = P, area
        o, r = k // P, k % P
        w = c.double() / rays
        self.nnz = k.numel()
        self.F = torch.sparse_coo_tensor(torch.stack((o, r)), w, (P, P), is_coalesced=True).to_sparse_csr()
        back, order = torch.sort(r * P + o)
        self.FT = torch.sparse_coo_tensor(torch.stack((back // P, back % P)), w[order], (P, P), is_coalesced=True).to_sparse_csr()
        self.nnz_sym = int(torch.unique(torch.cat((k, back))).numel())
        self.d = torch.ones(P, dtype=torch.float64, device="cuda")
        if balance:
            best, y, kept = math.inf, torch.zeros_like(self.d), 0
            for _ in range(3000):
                d = torch.exp(y)
                row = d * self.S(d) / area
                err = float((row - 1).abs().max())
                if err < best:
                    best, self.d, kept = err, d, 0
                else:
                    kept += 1
                if best < 1e-14 or kept > 20:
                    break
                y = y - 0.5 * torch.log(row)

    def S(self, x):
        return 0.5 * self.A * ((self.F @ x[:, None])[:, 0] + (self.FT @ x[:, None])[:, 0]) + 1e-15 * self.A * x

    def rmatvec(self, x):
        return self.d * self.S(self.d * (x / self.A))

    def absorbed(self, e, eps, tol=1e-16):
        total, flight, ref = torch.zeros_like(e), e.clone(), float(e.abs().sum())
        for _ in range(5000):
            inc = self.rmatvec(flight)
            total += eps * inc
            flight = (1 - eps) * inc
            if float(flight.abs().sum()) <= tol * ref:
                break
        return total


def _operator(case, pt, tables, rays, shape):
    return _Operator(pt, _pool(tables) if len(tables) > 1 else tables[0], rays, (H_M / shape[0]) ** 2)


def _exact_channels(case, pt, op, shape, T_cells, Th, Tc, ref):
    nx, ny, nz = shape
    T = torch.where(pt["cls"] == 0, Th, torch.where(pt["cls"] == 1, Tc, T_cells.reshape(-1)[pt["cell"]]))
    eps = case["eps"]
    e = eps * SIGMA * op.A * ((T - ref) * (T + ref) * (T * T + ref * ref))
    net = op.absorbed(e, eps) - e
    xs = ny * nz * (H_M / nx) ** 2
    q = [-float(net[pt["cls"] == c].sum()) / xs for c in range(3)]
    power = torch.zeros(nx * ny * nz, dtype=torch.float64, device="cuda")
    inner = pt["cls"] == 2
    power.index_add_(0, pt["cell"][inner], net[inner])
    coarse = power.reshape(shape).cpu().numpy()
    for axis, n in enumerate(shape):
        b = min(8, n)
        sizes = [n // b + (1 if j < n % b else 0) for j in range(b)]
        coarse = np.add.reduceat(coarse, np.cumsum([0] + sizes[:-1]), axis=axis)
    return [*q, coarse / xs]


def _line(shape, Tm, dT):
    nx = shape[0]
    x = torch.arange(nx, dtype=torch.float64, device="cuda") + 0.5
    return ((Tm + dT / 2) - x * dT / nx)[:, None, None].expand(shape).contiguous()


def _exact_coupled(case, pt, op, ph):
    """Newton on A T - b - Q_rad(T) = 0, corrections by Jacobi-preconditioned BiCGStab."""

    shape = ph.shape
    Th, Tc, eps = 750.0, 650.0, case["eps"]
    k = torch.where(pt["solid"], K_SOLID, K_GAS).double()
    dx = H_M / shape[0]
    g = [2 * k * torch.roll(k, -1, a) / (k + torch.roll(k, -1, a) + 1e-30) * dx for a in range(3)]
    g[0][-1] = 0.0
    hot, cold = torch.zeros_like(k), torch.zeros_like(k)
    hot[0], cold[-1] = 2 * k[0] * dx, 2 * k[-1] * dx
    diag = sum(x + torch.roll(x, 1, a) for a, x in enumerate(g)) + hot + cold
    b = hot * Th + cold * Tc

    def A(T):
        out = diag * T
        for a, x in enumerate(g):
            y = x * torch.roll(T, -1, a)
            out = out - y - torch.roll(x * T, 1, a)
        return out

    inner = pt["cls"] == 2
    owner = pt["cell"][inner]

    def cells(net):
        p = torch.zeros(k.numel(), dtype=torch.float64, device="cuda")
        return p.index_add_(0, owner, net[inner]).reshape(shape)

    def net(e, tol):
        return op.absorbed(e, eps, tol) - e

    def patch_T(T):
        return torch.where(pt["cls"] == 0, Th, torch.where(pt["cls"] == 1, Tc, T.reshape(-1)[pt["cell"]]))

    def solve(J, rhs, inv, tol):
        x = torch.zeros_like(rhs)
        r = rhs.clone()
        r0, rho, alpha, om = r.clone(), 1.0, 1.0, 1.0
        v, p = torch.zeros_like(r), torch.zeros_like(r)
        stop = tol * float(rhs.norm())
        for _ in range(2000):
            rho1 = float((r0 * r).sum())
            p = r + (rho1 / rho) * (alpha / om) * (p - om * v)
            y = inv * p
            v = J(y)
            alpha = rho1 / float((r0 * v).sum())
            s = r - alpha * v
            z = inv * s
            t = J(z)
            om = float((t * s).sum()) / max(float((t * t).sum()), 1e-300)
            x = x + alpha * y + om * z
            r, rho = s - om * t, rho1
            if float(r.norm()) <= stop:
                break
        return x

    T0 = solve(A, b - A(_line(shape, 700.0, 100.0)), 1 / diag, 1e-14) + _line(shape, 700.0, 100.0)
    T = T0
    for step in range(6):
        Tp = patch_T(T)
        e = eps * SIGMA * op.A * Tp**4
        R = A(T) - b - cells(net(e, 1e-15))
        slope = torch.where(inner, 4 * eps * SIGMA * op.A * Tp**3, 0.0)

        def J(x):
            return A(x) - cells(net(slope * x.reshape(-1)[pt["cell"]], 1e-12))

        shift = torch.zeros(k.numel(), dtype=torch.float64, device="cuda").index_add_(0, owner, slope[inner]).reshape(shape)
        dT = solve(J, -R, 1 / (diag + shift), 1e-9)
        T = T + dT
        if float(dT.abs().max()) < 1e-10:
            break
    n = net(eps * SIGMA * op.A * patch_T(T)**4, 1e-16)
    xs = shape[1] * shape[2] * dx * dx
    qch, qcc = float((2 * k[0] * (Th - T[0]) / dx).mean()), float((2 * k[-1] * (T[-1] - Tc) / dx).mean())
    qrh, qrc = -float(n[pt["cls"] == 0].sum()) / xs, float(n[pt["cls"] == 1].sum()) / xs
    th = qch + qrh
    return [T0, T, cells(n), n, [th, qcc + qrc, qrh, qrh / th, th * H_M / 100.0], None]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("counts", "statistics"):
        return None  # whole numbers, and statistics of a hashed ray stream
    phases = _phases(case, seed)
    ph = phases[0]
    if kind == "morphology":
        s = ph == 1
        area = sum(int(np.count_nonzero(np.diff(s, axis=a))) for a in range(3))
        per = [int(np.count_nonzero(s != np.roll(s, -1, a))) for a in range(3)]
        runs = [int(np.count_nonzero(~np.moveaxis(s, a, 0)[0]))
                + int(np.count_nonzero(np.diff((~np.moveaxis(s, a, 0)).astype(np.int8), axis=0) == 1)) for a in range(3)]
        pore = int((~s).sum())
        scalar = dict(phi_solid=float(s.mean()), interfacial_area_density=area / s.size, mean_beam_length=4.0 * pore / area,
                      mean_pore_chord=tuple(pore / r for r in runs), pore_percolates=None, pore_largest_cluster_fraction=None)
        return [scalar, [dict(interface_normal_fraction_axis=f / sum(per)) for f in per]]
    cells = math.prod(_shape(case))
    if _patches(case) * case["rays"] * cells ** (1 / 3) * {"sets": 2, "arrays": 2, "sweep": 2 * case.get("count", 1)}.get(kind, 1) > 3.5e10:
        return None
    seeds = _ray_seeds(seed, 2 * max(1, case.get("count", 1)))
    R, shape = case["rays"], ph.shape
    if kind == "sweep":
        out = []
        for k, x in enumerate(phases):
            pt = _patch_table(x)
            op = _operator(case, pt, [_counts(pt, R, q) for q in seeds[2 * k:2 * k + 2]], 2 * R, shape)
            q = _exact_channels(case, pt, op, shape, _line(shape, 700.0, 100.0), 750.0, 650.0, 700.0)
            out.append([op.d, np.array(q[:3]), q[3]])
        return out
    pt = _patch_table(ph)
    if kind in ("sets", "arrays"):
        a, b = (_counts(pt, R, q) for q in seeds[:2])
    if kind == "sets":
        out = []
        for tables, r in (([a], R), ([b], R), ([a, b], 2 * R)):
            op = _operator(case, pt, tables, r, shape)
            out.append([None, None, op.d, *_exact_channels(case, pt, op, shape, _line(shape, 700.0, 100.0), 750.0, 650.0, 700.0)])
        return out
    if kind == "arrays":
        op = _operator(case, pt, [a, b], 2 * R, shape)
        return [None, None, op.d, *_exact_channels(case, pt, op, shape, _line(shape, 650.0, 20.0), 660.0, 640.0, 650.0)]
    op = _operator(case, pt, [_counts(pt, R, seeds[0])], R, shape)
    if kind == "fields":
        return [_exact_channels(case, pt, op, shape, T, 710.0, 690.0, 700.0) for T in _fields(case, seed)]
    if kind == "coupled":
        return _exact_coupled(case, pt, op, ph)
    v = {k: torch.from_numpy(x).cuda() for k, x in _vectors(case, seed, pt["P"]).items()}
    if kind == "products":
        x, d, A = v["x"], op.d, op.A
        return [(d / A) * op.S(d * x), d * op.S(d * (x / A)), op.S(x), (op.F @ x[:, None])[:, 0], (op.FT @ x[:, None])[:, 0]]
    T, eps, A = v["T"], v["eps"], op.A
    e = eps * SIGMA * A * ((T - 700.0) * (T + 700.0) * (T * T + 700.0 * 700.0))
    f = eps * SIGMA * A * T**4
    g = 4.0 * eps * SIGMA * A * T**3 * v["dT"]
    a, b = op.absorbed(e, eps), op.absorbed(f, eps)
    return [e, a, a - e, f, b, op.absorbed(g, eps) - g]

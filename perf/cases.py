"""The ray-shooting work a program has this library do, as cases that can be timed and checked.

Every case goes through the Python classes of ``slsimlib_b200``: lenses of particle planes (simulation haloes),
alone or with an NSIE galaxy or field-halo planes, shot by grid or by lists of rays, in the plain FP64 form (the
classes' default) or the split form (the batch's and the server's default); bare trees; many lenses in one launch;
a resident server; and the adaptive smoothing that precedes a particle lens.

``exact`` restates the same quantities in 64 bits with plain torch: the quadtree of the particles (midpoint boxes,
monopole + quadrupole cells, B-spline softening) and the multi-plane recursion.
"""
import math

import numpy as np
import torch

import slsimlib_b200 as glb

ARCSEC = 0.000004848136811
GRAV = 4.7788e-20  # G / c^2 in Mpc / Msun
CLIGHT = 2.99792458e5
PRECISION = {"fp64": glb.PREC_FP64, "split": glb.PREC_SPLIT, "fp32": glb.PREC_FP32}


# ------------------------------------------------------------------ cases
def listed():
    return [
        # An image finder follows one image: 9 x 9 rays around it through the full light cone, one call at a time.
        {"name": "rays-81", "kind": "rays", "precision": "fp64", "rays": 81, "planes": 10, "particles": 4194304,
         "size_kpc": 0.5, "spread": 0.5, "own_zs": False},
        # A refinement round of a critical-curve search: a few thousand rays near the curve, each with its own
        # source redshift (the RAY overload).
        {"name": "refine-4097", "kind": "rays", "precision": "fp64", "rays": 4097, "planes": 10, "particles": 4194304,
         "size_kpc": 0.5, "spread": 4.0, "own_zs": True},
        # The map of one simulated cluster: 512^2 GridMap over 2^18 particles, the classes' default precision.
        {"name": "cluster-512-fp64", "kind": "grid", "precision": "fp64", "side": 512, "planes": 1, "particles": 262144,
         "size_kpc": 1.0, "arcsec": 30.0},
        # The same map in the split form.
        {"name": "cluster-512-split", "kind": "grid", "precision": "split", "side": 512, "planes": 1, "particles": 262144,
         "size_kpc": 1.0, "arcsec": 30.0},
        # A light cone at reference precision on an odd grid.
        {"name": "cone-511-fp64", "kind": "grid", "precision": "fp64", "side": 511, "planes": 10, "particles": 1048576,
         "size_kpc": 0.5, "arcsec": 60.0},
        # The benchmark's light cone: 10 planes, 4,194,304 particles, an NSIE galaxy, 2048^2 rays kept on the device.
        {"name": "cone-2048-split", "kind": "device", "precision": "split", "side": 2048, "planes": 10,
         "particles": 4194304, "size_kpc": 0.5, "arcsec": 60.0},
        # Light cone with field planes of NFW and NSIE haloes between the particle planes (LensPlaneTree).
        {"name": "field-384-fp64", "kind": "field", "precision": "fp64", "side": 384, "planes": 5, "particles": 524288,
         "size_kpc": 0.5, "arcsec": 60.0, "members": 404},
        # A new snapshot: its tree built from host records, then forces and potential at a ragged list of positions.
        {"name": "tree-65537", "kind": "tree", "precision": "fp64", "rays": 65537, "particles": 1048576, "size_kpc": 1.0,
         "theta": 0.1, "bucket": 5, "arcsec": 120.0},
        # The precision sweep's force evaluation on device arrays: a large triaxial cluster, tiled rays.
        {"name": "force-1448-split", "kind": "force", "precision": "split", "side": 1448, "particles": 4194304,
         "size_kpc": 1.0, "theta": 0.1, "bucket": 5, "arcsec": 40.0},
        # Many independent lenses of uneven size in one launch, replayed from its graph.
        {"name": "batch-48", "kind": "batch", "precision": "split", "lenses": 48, "side_min": 64, "side_max": 512,
         "log2_min": 14, "log2_max": 18},
        # Requests of uneven size to a server with resident light cones.
        {"name": "served-16", "kind": "served", "precision": "split", "requests": 16, "rays_min": 1000, "rays_max": 60000,
         "models": 2, "planes": 10, "particles": 524288, "size_kpc": 0.5},
        # A snapshot's softening lengths: Nsmooth-th neighbour distances of 2^20 particles, in place on host records.
        {"name": "smooth-1m", "kind": "smooth", "precision": "fp64", "particles": 1048576, "nsmooth": 64},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["rays", "grid", "grid", "device", "field", "tree", "force", "batch", "served", "smooth"])
    prec = rng.choice(["fp64", "split"])
    size = round(rng.uniform(0.3, 2.0), 2)
    planes = rng.randint(1, 10)
    if kind == "rays":
        return {"kind": kind, "precision": prec, "rays": _log(rng, 1, 60000), "planes": planes,
                "particles": _log(rng, 4000, 2000000), "size_kpc": size, "spread": round(rng.uniform(0.05, 20.0), 2),
                "own_zs": rng.random() < 0.5}
    if kind in ("grid", "device"):
        top = math.sqrt((4.0e6 if prec == "fp64" else 1.2e7) / planes)
        return {"kind": kind, "precision": prec, "side": _log(rng, 33, min(2048, top)), "planes": planes,
                "particles": _log(rng, 4000, 2000000), "size_kpc": size, "arcsec": round(rng.uniform(10.0, 90.0), 1)}
    if kind == "field":
        return {"kind": kind, "precision": prec, "side": _log(rng, 33, 400), "planes": rng.randint(1, 6),
                "particles": _log(rng, 4000, 500000), "size_kpc": size, "arcsec": round(rng.uniform(20.0, 90.0), 1),
                "members": _log(rng, 20, 1000)}
    if kind == "tree":
        return {"kind": kind, "precision": "fp64", "rays": _log(rng, 100, 200000), "particles": _log(rng, 1000, 2000000),
                "size_kpc": size, "theta": rng.choice([0.1, 0.3]), "bucket": rng.choice([1, 5, 20]),
                "arcsec": round(rng.uniform(10.0, 200.0), 1)}
    if kind == "force":
        return {"kind": kind, "precision": rng.choice(["fp64", "split", "split", "fp32"]), "side": _log(rng, 100, 1400),
                "particles": _log(rng, 4000, 4000000), "size_kpc": size, "theta": rng.choice([0.1, 0.2, 0.3]),
                "bucket": rng.choice([5, 20]), "arcsec": round(rng.uniform(10.0, 100.0), 1)}
    if kind == "batch":
        return {"kind": kind, "precision": prec, "lenses": rng.randint(4, 32), "side_min": 32,
                "side_max": rng.randint(64, 320), "log2_min": 12, "log2_max": 17}
    if kind == "served":
        return {"kind": kind, "precision": prec, "requests": rng.randint(1, 16), "rays_min": 100,
                "rays_max": _log(rng, 1000, 40000), "models": rng.randint(1, 2), "planes": rng.randint(1, 6),
                "particles": _log(rng, 20000, 500000), "size_kpc": size}
    return {"kind": kind, "precision": "fp64", "particles": _log(rng, 2000, 2000000), "nsmooth": rng.choice([16, 32, 64, 100])}


# ----------------------------------------------------------------- inputs
_NODES, _WEIGHTS = np.polynomial.legendre.leggauss(64)


def _distance(z):
    """Comoving distance in Mpc, flat LambdaCDM (0.3, 0.7, h = 0.7)."""
    zz = 0.5 * z * (_NODES + 1.0)
    return float(CLIGHT / 70.0 * 0.5 * z * np.sum(_WEIGHTS / np.sqrt(0.3 * (1 + zz) ** 3 + 0.7)))


def _r200(m, z):
    h = 70.0 * math.sqrt(0.3 * (1 + z) ** 3 + 0.7)
    rho = 3 * h * h / (8 * math.pi * 4.30091727e-9)
    return (3 * m / (4 * math.pi * 200 * rho)) ** (1.0 / 3.0)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed, stream):
    g = torch.Generator(device=_device())
    g.manual_seed((int(seed) * 1000003 + stream * 7919 + 17) % (1 << 62))
    return g


def _nfw(g, masses, counts, z, centres, c=5.0, axes=(1.0, 1.0, 1.0)):
    """Positions (n, 3) in Mpc of particles sampling NFW haloes of the given masses, counts and centres."""
    dev = _device()
    x = torch.linspace(0, c, 8193, dtype=torch.float64, device=dev)
    m = torch.log1p(x) - x / (1 + x)
    n = int(sum(counts))
    u = torch.rand(n, generator=g, dtype=torch.float64, device=dev) * m[-1]
    j = torch.searchsorted(m, u).clamp(1, 8192)
    r = x[j - 1] + (u - m[j - 1]) / (m[j] - m[j - 1]) * (x[j] - x[j - 1])
    rs = torch.tensor([_r200(float(q), z) / c for q in masses], dtype=torch.float64, device=dev)
    own = torch.repeat_interleave(torch.arange(len(counts), device=dev), torch.tensor(counts, device=dev))
    r = r * rs[own]
    mu = torch.rand(n, generator=g, dtype=torch.float64, device=dev) * 2 - 1
    ph = torch.rand(n, generator=g, dtype=torch.float64, device=dev) * (2 * math.pi)
    s = torch.sqrt(1 - mu * mu)
    out = torch.stack([r * s * torch.cos(ph), r * s * torch.sin(ph), r * mu], 1)
    scale = (axes[0] * axes[1] * axes[2]) ** (-1.0 / 3.0)
    out *= torch.tensor(axes, dtype=torch.float64, device=dev) * scale
    out[:, :2] += torch.tensor(np.asarray(centres), dtype=torch.float64, device=dev)[own]
    return out


def _records(pos, mass, size):
    p = np.zeros(len(pos), dtype=glb.PARTICLE_DTYPE)
    p["x"] = pos.to(torch.float32).cpu().numpy()
    p["Mass"] = np.float32(mass)
    p["Size"] = np.float32(size)
    return p


def _plane(seed, stream, n, z, arcsec, size_kpc, halos):
    """Particle records of one plane: `halos` NFW haloes (1e12-1e14 Msun) over the field, equal particle mass; one
    halo is a 1e14 Msun cluster in the middle."""
    r = np.random.default_rng([int(seed) % (1 << 32), stream])
    half = 0.5 * arcsec * ARCSEC * _distance(z) / (1 + z)
    masses = 10 ** r.uniform(12, 14, halos) if halos > 1 else np.array([1e14])
    centres = r.uniform(-half, half, (halos, 2)) if halos > 1 else np.zeros((1, 2))
    counts = np.floor(n * masses / masses.sum()).astype(np.int64)
    counts[np.argmax(counts)] += n - counts.sum()
    pos = _nfw(_generator(seed, stream), masses, counts.tolist(), z, centres)
    return _records(pos, masses.sum() / n, size_kpc * 1e-3)


def _planes(case, seed, stream=0):
    """[(z, records)] of a case's particle planes: one cluster at z = 0.3, or a light cone of z = 0.1, 0.3, ..."""
    k = case["planes"]
    arcsec = case.get("arcsec", 60.0)
    if k == 1:
        return [(0.3, _plane(seed, stream, case["particles"], 0.3, arcsec, case["size_kpc"], 1))]
    each = case["particles"] // k
    return [(0.1 + 0.2 * i, _plane(seed, stream + i, max(64, each), 0.1 + 0.2 * i, arcsec, case["size_kpc"], 32))
            for i in range(k)]


def _zsource(case):
    return 2.0 if case["planes"] == 1 else 2.5


def _lens(planes, zsource):
    lens = glb.Lens(zsource)
    for z, p in planes:
        lens.insertMainHalo(glb.LensHaloParticles(p, z), True)
    return lens


def _grid(n, range_rad):
    i = np.arange(n * n)
    return np.stack([range_rad * (1.0 * (i % n) / (n - 1) - 0.5), range_rad * (1.0 * (i // n) / (n - 1) - 0.5)], axis=1)


def _tiled(n):
    """Row-major indices of an n x n grid in 8 x 4 tiles (neighbouring rays side by side)."""
    i = np.arange(n * n).reshape(n, n)
    iy, ix = np.divmod(i, n)
    return np.lexsort((ix.ravel(), iy.ravel(), (ix // 8).ravel(), (iy // 4).ravel()))


def _blob_rays(case, seed):
    """Ray positions of a refinement round: a Gaussian blob of `spread` arcsec in the field; own source redshifts."""
    r = np.random.default_rng([int(seed) % (1 << 32), 77])
    x = r.uniform(-10, 10, 2) * ARCSEC + r.normal(0, case["spread"] * ARCSEC, (case["rays"], 2))
    return x, (r.uniform(1.0, 3.0, case["rays"]) if case["own_zs"] else None)


def _tree_inputs(case, seed):
    """A cluster's records (1e15 Msun, triaxial, a tenth as uniform background) and its plane positions (Mpc)."""
    n = case["particles"]
    nb = n // 11
    g = _generator(seed, 5)
    pos = _nfw(g, [1e15], [n - nb], 0.3, np.zeros((1, 2)), c=4.0, axes=(1.0, 0.8, 0.6))
    lo, hi = pos.min(0).values, pos.max(0).values
    back = torch.rand((nb, 3), generator=g, dtype=torch.float64, device=_device()) * (hi - lo) + lo
    p = _records(torch.cat([pos, back]), 1e15 / max(1, n - nb), case["size_kpc"] * 1e-3)
    da = _distance(0.3) / 1.3
    if case["kind"] == "force":
        rays = _grid(case["side"], case["arcsec"] * ARCSEC * da)[_tiled(case["side"])]
    else:
        r = np.random.default_rng([int(seed) % (1 << 32), 78])
        rays = r.normal(0, 0.25 * case["arcsec"] * ARCSEC * da, (case["rays"], 2))
    return p, np.ascontiguousarray(rays)


def _batch_inputs(case, seed):
    """[(side, zsource, planes)]: lenses of one or three planes, sizes log-uniform, 30 arcsec wide."""
    r = np.random.default_rng([int(seed) % (1 << 32), 79])
    out = []
    for i in range(case["lenses"]):
        # the i-th lens's sizes are the case's, so that every seed has the same work; its particles are the seed's
        f = (i * 0.6180339887) % 1.0
        h = (i * 0.7548776662) % 1.0
        side = int(round(case["side_min"] * (case["side_max"] / case["side_min"]) ** f))
        n = int(2 ** (case["log2_min"] + (case["log2_max"] - case["log2_min"]) * h))
        c = {"planes": 3 if i % 3 == 2 else 1, "particles": n, "size_kpc": 1.0, "arcsec": 30.0}
        out.append((side, float(r.uniform(1, 3)), _planes(c, seed, 1000 + 16 * i)))
    return out


def _requests(case, seed):
    """[(model, rays, zs)]: Gaussian blobs over the field, request sizes log-uniform."""
    r = np.random.default_rng([int(seed) % (1 << 32), 80])
    out = []
    for i in range(case["requests"]):
        f = (i * 0.6180339887 + 0.3) % 1.0
        n = int(round(case["rays_min"] * (case["rays_max"] / case["rays_min"]) ** f))
        nb = int(r.integers(1, 9))
        cen = r.uniform(-30, 30, (nb, 2)) * ARCSEC
        sig = 10 ** r.uniform(math.log10(0.05), 0) * ARCSEC
        out.append((i % case["models"], cen[r.integers(0, nb, n)] + r.normal(0, sig, (n, 2)), float(r.uniform(1, 3))))
    return out


def _members(case, seed, stream, z):
    """Field haloes of one plane: NFW (1e10-1e13 Msun) and one NSIE in a hundred over the field."""
    r = np.random.default_rng([int(seed) % (1 << 32), 81, stream])
    half = 0.5 * case["arcsec"] * ARCSEC
    out = []
    for i in range(case["members"]):
        if i % 101 == 100:
            h = glb.LensHaloRealNSIE(10 ** r.uniform(12, 13), z, r.uniform(150, 250), r.uniform(5e-5, 2e-4),
                                     r.uniform(0.6, 0.9), r.uniform(0, math.pi))
        else:
            m = 10 ** r.uniform(10, 13)
            h = glb.LensHaloNFW(m, _r200(m, z), z, 5.0 * (m / 1e14) ** -0.1)
        h.setTheta(*r.uniform(-half, half, 2))
        out.append(h)
    return out


_streams = {}


def _stream():
    """The program's stream for device-array calls."""
    if "s" not in _streams:
        _streams["s"] = torch.cuda.Stream()
    return _streams["s"]


def _snapshot(case, seed):
    n = case["particles"]
    r = np.random.default_rng([int(seed) % (1 << 32), 82])
    k = 8
    masses = 10 ** r.uniform(12, 14.5, k)
    counts = np.floor(n * masses / masses.sum()).astype(np.int64)
    counts[np.argmax(counts)] += n - counts.sum()
    pos = _nfw(_generator(seed, 9), masses, counts.tolist(), 0.3, r.uniform(-2, 2, (k, 2)))
    return _records(pos, masses.sum() / n, 0.0)


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "precision": PRECISION[case["precision"]]}
    if kind == "rays":
        st["lens"] = _lens(_planes(case, seed), _zsource(case))
        st["x"], st["zs"] = _blob_rays(case, seed)
    elif kind in ("grid", "device", "field"):
        lens = _lens(_planes(case, seed), _zsource(case))
        if kind == "device":
            zl = 0.5
            lens.insertMainHalo(glb.LensHaloRealNSIE(1e13, zl, 250.0, 0.05 * ARCSEC * _distance(zl) / (1 + zl), 0.7, 0.0), True)
            n = case["side"] ** 2
            st["x"] = torch.from_numpy(_grid(case["side"], case["arcsec"] * ARCSEC)).cuda()
            st["y"] = torch.empty((n, 2), dtype=torch.float64, device="cuda")
            st["A"] = torch.empty((n, 4), dtype=torch.float64, device="cuda")
            _stream().wait_stream(torch.cuda.current_stream())
        if kind == "field":
            for i in range(case["planes"]):
                z = 0.2 + 0.2 * i
                lens.insertFieldPlane(glb.LensPlaneTree(z, _members(case, seed, i, z)))
        st["lens"] = lens
    elif kind == "tree":
        st["particles"], st["x"] = _tree_inputs(case, seed)
    elif kind == "force":
        p, rays = _tree_inputs(case, seed)
        st["tree"] = glb.TreeQuadParticles(p, bucket=case["bucket"], theta_force=case["theta"])
        st["x"] = torch.from_numpy(rays).cuda()
        st["out"] = torch.empty((len(rays), 5), dtype=torch.float64, device="cuda")
        _stream().wait_stream(torch.cuda.current_stream())
    elif kind == "batch":
        specs = _batch_inputs(case, seed)
        st["batch"] = glb.GridBatch([_lens(p, zs) for _, zs, p in specs], [s for s, _, _ in specs],
                                    [(0.0, 0.0)] * len(specs), [30.0 * ARCSEC] * len(specs), st["precision"])
    elif kind == "served":
        models = [_lens(_planes(case, seed, 100 * m), _zsource(case)) for m in range(case["models"])]
        st["server"] = glb.Server(models, max_rays_per_batch=2_000_000, precision=st["precision"])
        st["requests"] = _requests(case, seed)
    else:
        st["particles"] = _snapshot(case, seed)
    return st


def run(st):
    case, prec = st["case"], st["precision"]
    kind = case["kind"]
    if kind == "rays":
        return st["lens"].rayshooterInternal(st["x"], st["zs"], precision=prec)
    if kind in ("grid", "field"):
        g = glb.GridMap(st["lens"], case["side"], (0.0, 0.0), case["arcsec"] * ARCSEC, prec)
        return g.y, g.A
    if kind == "device":
        st["lens"].rayshoot_device(len(st["x"]), st["x"].data_ptr(), None, st["y"].data_ptr(), st["A"].data_ptr(), prec,
                                   _stream().cuda_stream)
        return st["y"], st["A"]
    if kind == "tree":
        tree = glb.TreeQuadParticles(st["particles"], bucket=case["bucket"], theta_force=case["theta"])
        return tree.force2D_recur(st["x"])
    if kind == "force":
        st["tree"].force_device(len(st["x"]), st["x"].data_ptr(), st["out"].data_ptr(), prec, _stream().cuda_stream)
        return st["out"]
    if kind == "batch":
        st["batch"].run()
        got = [st["batch"].result(i) for i in range(case["lenses"])]
        return np.concatenate([y for y, _ in got]), np.concatenate([a for _, a in got])
    if kind == "served":
        tickets = [st["server"].submit(m, x, zs) for m, x, zs in st["requests"]]
        got = [st["server"].wait(t) for t in tickets]
        return np.concatenate([g[0] for g in got]), np.concatenate([g[1] for g in got])
    glb.calculate_smoothing(case["nsmooth"], st["particles"])
    return st["particles"]["Size"]


# ------------------------------------------------------------------- work
def _per_ray(n, theta, bucket):
    """Cells and particles that one ray meets in a tree of n particles (estimates: annuli of cells level by level)."""
    levels = max(1.0, math.log(max(n / bucket, 4.0), 4.0))
    cells = min(n / bucket, 400.0 * (0.1 / theta) ** 2 * levels)
    return cells, min(n, 200.0 * bucket * (0.1 / theta) ** 2)


def work(case):
    """Records and rays read once, results written once; 60 flops a far cell and 29 a particle for every ray and plane."""
    kind = case["kind"]
    if kind == "smooth":
        n, k = case["particles"], case["nsmooth"]
        return {"bytes": 28.0 * n, "flops": 8.0 * 8 * (k + 1) * n}
    if kind == "batch":
        b = f = 0.0
        for i in range(case["lenses"]):
            u, h = (i * 0.6180339887) % 1.0, (i * 0.7548776662) % 1.0
            rays = round(case["side_min"] * (case["side_max"] / case["side_min"]) ** u) ** 2
            n = 2 ** (case["log2_min"] + (case["log2_max"] - case["log2_min"]) * h)
            k = 3 if i % 3 == 2 else 1
            cells, parts = _per_ray(n / k, 0.1, 20)
            b += 24.0 * n + 48.0 * rays
            f += rays * k * (60 * cells + 29 * parts)
        return {"bytes": b, "flops": f}
    planes = case.get("planes", 1)
    if kind == "served":
        rays = sum(round(case["rays_min"] * (case["rays_max"] / case["rays_min"]) ** ((i * 0.6180339887 + 0.3) % 1.0))
                   for i in range(case["requests"]))
    else:
        rays = case["rays"] if "rays" in case else case["side"] ** 2
    cells, parts = _per_ray(case["particles"] / planes, case.get("theta", 0.1), case.get("bucket", 20))
    f = rays * planes * (60 * cells + 29 * parts)
    if kind == "field":
        f += rays * planes * 60.0 * case["members"]
    return {"bytes": 24.0 * case["particles"] + 64.0 * rays, "flops": float(f)}


# ------------------------------------------------------------------ exact
class _Quadtree:
    """The particles' quadtree in 64 bits: square root box, midpoint quarters down to `bucket` particles, cells opened
    within max(1.1547 rcom / theta, sqrt(5.83) width), particles softened in the cell whose half width they exceed."""

    def __init__(self, rec, bucket, theta, screen2):
        dev = _device()
        x = torch.from_numpy(np.ascontiguousarray(rec["x"][:, 0])).to(dev).double()
        y = torch.from_numpy(np.ascontiguousarray(rec["x"][:, 1])).to(dev).double()
        m = torch.from_numpy(np.ascontiguousarray(rec["Mass"])).to(dev).double()
        h = torch.from_numpy(np.ascontiguousarray(rec["Size"])).to(dev).double()
        self.x, self.y, self.m, self.h, self.screen2 = x, y, m, h, screen2
        n = len(x)
        lo = [float(x.min()), float(y.min())]
        w = max(float(x.max()) - lo[0], float(y.max()) - lo[1])
        cell = torch.zeros(n, dtype=torch.long, device=dev)  # the particles' cell at this level, of this level's
        live = torch.arange(n, device=dev)
        bx, by = torch.tensor([lo[0]], dtype=torch.float64, device=dev), torch.tensor([lo[1]], dtype=torch.float64, device=dev)
        bX, bY = bx + w, by + w
        if float(x.max()) - lo[0] <= float(y.max()) - lo[1]:
            bY = torch.full_like(bY, float(y.max()))
            bX = bx + (bY - by)
        else:
            bX = torch.full_like(bX, float(x.max()))
            bY = by + (bX - bx)
        self.levels = []
        last = None  # the cell a walk through the fourth children ends in
        level, last_cell = 0, 0
        while True:
            nc = len(bx)
            cnt = torch.bincount(cell, minlength=nc)
            px, py, pm = x[live], y[live], m[live]
            z = lambda v: torch.zeros(nc, dtype=torch.float64, device=dev).index_add_(0, cell, v)  # noqa: E731
            mass, absm = z(pm), z(pm.abs())
            cx, cy = z(pm.abs() * px) / absm, z(pm.abs() * py) / absm
            dx, dy = px - cx[cell], py - cy[cell]
            sxx, syy, sxy = z(pm * dx * dx), z(pm * dy * dy), z(pm * dx * dy)
            wid = bX - bx
            rcom2 = torch.maximum((cx - bx) ** 2, (cx - bX) ** 2) + torch.maximum((cy - by) ** 2, (cy - bY) ** 2)
            near2 = 5.83 * wid * wid
            open2 = torch.maximum((1.15470 * torch.sqrt(rcom2) / theta) ** 2, near2)
            inner = cnt > bucket
            L = {"cx": cx, "cy": cy, "mass": mass, "q0": syy - sxx, "q2": -2 * sxy, "open2": open2, "near2": near2,
                 "wid": wid, "inner": inner, "cnt": cnt}
            if last is None and last_cell is not None and not bool(inner[last_cell]):
                last = tuple(float(L[k][last_cell]) if int(cnt[last_cell]) else 0.0 for k in ("mass", "q0", "q2"))
            # particles of the leaves, padded to `bucket`, and the inner cells' softened particles
            order = torch.argsort(cell, stable=True)
            start = torch.cumsum(cnt, 0) - cnt
            leaf = (~inner) & (cnt > 0)
            slot = torch.full((nc,), -1, dtype=torch.long, device=dev)
            slot[leaf] = torch.arange(int(leaf.sum()), device=dev)
            pad = torch.arange(bucket, device=dev)
            at = start[leaf][:, None] + pad[None]
            have = pad[None] < cnt[leaf][:, None]
            L["slot"], L["parts"], L["have"] = slot, live[order[at.clamp(max=len(order) - 1)]], have
            hp, hw = h[live], wid[cell]
            big = inner[cell] & (hp > hw / 2) & ((hp <= hw) if level else torch.ones_like(hp, dtype=torch.bool))
            if bool(big.any()):
                b = order[big[order]]
                L["bigs"], L["nbig"] = live[b], torch.bincount(cell[b], minlength=nc)
                L["big0"] = torch.cumsum(L["nbig"], 0) - L["nbig"]
            self.levels.append(L)
            if not bool(inner.any()):
                break
            rank = torch.cumsum(inner.long(), 0) - 1
            L["child"] = 4 * rank
            if last_cell is not None:
                last_cell = int(4 * rank[last_cell] + 3) if bool(inner[last_cell]) else None
            mx, my = (bx + bX) / 2, (by + bY) / 2
            keep = inner[cell]
            live, c = live[keep], cell[keep]
            q = (x[live] <= mx[c]).long() + 2 * (y[live] <= my[c]).long()
            cell = 4 * rank[c] + q
            ax, aX, ay, aY, mx, my = bx[inner], bX[inner], by[inner], bY[inner], mx[inner], my[inner]
            bx = torch.stack([mx, ax, mx, ax], 1).reshape(-1)
            bX = torch.stack([aX, mx, aX, mx], 1).reshape(-1)
            by = torch.stack([my, my, ay, ay], 1).reshape(-1)
            bY = torch.stack([aY, aY, my, my], 1).reshape(-1)
            level += 1
        self.phi = last

    def _spline(self, f, ray, x0, x1, rr, m, h):
        """The softening correction of particles within two sizes."""
        k = rr < 4 * h * h
        ray, x0, x1, m, h = ray[k], x0[k], x1[k], m[k], h[k]
        r = torch.sqrt(rr[k])
        q = r / h
        s = (8 - 12 * q + 6 * q ** 2 - q ** 3) / 4
        far = q > 1
        c = 10 / (7 * math.pi) / (h * h)
        sig = torch.where(far, s * c, c * (s - 1 + 3 * q - 3 * q ** 2 + q ** 3))
        M = torch.where(far, (-1 + 20 * q ** 2 * (1 - q + 3 * q ** 2 / 8 - q ** 3 / 20)) / 7,
                        10 * q ** 2 * (1 - 3 * q / 4 + 3 * q ** 3 / 10) / 7)
        k0 = (120 * math.log(2.0) - 631.0) / 840 + 19.0 / 70
        phi = torch.where(far, (-1232.0 + 1200 * q ** 2 - 800 * q ** 3 + 225 * q ** 4 - 24 * q ** 5 + 120 * torch.log(2 / q)) / 840,
                          k0 + 10 * (q ** 2 / 2 - 3 * q ** 4 / 4 + 3 * q ** 5 / 50) / 7) - torch.log(r)
        a = (M - 1) / math.pi / r
        gt = a / r - sig
        f.index_add_(0, ray, torch.stack([-m * a * x0 / r, -m * a * x1 / r, m * sig, -gt * m * (x0 * x0 - x1 * x1) / r ** 2,
                                          -gt * m * 2 * x0 * x1 / r ** 2, m * phi / math.pi], 1))

    def _spread(self, start, count):
        own = torch.repeat_interleave(torch.arange(len(count), device=count.device), count)
        return own, start[own] + torch.arange(len(own), device=count.device) - (torch.cumsum(count, 0) - count)[own]

    def force(self, rx, ry):
        """(n, 6): deflection (pointing to the ray), kappa, shear, potential as the walk sums them."""
        out = torch.zeros((len(rx), 6), dtype=torch.float64, device=rx.device)
        for a in range(0, len(rx), 16384):
            self._force(rx[a:a + 16384], ry[a:a + 16384], out[a:a + 16384])
        return out

    def _force(self, rx, ry, f):
        pi, s2 = math.pi, self.screen2
        ray = torch.arange(len(rx), device=rx.device)
        cell = torch.zeros_like(ray)
        pm, pq0, pq2 = self.phi
        for i, L in enumerate(self.levels):
            dx, dy = L["cx"][cell] - rx[ray], L["cy"][cell] - ry[ray]
            r2 = dx * dx + dy * dy
            opened = r2 < L["open2"][cell]
            k = ~opened
            fx, fy, g, c, fr = dx[k], dy[k], r2[k], cell[k], ray[k]
            scr = torch.exp(-g * s2) / pi
            m, q0, q2 = L["mass"][c], L["q0"][c], L["q2"][c]
            t = -m / g * scr + 4 * (q0 * (fx * fx - fy * fy) + 2 * q2 * fx * fy) / g ** 3 * scr
            i4 = scr / (g * g)
            f.index_add_(0, fr, torch.stack([
                t * fx - (q0 * fx + q2 * fy) * i4, t * fy - (q2 * fx - q0 * fy) * i4, torch.zeros_like(t),
                -m * i4 * (fx * fx - fy * fy), -2 * m * i4 * fx * fy,
                0.5 * pm * torch.log(g) * scr - 0.5 * (pq0 * (fx * fx - fy * fy) + 2 * pq2 * fx * fy) * i4], 1))
            ray, cell, r2 = ray[opened], cell[opened], r2[opened]
            near = r2 < L["near2"][cell]
            leaf = ~L["inner"][cell]
            s, lr, ln, lw = L["slot"][cell[leaf]], ray[leaf], near[leaf], L["wid"][cell[leaf]]
            for a in range(0, len(s), 1 << 20):
                b = slice(a, a + (1 << 20))
                p, ok = L["parts"][s[b]], L["have"][s[b]]
                x0, x1 = self.x[p] - rx[lr[b]][:, None], self.y[p] - ry[lr[b]][:, None]
                rr = x0 * x0 + x1 * x1
                scr = torch.exp(-rr * s2)
                rr = rr.clamp(min=1e-20)
                pre = torch.where(ok, self.m[p], 0.0) * scr / rr / pi
                f.index_add_(0, lr[b], torch.stack([(-pre * x0).sum(1), (-pre * x1).sum(1), torch.zeros_like(lw[b]),
                                                    (-pre / rr * (x0 * x0 - x1 * x1)).sum(1), (-2 * pre / rr * x0 * x1).sum(1),
                                                    (0.5 * pre * rr * torch.log(rr)).sum(1)], 1))
                k = ok & ln[b][:, None] & (self.h[p] < lw[b][:, None]) & (rr < 4 * self.h[p] ** 2)
                who = lr[b][:, None].expand(k.shape)[k]
                self._spline(f, who, x0[k], x1[k], rr[k], self.m[p[k]], self.h[p[k]])
            ray, cell, near = ray[~leaf], cell[~leaf], near[~leaf]
            if "bigs" in L:
                br, bc = ray[near], cell[near]
                own, at = self._spread(L["big0"][bc], L["nbig"][bc])
                p, br = L["bigs"][at], br[own]
                x0, x1 = self.x[p] - rx[br], self.y[p] - ry[br]
                self._spline(f, br, x0, x1, (x0 * x0 + x1 * x1).clamp(min=1e-20), self.m[p], self.h[p])
            if not len(ray):
                break
            kids = (L["child"][cell][:, None] + torch.arange(4, device=ray.device)[None]).reshape(-1)
            ray = ray.repeat_interleave(4)
            k = self.levels[i + 1]["cnt"][kids] > 0
            ray, cell = ray[k], kids[k]


def _shoot(planes, zsource, x, zs=None):
    """The multi-plane recursion: positions and Jacobians at each ray's source."""
    dev = _device()
    x = torch.from_numpy(np.ascontiguousarray(x)).to(dev)
    planes = sorted(((float(np.float32(z)), p) for z, p in planes), key=lambda v: v[0])
    z = [v[0] for v in planes]
    D = [_distance(v) for v in z]
    n, np_ = len(x), len(z)
    zs = np.full(n, zsource) if zs is None else np.asarray(zs)
    last = np.searchsorted(z, zs, side="right")  # planes in front of the source
    uniq, inv = np.unique(zs, return_inverse=True)
    Ds = np.array([_distance(v) for v in uniq])[inv]
    Dl = np.array([0.0] + D)[last]
    aa = torch.from_numpy((Ds - Dl) / Ds).to(dev)
    bb = torch.from_numpy(Dl / Ds).to(dev)
    last = torch.from_numpy(last).to(dev)
    th, sa = x.clone(), x.clone()
    A = torch.tensor([1.0, 0, 0, 1.0], dtype=torch.float64, device=dev).repeat(n, 1)
    S = A.clone()
    charge = 4 * math.pi * GRAV
    for j in range(np_):
        do = torch.nonzero(last > j).reshape(-1)
        if not len(do):
            continue
        tree = _Quadtree(planes[j][1], 20, 0.1, 1.0)
        phys = D[j] / (1 + z[j])
        pos = th[do] * phys
        f = tree.force(pos[:, 0].contiguous(), pos[:, 1].contiguous())
        del tree
        G = charge * D[j] / (1 + z[j])
        k, g0, g1 = f[:, 2] * G, f[:, 3] * G, f[:, 4] * G
        s = sa[do] - charge * f[:, :2]
        fin = (last[do] == j + 1)[:, None]
        nxt = D[j + 1] if j + 1 < np_ else D[j]
        a = torch.where(fin, aa[do][:, None], torch.full((1, 1), (nxt - D[j]) / nxt, dtype=torch.float64, device=dev))
        b = torch.where(fin, bb[do][:, None], torch.full((1, 1), D[j] / nxt, dtype=torch.float64, device=dev))
        T = th[do]
        A0, S0 = A[do], S[do]
        S0 = S0 - torch.stack([(k + g0) * A0[:, 0] + g1 * A0[:, 2], (k + g0) * A0[:, 1] + g1 * A0[:, 3],
                               g1 * A0[:, 0] + (k - g0) * A0[:, 2], g1 * A0[:, 1] + (k - g0) * A0[:, 3]], 1)
        th[do], sa[do], S[do], A[do] = b * T + a * s, s, S0, A0 * b + S0 * a
    return th, A


def _neighbours(rec, k):
    """Distance of every particle to its k-th nearest (itself the first)."""
    p = torch.from_numpy(np.ascontiguousarray(rec["x"])).to(_device())
    out = torch.empty(len(p), dtype=torch.float64, device=p.device)
    step = max(1, (1 << 27) // len(p))
    for a in range(0, len(p), step):
        d = p[a:a + step, None, :] - p[None]
        r2 = d.double().square().sum(2)
        out[a:a + step] = torch.topk(r2, k, dim=1, largest=False).values[:, -1].sqrt()
    return out


MOST = 2.7e6  # ray-planes that take too long in plain torch above this


def exact(case, seed):
    kind = case["kind"]
    if kind == "field":
        return None  # the haloes' tables and their tree are the library's own definition
    if kind == "smooth":
        n, k = case["particles"], case["nsmooth"] + 1
        return _neighbours(_snapshot(case, seed), k) if n <= 65536 and n > 2 * k else None
    if kind in ("tree", "force"):
        n = case["rays"] if kind == "tree" else case["side"] ** 2
        if n * (0.1 / case["theta"]) ** 2 > MOST:
            return None
        p, rays = _tree_inputs(case, seed)
        r = torch.from_numpy(rays).to(_device())
        f = _Quadtree(p, case["bucket"], case["theta"], 0.0).force(r[:, 0].contiguous(), r[:, 1].contiguous())
        if kind == "force":
            return f[:, :5].contiguous()
        gamma = torch.cat([f[:, 3:5], torch.zeros_like(f[:, :1])], 1)
        return f[:, :2].contiguous(), f[:, 2].contiguous(), gamma, f[:, 5].contiguous()
    if kind == "batch":
        specs = _batch_inputs(case, seed)
        if sum(s * s * len(p) for s, _, p in specs) > MOST:
            return None
        got = [_shoot(p, zs, _grid(s, 30.0 * ARCSEC)) for s, zs, p in specs]
        return torch.cat([y for y, _ in got]), torch.cat([a for _, a in got])
    if kind == "served":
        req = _requests(case, seed)
        if sum(len(x) for _, x, _ in req) * case["planes"] > MOST:
            return None
        models = [_planes(case, seed, 100 * m) for m in range(case["models"])]
        got = [_shoot(models[m], _zsource(case), x, np.full(len(x), zs)) for m, x, zs in req]
        return torch.cat([y for y, _ in got]), torch.cat([a for _, a in got])
    n = case["rays"] if kind == "rays" else case["side"] ** 2
    if kind == "device" or n * case["planes"] > MOST:
        return None  # with the NSIE galaxy, or too many rays
    if kind == "rays":
        x, zs = _blob_rays(case, seed)
        return _shoot(_planes(case, seed), _zsource(case), x, zs)
    return _shoot(_planes(case, seed), _zsource(case), _grid(case["side"], case["arcsec"] * ARCSEC))

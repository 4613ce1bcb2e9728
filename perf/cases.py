"""Performance cases of the reconstruction path, through its public entry points.

Each case is one call (or one served burst of calls) as a program makes it: the handle is
kept, the clouds are device-resident tensors or host arrays, and the outputs are the meshes,
in the program's own buffers (zero beyond a mesh's count).  The clouds are the repository's synthetic families (noisy spheres, tori, a torus
united with an ellipsoid, superquadrics with a sinusoidal displacement; random scale and
rotation where noted), generated on the GPU from the seed.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "poisson-surface-reconstruction-gpu_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import psr  # noqa: E402
import serve  # noqa: E402

DEV = "cuda"


def _cloud(name, form, shape, n, depth, **more):
    """A single-cloud case; `form`: "device" (tensors in, tensors out), "host" (arrays in and
    out, the drop-in call, the mesh gathered into the program's arrays), "pinned" (pinned host
    memory in and out, submitted and waited for) or "unoriented" (positions alone, on the
    device: normals, then the mesh)."""
    c = dict(name=name, form=form, shape=shape, n=n, depth=depth, rgb=False, normals=False, weld=False, keep_all=False,
             cg_iterations=0)
    c.update(more)
    return c


def listed():
    return [
        # the smallest call a program makes: a preview of a few thousand points, host arrays, a
        # fixed number of CG iterations; latency and launches count
        _cloud("sphere4k_d5_host", "host", "sphere", 4000, 5, rgb=True, cg_iterations=8),
        # the plain single-cloud configuration: 20,000 points of a sphere, depth 6, 8 iterations,
        # inputs and mesh in pinned host memory
        _cloud("sphere20k_d6_pinned", "pinned", "sphere", 20000, 6, cg_iterations=8),
        # a scan without normals (xyz only, odd size): normal estimation, then the mesh, as a file of
        # bare positions goes through
        _cloud("scan31k_d7_unoriented", "unoriented", "ellipsoid", 31337, 7),
        # the repository's headline workload: 200,000 coloured points, depth 7, device to device
        _cloud("torus200k_d7", "device", "torus_ellipsoid", 200000, 7, rgb=True),
        # a small cloud with every option of the mesh: colours, normals, welded vertices, odd size
        _cloud("mix61k_d7_weld", "device", "superquadric", 61803, 7, rgb=True, normals=True, weld=True),
        # a depth-8 scan of the multi-cloud mix's largest size with normals
        _cloud("mix150k_d8", "device", "torus", 149999, 8, normals=True),
        # the largest cloud of the serving mix at its largest depth, coloured, every Laplacian entry kept
        _cloud("serve500k_d9", "device", "torus", 500000, 9, rgb=True, normals=True, keep_all=True),
        # the large-cloud workload: 2M points, depth 9, with normals
        _cloud("superquadric2m_d9", "device", "superquadric", 2000000, 9, normals=True, keep_all=True),
        # a multi-cloud launch: 16 clouds of uneven size, one pass per depth
        dict(name="batch16_d7", form="batch", count=16, lo=20000, hi=150000, depth=7),
        # the served form: a burst of 16 requests of the headline size over 8 resident slots
        dict(name="served16_d7", form="served", count=16, slots=8, lo=200000, hi=200000, depth=7),
        # the served form on small clouds of uneven size (many short reconstructions in flight)
        dict(name="served16_d6", form="served", count=16, slots=8, lo=10000, hi=100000, depth=6),
        # normals of an unoriented cloud on the device (its own entry point)
        dict(name="normals200k", form="normals", shape="torus_ellipsoid", n=200000),
    ]


def draw(rng):
    def size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi)))) | 1

    form = rng.choice(["host", "pinned", "unoriented", "device", "device", "device", "batch", "served", "normals"])
    shape = rng.choice(["sphere", "torus", "torus_ellipsoid", "superquadric"])
    if form == "normals":
        return dict(form=form, shape=shape, n=size(2000, 500000))
    if form == "batch":
        depth = rng.choice([6, 7])
        lo = size(5000, 30000) if depth == 6 else size(20000, 50000)
        return dict(form=form, count=rng.randint(3, 16), lo=lo, hi=size(2 * lo, 150000), depth=depth)
    if form == "served":
        depth = rng.choice([6, 7])
        lo = size(10000, 60000) if depth == 6 else size(20000, 60000)
        return dict(form=form, count=rng.randint(5, 16), slots=8, lo=lo, hi=size(lo, 200000), depth=depth)
    if form in ("host", "pinned", "unoriented"):
        depth = rng.choice([5, 6, 7])
        n = size(4000 << (depth - 5), 30000 << (depth - 5))
        c = _cloud("", form, shape, n, depth, rgb=rng.random() < 0.5,
                   cg_iterations=8 if form != "unoriented" and rng.random() < 0.5 else 0)
        del c["name"]
        return c
    depth = rng.choice([6, 7, 7, 8, 8, 9])
    n = size(*{6: (10000, 150000), 7: (30000, 500000), 8: (120000, 700000), 9: (400000, 1900000)}[depth])
    c = _cloud("", form, shape, n, depth, rgb=rng.random() < 0.5, normals=rng.random() < 0.5, weld=rng.random() < 0.25,
               keep_all=depth == 9)
    del c["name"]
    return c


# ---- clouds ------------------------------------------------------------------------------
def _unit(v):
    return v / v.norm(dim=1, keepdim=True).clamp_min(1e-30)


def _rand(g, n, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(n, generator=g, device=DEV, dtype=torch.float64)


def _kept(n, make):
    """n rows of make()'s accepted candidates."""
    got = []
    while sum(len(x) for x in got) < n:
        got.append(make())
    return torch.cat(got)[:n]


def _sphere(n, g):
    d = _unit(torch.randn(n, 3, generator=g, device=DEV, dtype=torch.float64))
    return d, d


def _torus(n, g, R=1.0, r=0.35):
    def make():
        v = _rand(g, 2 * n, 0, 2 * math.pi)
        return v[_rand(g, 2 * n, 0, R + r) < R + r * torch.cos(v)]
    v, u = _kept(n, make), _rand(g, n, 0, 2 * math.pi)
    nrm = torch.stack([torch.cos(v) * torch.cos(u), torch.cos(v) * torch.sin(u), torch.sin(v)], 1)
    ring = torch.stack([torch.cos(u), torch.sin(u), torch.zeros_like(u)], 1)
    return R * ring + r * nrm, nrm


def _ellipsoid(n, g, radii=(0.6, 0.4, 0.3)):
    a = torch.tensor(radii, device=DEV, dtype=torch.float64)
    across = a.prod() / a

    def make():
        u = _unit(torch.randn(2 * n, 3, generator=g, device=DEV, dtype=torch.float64))
        return u[_rand(g, 2 * n) * across.max() < (u * across).norm(dim=1)]
    u = _kept(n, make)
    return u * a, _unit(u / a)


def _torus_ellipsoid(n, g):
    area_e = 4 * math.pi * (((0.24 ** 1.6075) + (0.18 ** 1.6075) + (0.12 ** 1.6075)) / 3) ** (1 / 1.6075)
    area_t = 4 * math.pi ** 2 * 0.35
    nt = round(n * area_t / (area_t + area_e))
    p1, n1 = _torus(nt, g)
    p2, n2 = _ellipsoid(n - nt, g)
    p2 = p2 + torch.tensor([0.0, 0.0, 0.8], device=DEV, dtype=torch.float64)
    order = torch.randperm(n, generator=g, device=DEV)
    return torch.cat([p1, p2])[order], torch.cat([n1, n2])[order]


def _superquadric(n, g, e=0.5, amp=0.05, freq=8.0):
    def power(x):
        return torch.sign(x) * x.abs() ** e

    def point(eta, om):
        s = 1.0 + amp * torch.sin(freq * eta) * torch.sin(freq * om)
        x = power(torch.cos(eta)) * power(torch.cos(om))
        y = power(torch.cos(eta)) * power(torch.sin(om))
        return torch.stack([x * s, y * s, power(torch.sin(eta)) * s], 1)

    def make():
        h, m = 1e-5, 2 * n
        eta, om = _rand(g, m, -math.pi / 2 + 1e-4, math.pi / 2 - 1e-4), _rand(g, m, -math.pi, math.pi)
        pe = (point(eta + h, om) - point(eta - h, om)) / (2 * h)
        po = (point(eta, om + h) - point(eta, om - h)) / (2 * h)
        cr = torch.linalg.cross(po, pe)
        area = cr.norm(dim=1)
        top = area.kthvalue(int(0.999 * m)).values
        keep = _rand(g, m) * top < area
        return torch.cat([point(eta, om), cr], 1)[keep]
    q = _kept(n, make)
    p, nrm = q[:, :3], _unit(q[:, 3:])
    return p, nrm * torch.where((nrm * p).sum(1, keepdim=True) < 0, -1.0, 1.0)


_SHAPES = {"sphere": _sphere, "torus": _torus, "ellipsoid": _ellipsoid, "torus_ellipsoid": _torus_ellipsoid,
           "superquadric": _superquadric}


def _points(shape, n, g, rgb, place=False):
    """(xyz float32, unit normals float32, uint8 colours or None) on the GPU; `place`: a random
    rotation and scale."""
    p, nrm = _SHAPES[shape](n, g)
    if place:
        q, r = torch.linalg.qr(torch.randn(3, 3, generator=g, device=DEV, dtype=torch.float64))
        q = q * torch.sign(torch.diagonal(r))
        p, nrm = p @ q.T * float(_rand(g, 1, 0.5, 2.0)), nrm @ q.T
    p = p + 0.002 * torch.randn(n, 3, generator=g, device=DEV, dtype=torch.float64)
    p = p.float().contiguous()
    col = None
    if rgb:   # a linear function of position
        lo, hi = p.min(0).values, p.max(0).values
        col = (255 * (p - lo) / (hi - lo)).round().clamp(0, 255).to(torch.uint8).contiguous()
    return p, _unit(nrm).float().contiguous(), col


def _sizes(case, g):
    """Cloud sizes of a batch or burst: log-uniform in [lo, hi], the largest included."""
    lo, hi = case["lo"], case["hi"]
    u = torch.rand(case["count"], generator=g, device=DEV).tolist()
    return [hi if k == 0 else int(lo * (hi / lo) ** u[k]) for k in range(case["count"])]


def _caps(depth, n):
    """Output and subdivision capacities a program sets for its depth."""
    if depth <= 7:
        return dict(max_triangles=1000000, max_mesh_vertices=300000)
    if depth == 8:
        return dict(max_triangles=2000000, max_mesh_vertices=1000000, max_subdivision_nodes=max(4000000, 8 * n))
    return dict(max_triangles=12000000, max_mesh_vertices=6000000, max_subdivision_nodes=max(8000000, 8 * n))


def _buffers(depth, colors, normals, where="device"):
    """The program's mesh buffers: room for about four times the mesh of a closed surface at
    the depth (from depth 8 on, where noise folds the surface, ten times)."""
    v = (9 if depth < 8 else 22) * 4 ** depth
    def rows(m, dtype):
        if where == "device":
            return torch.zeros(m, 3, dtype=dtype, device=DEV)
        return torch.zeros(m, 3, dtype=dtype).pin_memory() if where == "pinned" else torch.zeros(m, 3, dtype=dtype).numpy()
    return dict(vertices=rows(v, torch.float32), triangles=rows(2 * v, torch.int32),
                colors=rows(v, torch.float32) if colors else None, normals=rows(v, torch.float32) if normals else None)


def _ptr(x):
    return None if x is None else x.data_ptr()


def _mesh(b, location=psr.PSR_DEVICE):
    return psr.PsrMesh(_ptr(b["vertices"]), _ptr(b["triangles"]), _ptr(b["colors"]), _ptr(b["normals"]),
                       b["vertices"].shape[0], b["triangles"].shape[0], location, 0, 0)


def _gather(b, vertices, triangles, colors=None):
    """A finished mesh into the program's buffers."""
    b["vertices"][:len(vertices)] = vertices
    b["triangles"][:len(triangles)] = triangles
    if colors is not None:
        b["colors"][:len(colors)] = colors


def _place(meshes):
    return np.array([[*m.center, m.scale] for m in meshes], np.float32)


# ---- the cases ---------------------------------------------------------------------------
def _burst(case, g):
    """The clouds of a batch or a served burst."""
    sizes = _sizes(case, g)
    uneven = case["lo"] < case["hi"]
    shapes = ["sphere", "torus", "superquadric"] if uneven else ["torus_ellipsoid"]
    return [_points(shapes[k % len(shapes)], n, g, case["form"] == "served", place=uneven) for k, n in enumerate(sizes)]


def prepare(case, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    form, s = case["form"], dict(case=case)
    if form == "normals":
        s["xyz"] = _points(case["shape"], case["n"], g, False)[0]
        s["out"] = torch.empty_like(s["xyz"])
        s["recon"] = psr.PoissonReconstruction(max_depth=7, max_points=case["n"])
        return s
    depth = case["depth"]
    if form in ("batch", "served"):
        s["clouds"] = _burst(case, g)
        caps = _caps(depth, case["hi"])
        s["buffers"] = [_buffers(depth, form == "served", form == "batch") for _ in s["clouds"]]
        if form == "batch":
            s["recon"] = psr.PoissonReconstruction(max_depth=depth, max_points=case["hi"], batch_clouds=case["count"],
                                                   compute_normals=True, **caps)
        else:
            # a slot keeps as many finished meshes as the burst may hand it
            s["server"] = serve.Server(slots=case["slots"], max_depth=depth, max_points=case["hi"], compute_colors=True,
                                       compute_normals=False, out_sets=case["count"], **caps)
        return s
    xyz, nrm, rgb = _points(case["shape"], case["n"], g, case["rgb"])
    s["recon"] = psr.PoissonReconstruction(
        max_depth=depth, max_points=case["n"] if depth > 7 else max(300000, case["n"]), compute_colors=case["rgb"],
        compute_normals=case["normals"], weld_vertices=case["weld"], laplacian_epsilon=0.0 if case["keep_all"] else 1e-6,
        **_caps(depth, case["n"]))
    s["buffers"] = _buffers(depth, case["rgb"], case["normals"], form if form in ("host", "pinned") else "device")
    if form == "pinned":
        xyz, nrm, rgb = (None if x is None else x.cpu().pin_memory() for x in (xyz, nrm, rgb))
    if form == "host":
        xyz, nrm, rgb = (None if x is None else x.cpu().numpy() for x in (xyz, nrm, rgb))
    if form == "unoriented":
        nrm = torch.empty_like(nrm)
    s.update(xyz=xyz, nrm=nrm, rgb=rgb)
    return s


def run(state):
    case, n = state["case"], state["case"].get("n")
    form, r, b = case["form"], state.get("recon"), state.get("buffers")
    if form == "normals":
        r.estimate_normals_device(state["xyz"].data_ptr(), n, state["out"].data_ptr())
        return state["out"]
    if form == "batch":
        n = case["count"]
        pts, meshes = (psr.PsrPoints * n)(), (psr.PsrMesh * n)()
        for k, (xyz, nrm, _) in enumerate(state["clouds"]):
            pts[k] = psr.PsrPoints(xyz.data_ptr(), nrm.data_ptr(), None, xyz.shape[0], psr.PSR_DEVICE)
            meshes[k] = _mesh(b[k])
        r.submit_batch_device(pts, meshes, depth=case["depth"])
        try:
            r.wait()
        except psr.PsrError as e:
            # one cloud in a thousand or so has an octree that the algorithm cannot mesh: it fails
            # alone and the program goes on with the others
            if e.status != psr.PSR_INVALID_INPUT:
                raise
        return [*b, _place([m for m in meshes if m.scale > 0])]
    if form == "served":
        reqs = [serve.Request(xyz, nrm, rgb, depth=case["depth"], tag=k)
                for k, (xyz, nrm, rgb) in enumerate(state["clouds"])]
        state["server"].run(reqs)
        for k, q in enumerate(reqs):
            if not q.error:
                _gather(b[k], q.vertices, q.triangles, q.colors)
            elif "invalid input" not in q.error:
                raise RuntimeError(q.error)
        return [*b, _place([q for q in reqs if not q.error])]
    xyz, nrm, rgb = state["xyz"], state["nrm"], state["rgb"]
    options = dict(depth=case["depth"], cg_iterations=case["cg_iterations"])
    if form == "host":
        m = r.SolvePoissionReconstructionMesh(xyz, nrm, rgb, **options)
        _gather(b, m.vertices, m.triangles, m.colors)
        return dict(b, place=_place([m]))
    if form == "pinned":
        m = _mesh(b, psr.PSR_HOST)
        r.submit_device(xyz.data_ptr(), nrm.data_ptr(), _ptr(rgb), n, m, location=psr.PSR_HOST, **options)
        r.wait()
        return dict(b, place=_place([m]))
    if form == "unoriented":
        r.estimate_normals_device(xyz.data_ptr(), n, nrm.data_ptr())
    m = r.reconstruct_device(xyz.data_ptr(), nrm.data_ptr(), _ptr(rgb), n, out=_mesh(b), **options)
    out = dict(b, place=_place([m]))
    if form == "unoriented":
        out["estimated"] = nrm
    return out


def work(case):
    """Inputs read once, meshes written once; the arithmetic of the CG systems (27-point rows, about
    55 iterations to the tolerance, or the fixed count) and of the sample and vertex values."""
    if case["form"] == "normals":
        # positions in, normals out; 27 cells of candidates per point and a 3x3 eigenproblem
        return dict(bytes=24.0 * case["n"], flops=case["n"] * (9 * 30 + 27 * 10 + 200.0))
    if case["form"] in ("batch", "served"):
        lo, hi = case["lo"], case["hi"]
        mean = (hi - lo) / math.log(hi / lo) if hi > lo else hi
        sizes = [hi] + [mean] * (case["count"] - 1)
        one = [_work(n, case["depth"], case["form"] == "served", case["form"] == "batch", 55) for n in sizes]
    else:
        one = [_work(case["n"], case["depth"], case["rgb"], case["normals"], case["cg_iterations"] or 55)]
        if case["form"] == "unoriented":
            one.append((24.0 * case["n"], 740.0 * case["n"]))
    return dict(bytes=sum(b for b, _ in one), flops=sum(f for _, f in one))


def _work(n, depth, rgb, normals, iterations):
    cells = min(4.5 * 4 ** depth, 8 * n)               # depth-D nodes of a closed surface
    nodes = cells * 4 / 3
    verts = min(2.2 * 4 ** depth, 2.0 * n)
    size = n * (24 + 3 * rgb) + verts * (12 + 24 + 12 * rgb + 12 * normals)
    flops = nodes * iterations * (54 + 10) + (n + 1.5 * nodes) * 27 * 4 * depth + n * 27 * 15
    return size, flops


# ---- 64-bit values -------------------------------------------------------------------------
def _exact_place(clouds):
    """Bounding-box placement: the box enlarged 1.25 times around its middle, its lower corner
    and edge."""
    rows = []
    for xyz in clouds:
        p = xyz.double().cpu().numpy()
        lo, hi = p.min(0), p.max(0)
        edge = 1.25 * (hi - lo).max()
        rows.append([*((lo + hi) / 2 - edge / 2), edge])
    return np.array(rows)


def _exact_normals(xyz, k=10):
    """Smallest eigenvector of each point's k nearest neighbours' covariance (itself one of them),
    towards the origin."""
    p32 = xyz - xyz.mean(0)
    p = xyz.double()
    n = p.shape[0]
    sq = (p32 * p32).sum(1)
    near = []
    step = max(1, (1 << 28) // n)
    for a in range(0, n, step):   # candidates by float distances, then the nearest of them in 64 bits
        d = sq[a:a + step, None] + sq[None, :] - 2.0 * (p32[a:a + step] @ p32.T)
        c = d.topk(min(n, 40), largest=False).indices
        e = (p[c] - p[a:a + step, None, :]).square().sum(2)
        near.append(c.gather(1, e.topk(min(n, k), largest=False).indices))
    q = p[torch.cat(near)]
    q = (q - q.mean(1, keepdim=True)).cpu().numpy()
    _, v = np.linalg.eigh(np.einsum("nki,nkj->nij", q, q))
    v = torch.from_numpy(v[:, :, 0]).to(p.device)
    return v * torch.where((v * p).sum(1, keepdim=True) > 0, -1.0, 1.0)


def exact(case, seed):
    """The placement of every mesh and, where they are asked for, the estimated normals.  The mesh
    itself (a multi-level Poisson solution and its level set) has no short 64-bit statement."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    form = case["form"]
    if form == "normals":
        return _exact_normals(_points(case["shape"], case["n"], g, False)[0])
    if form in ("batch", "served"):
        clouds = [c[0] for c in _burst(case, g)]
        return [None for _ in clouds] + [_exact_place(clouds)]
    xyz = _points(case["shape"], case["n"], g, case["rgb"])[0]
    out = dict(place=_exact_place([xyz]))
    if form == "unoriented":
        out["estimated"] = _exact_normals(xyz)
    return out

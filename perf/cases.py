"""The work that users of this framework have it do, as measurable cases.

A case names a kind of call (its "kind") and the sizes of one call.  The kinds are the ways the
package is used: depth pre-processing, rigid integration, surface extraction, the dense per-voxel
warp chain, the motion-graph stage, the two Gauss-Newton solvers, the rigid multi-camera stream,
whole non-rigid sequences, and many sessions at once.  Sizes come from configs.py, bench.py and the
tests.  Scenes are rendered here from the seed (depth in millimetres with the depth-dependent sensor
noise of synth.py), so the inputs of a case do not depend on the code that is measured.
"""
import math
import random

import numpy as np
import torch

from volumefusion_gb300 import af, configs
from volumefusion_gb300.batch import Batch
from volumefusion_gb300.fusion import FusionSession
from volumefusion_gb300.rigid_stream import RigidStream

DEV = "cuda"
F64 = torch.float64


def listed():
    return [
        # One frame of the small camera made into filtered depth, vertices, normals and centroid: the
        # smallest call a caller makes per frame, where launches and host time count.
        dict(name="prep_320x288", kind="prep", width=320, height=288, radius=2),
        # The reference's static reconstruction: one frame into a large FP32 volume at a given pose.
        dict(name="integrate_512", kind="integrate", x=512, y=512, z=512, width=640, height=576),
        # Canonical point cloud of a volume: marching cubes, then sort + unique; an odd, ragged volume.
        dict(name="mc_cloud_257x230x301", kind="mc", x=257, y=230, z=301),
        # The reference's dense non-rigid integration, step by step, on per-voxel arrays.
        dict(name="voxel_chain_200", kind="voxel", x=200, y=200, z=200, nodes=600, knn=4, width=640, height=576),
        # The motion-graph stage of a frame, step by step: graph, KNN, weights, warp, correspondences.
        dict(name="cloud_stage_60k", kind="cloud", points=60000, spacing=0.020, knn=4, kreg=8, width=640, height=576),
        # Gauss-Newton system and PCG solve at the graph size of the usual 25 mm node radius ...
        dict(name="gn_140", kind="gn", points=20000, nodes=140, knn=4, kreg=8, iterations=10),
        # ... and at that of a dense graph.
        dict(name="gn_1500", kind="gn", points=60000, nodes=1500, knn=4, kreg=8, iterations=10),
        # The reference's dense solver (LU with partial pivoting) on a system of 137 nodes.
        dict(name="lu_822", kind="lu", n=822),
        # Rigid multi-camera stream, 3 cameras into the default 400^3 volume, 4 frames and the outputs.
        dict(name="stream_3x640_400", kind="stream", cameras=3, width=640, height=576, dims=400, frames=4),
        # The headline: a 30-frame non-rigid sequence from an empty 256^3 FP32 volume.
        dict(name="session_256_fp32", kind="session", dims=256, voxel=0.004, width=640, height=576, graph_radius=0.025,
             precision="fp32", frames=30),
        # The precision form at 512^3 with a dense graph: the largest volume, cloud and graph.
        dict(name="session_512_fp16", kind="session", dims=512, voxel=0.002, width=640, height=576, graph_radius=0.009,
             precision="fp16", frames=8),
        # Many uneven sessions advanced together.
        dict(name="batch_8", kind="batch", sessions=8, mix=7, frames=12),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["prep", "integrate", "mc", "voxel", "cloud", "gn", "gn", "lu", "stream", "session", "session",
                       "batch"])
    if kind == "prep":
        w = _log(rng, 160, 1280)
        return dict(kind=kind, width=w, height=max(120, int(w * 0.9) - rng.randrange(16)), radius=rng.choice([1, 2, 2, 3, 5]))
    if kind == "integrate":
        x, y, z = (_log(rng, 96, 512) for _ in range(3))
        return dict(kind=kind, x=x, y=y, z=z, width=rng.choice([320, 640]), height=rng.choice([288, 480, 576]))
    if kind == "mc":
        x, y, z = (_log(rng, 64, 384) for _ in range(3))
        return dict(kind=kind, x=x, y=y, z=z)
    if kind == "voxel":
        x, y, z = (_log(rng, 64, 200) for _ in range(3))
        return dict(kind=kind, x=x, y=y, z=z, nodes=_log(rng, 40, 600), knn=rng.choice([4, 4, 6]), width=640, height=576)
    if kind == "cloud":
        return dict(kind=kind, points=_log(rng, 2000, 200000), spacing=round(rng.uniform(0.012, 0.035), 4),
                    knn=rng.choice([4, 4, 6]), kreg=rng.choice([4, 8]), width=rng.choice([320, 640]),
                    height=rng.choice([288, 576]))
    if kind == "gn":
        nodes = _log(rng, 60, 2500)
        return dict(kind=kind, points=nodes * rng.randrange(30, 140), nodes=nodes, knn=rng.choice([4, 4, 6]),
                    kreg=rng.choice([4, 8]), iterations=rng.choice([10, 10, 20]))
    if kind == "lu":
        return dict(kind=kind, n=6 * _log(rng, 12, 260))
    if kind == "stream":
        w, h = rng.choice([(320, 288), (640, 576), (512, 424)])
        return dict(kind=kind, cameras=rng.randrange(1, 5), width=w, height=h, dims=_log(rng, 128, 400), frames=4)
    if kind == "session":
        if rng.random() < 0.3:
            dims, radius, precision, frames = _log(rng, 320, 512), 0.010, "fp16", 6
        else:
            dims, radius, precision, frames = _log(rng, 96, 320), rng.uniform(0.020, 0.035), rng.choice(["fp32", "fp32", "fp16"]), 16
        w, h = rng.choice([(320, 288), (640, 576)])
        return dict(kind=kind, dims=dims, voxel=round(1.024 / dims, 6), width=w, height=h, graph_radius=round(radius, 4),
                    precision=precision, frames=frames)
    return dict(kind=kind, sessions=rng.randrange(3, 9), mix=rng.randrange(1000), frames=10)


# ---- scenes ----

def _cuda_rng(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFF)
    return g


def _K(width, height):
    f = 504.0 * width / 640.0
    return np.array([[f, 0.0, width / 2.0], [0.0, f, height / 2.0], [0.0, 0.0, 1.0]])


def _rays(width, height, K, device):
    v, u = torch.meshgrid(torch.arange(height, dtype=F64, device=device), torch.arange(width, dtype=F64, device=device),
                          indexing="ij")
    return torch.stack([(u - K[0, 2]) / K[0, 0], (v - K[1, 2]) / K[1, 1], torch.ones_like(u)], -1)


def _hit_sphere(d, c, r):
    c = torch.as_tensor(c, dtype=F64, device=d.device)
    dd, dc = (d * d).sum(-1), d @ c
    disc = dc * dc - dd * (c @ c - r * r)
    t = (dc - disc.clamp(min=0).sqrt()) / dd
    return torch.where((disc >= 0) & (t > 0), t, torch.full_like(t, math.inf))


def _hit_capsule(d, a, b, r):
    a, b = (torch.as_tensor(x, dtype=F64, device=d.device) for x in (a, b))
    L = (b - a).norm()
    ax = (b - a) / L
    dpar = d @ ax
    dperp = d - dpar[..., None] * ax
    apar = -(a @ ax)
    aperp = -a - apar * ax
    A = (dperp * dperp).sum(-1)
    B = 2.0 * (dperp @ aperp)
    C = aperp @ aperp - r * r
    disc = B * B - 4 * A * C
    t = (-B - disc.clamp(min=0).sqrt()) / (2 * A.clamp(min=1e-15))
    s = t * dpar + apar
    body = (disc >= 0) & (A > 1e-15) & (t > 0) & (s >= 0) & (s <= L)
    t = torch.where(body, t, torch.full_like(t, math.inf))
    return torch.minimum(t, torch.minimum(_hit_sphere(d, a, r), _hit_sphere(d, b, r)))


def _scene(name, rnd):
    """Geometry of a scene, shifted a little by the seed: capsule pair or sphere, around 0.8 m away."""
    j = np.array([rnd.uniform(-0.01, 0.01), rnd.uniform(-0.01, 0.01), 0.8 + rnd.uniform(-0.01, 0.01)])
    return dict(name=name, joint=j, radius=(0.06 if name == "capsule" else 0.15) * rnd.uniform(0.97, 1.03), length=0.3)


def _capsules(sc, u):
    """End points of the two capsules at time u in [0, 1] (the second bends by 45 degrees)."""
    th = math.radians(45.0) * u
    j, L = sc["joint"], sc["length"]
    return (j + L * np.array([-1.0, 0.0, 0.0]), j), (j, j + L * np.array([math.cos(th), 0.0, -math.sin(th)]))


def _depth(sc, u, width, height, K, device=DEV):
    """Noise-free depth in metres (inf where nothing is hit)."""
    d = _rays(width, height, K, device)
    if sc["name"] == "capsule":
        p, q = _capsules(sc, u)
        return torch.minimum(_hit_capsule(d, *p, sc["radius"]), _hit_capsule(d, *q, sc["radius"]))
    return _hit_sphere(d, sc["joint"] + np.array([0.1 * u - 0.05, 0.02 * u, 0.05 * u]), sc["radius"])


def _frame(sc, u, width, height, K, gen):
    """One depth frame in millimetres: int16 holding the uint16 image, 0 where nothing is seen."""
    z = _depth(sc, u, width, height, K)
    ok = torch.isfinite(z)
    z = torch.where(ok, z, torch.zeros_like(z))
    z = z + 0.001 * z * z * torch.randn(z.shape, generator=gen, dtype=F64, device=DEV)
    return torch.where(ok, (z * 1000.0).round(), torch.zeros_like(z)).to(torch.int16).contiguous()


def _frames(sc, n, total, width, height, K, seed, salt=0):
    gen = _cuda_rng(seed, salt)
    return [_frame(sc, f / max(total - 1, 1), width, height, K, gen) for f in range(n)]


def _surface(sc, count, gen):
    """`count` points on the camera side of the capsule pair's surface, sorted as a canonical cloud is."""
    pts = []
    for a, b in _capsules(sc, 0.0):
        a, b = (torch.as_tensor(x, dtype=F64, device=DEV) for x in (a, b))
        n = (count + 1) // 2
        t = torch.rand(n, generator=gen, dtype=F64, device=DEV)
        phi = math.pi * (1.0 + torch.rand(n, generator=gen, dtype=F64, device=DEV))
        ring = torch.stack([torch.zeros_like(phi), phi.cos(), phi.sin()], -1)
        pts.append(a + t[:, None] * (b - a) + sc["radius"] * ring)
    p = torch.cat(pts)[:count]
    p = p + 0.0005 * torch.randn(p.shape, generator=gen, dtype=F64, device=DEV)
    p = p.float().cpu().numpy()
    return torch.from_numpy(p[np.lexsort(p.T[::-1])]).to(DEV).contiguous()


def _spread(points, count):
    """About `count` of the points, one per cell of a grid over them, and the cell size."""
    p = points.cpu().numpy()
    lo, hi = 1e-3, 0.3
    for _ in range(24):
        cell = math.sqrt(lo * hi)
        _, first = np.unique(np.floor(p / cell).astype(np.int64), axis=0, return_index=True)
        lo, hi = (cell, hi) if len(first) > count else (lo, cell)
    return points[torch.from_numpy(np.sort(first)).to(DEV)].contiguous(), cell


def _exactly(points, count):
    """`count` of the points, spread evenly over them, and the distance that keeps them apart."""
    some, cell = _spread(points, count)
    while some.shape[0] < count:
        cell *= 0.97
        _, first = np.unique(np.floor(points.cpu().numpy() / cell).astype(np.int64), axis=0, return_index=True)
        some = points[torch.from_numpy(np.sort(first)).to(DEV)]
    take = torch.linspace(0, some.shape[0] - 1, count, dtype=F64, device=DEV).round().long()
    return some[take].contiguous(), cell


def _padded(x, rows):
    """The rows of a result whose number depends on the data, in a buffer of the caller's size."""
    out = x.new_zeros((rows,) + tuple(x.shape[1:]))
    out[:x.shape[0]] = x
    return out


def _rigid_near_identity(count, gen, angle=0.05, shift=0.004):
    """`count` small rigid motions as column-major 4x4 rows."""
    w = angle * torch.randn((count, 3), generator=gen, dtype=F64, device=DEV)
    S = torch.zeros((count, 3, 3), dtype=F64, device=DEV)
    S[:, 0, 1], S[:, 0, 2], S[:, 1, 2] = -w[:, 2], w[:, 1], -w[:, 0]
    R = torch.matrix_exp(S - S.transpose(1, 2))
    T = torch.eye(4, dtype=F64, device=DEV).repeat(count, 1, 1)
    T[:, :3, :3] = R
    # about the capsules' joint, 0.8 m in front of the camera
    c = torch.tensor([0.0, 0.0, 0.8], dtype=F64, device=DEV)
    T[:, :3, 3] = c - R @ c + shift * torch.randn((count, 3), generator=gen, dtype=F64, device=DEV)
    return T.transpose(1, 2).reshape(count, 16).float().contiguous()


def _nearest(queries, nodes, k, skip=0):
    """Indices and distances of the k nearest nodes (64 bits, in chunks)."""
    idx, dist = [], []
    n = nodes.double()
    for q in queries.double().split(16384):
        d, i = torch.cdist(q, n, compute_mode="donot_use_mm_for_euclid_dist").topk(k + skip, largest=False)
        idx.append(i[:, skip:])
        dist.append(d[:, skip:])
    return torch.cat(idx), torch.cat(dist)


def _frame_vertices(depth, K):
    d = _rays(depth.shape[1], depth.shape[0], K, DEV)
    return torch.where(torch.isfinite(depth), depth, torch.zeros_like(depth))[..., None] * d


def _rot(axis, deg):
    a = math.radians(deg)
    c, s = math.cos(a), math.sin(a)
    return np.array({"x": [[1, 0, 0], [0, c, -s], [0, s, c]], "y": [[c, 0, s], [0, 1, 0], [-s, 0, c]],
                     "z": [[c, -s, 0], [s, c, 0], [0, 0, 1]]}[axis])


def _session_cfg(case):
    cfg = configs.nonrigid_capsules_256(n_frames=case["frames"], dims=(case["dims"],) * 3, voxel=case["voxel"])
    cfg.update(width=case["width"], height=case["height"], K=_K(case["width"], case["height"]),
               graph_radius=case["graph_radius"], precision=case["precision"], delta=max(0.016, 4 * case["voxel"]))
    return cfg


def _mix(case):
    """The sessions of a batch, drawn as configs.session_mix draws them (spheres and capsules)."""
    rnd = random.Random(case["mix"])
    out = []
    for _ in range(case["sessions"]):
        dims, voxel = rnd.choice([(128, 0.008), (192, 0.006), (256, 0.004), (384, 0.003)])
        w, h, f = rnd.choice([(320, 288, 252.0), (640, 576, 504.0)])
        out.append(configs.session_config(dims, voxel, w, h, f, rnd.uniform(0.020, 0.035), rnd.choice(["sphere", "capsule"]),
                                          rnd.randrange(1 << 30)))
    return out


# ---- prepare ----

def prepare(case, seed):
    rnd = random.Random(seed)
    s = dict(case=case)
    kind = case["kind"]
    if kind == "prep":
        K = _K(case["width"], case["height"])
        s.update(K=K, mm=_frames(_scene("sphere", rnd), 1, 1, case["width"], case["height"], K, seed)[0])
    elif kind == "integrate":
        W, H = case["width"], case["height"]
        K = _K(W, H)
        sc = _scene("capsule", rnd)
        depth = _frames(sc, 1, 1, W, H, K, seed)[0].float() * 0.001
        dims = (case["x"], case["y"], case["z"])
        size = tuple(1.024 * v / max(dims) for v in dims)
        S = dims[0] * dims[1] * dims[2]
        s.update(K=K, dims=dims, size=size, vs=tuple(np.float32(a) / np.float32(b) for a, b in zip(size, dims)),
                 depth=torch.where(depth > 0, depth, torch.full_like(depth, math.inf)).contiguous(), R=_rot("y", 10.0),
                 t=sc["joint"], tsdf=torch.full((S,), -1.0, device=DEV), weights=torch.zeros(S, device=DEV))
    elif kind == "mc":
        s.update(_mc_volume(case, seed, rnd))
    elif kind == "voxel":
        s.update(_voxel_inputs(case, seed, rnd))
    elif kind == "cloud":
        s.update(_cloud_inputs(case, seed, rnd))
    elif kind == "gn":
        s.update(_gn_inputs(case, seed, rnd))
        s["system"] = af.GaussNewtonSystem(case["points"], s["n"], case["knn"], case["kreg"])
    elif kind == "lu":
        n = case["n"]
        g = _cuda_rng(seed)
        G = torch.randn((2 * n, n), generator=g, device=DEV) * (torch.rand((2 * n, n), generator=g, device=DEV) < 0.1)
        # symmetric as J^T J is: column-major and row-major are the same matrix
        s.update(A=((G.double().T @ G.double()) / (0.2 * n) + 0.05 * torch.eye(n, dtype=F64, device=DEV)).float().contiguous(),
                 b=torch.randn(n, generator=g, device=DEV), ipiv=torch.zeros(n, dtype=torch.int32, device=DEV),
                 x=torch.zeros(n, device=DEV))
    elif kind == "stream":
        W, H, n = case["width"], case["height"], case["cameras"]
        K = _K(W, H)
        poses = [np.eye(4) for _ in range(n)]
        for c in range(1, n):
            poses[c][:3, :3] = _rot("xyz"[c % 3], 12.0 * c)
            poses[c][:3, 3] = [0.1 * c, -0.05 * c, 0.02]
        sc = _scene("capsule", rnd)
        s.update(K=K, poses=poses, center=sc["joint"], R=_rot("z", 8.0),
                 frames=[_frames(sc, case["frames"], case["frames"], W, H, K, seed, c) for c in range(n)])
        s["stream"] = RigidStream([K] * n, poses, W, H, (case["dims"],) * 3, (1.0,) * 3, 0.016, s["center"], s["R"])
    elif kind == "session":
        cfg = _session_cfg(case)
        s.update(cfg=cfg, frames=_frames(_scene("capsule", rnd), case["frames"], 30, cfg["width"], cfg["height"], cfg["K"], seed),
                 session=FusionSession(cfg))
    else:
        cfgs = _mix(case)
        s["frames"] = [_frames(_scene(c["scene"], rnd), case["frames"], 30, c["width"], c["height"], c["K"], seed, i)
                       for i, c in enumerate(cfgs)]
        s["sessions"] = [FusionSession(c) for c in cfgs]
        s["batch"] = Batch(s["sessions"])
    return s


def _mc_volume(case, seed, rnd):
    """A fused volume: a noisy capsule pair, weights only in front of and inside its truncation band."""
    dims = (case["x"], case["y"], case["z"])
    voxel = 0.75 / max(dims)
    size = tuple(d * voxel for d in dims)
    vs = tuple(np.float32(a) / np.float32(b) for a, b in zip(size, dims))
    sc = _scene("capsule", rnd)
    sc["joint"] = sc["joint"] - np.array([0.0, 0.0, 0.8])
    sc["radius"] = 0.1
    gen = _cuda_rng(seed)
    ax = [torch.arange(d, device=DEV) * float(v) - 0.5 * float(s) for d, v, s in zip(dims, vs, size)]
    delta = 4 * voxel
    dist = None
    for a, b in _capsules(sc, 0.6):
        ab = b - a
        h = ((ax[0] - a[0]) * ab[0])[None, None, :] + ((ax[1] - a[1]) * ab[1])[None, :, None] + ((ax[2] - a[2]) * ab[2])[:, None, None]
        h = (h / float(ab @ ab)).clamp_(0, 1)
        d = ((ax[0] - a[0])[None, None, :] - h * ab[0]).square_()
        d += ((ax[1] - a[1])[None, :, None] - h * ab[1]).square_()
        d += ((ax[2] - a[2])[:, None, None] - h * ab[2]).square_()
        d = d.sqrt_()
        dist = d if dist is None else torch.minimum(dist, d)
    inside = sc["radius"] - dist + 0.1 * voxel * torch.randn(dist.shape, generator=gen, device=DEV)
    weights = ((inside <= delta) & (ax[2] < sc["joint"][2] + 0.02)[:, None, None]).float() * 3.0
    tsdf = torch.where(weights > 0, (inside / delta).clamp(-1, 1), torch.full_like(inside, -1.0))
    cap = 1_000_000
    return dict(dims=dims, size=size, vs=vs, tsdf=tsdf.reshape(-1).contiguous(), weights=weights.reshape(-1).contiguous(),
                points=torch.empty((cap, 3), device=DEV), count=torch.zeros(1, dtype=torch.int32, device=DEV))


def _voxel_inputs(case, seed, rnd):
    W, H, k = case["width"], case["height"], case["knn"]
    K = _K(W, H)
    dims = (case["x"], case["y"], case["z"])
    size = tuple(0.8 * d / max(dims) for d in dims)
    vs = tuple(np.float32(a) / np.float32(b) for a, b in zip(size, dims))
    gen = _cuda_rng(seed)
    sc = _scene("capsule", rnd)
    nodes, cell = _exactly(_surface(sc, 20000, gen), case["nodes"])
    centre = np.array([np.float32(v) for v in sc["joint"]])
    nodes_t = (nodes - torch.from_numpy(centre).to(DEV)).contiguous()
    n, S = nodes.shape[0], dims[0] * dims[1] * dims[2]
    radius = np.float32(cell)
    per = tuple(2 * (int(radius / v) + 1) + 1 for v in vs)
    depth = _frame(sc, 0.1, W, H, K, gen).float() * 0.001
    i32 = dict(dtype=torch.int32, device=DEV)
    return dict(K=K, dims=dims, size=size, vs=vs, S=S, centre=centre, nodes_t=nodes_t, n=n, per=per,
                radii=torch.full((n,), float(radius), device=DEV), T=_rigid_near_identity(n, gen, 0.02, 0.002),
                depth=torch.where(depth > 0, depth, torch.full_like(depth, math.inf)).contiguous(), delta=4 * float(max(vs)),
                idx=torch.full((S, k), -1, **i32), dist=torch.zeros((S, k), device=DEV), cnt=torch.zeros(S, **i32),
                w=torch.zeros((S, k), device=DEV), verts=torch.zeros((S, 3), device=DEV), coll=torch.zeros(S, **i32),
                tsdf=torch.full((S,), -1.0, device=DEV), weights=torch.zeros(S, device=DEV))


def _cloud_inputs(case, seed, rnd):
    W, H, m, k, kreg = case["width"], case["height"], case["points"], case["knn"], case["kreg"]
    K = _K(W, H)
    gen = _cuda_rng(seed)
    sc = _scene("capsule", rnd)
    points = _surface(sc, m, gen)
    depth = _depth(sc, 0.05, W, H, K)
    cap = 8192
    i32 = dict(dtype=torch.int32, device=DEV)
    return dict(K=K, points=points, n_points=torch.tensor([m], **i32), depth=depth.float().contiguous(),
                frame=_frame_vertices(depth, K).float().contiguous(), T=_rigid_near_identity(cap, gen, 0.01, 0.001),
                nodes=torch.zeros((cap, 3), device=DEV), radii=torch.zeros(cap, device=DEV),
                graph_T=torch.zeros((cap, 16), device=DEV), n_nodes=torch.zeros(1, **i32),
                idx=torch.empty((m, k), **i32), dist=torch.empty((m, k), device=DEV), w=torch.empty((m, k), device=DEV),
                gidx=torch.empty((cap, kreg), **i32), gdist=torch.empty((cap, kreg), device=DEV),
                warped=torch.empty((m, 3), device=DEV), corr=torch.empty((m, 2), **i32), n_corr=torch.zeros(1, **i32))


def _gn_inputs(case, seed, rnd):
    m, k, kreg = case["points"], case["knn"], case["kreg"]
    gen = _cuda_rng(seed)
    sc = _scene("capsule", rnd)
    points = _surface(sc, m, gen)
    n = case["nodes"]
    nodes, cell = _exactly(points, n)
    idx, dist = _nearest(points, nodes, k)
    r = 1.2 * cell
    w = torch.where(dist < r, torch.exp(-dist * dist / (2 * r * r)), torch.zeros_like(dist))
    w = (w / w.sum(1, keepdim=True).clamp(min=1e-30)).float()
    gidx, gdist = _nearest(nodes, nodes, kreg, skip=1)
    gidx = torch.where(gdist <= 2.0 * r, gidx, torch.full_like(gidx, -1))
    # a depth pixel near three in four vertices, a few millimetres off along its normal
    has = torch.randperm(m, generator=gen, device=DEV)[:3 * m // 4].sort()[0]
    pix = has[torch.randperm(has.numel(), generator=gen, device=DEV)]
    corr = torch.stack([has, pix], 1).int().contiguous()
    normals = torch.zeros((m, 3), dtype=F64, device=DEV)
    normals[pix] = points[has].double() - torch.as_tensor(sc["joint"], dtype=F64, device=DEV)
    normals[:, 0] *= 0.05
    normals = normals / normals.norm(dim=1, keepdim=True).clamp(min=1e-9)
    warped = points.double() + 0.002 * torch.randn((m, 3), generator=gen, dtype=F64, device=DEV)
    frame = torch.zeros((m, 3), dtype=F64, device=DEV)
    frame[pix] = points[has].double() + 0.003 * normals[pix]
    i32 = dict(dtype=torch.int32, device=DEV)
    return dict(points=points, n=n, n_points=torch.tensor([m], **i32), idx=idx.int().contiguous(), w=w.contiguous(), corr=corr,
                n_corr=torch.tensor([corr.shape[0]], **i32), frame=frame.float().contiguous(), normals=normals.float().contiguous(),
                warped=warped.float().contiguous(), nodes=nodes, T=_rigid_near_identity(n, gen, 0.002, 0.0005),
                n_nodes=torch.tensor([n], **i32), gidx=gidx.int().contiguous(), lam_d=1.0, lam_r=math.sqrt(200.0))


# ---- run ----

def run(s):
    return _RUN[s["case"]["kind"]](s)


def _run_prep(s):
    return list(af.loadProcessFrame(s["mm"], s["K"], bilateral_r=s["case"]["radius"]))


def _run_integrate(s):
    af.runIntegrateTSDFFromFrameKernel(s["tsdf"], s["weights"], s["depth"], (s["case"]["width"], s["case"]["height"]), 0.016,
                                       s["dims"], s["vs"], s["size"], s["R"], s["t"], s["K"])
    return [s["tsdf"], s["weights"]]


def _run_mc(s):
    s["count"].zero_()
    af.runMarchingCubesMeshKernel(s["points"], s["count"], s["tsdf"], s["weights"], s["dims"], s["vs"], s["size"])
    af.sortUnique(s["points"], s["count"])
    n = int(s["count"].item())
    return [_padded(s["points"][:n], s["points"].shape[0]), n]


def _run_voxel(s):
    dims, size, vs, S = s["dims"], s["size"], s["vs"], s["S"]
    I3 = np.eye(3)
    s["coll"].zero_()
    af.runTsdfKNNGraph(s["idx"], s["dist"], s["cnt"], s["nodes_t"], s["radii"], s["n"], vs, size, dims, s["per"])
    af.runComputeTsdfWarpWeightsKernel(s["w"], s["radii"], s["idx"], s["dist"], s["cnt"], S)
    af.runGenerateTsdfVerticesKernel(s["verts"], vs, size, dims)
    af.runTranslateKernel(s["verts"], S, s["centre"])
    af.runWarpTsdfKernel(s["verts"], s["T"], s["idx"], s["w"], s["cnt"], vs, size, dims)
    af.runCountCollisionsPerVoxelKernel(s["coll"], s["verts"], s["cnt"], vs, size, dims, I3, s["centre"])
    af.runIntegrateWarpedTSDFFromFrameKernel(s["tsdf"], s["weights"], s["verts"], s["coll"], s["cnt"], s["depth"],
                                             (s["case"]["width"], s["case"]["height"]), s["delta"], vs, size, dims, I3,
                                             s["centre"], s["K"])
    return [s["cnt"], s["coll"], s["verts"], s["tsdf"], s["weights"]]


def _run_cloud(s):
    c = s["case"]
    m = c["points"]
    s["n_nodes"].zero_()
    s["n_corr"].zero_()
    af.buildGraph(s["nodes"], s["radii"], s["graph_T"], s["n_nodes"], s["points"], s["n_points"], c["knn"], c["spacing"])
    n = int(s["n_nodes"].item())
    af.getKnnData(s["idx"], s["dist"], s["nodes"], s["n_nodes"], s["points"])
    gi, gd = s["gidx"][:n], s["gdist"][:n]
    af.getKnnData(gi, gd, s["nodes"], s["n_nodes"], s["nodes"][:n], excludeClosest=True)
    af.filterDisconnected(gi, gd, s["n_nodes"], s["radii"])
    af.runComputeWarpWeightsKernel(s["w"], s["radii"], s["idx"], s["dist"], m, s["n_nodes"])
    af.runWarpKernel(s["warped"], s["points"], s["T"], s["idx"], s["w"], m)
    af.runCorrespondencePairsKernel(s["corr"], s["n_corr"], s["warped"], m, s["K"], s["depth"], (c["height"], c["width"]),
                                    s["frame"], 0.01)
    nc = int(s["n_corr"].item())
    return [_padded(s["nodes"][:n], s["nodes"].shape[0]), s["idx"], s["dist"], _padded(gi, s["nodes"].shape[0]), s["w"], s["warped"],
            _padded(s["corr"][:nc], m), n, nc]


def _run_gn(s):
    g = s["system"]
    g.build(s["points"], s["n_points"], s["idx"], s["w"], s["corr"], s["n_corr"], s["frame"], s["normals"], s["warped"],
            s["nodes"], s["T"], s["n_nodes"], s["gidx"], s["lam_d"], s["lam_r"])
    x = g.solve(iterations=s["case"]["iterations"])
    jtj, jtr, rd, rr = g.export(s["n"], s["corr"].shape[0])
    return [x, jtj, jtr, rd, rr]


def _run_lu(s):
    n = s["case"]["n"]
    ok = af.linearSolverLUStable(None, n, s["A"], n, s["b"], s["ipiv"], s["x"])
    return [s["x"], ok]


def _run_stream(s):
    for f in range(s["case"]["frames"]):
        s["stream"].process([cam[f] for cam in s["frames"]])
    cloud, _, faces, tsdf, weights = s["stream"].outputs()
    return [cloud, tsdf, weights, faces.shape[0]]


_NODES, _CLOUD = 16384, 600_000


def _session_outputs(session):
    # the triangles' order is not defined, so the mesh stands here by its counts
    st = session.stats()
    tsdf, weights = session.tsdf()
    nodes, _, T = session.graph()
    return [tsdf, weights, _padded(nodes, _NODES), _padded(T, _NODES), _padded(session.point_cloud(), _CLOUD), st["n_nodes"], st["mesh_points"], st["correspondences"],
            st["gn_iterations_done"], st["mesh_vertices"], st["mesh_faces"]]


def _run_session(s):
    s["session"].reset()
    for f in s["frames"]:
        s["session"].process(f)
    return _session_outputs(s["session"])


def _run_batch(s):
    for session in s["sessions"]:
        session.reset()
    for f in range(s["case"]["frames"]):
        s["batch"].process([cam[f] for cam in s["frames"]])
    out = []
    for session in s["sessions"]:
        _, _, T = session.graph()
        tsdf, weights = session.tsdf()
        out.append([tsdf, weights, _padded(T, _NODES), _padded(session.point_cloud(), _CLOUD)])
    return out


_RUN = dict(prep=_run_prep, integrate=_run_integrate, mc=_run_mc, voxel=_run_voxel, cloud=_run_cloud, gn=_run_gn, lu=_run_lu,
            stream=_run_stream, session=_run_session, batch=_run_batch)


# ---- work ----

def _seen_fraction(dims, size, R, t, width, height, delta=0.016):
    """Share of a volume's voxels that one frame of the capsule pair updates, on a coarse grid."""
    K = _K(width, height)
    z = _depth(_scene("capsule", random.Random(0)), 0.0, width, height, K, "cpu").numpy()
    g = np.stack(np.meshgrid(*[(np.arange(40) + 0.5) / 40 - 0.5] * 3, indexing="ij"), -1).reshape(-1, 3) * np.asarray(size)
    p = g @ np.asarray(R).T + np.asarray(t)
    u = (K[0, 0] * p[:, 0] / p[:, 2] + K[0, 2] + 0.5).astype(int)
    v = (K[1, 1] * p[:, 1] / p[:, 2] + K[1, 2] + 0.5).astype(int)
    ok = (p[:, 2] > 1e-4) & (u >= 0) & (u < width) & (v >= 0) & (v < height)
    D = z[v.clip(0, height - 1), u.clip(0, width - 1)]
    return float((ok & np.isfinite(D) & (p[:, 2] - D <= delta)).mean())


def work(case):
    kind = case["kind"]
    if kind == "prep":
        P = case["width"] * case["height"]
        return dict(bytes=30 * P, flops=P * (60 + 8 * (2 * case["radius"] + 1) ** 2))
    if kind == "integrate":
        S = case["x"] * case["y"] * case["z"]
        dims = np.array([case["x"], case["y"], case["z"]])
        share = _seen_fraction(dims, 1.024 * dims / dims.max(), _rot("y", 10.0), [0.0, 0.0, 0.8], case["width"], case["height"])
        return dict(bytes=16 * share * S + 4 * case["width"] * case["height"], flops=30 * S)
    if kind == "mc":
        S, m = case["x"] * case["y"] * case["z"], max(case["x"], case["y"], case["z"])
        # the surface of the capsule pair, in voxel faces, with about three edges crossed per face
        return dict(bytes=8 * S + 12 * 3 * (0.22 / (0.75 / m) ** 2), flops=16 * S)
    if kind == "voxel":
        # counts, collisions, vertices and volume of every voxel, KNN and weights of the supported ones
        S = case["x"] * case["y"] * case["z"]
        return dict(bytes=S * (4 + 4 + 12) + 0.15 * S * (12 * case["knn"] + 16), flops=0.15 * S * 200)
    if kind == "cloud":
        m, P = case["points"], case["width"] * case["height"]
        n = min(8000, 0.12 / case["spacing"] ** 2)
        return dict(bytes=m * (12 + 12 * case["knn"] + 12 + 8) + n * (12 + 64 + 8 * case["kreg"]) + 16 * min(m, P), flops=m * n * 8)
    if kind == "gn":
        m, n, k = case["points"], case["nodes"], case["knn"]
        blocks = 14 * n  # a node, the nodes it shares vertices with and its regularisation edges
        return dict(bytes=m * (12 + 8 * k + 12) + 0.75 * m * 32 + n * 76 + (6 * n) ** 2 * 4 + 48 * n,
                    flops=0.75 * m * k * k * 72 + case["iterations"] * blocks * 72)
    if kind == "lu":
        n = case["n"]
        return dict(bytes=4 * n * n + 8 * n, flops=2 * n ** 3 / 3)
    if kind == "stream":
        P, S = case["width"] * case["height"], case["dims"] ** 3
        return dict(bytes=case["frames"] * (case["cameras"] * 14 * P + 8 * S), flops=case["frames"] * (30 * S + 300 * P * case["cameras"]))
    if kind == "session":
        return _session_work(case["dims"], case["voxel"], case["width"] * case["height"], case["graph_radius"],
                             4 if case["precision"] == "fp16" else 8, case["frames"])
    total = dict(bytes=0.0, flops=0.0)
    for c in _mix(case):
        w = _session_work(c["dims"][0], c["volume_size"][0] / c["dims"][0], c["width"] * c["height"], c["graph_radius"], 8,
                          case["frames"])
        total = {k: total[k] + w[k] for k in total}
    return total


def _session_work(dims, voxel, P, graph_radius, voxel_bytes, frames):
    """Reset of the volume, then per frame the depth in, its maps out, the voxels around the seen surface
    (0.1 m^2) read and written, the cloud and triangles out, and five solves of ten PCG iterations."""
    area = 0.1
    nodes, near, cloud = area / graph_radius ** 2, area * 4 * graph_radius / voxel ** 3, 3 * area / voxel ** 2
    return dict(bytes=voxel_bytes * dims ** 3 + frames * (30 * P + 2 * voxel_bytes * near + cloud * (12 + 32)),
                flops=frames * (near * 150 + nodes * 14 * 72 * 50 + cloud * 16 * 72))


# ---- exact ----

def exact(case, seed):
    f = _EXACT.get(case["kind"])
    return f(prepare(case, seed)) if f else None


def _f64(values):
    """The 64-bit values of the 32-bit numbers that the entry points take."""
    return torch.as_tensor(np.asarray(values, np.float32).astype(np.float64), device=DEV)


def _bilateral64(d32, r):
    """Range / spatial filter in 64 bits; the range bucket of a pair of pixels is the 32-bit one."""
    sI, sS, thr = 0.03, 2.0, 0.09
    H, W = d32.shape
    fc = [np.float32(math.exp(-((i / 10.0) ** 2) / 2)) for i in range(31)]
    clr = torch.tensor([int(v / fc[30]) for v in fc], dtype=F64, device=DEV)
    norm = torch.tensor(np.float32(30 / (3 * sI)), device=DEV)
    ys, xs = torch.arange(H, device=DEV), torch.arange(W, device=DEV)
    num, den = torch.zeros((H, W), dtype=F64, device=DEV), torch.zeros((H, W), dtype=F64, device=DEV)
    for dy in range(-r, r + 1):
        for dx in range(-r, r + 1):
            cur = d32[(ys + dy).clamp(0, H - 1)][:, (xs + dx).clamp(0, W - 1)]
            diff = (d32 - cur).abs()
            ok = torch.isfinite(cur) & (diff <= np.float32(thr))
            bucket = torch.where(ok, diff * norm, torch.zeros_like(diff)).clamp(max=30).long()
            # the table's entry for column offset a and row offset b is g[a] g[b]: symmetric
            w = torch.where(ok, math.exp(-(dx * dx + dy * dy) / (2 * sS * sS)) * clr[bucket], torch.zeros_like(num))
            num += torch.where(ok, cur.double(), torch.zeros_like(num)) * w
            den += w
    return torch.where(torch.isfinite(d32), num / den, torch.full_like(num, math.inf))


def _filtered(mm, r):
    d = mm.float() * torch.tensor(np.float32(0.001), device=DEV)
    d = torch.where((d > 1.2) | (d < 1e-4), torch.full_like(d, math.inf), d)
    return _bilateral64(d, r)


def _exact_prep(s):
    d = _filtered(s["mm"], s["case"]["radius"])
    V = _frame_vertices(d, s["K"])
    N = torch.zeros_like(V)
    H, W = d.shape
    ok = V[..., 2] > 1e-4
    inner = ok[1:-1, 1:-1] & ok[1:-1, 2:] & ok[1:-1, :-2] & ok[2:, 1:-1] & ok[:-2, 1:-1]
    dX, dY = V[1:-1, 2:] - V[1:-1, :-2], V[2:, 1:-1] - V[:-2, 1:-1]
    gX, gY = (g / g[..., :2].norm(dim=-1, keepdim=True) for g in (dX, dY))
    n = torch.linalg.cross(gY, gX)
    n = n / n.norm(dim=-1, keepdim=True)
    ang = torch.acos(n[..., 2].clamp(-1, 1))
    keep = inner & ~((ang > 1.3) & (ang < 2.1))
    N[1:-1, 1:-1] = torch.where(keep[..., None], n, torch.zeros_like(n))
    border = torch.ones((H, W), dtype=torch.bool, device=DEV)
    border[1:-1, 1:-1] = keep
    d = torch.where(border, d, torch.full_like(d, math.inf))
    V = torch.where(border[..., None], V, torch.zeros_like(V))
    return [d, V, N, V.reshape(-1, 3).sum(0) / (V[..., 2] > 1e-4).sum()]


def _update64(p, depth, K, delta):
    """New signed distance of camera-space points and whether they are updated."""
    H, W = depth.shape
    z = p[:, 2]
    zi = 1.0 / torch.where(z < 1e-4, torch.ones_like(z), z)
    u = (K[0, 0] * p[:, 0] * zi + K[0, 2] + 0.5).trunc()
    v = (K[1, 1] * p[:, 1] * zi + K[1, 2] + 0.5).trunc()
    ok = (z >= 1e-4) & (u >= 0) & (u < W) & (v >= 0) & (v < H)
    D = depth.reshape(-1)[torch.where(ok, v * W + u, torch.zeros_like(u)).long()].double()
    sdf = z - D
    ok &= torch.isfinite(D) & (D >= 1e-4) & (sdf <= delta)
    return torch.where(sdf < -delta, torch.full_like(sdf, -1.0), sdf / delta), ok


def _voxel_centres(dims, vs, size, z0, z1):
    ax = [torch.arange(a, b, dtype=F64, device=DEV) * v - 0.5 * h
          for (a, b), v, h in zip(((0, dims[0]), (0, dims[1]), (z0, z1)), _f64(vs), _f64(size))]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    return torch.stack([x, y, z], -1).reshape(-1, 3)


def _fresh64(depth, K, delta, dims, vs, size, R, t):
    tsdf, weights = [], []
    step = max(1, (1 << 23) // (dims[0] * dims[1]))
    for z0 in range(0, dims[2], step):
        p = _voxel_centres(dims, vs, size, z0, min(dims[2], z0 + step)) @ _f64(R).T + _f64(t)
        tn, ok = _update64(p, depth, np.asarray(K, np.float32).astype(np.float64), float(np.float32(delta)))
        tsdf.append(torch.where(ok, tn, torch.full_like(tn, -1.0)))
        weights.append(ok.double())
    return torch.cat(tsdf), torch.cat(weights)


def _exact_integrate(s):
    return list(_fresh64(s["depth"], s["K"], 0.016, s["dims"], s["vs"], s["size"], s["R"], s["t"]))


def _exact_voxel(s):
    dims, vs, size, k, S, n = s["dims"], s["vs"], s["size"], s["case"]["knn"], s["S"], s["n"]
    r = float(s["radii"][0])
    C = _voxel_centres(dims, vs, size, 0, dims[2])
    best = torch.full((S, k + 1), math.inf, dtype=F64, device=DEV)
    who = torch.full((S, k + 1), -1, dtype=torch.int64, device=DEV)
    half, inv = 0.5 * _f64(size), 1.0 / _f64(vs)
    base = ((s["nodes_t"].double() + half) * inv).trunc().long().cpu()
    for j in range(n):
        lo = [max(int(base[j, c]) - (s["per"][c] - 1) // 2, 0) for c in range(3)]
        hi = [min(int(base[j, c]) - (s["per"][c] - 1) // 2 + s["per"][c] - 1, dims[c] - 1) for c in range(3)]
        if any(a > b for a, b in zip(lo, hi)):
            continue
        z, y, x = torch.meshgrid(*[torch.arange(lo[c], hi[c] + 1, device=DEV) for c in (2, 1, 0)], indexing="ij")
        v = ((z * dims[1] + y) * dims[0] + x).reshape(-1)
        d = (C[v] - s["nodes_t"][j].double()).norm(dim=1)
        v, d = v[d <= 2.0 * r], d[d <= 2.0 * r]
        best[v, k], who[v, k] = d, j
        order = torch.argsort(best[v], dim=1, stable=True)
        best[v], who[v] = best[v].gather(1, order), who[v].gather(1, order)
        best[v, k] = math.inf
    best, who = best[:, :k], who[:, :k]
    near = torch.isfinite(best)
    w = torch.where(near, torch.exp(-best * best / (2 * r * r)), torch.zeros_like(best))
    w = w / w.sum(1, keepdim=True).clamp(min=1e-300)
    c64 = _f64(s["centre"])
    p0 = C + c64
    T = s["T"].double().reshape(-1, 4, 4).transpose(1, 2)
    q = torch.zeros_like(p0)
    for a in range(k):
        M = T[who[:, a].clamp(min=0)]
        q += w[:, a, None] * ((M[:, :3, :3] @ p0[..., None])[..., 0] + M[:, :3, 3])
    has = near[:, 0]
    q = torch.where(has[:, None], q, p0)
    tv = ((q - c64 + half) * inv).trunc()
    D = torch.tensor(dims, device=DEV)
    inside = has & (tv >= 0).all(1) & (tv < D).all(1)
    target = torch.where(inside, (tv[:, 2] * dims[1] + tv[:, 1]) * dims[0] + tv[:, 0], torch.zeros_like(tv[:, 0])).long()
    coll = torch.zeros(S, device=DEV).index_add_(0, target[inside], torch.ones(int(inside.sum()), device=DEV))
    tn, ok = _update64(q, s["depth"], s["K"], float(np.float32(s["delta"])))
    ok &= inside & (coll[target] <= 1)
    return [None, None, q, torch.where(ok, tn, torch.full_like(tn, -1.0)), ok.double()]


def _exact_cloud(s):
    c = s["case"]
    p = s["points"]
    r = torch.tensor(np.float32(c["spacing"]), device=DEV)
    # greedy subsampling in order; which point a node covers is the 32-bit comparison of the path
    free = torch.ones(p.shape[0], dtype=torch.bool, device=DEV)
    chosen = []
    at = 0
    while True:
        at = int(free.to(torch.uint8).argmax())
        if not bool(free[at]):
            break
        chosen.append(at)
        d = (p - p[at]).square()
        free &= ~(((d[:, 0] + d[:, 1]) + d[:, 2]).sqrt() < r)
        free[at] = False
    nodes = p[torch.tensor(chosen, device=DEV)]
    idx, dist = _nearest(p, nodes, c["knn"])
    w = torch.where(dist < float(r), torch.exp(-dist * dist / (2 * float(r) ** 2)), torch.zeros_like(dist))
    tot = w.sum(1, keepdim=True)
    w = torch.where(tot > 0, w / tot.clamp(min=1e-300), w)
    T = s["T"].double().reshape(-1, 4, 4).transpose(1, 2)
    q = torch.zeros((p.shape[0], 3), dtype=F64, device=DEV)
    for a in range(c["knn"]):
        M = T[idx[:, a]]
        q += w[:, a, None] * ((M[:, :3, :3] @ p.double()[..., None])[..., 0] + M[:, :3, 3])
    q = torch.where(tot > 0, q, p.double())
    return [_padded(nodes.double(), s["nodes"].shape[0]), None, dist, None, w, q, None, None, None]


def _grad64(p):
    G = torch.zeros((p.shape[0], 3, 6), dtype=F64, device=DEV)
    G[:, 0, 1], G[:, 0, 2] = p[:, 2], -p[:, 1]
    G[:, 1, 0], G[:, 1, 2] = -p[:, 2], p[:, 0]
    G[:, 2, 0], G[:, 2, 1] = p[:, 1], -p[:, 0]
    G[:, 0, 3] = G[:, 1, 4] = G[:, 2, 5] = 1.0
    return G


def _exact_gn(s):
    n, k, kreg = s["n"], s["case"]["knn"], s["case"]["kreg"]
    lam_r = float(np.float32(s["lam_r"]))
    A = torch.zeros((n, n, 6, 6), dtype=F64, device=DEV).reshape(n * n, 6, 6)
    g = torch.zeros((n, 6), dtype=F64, device=DEV)
    v, px = s["corr"][:, 0].long(), s["corr"][:, 1].long()
    nrm = s["normals"][px].double()
    rd = (nrm * (s["warped"][v].double() - s["frame"][px].double())).sum(1)
    row = (nrm[:, None, :] @ _grad64(s["points"][v].double()))[:, 0]
    w = s["w"][v].double()
    J = torch.where(w < 1e-4, torch.zeros_like(w), w)[..., None] * row[:, None, :]
    nd = s["idx"][v].long()
    for a in range(k):
        g.index_add_(0, nd[:, a], J[:, a] * rd[:, None])
        for b in range(k):
            A.index_add_(0, nd[:, a] * n + nd[:, b], J[:, a, :, None] * J[:, b, None, :])
    gi = s["gidx"].long()
    own = torch.arange(n, device=DEV)[:, None].expand(-1, kreg)
    live = (gi >= 0) & (gi < n)
    P = s["nodes"].double()
    T = s["T"].double().reshape(-1, 4, 4).transpose(1, 2)
    move = lambda j, q: (T[j][..., :3, :3] @ q[..., None])[..., 0] + T[j][..., :3, 3]  # noqa: E731
    rr = (move(own, P[own]) - move(gi.clamp(min=0), P[own])) * lam_r * live[..., None]
    G = _grad64(P) * lam_r
    src, dst = own[live], gi[live]
    GtG = (G.transpose(1, 2) @ G)[src]
    Gtr = (G[src].transpose(1, 2) @ rr[live][..., None])[..., 0]
    for a, b, sign in ((src, src, 1.0), (dst, dst, 1.0), (src, dst, -1.0), (dst, src, -1.0)):
        A.index_add_(0, a * n + b, sign * GtG)
    g.index_add_(0, src, Gtr)
    g.index_add_(0, dst, -Gtr)
    D = A.reshape(n, n, 6, 6)[torch.arange(n), torch.arange(n)]
    untouched = D.abs().sum((1, 2)) == 0
    D = torch.where(untouched[:, None, None], torch.eye(6, dtype=F64, device=DEV), D)
    A.reshape(n, n, 6, 6)[torch.arange(n), torch.arange(n)] = D
    A = A.reshape(n, n, 6, 6).transpose(1, 2).reshape(6 * n, 6 * n)
    b = g.reshape(-1)
    Minv = torch.linalg.inv(D)
    z_of = lambda r: (Minv @ r.reshape(n, 6, 1)).reshape(-1)  # noqa: E731
    x, r = torch.zeros_like(b), b.clone()
    z = z_of(r)
    p, rz = z.clone(), r @ z
    for _ in range(s["case"]["iterations"]):
        Ap = A @ p
        alpha = rz / (p @ Ap)
        x, r = x + alpha * p, r - alpha * Ap
        z = z_of(r)
        new = r @ z
        p, rz = z + (new / rz) * p, new
    return [x, A, b, rd, rr.reshape(-1)]


def _exact_lu(s):
    return [torch.linalg.solve(s["A"].double(), s["b"].double()), None]


def _exact_stream(s):
    c = s["case"]
    clouds, depth0 = [], None
    for cam in range(c["cameras"]):
        d = _filtered(s["frames"][cam][-1], 2)
        depth0 = d if cam == 0 else depth0
        V = _frame_vertices(d, s["K"]).reshape(-1, 3)
        M = _f64(s["poses"][cam])
        clouds.append(V @ M[:3, :3].T + M[:3, 3])
    n = c["dims"]
    size = (1.0,) * 3
    vs = (np.float32(1.0) / np.float32(n),) * 3
    return [torch.cat(clouds), *_fresh64(depth0, s["K"], 0.016, (n,) * 3, vs, size, s["R"], s["center"]), None]


_EXACT = dict(prep=_exact_prep, integrate=_exact_integrate, voxel=_exact_voxel, cloud=_exact_cloud, gn=_exact_gn, lu=_exact_lu,
              stream=_exact_stream)

"""The work that programs on the `wos` package have it do, as cases that can be
timed: what a program holds before the call (`prepare`), one pass through the
package's public entry points (`run`), the bytes and operations a pass cannot do
without (`work`) and, where there is one, the pass's result in 64 bits
(`exact`).  Sizes are those of the repository's workloads (bench.py, tests/) or
lie between them; every input is made from the seed.
"""
from __future__ import annotations

import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "diff-wos_b200"))
import wos  # noqa: E402
from wos.native import AdjointSettings, WalkSettings  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # u at a few points that a user clicks on or probes: all latency
        dict(name="probe2d", kind="solve2d", segments=301, lobes=3, points=37, nwalks=16, nsteps=64, source="none"),
        # the plain primal solve on a pixel grid inside a circle of 1,024 segments
        dict(name="grid2d", kind="solve2d", segments=1024, lobes=0, points=14592, nwalks=64, nsteps=32,
             source="none"),
        # Poisson problem with the Green's function importance sampled
        dict(name="source2d", kind="solve2d", segments=4096, lobes=5, points=12500, nwalks=64, nsteps=64,
             source="green"),
        # the 2D differentiable solve: values, source and vertices, 512^2 grid
        dict(name="grad2d", kind="grad2d", segments=4096, lobes=5, points=80222, nwalks=256, nsteps=64,
             source="green"),
        # one iteration of the inverse problem in the boundary values
        dict(name="inverse2d", kind="inverse2d", segments=8192, lobes=5, points=19988, nwalks=32, nsteps=64),
        # one iteration of a shape optimisation: the scene is built anew from
        # the moved vertices, solved and differentiated
        dict(name="shape2d", kind="shape2d", segments=1024, lobes=5, points=1600, nwalks=128, nsteps=64),
        # a derivative image (forward mode) over a detector's pixels
        dict(name="image2d", kind="image2d", segments=777, lobes=4, res=128, nwalks=16, nsteps=64),
        # 3D primal solve on a displaced sphere of 20,480 triangles
        dict(name="solve3d", kind="solve3d", level=5, points=20000, nwalks=64, nsteps=64),
        # 3D differentiable solve (values and vertices), 81,920 triangles
        dict(name="grad3d", kind="grad3d", level=6, points=100000, nwalks=16, nsteps=64),
        # closest points and signed distances of a point cloud
        dict(name="closest3d", kind="closest3d", level=5, points=200003),
        # a mesh that deforms: trees and normals rebuilt, then signed distances
        dict(name="move3d", kind="move3d", level=6, points=10007),
        # many scenes of uneven sizes, forward and adjoint, as one plan
        dict(name="batch", kind="batch", scenes=6, least=1000, most=20000, nwalks=40, segments=2500, level=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve2d", "solve2d", "grad2d", "inverse2d", "shape2d", "image2d", "solve3d", "grad3d",
                       "closest3d", "move3d", "batch"])
    c = dict(kind=kind)
    if kind == "solve2d":
        c.update(segments=_log(rng, 128, 16384), lobes=rng.choice([0, 3, 4, 5, 7, 9]), points=_log(rng, 1, 40000),
                 nwalks=_log(rng, 1, 256), nsteps=rng.choice([32, 64]), source=rng.choice(["none", "disk", "green"]))
    elif kind == "grad2d":
        c.update(segments=_log(rng, 256, 16384), lobes=rng.randint(3, 9), points=_log(rng, 100, 40000),
                 nwalks=_log(rng, 8, 128), nsteps=64, source=rng.choice(["none", "disk", "green"]))
    elif kind == "inverse2d":
        c.update(segments=_log(rng, 256, 16384), lobes=rng.randint(3, 9), points=_log(rng, 200, 60000),
                 nwalks=_log(rng, 8, 64), nsteps=64)
    elif kind == "shape2d":
        c.update(segments=_log(rng, 100, 16384), lobes=rng.randint(3, 9), points=_log(rng, 100, 5000),
                 nwalks=_log(rng, 8, 128), nsteps=64)
    elif kind == "image2d":
        c.update(segments=_log(rng, 100, 8192), lobes=rng.randint(3, 9), res=rng.randint(32, 200),
                 nwalks=_log(rng, 2, 32), nsteps=64)
    elif kind == "solve3d":
        c.update(level=rng.randint(2, 6), points=_log(rng, 10, 30000), nwalks=_log(rng, 1, 64), nsteps=64)
    elif kind == "grad3d":
        c.update(level=rng.randint(3, 6), points=_log(rng, 100, 60000), nwalks=_log(rng, 4, 16), nsteps=64)
    elif kind == "closest3d":
        c.update(level=rng.randint(2, 6), points=_log(rng, 10, 400000))
    elif kind == "move3d":
        c.update(level=rng.randint(2, 6), points=_log(rng, 10, 40000))
    else:
        c.update(scenes=rng.randint(3, 9), least=_log(rng, 100, 1000), most=_log(rng, 2000, 20000),
                 nwalks=_log(rng, 16, 48), segments=_log(rng, 256, 16384), level=rng.randint(3, 5))
    return c


# ---------------------------------------------------------------- inputs
def _gen(seed, k=0):
    return torch.Generator(device=DEV).manual_seed((int(seed) * 1000003 + 7919 * k + 12345) & 0x7FFFFFFFFFFFFFFF)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)


def _star(segments, lobes, g):
    """A closed counter-clockwise star (a circle for no lobes): vertices, faces
    and the radius as a function of the angle."""
    amp = float(0.15 + 0.15 * _rand(g, 1)) if lobes else 0.0
    phase = float(2 * math.pi * _rand(g, 1))
    base = 0.6 if lobes else 1.0
    th = 2 * math.pi * torch.arange(segments, device=DEV, dtype=torch.float64) / segments
    radius = lambda t: base + amp * torch.cos(lobes * t + phase)  # noqa: E731
    r = radius(th)
    V = torch.stack([r * torch.cos(th), r * torch.sin(th)], 1).float().contiguous()
    i = torch.arange(segments, device=DEV, dtype=torch.int32)
    F = torch.stack([i, (i + 1) % segments], 1).to(torch.int32).contiguous()
    return V, F, radius


def _grid_points(n, radius, g):
    """n interior points of a pixel grid: the rows of the finest grid needed,
    thinned evenly to the count, in row-major order."""
    res = int(math.sqrt(n)) + 2
    ext = 0.9
    while True:
        s = torch.linspace(-ext, ext, res, device=DEV, dtype=torch.float64)
        s = s + (float(_rand(g, 1)) - 0.5) * 1e-3
        Y, X = torch.meshgrid(s.flip(0), s, indexing="ij")
        x, y = X.reshape(-1), Y.reshape(-1)
        m = torch.hypot(x, y) < radius(torch.atan2(y, x)) - 0.002
        P = torch.stack([x[m], y[m]], 1)
        if P.shape[0] >= n:
            keep = torch.linspace(0, P.shape[0] - 1, n, device=DEV, dtype=torch.float64).round().long()
            return P[keep].float().contiguous()
        res = int(res * 1.1) + 2


def _values2(V, g):
    c = 2 * _rand(g, 3) - 1
    x, y = V[:, 0].double(), V[:, 1].double()
    return (torch.sin(3 * x + c[0]) * torch.cos(2 * y + c[1]) + 0.3 * c[2] * x * y).float().contiguous()


@functools.lru_cache(maxsize=None)
def _sphere(level):
    return wos.shapes.icosphere(level)


def _mesh(level, g):
    """A sphere displaced radially by up to 15 % with a few seeded waves."""
    V, F = _sphere(level)
    V = torch.as_tensor(V, device=DEV, dtype=torch.float64)
    k = 6 * (2 * _rand(g, 8, 3) - 1)
    ph = 2 * math.pi * _rand(g, 8)
    a = _rand(g, 8)
    d = (torch.sin(V @ k.T + ph) * a).sum(1) / a.sum()
    return (V * (1 + 0.15 * d)[:, None]).float().contiguous(), torch.as_tensor(F, device=DEV, dtype=torch.int32)


def _points3(n, V, F, g, outside=False):
    """Points inside the (star-shaped) mesh: a random boundary point scaled by
    u^(1/3); with `outside`, by up to 1.3."""
    f = F.long()[(_rand(g, n) * F.shape[0]).long().clamp_max(F.shape[0] - 1)]
    b = _rand(g, n, 2)
    s = torch.sqrt(b[:, :1])
    w = torch.cat([1 - s, s * (1 - b[:, 1:]), s * b[:, 1:]], 1)
    p = (V.double()[f] * w[:, :, None]).sum(1)
    u = _rand(g, n) ** (1.0 / 3.0) * (1.3 if outside else 0.998)
    return (p * u[:, None]).float().contiguous()


def _values3(V, g):
    c = 2 * _rand(g, 2) - 1
    x, y, z = V.double().unbind(1)
    return (x * x - y * y + z + 0.2 * c[0] * x * y + 0.2 * c[1] * y * z).float().contiguous()


def _source(kind, g):
    """(source_type, parameters) of a scene: a constant for the importance
    sampled Green's function, a Gaussian bump otherwise."""
    if kind == "none":
        return 0, None
    a = float(_rand(g, 1))
    if kind == "green":
        return 2, torch.tensor([1.0, 2.0, a, 0.25, 1.0], device=DEV)
    return 1, torch.tensor([0.1 * a, -0.1, 0.3, 0.25, 2.0], device=DEV)


def _scene2(c, seed):
    g = _gen(seed)
    V, F, radius = _star(c["segments"], c["lobes"], g)
    val = _values2(V, g)
    st, sp = _source(c.get("source", "none"), g)
    P = _grid_points(c["points"], radius, g) if "points" in c else None
    return V, F, val, st, sp, P


def _solver2(c):
    kw = dict(nwalks=c["nwalks"], nsteps=c["nsteps"], epsilon=1e-3)
    if c.get("source", "none") == "none":
        return wos.WoSCUDA(**kw)
    return wos.WoSWithSourceCUDA(use_IS_for_greens=c["source"] == "green", **kw)


def _shape_solver(c, fwd, **more):
    bwd = wos.OursCUDA(nwalks=c["nwalks"], nsteps=c["nsteps"], epsilon=1e-3, epsilon2=1e-3, clamping=0.1,
                       use_IS_for_greens=c.get("source") == "green", **more)
    return wos.CustomSolver(fwd_solver=fwd, bwd_solver=bwd)


def _batch_sizes(c, i):
    """Points and walks of item i of a batch: spread over the case's ranges."""
    u, v = (0.13 + 0.618034 * i) % 1.0, (0.71 + 0.754878 * i) % 1.0
    return int(c["least"] * (c["most"] / c["least"]) ** u), max(1, int(c["nwalks"] * (0.4 + 1.2 * v)))


# ---------------------------------------------------------------- passes
def prepare(case, seed):
    c, kind = case, case["kind"]
    s = dict(kind=kind, seed=int(seed) & 0x7FFFFFFF)
    if kind == "solve2d":
        V, F, val, st, sp, P = _scene2(c, seed)
        s.update(scene=wos.Polyline(V, F, val, source_type=st, source_params=sp), P=P, solver=_solver2(c))
    elif kind == "grad2d":
        V, F, val, st, sp, P = _scene2(c, seed)
        V.requires_grad_(True)
        val.requires_grad_(True)
        leaves = [V, val]
        if sp is not None:
            sp.requires_grad_(True)
            leaves.append(sp)
        s.update(scene=wos.Polyline(V, F, val, source_type=st, source_params=sp), P=P, leaves=leaves,
                 solver=_shape_solver(c, _solver2(c), grad_values=True, grad_source=sp is not None,
                                      source_in_normal_derivative=sp is not None))
    elif kind == "inverse2d":
        V, F, val, _, _, P = _scene2(c, seed)
        scene = wos.Polyline(V, F, val)
        target = wos.WoSCUDA(nwalks=c["nwalks"], nsteps=c["nsteps"]).solve(P, scene, seed=s["seed"] + 1)
        s.update(scene=scene, P=P, target=target, values=(0.5 * val).requires_grad_(True),
                 solver=wos.WoSCUDA(nwalks=c["nwalks"], nsteps=c["nsteps"], epsilon=1e-3))
    elif kind == "shape2d":
        V, F, val, _, _, P = _scene2(c, seed)
        fwd = _solver2(c)
        target = fwd.solve(0.5 * P, wos.Polyline(V, F, val), seed=s["seed"] + 1)
        t = torch.tensor([0.05, -0.03], device=DEV, requires_grad=True)
        s.update(V=V, F=F, values=val, P=(0.5 * P).contiguous(), target=target, t=t, solver=_shape_solver(c, fwd))
    elif kind == "image2d":
        V, F, val, _, _, _ = _scene2(c, seed)
        g = _gen(seed, 1)
        dV = (2 * _rand(g, 1, 2) - 1).float().expand_as(V).contiguous()
        s.update(V=V, F=F, values=val, dV=dV, scene=wos.Polyline(V, F, val),
                 detector=wos.Detector(vmin=(-0.8, -0.8), vmax=(0.8, 0.8), res=(c["res"], c["res"])),
                 solver=_shape_solver(c, _solver2(c)))
    elif kind in ("solve3d", "grad3d"):
        g = _gen(seed)
        V, F = _mesh(c["level"], g)
        val = _values3(V, g)
        P = _points3(c["points"], V, F, g)
        fwd = wos.WoS3DCUDA(nwalks=c["nwalks"], nsteps=c["nsteps"], epsilon=1e-3)
        if kind == "solve3d":
            s.update(scene=wos.Scene3D(V, F, val), P=P, solver=fwd)
        else:
            V.requires_grad_(True)
            val.requires_grad_(True)
            bwd = wos.Ours3D(nwalks=c["nwalks"], nsteps=c["nsteps"], epsilon=1e-3, grad_values=True)
            s.update(scene=wos.Scene3D(V, F, val), P=P, leaves=[V, val],
                     solver=wos.CustomSolver(fwd_solver=fwd, bwd_solver=bwd))
    elif kind == "closest3d":
        g = _gen(seed)
        V, F = _mesh(c["level"], g)
        s.update(scene=wos.Scene3D(V, F, _values3(V, g)), P=_points3(c["points"], V, F, g, outside=True))
    elif kind == "move3d":
        g = _gen(seed)
        V, F = _mesh(c["level"], g)
        scene = wos.Scene3D(V, F, _values3(V, g))
        s.update(scene=scene, V=_mesh(c["level"], g)[0], P=_points3(c["points"], V, F, g, outside=True))
    else:
        items = []
        for i in range(c["scenes"]):
            g = _gen(seed, i)
            n, nw = _batch_sizes(c, i)
            st = WalkSettings(nwalks=nw, nsteps=64, epsilon=1e-3, seed=s["seed"] + i)
            if i % 2 == 0:
                V, F, radius = _star(max(64, c["segments"] >> (i // 2)), 3 + i, g)
                P = _grid_points(n, radius, g)
                scene = wos.Polyline(V, F, _values2(V, g))
            else:
                V, F = _mesh(max(2, c["level"] - i // 2), g)
                P = _points3(n, V, F, g)
                scene = wos.Scene3D(V, F, _values3(V, g))
            items.append(wos.BatchItem(scene, P, st, loss_kind=1))
        s.update(plan=wos.BatchPlan(items, AdjointSettings(want_dV=True, want_dg=True)), n=len(items))
    return s


def run(s):
    kind = s["kind"]
    if kind in ("solve2d", "solve3d"):
        return s["solver"].solve(s["P"], s["scene"], seed=s["seed"])
    if kind in ("grad2d", "grad3d"):
        u = s["solver"].walk(s["P"], s["scene"], seed=s["seed"])
        loss = (u * u).mean()
        return dict(u=u.detach(), grads=list(torch.autograd.grad(loss, s["leaves"])))
    if kind == "inverse2d":
        s["scene"].update_values(s["values"])
        u = s["solver"].walk(s["P"], s["scene"], seed=s["seed"])
        loss = ((u - s["target"]) ** 2).mean()
        return dict(u=u.detach(), grad=torch.autograd.grad(loss, s["values"])[0])
    if kind == "shape2d":
        scene = wos.Polyline(s["V"] + s["t"], s["F"], s["values"])
        u = s["solver"].walk(s["P"], scene, seed=s["seed"])
        loss = ((u - s["target"]) ** 2).mean()
        return dict(u=u.detach(), grad=torch.autograd.grad(loss, s["t"])[0])
    if kind == "image2d":
        import torch.autograd.forward_ad as fwAD
        with fwAD.dual_level():
            scene = s["scene"]
            scene.vertices = fwAD.make_dual(s["V"], s["dV"])
            image = s["solver"].walk_detector(scene, s["detector"], seed=s["seed"])
            u, du = fwAD.unpack_dual(image)
            scene.vertices = s["V"]
        return dict(u=u, du=du)
    if kind == "closest3d":
        its = s["scene"].closest_point(s["P"])
        return dict(prim=its.prim_id, p=its.p, uv=its.uv, sdf=s["scene"].sdf(s["P"]))
    if kind == "move3d":
        s["scene"].update_vertices(s["V"])
        return dict(normals=s["scene"].normals, sdf=s["scene"].sdf(s["P"]))
    s["plan"].run()
    out = [s["plan"].outputs(i) for i in range(s["n"])]
    return [{k: o[k] for k in ("mean", "var", "loss", "dV", "dg")} for o in out]


# ---------------------------------------------------------------- work
#: Nearest queries of one walk, and of one sample of the shape estimator beside its walk (bisection of the ball and
#: two walks), in 2D and 3D; operations of one exact point-to-primitive distance.
QUERIES, SAMPLE, DISTANCE = {2: 10, 3: 18}, {2: 22, 3: 40}, {2: 14, 3: 45}


def _walks(dim, n, nwalks, faces, gradient):
    """Work of n x nwalks walks: a query cannot do with less than the depth of
    a binary tree in boxes and one exact distance."""
    q = n * nwalks * (QUERIES[dim] + (SAMPLE[dim] if gradient else 0))
    return q * (DISTANCE[dim] + 4 * dim * math.log2(max(2, faces)))


def work(case):
    c, kind = case, case["kind"]
    if kind == "batch":
        flops = nbytes = 0
        for i in range(c["scenes"]):
            dim = 2 if i % 2 == 0 else 3
            faces = max(64, c["segments"] >> (i // 2)) if dim == 2 else 20 * 4 ** max(2, c["level"] - i // 2)
            n, nw = _batch_sizes(c, i)
            flops += _walks(dim, n, nw, faces, True)
            nbytes += n * (4 * dim + 16) + faces * (8 * dim + 12)
        return dict(bytes=float(nbytes), flops=float(flops))
    dim = 3 if kind.endswith("3d") else 2
    faces = 20 * 4 ** c["level"] if dim == 3 else c["segments"]
    nv = faces // 2 + 2 if dim == 3 else faces
    n = c["res"] ** 2 if kind == "image2d" else c["points"]
    scene = 4 * nv * (dim + 1) + 4 * faces * dim
    if kind == "closest3d":
        return dict(bytes=float(scene + n * 4 * (3 + 1 + 3 + 2 + 1)), flops=float(2 * _walks(3, n, 1, faces, False) / 18))
    if kind == "move3d":
        return dict(bytes=float(scene + 12 * nv * 2 + n * 16),
                    flops=float(_walks(3, n, 1, faces, False) / 18 + 200 * faces))
    grad = kind in ("grad2d", "grad3d", "shape2d", "image2d")
    nbytes = scene + n * 4 * (dim + 1) + (4 * nv * (dim + 1) if grad or kind == "inverse2d" else 0)
    return dict(bytes=float(nbytes), flops=float(_walks(dim, n, c["nwalks"], faces, grad)))


# ---------------------------------------------------------------- 64 bits
#: Most point-primitive pairs that a plain search in 64 bits gets through in a few seconds.
PAIRS = 8e9


def _nearest2(p, V, F):
    """(distance, segment, parameter) of the nearest segment, by brute force."""
    a, e = V[F[:, 0]], V[F[:, 1]] - V[F[:, 0]]
    ee = (e * e).sum(1)
    out = []
    for q in p.split(max(1, int(2e8 // F.shape[0]))):
        x, y = q[:, :1] - a[:, 0], q[:, 1:] - a[:, 1]
        t = ((x * e[:, 0] + y * e[:, 1]) / ee).clamp(0, 1)
        d2 = (x - t * e[:, 0]) ** 2 + (y - t * e[:, 1]) ** 2
        m, i = d2.min(1)
        out.append((m.sqrt(), i, t.gather(1, i[:, None])[:, 0]))
    return tuple(torch.cat(v) for v in zip(*out))


def _closest_on(p, a, ab, ac):
    """Closest points of triangles, element by element: the face's foot point if
    it is inside, else the nearest of the three edges'."""
    def edge(o, d):
        t = (((p - o) * d).sum(-1) / (d * d).sum(-1)).clamp(0, 1)
        return o + t[..., None] * d

    n = torch.linalg.cross(ab, ac)
    nn = (n * n).sum(-1)
    ap = p - a
    v = (torch.linalg.cross(ap, ac.expand_as(ap)) * n).sum(-1) / nn
    w = (torch.linalg.cross(ab.expand_as(ap), ap) * n).sum(-1) / nn
    inside = (v >= 0) & (w >= 0) & (v + w <= 1)
    best = a + v[..., None] * ab + w[..., None] * ac
    d = torch.where(inside, ((p - best) ** 2).sum(-1), math.inf)
    for c in (edge(a, ab), edge(a, ac), edge(a + ab, ac - ab)):
        e = ((p - c) ** 2).sum(-1)
        best = torch.where((e < d)[..., None], c, best)
        d = torch.minimum(d, e)
    return best


def _nearest3(p, V, F):
    """(distance, closest point, triangle) by a search over every triangle in
    32 bits for candidates and in 64 bits among the nearest of them."""
    a, ab, ac = V[F[:, 0]], V[F[:, 1]] - V[F[:, 0]], V[F[:, 2]] - V[F[:, 0]]
    a4, ab4, ac4 = a.float(), ab.float(), ac.float()
    out = []
    for q in p.split(max(1, int(4e7 // F.shape[0]))):
        c4 = _closest_on(q.float()[:, None, :], a4[None], ab4[None], ac4[None])
        d4 = ((c4 - q.float()[:, None, :]) ** 2).sum(-1)
        i = d4.topk(min(8, F.shape[0]), 1, largest=False).indices
        c = _closest_on(q[:, None, :], a[i], ab[i], ac[i])
        d, j = ((c - q[:, None, :]) ** 2).sum(-1).min(1)
        out.append((d.sqrt(), c.gather(1, j[:, None, None].expand(-1, 1, 3))[:, 0], i.gather(1, j[:, None])[:, 0]))
    return tuple(torch.cat(v) for v in zip(*out))


def _philox(key, c0, c1, c2, c3):
    """Philox-4x32-10 on int64 tensors holding 32-bit words."""
    M = 0xFFFFFFFF
    k0, k1 = key
    for _ in range(10):
        p0, p1 = 0xD2511F53 * c0, 0xCD9E8D57 * c2
        h0, h1 = (p0 >> 32) & M, (p1 >> 32) & M
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, p1 & M, h0 ^ c3 ^ k1, p0 & M
        k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
    return c0, c1, c2, c3


def _u01(x):
    return (x >> 9).double() / 8388608.0


def _green_cdf():
    r = (torch.arange(10000, device=DEV, dtype=torch.float64) + 0.5) / 10000
    c = torch.cumsum(r * torch.log(1 / r), 0)
    c = (c / c[-1]).float().double()
    c[-1] = 1.0
    return c


def _solve2_exact(c, seed):
    """The 2D walks of the case in 64 bits, from the same Philox numbers."""
    V, F, val, st, sp, P = _scene2(c, seed)
    seed = int(seed) & 0x7FFFFFFF
    key = (seed & 0xFFFFFFFF, 0x5BD1E995)
    V, F, val = V.double(), F.long(), val.double()
    n, nw, eps = c["points"], c["nwalks"], float(np.float32(1e-3))
    ids = torch.arange(n * nw, device=DEV)
    p = P.double().repeat_interleave(nw, 0)
    total = torch.zeros(n * nw, device=DEV, dtype=torch.float64)
    contrib = torch.zeros_like(total)
    cdf = _green_cdf() if c.get("source") == "green" else None
    q = sp.double().tolist() if sp is not None else None
    for i in range(c["nsteps"]):
        d, f, t = _nearest2(p, V, F)
        done = d < eps
        va, vb = val[F[f, 0]], val[F[f, 1]]
        total[ids[done]] = (va + t * (vb - va) + contrib[ids])[done]
        if i == c["nsteps"] - 1 or bool(done.all()):
            break
        keep = ~done
        ids, p, d = ids[keep], p[keep], d[keep]
        z = torch.zeros_like(ids)
        r0, _, r2, r3 = _philox(key, ids // nw, ids % nw, z + i, z)
        if st != 0:
            if cdf is not None:
                u = _u01(r2)
                l = torch.searchsorted(cdf, u, right=True).clamp_max(9999)
                prev = torch.where(l > 0, cdf[(l - 1).clamp_min(0)], torch.zeros_like(u))
                pmf = cdf[l] - prev
                rad = d * (l + (u - prev) / pmf) / 10000
                pdf, weight = pmf * 10000 / d / (2 * math.pi), rad
                ang = 2 * math.pi * _u01(r3)
            else:
                rad = torch.sqrt(_u01(r3)) * d
                pdf, weight = 1 / (math.pi * d * d), torch.ones_like(d)
                ang = 2 * math.pi * _u01(r2)
            y = p + rad[:, None] * torch.stack([torch.cos(ang), torch.sin(ang)], 1)
            G = torch.log(d / rad.clamp_min(1e-4)) / (2 * math.pi)
            if st == 1:
                fy = q[4] * torch.exp(-(y[:, 0] - q[0]) ** 2 / (2 * q[2] ** 2) - (y[:, 1] - q[1]) ** 2 / (2 * q[3] ** 2))
            else:
                fy = q[3] * torch.sin(q[0] * y[:, 0] + q[1] * y[:, 1] + q[2]) + q[4]
            contrib[ids] += torch.where(pdf > 1e-5, fy * G * weight / pdf, torch.zeros_like(G))
        ang = 2 * math.pi * _u01(r0)
        p = p + d[:, None] * torch.stack([torch.cos(ang), torch.sin(ang)], 1)
    return total.reshape(n, nw).mean(1)


def _normals3_exact(V, F):
    """Vertex normals weighted by the face's angle there."""
    p = [V[F[:, k]] for k in range(3)]
    n = torch.linalg.cross(p[1] - p[0], p[2] - p[0])
    n = n / torch.linalg.norm(n, dim=1, keepdim=True)
    out = torch.zeros_like(V)
    for k in range(3):
        a, b = p[(k + 1) % 3] - p[k], p[(k + 2) % 3] - p[k]
        ang = torch.atan2(torch.linalg.norm(torch.linalg.cross(a, b), dim=1), (a * b).sum(1))
        out.index_add_(0, F[:, k], ang[:, None] * n)
    return out / torch.linalg.norm(out, dim=1, keepdim=True)


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "solve2d":
        if c["points"] * c["nwalks"] * 12.0 * c["segments"] > 8 * PAIRS:
            return None
        return _solve2_exact(c, seed)
    if kind not in ("closest3d", "move3d") or c["points"] * 20.0 * 4 ** c["level"] > PAIRS:
        return None  # gradients and 3D walks: no plain restatement runs in seconds
    g = _gen(seed)
    V, F = _mesh(c["level"], g)
    _values3(V, g)
    Vn = _mesh(c["level"], g)[0] if kind == "move3d" else V
    P = _points3(c["points"], V, F, g, outside=True).double()
    V, F = Vn.double(), F.long()
    d, pt, f = _nearest3(P, V, F)
    p = [V[F[f, k]] for k in range(3)]
    side = (torch.linalg.cross(p[1] - p[0], p[2] - p[0]) * (P - pt)).sum(1)
    sdf = torch.where(side > 0, d, -d)
    if kind == "move3d":
        return dict(normals=_normals3_exact(V, F), sdf=sdf)
    return dict(prim=None, p=pt, uv=None, sdf=sdf)

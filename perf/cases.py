"""The framework's measured workloads: what a program calls it for, through the package's public entry points.

A case is a dict of plain values.  ``kind`` says which call it is:

* ``mesh``   -- the generalized winding number of an open triangle mesh (an icosphere with a 30 degree cap removed
                and vertex noise, or the reference tests' open cube) at many points: eval_gwnr_mesh_batch and its two
                terms, in either precision, on host (numpy) or device (torch) arrays.
* ``remesh`` -- the same on a mesh that is new on every pass (a deforming surface): boundary extraction, intersector
                and evaluation.
* ``robust`` -- CudaRobustMeshGwn on two interpenetrating tori with holes, half of the points next to the surface.
* ``batch``  -- CudaRobustBatch: many small meshes with their own points in one launch.
* ``param``  -- the parametric winding number over bicubic Bezier patches: adaptive GK15 over the boundary curves and
                the patches' signed crossings.

``prepare`` makes a program's state (inputs from the seed alone, dispatcher, geometry handles), ``run`` is one pass,
``work`` the bytes and operations no implementation can do without, ``exact`` the result in plain 64-bit torch.
"""

import functools
import math

import numpy as np
import torch

import antipodal_gb300 as ag
from antipodal_gb300 import synth

# ----------------------------------------------------------------------------------------------------------------
# the cases
# ----------------------------------------------------------------------------------------------------------------


def listed():
    return [
        # a few points probed interactively on a small mesh from numpy, default precision: latency
        dict(name="probe_f64", kind="mesh", dtype="f64", precision="exact", level=3, points="random", n=257,
             term="full", host=True),
        # the reference tests' open cube under a random rotation, 1e5 points, default precision
        dict(name="cube_f64", kind="mesh", dtype="f64", precision="exact", level=0, points="random", n=100_000,
             term="full", host=False),
        # a plane slice of a mesh as the slice example draws it: host arrays, default precision, one row short of square
        dict(name="slice_f64", kind="mesh", dtype="f64", precision="exact", level=5, points="slice", n=512 * 511,
             term="full", host=True),
        # a sampled volume in single precision (a signed field for a float pipeline)
        dict(name="volume_f32", kind="mesh", dtype="f32", precision="exact", level=5, points="grid", n=96 ** 3,
             term="full", host=False),
        # scattered points (a particle cloud) on a mid-size mesh, mixed precision
        dict(name="cloud_f64_mixed", kind="mesh", dtype="f64", precision="mixed", level=5, points="random",
             n=200_003, term="full", host=False),
        # the benchmark's headline: a 256^3 grid around the level-6 icosphere, mixed precision
        dict(name="volume_f64_mixed", kind="mesh", dtype="f64", precision="mixed", level=6, points="grid",
             n=256 ** 3, term="full", host=False),
        # one frame of a deforming mesh: new vertices, so a new boundary, intersector and evaluation every pass
        dict(name="remesh_f64_mixed", kind="remesh", level=6, n=100_000),
        # the robust evaluator's default for float meshes, points half on a coarse-to-fine band about the surface
        dict(name="robust_f32", kind="robust", dtype="f32", policy="int64_grid", precision="exact", tris=20_000,
             holes=6, n=150_000),
        # a large self-intersecting mesh, doubles, exact predicates with the mixed fractional term
        dict(name="robust_f64_mixed", kind="robust", dtype="f64", policy="exact_float", precision="mixed",
             tris=250_000, holes=20, n=1_500_000),
        # many meshes (an asset library), a grid of points each, in one persistent launch
        dict(name="batch_f32_mixed", kind="batch", meshes=16, tris=20_000, side=72, precision="mixed"),
        # parametric surfaces in the default precision: the reference's own adaptive quadrature
        dict(name="param_f64", kind="param", precision="exact", learned=False, patches=24, n=3_001, tol=1e-8),
        # the parametric benchmark's form (learned start depths, mixed precision) on a sample of its points
        dict(name="param_f64_mixed", kind="param", precision="mixed", learned=True, patches=256, n=20_000, tol=1e-10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mesh", "mesh", "mesh", "mesh", "remesh", "robust", "robust", "batch", "param", "param"])
    if kind == "mesh":
        dtype = rng.choice(["f64", "f64", "f32"])
        precision = rng.choice(["exact", "mixed"]) if dtype == "f64" else "exact"
        level = rng.choice([0, 2, 3, 4, 5, 6])
        segments = (4, 6, 12, 24, 56, 102, 212)[level]
        pairs = {"exact": 3.0e7, "mixed": 3.5e9}[precision] * (8 if dtype == "f32" else 1)
        host = rng.random() < 0.3
        top = min(pairs / segments, 2e6 if host else 1.6e7, 3e5 if level == 0 else 1.6e7)
        return dict(kind="mesh", dtype=dtype, precision=precision, level=level,
                    points=rng.choice(["random", "grid", "slice"]), n=_log_int(rng, 200, top),
                    term=rng.choice(["full", "full", "fractional", "integer"]), host=host)
    if kind == "remesh":
        return dict(kind="remesh", level=rng.choice([4, 5, 6]), n=_log_int(rng, 2_000, 200_000))
    if kind == "robust":
        if rng.random() < 0.5:
            return dict(kind="robust", dtype="f32", policy=rng.choice(["int64_grid", "int64_grid", "int128_grid"]),
                        precision="exact", tris=_log_int(rng, 4_000, 20_000), holes=rng.randint(2, 6),
                        n=_log_int(rng, 1_000, 150_000))
        return dict(kind="robust", dtype="f64", policy="exact_float", precision="mixed",
                    tris=_log_int(rng, 20_000, 250_000), holes=rng.randint(4, 20), n=_log_int(rng, 20_000, 1_500_000))
    if kind == "batch":
        return dict(kind="batch", meshes=rng.randint(4, 16), tris=_log_int(rng, 2_000, 20_000),
                    side=rng.randint(32, 72), precision=rng.choice(["mixed", "mixed", "exact"]))
    if rng.random() < 0.5:
        return dict(kind="param", precision="exact", learned=False, patches=rng.randint(4, 24),
                    n=_log_int(rng, 200, 3_001), tol=rng.choice([1e-6, 1e-8]))
    return dict(kind="param", precision="mixed", learned=rng.random() < 0.5, patches=_log_int(rng, 32, 256),
                n=_log_int(rng, 2_000, 20_000), tol=rng.choice([1e-8, 1e-10]))


# ----------------------------------------------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _sphere(level):
    """The open icosphere without its noise, and its boundary's vertex pairs (the topology is the level's alone)."""
    v, idx, bnd, _, _ = synth.open_icosphere(seed=0, level=level, sigma=0.0, grid=0)
    key = {tuple(p): k for k, p in enumerate(v)}
    return v, idx, np.array([[key[tuple(r[0:3])], key[tuple(r[3:6])]] for r in bnd])


def _mesh(level, seed, dtype):
    """(vertices, indices, boundary, x0): the open cube for level 0, else the noisy open icosphere."""
    rng = np.random.default_rng(seed)
    if level == 0:
        v, idx, bnd, _, x0 = synth.rotated_open_cube(seed=seed, n_queries=0, dtype=dtype)
        return v, idx, bnd, x0
    v0, idx, ends = _sphere(level)
    v = (v0 + rng.normal(0.0, 1e-3, size=v0.shape)).astype(dtype)
    bnd = np.concatenate([v[ends[:, 0]], v[ends[:, 1]], np.ones((len(ends), 1), dtype)], axis=1)
    return v, idx, bnd, synth.random_unit(rng).astype(dtype)


def _points(case, lo, hi, seed, dtype):
    """``n`` points over the bounding box scaled by 1.2: uniform, a grid (x fastest) or a plane (row by row)."""
    n, g = case["n"], torch.Generator(device="cuda").manual_seed(seed)
    lo, hi = torch.tensor(lo, device="cuda"), torch.tensor(hi, device="cuda")
    c, h = (lo + hi) / 2, (hi - lo) / 2 * 1.2
    if case["points"] == "random":
        p = c + h * (2 * torch.rand(n, 3, generator=g, dtype=torch.float64, device="cuda") - 1)
    elif case["points"] == "grid":
        s = max(2, math.ceil(round(n ** (1 / 3), 6)))
        k = torch.arange(n, device="cuda")
        i = torch.stack([k % s, k // s % s, k // (s * s)], 1).double()
        p = c + h * (2 * i / (s - 1) - 1)
    else:
        s = max(2, math.ceil(math.sqrt(n)))
        k = torch.arange(n, device="cuda")
        a, b = (k % s + 0.5) / s * 2 - 1, (k // s + 0.5) / s * 2 - 1
        f = torch.rand(1, generator=g, dtype=torch.float64, device="cuda") - 0.5
        p = c + h * torch.stack([a.double(), b.double(), f.expand(n)], 1)
    return p.to(torch.float64 if dtype == np.float64 else torch.float32).contiguous()


def _dtype(case):
    return np.float32 if case.get("dtype") == "f32" else np.float64


def _tensor(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _robust_inputs(case, seed):
    """Two noisy tori with holes, and points of which half lie 1e-9 to 1e-3 off the surface."""
    return synth.two_tori(seed=seed, n_tris=case["tris"], n_holes=case["holes"], n_queries=case["n"],
                          dtype=_dtype(case))


def _batch_inputs(case, seed):
    """Meshes of 0.3 to 1 times ``tris`` triangles with 1 to 11 holes, grids of 0.6 to 1 times ``side`` points a side."""
    rng, sizes = np.random.default_rng(seed), np.random.default_rng(1)
    out = []
    for k in range(case["meshes"]):
        v, i = synth.noisy_mesh("icosphere" if k % 2 else "torus", int(case["tris"] * sizes.uniform(0.3, 1.0)),
                                int(sizes.integers(1, 12)), rng)
        b = synth.boundary_segments(v, i)
        side = int(case["side"] * sizes.uniform(0.6, 1.0))
        q = synth.grid_queries(v.min(0), v.max(0), side, 1.2, np.float32)
        out.append((v.astype(np.float32), i, b.astype(np.float32), q))
    return out


def _param_inputs(case, seed):
    """Patches with N(0, 1) control points; 30% of the points lie within 1e-2 of a boundary curve."""
    return synth.bezier_patches(seed=seed, n_patches=case["patches"], n_queries=case["n"], near_dist=1e-2,
                                return_patches=True)


# ----------------------------------------------------------------------------------------------------------------
# state and pass
# ----------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind, dtype = case["kind"], _dtype(case)
    disp = ag.CudaDispatcher(stream=torch.cuda.current_stream())
    s = dict(case=case, disp=disp)
    if kind in ("mesh", "remesh"):
        v, idx, bnd, x0 = _mesh(case["level"], seed, dtype)
        p = _points(dict(case, points=case.get("points", "random")), v.min(0), v.max(0), seed, dtype)
        out = torch.empty(len(p), dtype=torch.int32 if case.get("term") == "integer" else p.dtype, device="cuda")
        if case.get("host"):
            s.update(p=p.cpu().numpy(), out=out.cpu().numpy(), bnd=bnd, x0=x0)
        else:
            s.update(p=p, out=out, bnd=_tensor(bnd), x0=x0)
        disp.set_precision(case.get("precision", "mixed"))
        if kind == "mesh":
            s["isect"] = ag.CudaIntersector(disp, v, idx)
        else:
            s.update(v=_tensor(v), idx=_tensor(idx))
    elif kind == "robust":
        v, idx, bnd, q = _robust_inputs(case, seed)
        disp.set_robust_precision(case["precision"])
        s["mesh"] = ag.CudaRobustMeshGwn(disp, v, idx, bnd, precision=case["policy"])
        s["p"] = _tensor(q)
        s["out"] = torch.empty(len(q), dtype=s["p"].dtype, device="cuda")
        s["counts"] = torch.empty(len(q), dtype=torch.int32, device="cuda")
    elif kind == "batch":
        disp.set_robust_precision(case["precision"])
        meshes, p, out = [], [], []
        for v, i, b, q in _batch_inputs(case, seed):
            meshes.append(ag.CudaRobustMeshGwn(disp, v, i, b, precision="int64_grid"))
            p.append(_tensor(q))
            out.append(torch.empty(len(q), dtype=torch.float32, device="cuda"))
        s.update(out=out, batch=ag.CudaRobustBatch(disp, meshes, p, out))
    else:
        curves, q, x0, patches = _param_inputs(case, seed)
        s.update(p=_tensor(q), curves=_tensor(curves), x0=x0, cfg=ag.IntegrateConfig(tol=case["tol"]), net=None)
        s["patches"] = ag.CudaBezierPatchIntersector(disp, patches)
        s["out"] = torch.empty(len(q), dtype=torch.float64, device="cuda")
        s["counts"] = torch.empty(len(q), dtype=torch.int32, device="cuda")
        disp.set_param_precision("exact")
        if case["learned"]:  # trained once on the plain integrator's labels of a few points, as a program would
            s["net"] = ag.LearnedGK15Proposal(disp, seed=1, alpha=0.9)
            few = s["p"][: max(1, min(len(q), 200_000 // len(curves)))].contiguous()
            s["net"].fit(few, x0, s["curves"], s["cfg"], steps=2_000)
        disp.set_param_precision(case["precision"])
    torch.cuda.synchronize()
    return s


def run(s):
    kind, disp = s["case"]["kind"], s["disp"]
    if kind == "mesh":
        term = s["case"]["term"]
        if term == "full":
            ag.eval_gwnr_mesh_batch(disp, s["isect"], s["p"], s["out"], s["x0"], s["bnd"])
        elif term == "fractional":
            ag.eval_gwnr_mesh_batch_fractional(disp, s["p"], s["out"], s["x0"], s["bnd"])
        else:
            ag.eval_gwnr_mesh_batch_integer(disp, s["isect"], s["p"], s["out"], s["x0"])
        return s["out"]
    if kind == "remesh":
        bnd = ag.build_boundary_segments(disp, s["v"], s["idx"])
        isect = ag.CudaIntersector(disp, s["v"], s["idx"])
        ag.eval_gwnr_mesh_batch(disp, isect, s["p"], s["out"], s["x0"], bnd)
        isect.close()
        return s["out"]
    if kind == "robust":
        s["mesh"].evaluate(s["p"], s["out"], s["counts"])
        return [s["out"], s["counts"]]
    if kind == "batch":
        s["batch"].run(graph=True)
        return s["out"]
    ag.eval_gwnr_parametric_batch_fractional(disp, s["p"], s["out"], s["x0"], s["curves"], s["cfg"], s["net"])
    ag.eval_gwnr_parametric_batch_integer(disp, s["patches"], s["p"], s["counts"], s["x0"])
    return [s["out"], s["counts"]]


# ----------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------------------------------------------
_PAIR = 56      # operations of one (point, segment) term: two vertex differences, dot products, atan2
_CROSS = 120    # per point: the few triangles its ray meets
_NODE = 150     # one evaluation of the parametric integrand
_PANELS = 8     # panels of 15 nodes per (point, curve) pair
_PATCH = 5_000  # per (point, patch): the cells next to the ray


def work(case):
    kind = case["kind"]
    size = _dtype(case)().itemsize
    n = case.get("n", 0)
    if kind in ("mesh", "remesh"):
        segments = (4, 6, 12, 24, 56, 102, 212)[case["level"]]
        tris = 10 if case["level"] == 0 else int(0.93 * 20 * 4 ** case["level"])
        term = case.get("term", "full")
        pairs = 0 if term == "integer" else n * segments
        flops = _PAIR * pairs + (0 if term == "fractional" else _CROSS * n)
        out = 4 if term == "integer" else size
        geometry = 0 if term == "fractional" else tris * 9 * size
        return {"bytes": n * (3 * size + out) + segments * 7 * size + geometry, "flops": flops}
    if kind == "robust":
        segments = int(41 * math.sqrt(case["tris"] / 20_000) * case["holes"] / 6)
        return {"bytes": n * (4 * size + 4) + case["tris"] * 9 * size, "flops": n * (_PAIR * segments + _CROSS)}
    if kind == "batch":
        q = case["meshes"] * (0.8 * case["side"]) ** 3
        return {"bytes": q * 16 + case["meshes"] * case["tris"] * 36, "flops": q * (_PAIR * 250 + _CROSS)}
    pairs = n * 4 * case["patches"]
    return {"bytes": n * 36 + case["patches"] * 100 * 8,
            "flops": pairs * _PANELS * 15 * _NODE + n * case["patches"] * _PATCH}


# ----------------------------------------------------------------------------------------------------------------
# the results in 64 bits
# ----------------------------------------------------------------------------------------------------------------
def _chunks(n, width, limit=3e7):
    step = max(1, int(limit / max(1, width)))
    return [(a, min(n, a + step)) for a in range(0, n, step)]


def _fractional(p, bnd, x0):
    """sum w atan2(x1 . (v0 x v1), l0 l1 + l1 x1.v0 + l0 x1.v1 + v0.v1) / (2 pi) with x1 = -x0."""
    out = torch.zeros(len(p), dtype=torch.float64, device="cuda")
    for a, b in _chunks(len(p), len(bnd)):
        v0, v1 = bnd[None, :, 0:3] - p[a:b, None], bnd[None, :, 3:6] - p[a:b, None]
        l0, l1 = v0.square().sum(-1).sqrt(), v1.square().sum(-1).sqrt()
        num = (torch.cross(v0, v1, dim=-1) * -x0).sum(-1)
        den = l0 * l1 + l1 * (v0 * -x0).sum(-1) + l0 * (v1 * -x0).sum(-1) + (v0 * v1).sum(-1)
        out[a:b] = (bnd[None, :, 6] * torch.atan2(num, den)).sum(-1) / (2 * math.pi)
    return out


def _crossings(p, tri, x0):
    """Signed crossings of the rays p + t x0, t >= 0, with the triangles (n, 3, 3), each rounded operation by itself."""
    e1, e2 = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    h = torch.linalg.cross(x0.expand_as(e2), e2)
    det = (e1 * h).sum(-1)
    sign = torch.where((torch.linalg.cross(e1, e2) * x0).sum(-1) > 0, 1, -1)
    ok = det != 0
    inv = 1 / det
    out = torch.zeros(len(p), dtype=torch.int64, device="cuda")
    for a, b in _chunks(len(p), len(tri)):
        s = [p[a:b, k, None] - tri[None, :, 0, k] for k in range(3)]
        u = inv * (s[0] * h[:, 0] + s[1] * h[:, 1] + s[2] * h[:, 2])
        hit = ok & (u >= 0) & (u <= 1)
        q = [s[1] * e1[:, 2] - s[2] * e1[:, 1], s[2] * e1[:, 0] - s[0] * e1[:, 2], s[0] * e1[:, 1] - s[1] * e1[:, 0]]
        v = inv * (q[0] * x0[0] + q[1] * x0[1] + q[2] * x0[2])
        t = inv * (q[0] * e2[:, 0] + q[1] * e2[:, 1] + q[2] * e2[:, 2])
        hit &= (v >= 0) & (u + v <= 1) & (t >= 0)
        out[a:b] = (hit * sign).sum(-1)
    return out


def _f64(a):
    return torch.as_tensor(np.asarray(a), dtype=torch.float64, device="cuda") if isinstance(a, np.ndarray) \
        else a.to("cuda", torch.float64)


def _on_grid(v, idx, bnd, q, bits=20):
    """The vertices, segments and points on the integer grid of RobustMeshGwn's int64_grid policy, as doubles."""
    lo, hi = v.min(0).values, v.max(0).values
    c, half = lo + (hi - lo) * 0.5, 0.5 * float((hi - lo).max())
    scale = (2 ** bits - 1) / half
    far = 2.0 ** (bits + 10)

    def on(x):
        t = ((x - c) * scale).clamp(-far, far)
        return torch.sign(t) * torch.floor(t.abs() + 0.5)
    return on(v)[idx.long()].view(-1, 3, 3), torch.cat([on(bnd[:, 0:3]), on(bnd[:, 3:6]), bnd[:, 6:7]], 1), on(q)


_GK_X = [0.0, 0.9914553711208126, 0.9491079123427585, 0.8648644233597691, 0.7415311855993945, 0.5860872354676911,
         0.4058451513773972, 0.2077849550078985]
_GK_K = [0.2094821410847278, 0.0229353220105292, 0.0630920926299786, 0.1047900103222502, 0.1406532597155259,
         0.1690047266392679, 0.1903505780647854, 0.2044329400752989]
_GK_G = {0: 0.4179591836734694, 2: 0.1294849661688697, 4: 0.2797053914892767, 6: 0.3818300505051189}


def _parametric(p, curves, x0, tol, max_depth=10):
    """sum over curves of the adaptive G7-K15 integral of w - d_eta, over 4 pi: level by level, all panels at once."""
    c = curves.view(-1, 4, 3)
    out = torch.zeros(len(p), dtype=torch.float64, device="cuda")

    def f(cp, t):
        u = 1 - t
        r = (u ** 3)[:, None] * cp[:, 0] + (3 * u * u * t)[:, None] * cp[:, 1] \
            + (3 * u * t * t)[:, None] * cp[:, 2] + (t ** 3)[:, None] * cp[:, 3]
        d = 3 * ((u * u)[:, None] * (cp[:, 1] - cp[:, 0]) + (2 * u * t)[:, None] * (cp[:, 2] - cp[:, 1])
                 + (t * t)[:, None] * (cp[:, 3] - cp[:, 2]))
        xr = torch.linalg.cross(x0.expand_as(r), r)
        s, m, rho, big_t = r.norm(dim=1), r @ x0, (xr * xr).sum(1), (d * xr).sum(1)
        return torch.where(m < 0, -big_t / (s * (s - m)), -big_t * (s + m) / (s * rho))

    for a, b in _chunks(len(p), len(c), 2e6):
        m = b - a
        pair = torch.arange(m * len(c), device="cuda")
        j = torch.zeros_like(pair, dtype=torch.float64)
        acc = torch.zeros(m, dtype=torch.float64, device="cuda")
        for depth in range(max_depth + 1):
            cp = c[pair % len(c)] - p[a + pair // len(c), None]
            h = 0.5 ** (depth + 1)
            mid = (2 * j + 1) * h
            k_sum = torch.zeros_like(mid)
            g_sum = torch.zeros_like(mid)
            for k, x in enumerate(_GK_X):
                y = f(cp, mid) if k == 0 else f(cp, mid - h * x) + f(cp, mid + h * x)
                k_sum += _GK_K[k] * y
                if k in _GK_G:
                    g_sum += _GK_G[k] * y
            done = ((k_sum - g_sum).abs() * h <= tol * 0.5 ** depth) | (depth == max_depth)
            acc.index_add_(0, (pair // len(c))[done], (k_sum * h)[done])
            pair, j = pair[~done].repeat(2), torch.cat([2 * j[~done], 2 * j[~done] + 1])
            if not len(pair):
                break
        out[a:b] = acc / (4 * math.pi)
    return out


def exact(case, seed):
    kind, dtype = case["kind"], _dtype(case)
    most = 4e10  # (point, triangle) pairs that are counted in a few seconds
    if kind in ("mesh", "remesh"):
        v, idx, bnd, x0 = _mesh(case["level"], seed, dtype)
        if case["n"] * len(idx) / 3 > most and case.get("term", "full") == "full":
            return None
        p = _f64(_points(dict(case, points=case.get("points", "random")), v.min(0), v.max(0), seed, dtype))
        d = _f64(x0)
        if case.get("term") == "integer":
            return None
        out = _fractional(p, _f64(bnd), d)
        if case.get("term") != "fractional":
            out += _crossings(p, _f64(v)[torch.from_numpy(idx).cuda().long()].view(-1, 3, 3), d)
        return out
    if kind == "robust":
        if case["policy"] == "int128_grid" or case["n"] * case["tris"] > most:
            return None
        v, idx, bnd, q = _robust_inputs(case, seed)
        v, bnd, q, idx = _f64(v), _f64(bnd), _f64(q), torch.from_numpy(idx).cuda()
        tri, bnd, q = _on_grid(v, idx, bnd, q) if case["policy"] == "int64_grid" else (v[idx.long()].view(-1, 3, 3),
                                                                                    bnd, q)
        d = torch.tensor([-1.0, 0.0, 0.0], dtype=torch.float64, device="cuda")
        return [_fractional(q, bnd, d) + _crossings(q, tri, d), None]
    if kind == "batch":
        out = []
        d = torch.tensor([-1.0, 0.0, 0.0], dtype=torch.float64, device="cuda")
        if case["meshes"] * case["tris"] * (0.8 * case["side"]) ** 3 > 2 * most:
            return None
        for v, idx, bnd, q in _batch_inputs(case, seed):
            tri, bnd, q = _on_grid(_f64(v), torch.from_numpy(idx).cuda(), _f64(bnd), _f64(q))
            out.append(_fractional(q, bnd, d) + _crossings(q, tri, d))
        return out
    curves, q, x0, _ = _param_inputs(case, seed)
    return [_parametric(_f64(q), _f64(curves), _f64(x0), case["tol"]), None]

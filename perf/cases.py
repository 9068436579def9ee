"""The work that programs give this framework, as measured cases.

A case is a dict of plain values; its "kind" names the call:

  solve       one map, GridBasedTransportSolver.solve, host density in, host mesh out (the
              calling convention of the reference's solver class), FP64
  batch       many maps in one otm_solve_batch call on device buffers, FP64 or split
              precision (a throughput service; also the single large solve with count 1)
  gradient    transport_map() of torch.autograd, forward and backward (Krylov adjoint)
  locate      a new map: point locator built, then points pulled back through it, device
              buffers (the inverse maps of composition, barycenters and resampling)
  raster      otm_rasterize_mode of a forward mesh with its density, device buffers
  barycenter  barycenter_image: four inverse meshes blended, rasterized, rescaled
  loss        barycenter_loss() of torch.autograd: solves, inversions, blend, raster and
              the gradient with respect to every density

Densities are the repository's synthetic families (otmap_b200/workloads.py) drawn on the
GPU: Gaussian mixtures with a floor, blurred disks and polygons, blurred softmax logits.
Meshes that a case starts from come from `solve64`, a plain torch FP64 restatement of the
reference's iteration, so they do not depend on the code that is measured; `exact` uses
the same restatement.
"""

import ctypes
import math

import numpy as np
import torch

from otmap_b200 import autograd, native
from otmap_b200 import otmap as ot

F64 = torch.float64
DEV = "cuda"


def listed():
    return [
        # the smallest map that is worth a GPU: launch latency and the host path
        {"name": "solve 64", "kind": "solve", "n": 64, "parts": 8, "threshold": 1e-7},
        # the reference's own CPU-sized configuration: 8 Gaussians on 256^2, residual 1e-7
        {"name": "solve 256", "kind": "solve", "n": 256, "parts": 8, "threshold": 1e-7},
        # images are seldom powers of two: any other side takes the general transform
        {"name": "solve 500", "kind": "solve", "n": 500, "parts": 8, "threshold": 1e-7},
        # an image above 1024^2, the largest transform held in shared memory but one
        {"name": "solve 2048", "kind": "solve", "n": 2048, "parts": 8, "threshold": 1e-6},
        # the single large solve of the parity configuration: blurred shapes, 1024^2, FP64
        {"name": "shapes 1024 fp64", "kind": "batch", "family": "shapes", "n": 1024, "count": 1, "split": False,
         "threshold": 1e-7},
        # the benchmark's step: 8 x 1024^2 blurred shapes in split precision
        {"name": "shapes 8x1024 split", "kind": "batch", "family": "shapes", "n": 1024, "count": 8, "split": True,
         "threshold": 1e-7},
        # a service's mixed queue: uneven sizes in one call
        {"name": "mixed 24 fp64", "kind": "batch", "family": "mixed", "n": 1024, "count": 24, "split": False,
         "threshold": 1e-6},
        # learning through a map: blurred softmax logits, forward and backward
        {"name": "gradient 512", "kind": "gradient", "n": 512, "sigma": 8.0},
        # inverse map of a new 1024^2 map at 2^20 points, with faces and hit counts
        {"name": "locate 1024", "kind": "locate", "n": 1024, "parts": 8, "points": 1 << 20, "fast": False},
        # the forward mesh rendered at its own resolution
        {"name": "raster 1024", "kind": "raster", "n": 1024, "parts": 8, "rows": 1024, "cols": 1024,
         "per_vertex": False},
        # one frame of the bilinear barycenters demo
        {"name": "barycenter 512", "kind": "barycenter", "n": 512, "parts": 6, "res": 512},
        # a training step on a barycenter of four densities
        {"name": "loss 256", "kind": "loss", "n": 256, "parts": 6, "res": 256},
    ]


def draw(rng):
    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["solve", "solve", "solve", "batch", "batch", "gradient", "locate", "raster", "barycenter",
                       "loss"])
    parts = rng.randint(4, 16)
    if kind == "solve":
        # any side: odd and prime ones, smooth composites and powers of two
        n = rng.choice([log_int(48, 1100), log_int(48, 1100), 1 << rng.randint(6, 11)])
        return {"kind": kind, "n": n, "parts": parts, "threshold": rng.choice([1e-6, 1e-7])}
    if kind == "batch":
        family = rng.choice(["shapes", "mixed"])
        n = rng.choice([256, 512, 1024]) if family == "shapes" else 1024
        return {"kind": kind, "family": family, "n": n, "count": rng.randint(1, 8) if family == "shapes" else
                rng.randint(4, 24), "split": rng.random() < 0.5, "threshold": rng.choice([1e-6, 1e-7])}
    if kind == "gradient":
        n = rng.choice([128, 256, 512, log_int(96, 512)])
        return {"kind": kind, "n": n, "sigma": round(rng.uniform(n / 96, n / 48), 2)}
    if kind == "locate":
        return {"kind": kind, "n": log_int(64, 1100), "parts": parts, "points": log_int(1 << 12, 1 << 20),
                "fast": rng.random() < 0.3}
    if kind == "raster":
        return {"kind": kind, "n": log_int(64, 1100), "parts": parts, "rows": log_int(100, 1400),
                "cols": log_int(100, 1400), "per_vertex": rng.random() < 0.4}
    if kind == "barycenter":
        return {"kind": kind, "n": log_int(64, 512), "parts": parts, "res": log_int(64, 1024)}
    return {"kind": kind, "n": rng.choice([64, 128, 256, log_int(48, 160)]), "parts": rng.randint(4, 8),
            "res": log_int(64, 256)}


# ---- densities (per cell, face order f = j + i n: tensors indexed [i, j]) ----


def _mixture(n, rng, parts):
    """Isotropic Gaussians (centres U[0.1,0.9]^2, sigma U[0.03,0.15], amplitude U[0.5,2])
    plus 1e-3, mean 1."""
    c = (torch.arange(n, dtype=F64, device=DEV) + 0.5) / n
    img = torch.full((n, n), 1e-3, dtype=F64, device=DEV)
    for _ in range(parts):
        cx, cy = rng.uniform(0.1, 0.9, size=2)
        s, a = rng.uniform(0.03, 0.15), rng.uniform(0.5, 2.0)
        img += a * torch.exp(-((c[:, None] - cx) ** 2 + (c[None, :] - cy) ** 2) / (2.0 * s * s))
    return img / img.mean()


def _blur(img, sigma):
    """Separable Gaussian blur, radius ceil(3 sigma), mirror borders."""
    n, r = img.shape[0], max(1, math.ceil(3.0 * sigma))
    t = np.arange(-r, r + 1)
    k = np.exp(-0.5 * (t / sigma) ** 2)
    k /= k.sum()
    B = np.zeros((n, n))
    src = np.arange(n)[:, None] + t[None, :]
    src = np.where(src < 0, -src - 1, src)
    src = np.where(src >= n, 2 * n - 1 - src, src)
    np.add.at(B, (np.repeat(np.arange(n), 2 * r + 1), src.ravel()), np.tile(k, n))
    B = torch.from_numpy(B).to(DEV)
    return B @ img @ B.T


def _shapes(n, rng, count=6):
    """Filled disks or convex polygons on 1e-3, blurred by 5 pixels of a 1024^2 grid, mean 1."""
    c = (torch.arange(n, dtype=F64, device=DEV) + 0.5) / n
    x, y = c[:, None], c[None, :]
    img = torch.full((n, n), 1e-3, dtype=F64, device=DEV)
    for _ in range(count):
        cx, cy = rng.uniform(0.2, 0.8, size=2)
        rad = rng.uniform(0.05, 0.15)
        if rng.uniform() < 0.5:
            inside = (x - cx) ** 2 + (y - cy) ** 2 <= rad * rad
        else:
            ang = np.sort(rng.uniform(0.0, 2.0 * math.pi, size=int(rng.integers(3, 9))))
            px, py = cx + rad * np.cos(ang), cy + rad * np.sin(ang)
            inside = torch.ones((n, n), dtype=torch.bool, device=DEV)
            for q in range(len(ang)):
                ax, ay, bx, by = px[q - 1], py[q - 1], px[q], py[q]
                inside &= (bx - ax) * (y - ay) - (by - ay) * (x - ax) >= 0.0
        img[inside] = 1.0
    img = _blur(img, 5.0 * n / 1024)
    return img / img.mean()


def _logits(n, rng, sigma):
    g = torch.Generator(DEV).manual_seed(int(rng.integers(1 << 40)))
    z = torch.randn((n, n), dtype=F64, device=DEV, generator=g)
    img = _blur(torch.softmax(z.ravel(), 0).reshape(n, n), sigma)
    return img / img.mean()


def _batch_densities(case, rng):
    if case["family"] == "shapes":
        return [_shapes(case["n"], rng) for _ in range(case["count"])]
    sizes = (256, 1024, 128, 512)
    return [_mixture(sizes[k % 4], rng, int(rng.integers(4, 17))) for k in range(case["count"])]


# ---- the reference's iteration in plain torch, FP64 ----


def _basis(n):
    """Orthonormal DCT-II basis C[k, i] and the eigenvalues of the pseudo-Laplacian."""
    k = torch.arange(n, dtype=F64, device=DEV)
    C = math.sqrt(2.0 / n) * torch.cos(math.pi * k[:, None] * (k[None, :] + 0.5) / n)
    C[0] = math.sqrt(1.0 / n)
    ck = torch.cos(math.pi * k / n)
    lam = 2.0 - 2.0 * ck[:, None] * ck[None, :]
    lam[0, 0] = math.inf
    return C, lam


def _poisson(r, C, lam):
    return C.T @ (((C @ r) @ C.T) / lam) @ C


def _vertex_gradients(p):
    """(gx, gy) at the (n+1)^2 vertices from the clamped cells around each."""
    n = p.shape[0]
    q = torch.nn.functional.pad(p[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
    p00, p01, p10, p11 = q[:-1, :-1], q[:-1, 1:], q[1:, :-1], q[1:, 1:]
    return 0.5 * n * ((p10 + p11) - (p00 + p01)), 0.5 * n * ((p01 + p11) - (p00 + p10))


def _diagonals(g):
    return g[1:, 1:] - g[:-1, :-1], g[:-1, 1:] - g[1:, :-1]


def _areas(p):
    """Quad areas of the grid displaced by the vertex gradients of p."""
    e = 1.0 / p.shape[0]
    (ax, bx), (ay, by) = (_diagonals(g) for g in _vertex_gradients(p))
    return 0.5 * ((ax + e) * (by + e) - (ay + e) * (bx - e))


def _grid(n):
    t = torch.arange(n + 1, dtype=F64, device=DEV) * (1.0 / n)
    return torch.stack(torch.meshgrid(t, t, indexing="ij"), -1)


def solve64(rho, threshold, max_iter=1000):
    """(potential, forward mesh [n+1, n+1, 2], normalised density, iterations)."""
    n = rho.shape[0]
    e, ea = 1.0 / n, 1.0 / (n * n)
    C, lam = _basis(n)
    rho = rho / (rho.sum() * ea)
    psi = torch.zeros_like(rho)
    r = e * e - ea * rho
    residual = float((r * r).sum() / ea)
    alpha, it, rp, dp = 0.0, 0, r, psi
    while it < max_iter and residual > threshold:
        d = _poisson(r, C, lam)
        if it:
            eps, jd = alpha / 2.0, r - rp
            reps = _areas(psi - eps * d) - ea * rho
            d = d + max(-1.0, float((jd * (reps - r)).sum() / (jd * jd).sum()) / eps * alpha) * dp
        (ax, bx), (ay, by) = (_diagonals(g) for g in _vertex_gradients(psi))
        (hx, kx), (hy, ky) = (_diagonals(g) for g in _vertex_gradients(d))
        a = 0.5 * (hx * ky - hy * kx)
        b = 0.5 * (hx * (by + e) - hy * (bx - e) + (ax + e) * ky - (ay + e) * kx)
        s = torch.stack([(b * r).sum(), (b * b).sum() + 2 * (a * r).sum(), (a * b).sum(), (a * a).sum()]).tolist()
        z = [residual * ea, 2 * s[0], s[1], 2 * s[2], s[3]]
        t = np.roots([4 * z[4], 3 * z[3], 2 * z[2], z[1]])
        t = [x.real for x in t if abs(x.imag) <= 1e-12 * max(1.0, abs(x)) and -10 <= x.real <= 10] or [0.5]
        residual, alpha = min((z[0] + x * (z[1] + x * (z[2] + x * (z[3] + x * z[4]))), x) for x in t)
        residual /= ea
        psi = psi + alpha * d
        rp, r, dp = r, a * alpha * alpha + b * alpha + r, d
        it += 1
    return psi, _grid(n) + torch.stack(_vertex_gradients(psi), -1), rho, it


def _corners(mesh, i, j):
    return mesh[i, j], mesh[i + 1, j], mesh[i + 1, j + 1], mesh[i, j + 1]


def _locate64(mesh, pts):
    """Cell (i, j) and bilinear coordinates (u, v) of points in a mesh without folds: Newton
    steps that walk from cell to cell, started at the nearest of a coarse set of vertices."""
    n = mesh.shape[0] - 1
    at = torch.linspace(0, n, min(n, 32) + 1, device=DEV).long()
    coarse = mesh[at][:, at].reshape(-1, 2)
    near = torch.cat([torch.cdist(p, coarse).argmin(1) for p in pts.split(1 << 16)])
    s = torch.stack([at[near // len(at)], at[near % len(at)]], -1).to(F64).clamp(1e-3, n - 1e-3)
    for step in range(300):
        c = s.floor().clamp(0, n - 1)
        i, j = c[:, 0].long(), c[:, 1].long()
        u, v = (s[:, 0] - c[:, 0])[:, None], (s[:, 1] - c[:, 1])[:, None]
        p0, p1, p2, p3 = _corners(mesh, i, j)
        f = pts - ((1 - u) * (1 - v) * p0 + u * (1 - v) * p1 + u * v * p2 + (1 - u) * v * p3)
        gu, gv = (1 - v) * (p1 - p0) + v * (p2 - p3), (1 - u) * (p3 - p0) + u * (p2 - p1)
        det = gu[:, 0] * gv[:, 1] - gu[:, 1] * gv[:, 0]
        d = torch.stack([f[:, 0] * gv[:, 1] - f[:, 1] * gv[:, 0], gu[:, 0] * f[:, 1] - gu[:, 1] * f[:, 0]], -1)
        d = torch.nan_to_num(d / det[:, None], nan=0.1, posinf=1.0, neginf=-1.0)
        size = d.abs().amax(1, keepdim=True)
        if float(size.max()) < 1e-13 * n:
            break
        reach = 8.0 if step < 60 else 1.0 if step < 160 else 0.3
        new = s + d * (reach / size.clamp(min=reach))
        # a step that leaves the cell stops just beyond its edge, so that no cell is skipped late
        if step >= 60:
            new = torch.minimum(torch.maximum(new, c - 1e-9 * (n + 1)), c + 1 + 1e-9 * (n + 1))
        s = new.clamp(0, n)
    c = s.floor().clamp(0, n - 1)
    return c[:, 0].long(), c[:, 1].long(), s


def _inverse_mesh(mesh):
    """Inverse positions of the origin grid's vertices, (n+1)^2 x 2."""
    n = mesh.shape[0] - 1
    return _locate64(mesh, _grid(n).reshape(-1, 2))[2] / n


def _face_areas(mesh):
    p0, p1, p2, p3 = mesh[:-1, :-1], mesh[1:, :-1], mesh[1:, 1:], mesh[:-1, 1:]
    d, k = p2 - p0, p3 - p1
    return 0.5 * (d[..., 0] * k[..., 1] - d[..., 1] * k[..., 0])


def _folded(mesh):
    """Whether a face of the mesh is turned over at a corner: points there lie in several faces, and which
    one a call takes is its rule, not a computed value."""
    p = _corners(mesh, *torch.meshgrid(*[torch.arange(mesh.shape[0] - 1, device=DEV)] * 2, indexing="ij"))
    for k in range(4):
        a, b = p[(k + 1) % 4] - p[k], p[k - 1] - p[k]
        if bool((a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0] <= 0).any()):
            return True
    return False


def _owners(mesh, rows, cols):
    """Cell of every pixel centre, [rows, cols] each (row = y)."""
    y = (torch.arange(rows, dtype=F64, device=DEV) + 0.5) / rows
    x = (torch.arange(cols, dtype=F64, device=DEV) + 0.5) / cols
    p = torch.stack([x[None, :].expand(rows, cols), y[:, None].expand(rows, cols)], -1).reshape(-1, 2)
    i, j, _ = _locate64(mesh, p)
    return i.reshape(rows, cols), j.reshape(rows, cols)


def _adjoint64(psi, rho_raw, q, tol=1e-13, steps=400):
    """dL/ddensity for dL/dmesh = q: J^T l = G^T q by GMRES, preconditioned with the
    pseudo-inverse of the Laplacian, then through the normalisation."""
    n = psi.shape[0]
    C, lam = _basis(n)

    def transposed(f, w):
        with torch.enable_grad():
            p = psi.detach().requires_grad_()
            return torch.autograd.grad(f(p), p, w)[0]

    b = transposed(lambda p: torch.stack(_vertex_gradients(p), -1), q)
    bn = b.norm()
    V, Z, H = [b / bn], [], torch.zeros(steps + 1, steps, dtype=F64)
    for k in range(steps):
        Z.append(_poisson(V[k], C, lam))
        w = transposed(_areas, Z[k])
        for _ in range(2):
            B = torch.stack([v.ravel() for v in V])
            h = B @ w.ravel()
            H[: k + 1, k] += h.cpu()
            w = w - (h @ B).reshape(n, n)
        H[k + 1, k] = w.norm()
        V.append(w / H[k + 1, k])
        e1 = torch.zeros(k + 2, dtype=F64)
        e1[0] = float(bn)
        y = torch.linalg.lstsq(H[: k + 2, : k + 1], e1[:, None], driver="gelsd").solution[:, 0]
        if float((H[: k + 2, : k + 1] @ y - e1).norm()) <= tol * float(bn):
            break
    l = sum(float(c) * z for c, z in zip(y, Z))
    S = rho_raw.sum()
    return (l - (l * rho_raw).sum() / S) / S


# ---- the cases ----

_contexts = {}


def _context(split):
    """One context per precision, kept by the program."""
    if split not in _contexts:
        _contexts[split] = native.Context(torch.cuda.current_device())
        _contexts[split].set_precision(native.PRECISION_SPLIT if split else native.PRECISION_FP64)
    return _contexts[split]


def _arr(tensors):
    return (ctypes.c_void_p * len(tensors))(*[t.data_ptr() for t in tensors])


def _map_of(case, rng):
    """(potential, mesh, density) of a Gaussian mixture's map."""
    return solve64(_mixture(case["n"], rng, case["parts"]), 1e-7, 200)[:3]


def _weights(rng):
    return [float(x) for x in rng.uniform(0.1, 0.9, size=2)]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind, n = case["kind"], case["n"]
    s = {"case": case, "ctx": _context(bool(case.get("split", False)))}
    if kind == "solve":
        s["density"] = _mixture(n, rng, case["parts"]).reshape(-1).cpu().numpy()
        s["solver"] = ot.GridBasedTransportSolver(s["ctx"])
        s["solver"].set_verbose_level(0)
        s["solver"].init(n)
        s["opt"] = ot.SolverOptions(threshold=case["threshold"])
    elif kind == "batch":
        s["density"] = [d.contiguous() for d in _batch_densities(case, rng)]
        s["ns"] = [d.shape[0] for d in s["density"]]
        for m in set(s["ns"]):
            s["ctx"].init(m)
        s["fwd"] = [torch.empty(((m + 1) ** 2, 2), dtype=F64, device=DEV) for m in s["ns"]]
        s["opt"] = native.default_options()
        s["opt"].threshold = case["threshold"]
    elif kind == "gradient":
        s["density"] = _logits(n, rng, case["sigma"]).reshape(-1)
        g = torch.Generator(DEV).manual_seed(seed)
        s["q"] = torch.randn(((n + 1) ** 2, 2), dtype=F64, device=DEV, generator=g)
        s["ctx"].init(n)
    elif kind == "locate":
        _, mesh, rho = _map_of(case, rng)
        s["mesh"], s["density"] = mesh.reshape(-1, 2).contiguous(), rho.reshape(-1).contiguous()
        g = torch.Generator(DEV).manual_seed(seed)
        s["points"] = torch.rand((case["points"], 2), dtype=torch.float32, device=DEV, generator=g).to(F64)
    elif kind == "raster":
        _, mesh, rho = _map_of(case, rng)
        s["mesh"], s["density"] = mesh.reshape(-1, 2).contiguous(), rho.reshape(-1).contiguous()
        s["image"] = torch.empty((case["rows"], case["cols"]), dtype=F64, device=DEV)
    elif kind == "barycenter":
        s["inverse"] = [_inverse_mesh(_map_of(case, rng)[1]).contiguous() for _ in range(4)]
        s["weights"] = _weights(rng)
        s["means"] = [float(x) for x in rng.uniform(0.5, 1.5, size=4)]
    else:
        s["density"] = torch.stack([_mixture(n, rng, case["parts"]).reshape(-1) for _ in range(4)])
        s["weights"] = ot.bilinear_weights(*_weights(rng))
        s["target"] = _mixture(case["res"], rng, case["parts"])
        s["ctx"].init(n)
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind, n = case["kind"], case["n"]
    if kind == "solve":
        m = s["solver"].solve(s["density"], s["opt"])
        return {"mesh": m.fwd_mesh(), "density": m.density(), "iterations": m.stats.iterations}
    if kind == "batch":
        count = len(s["ns"])
        stats = (native.SolveStatsC * count)()
        native.check(native.lib().otm_solve_batch(ctx.handle, count, (ctypes.c_int * count)(*s["ns"]),
                                                  _arr(s["density"]), ctypes.byref(s["opt"]), _arr(s["fwd"]), None,
                                                  stats))
        return {"mesh": s["fwd"], "iterations": np.array([st.iterations for st in stats])}
    if kind == "gradient":
        d = s["density"].detach().clone().requires_grad_()
        fwd = autograd.transport_map(d, n, context=ctx)
        (fwd * s["q"]).sum().backward()
        return {"mesh": fwd.detach(), "gradient": d.grad}
    if kind == "locate":
        points = s["points"].clone()
        face = torch.empty(len(points), dtype=torch.int32, device=DEV)
        hits = torch.empty(len(points), dtype=torch.int32, device=DEV)
        handle, missing = ctypes.c_void_p(), ctypes.c_long(0)
        torch.cuda.current_stream().synchronize()  # the library works on its context's stream
        lib = native.lib()
        native.check(lib.otm_map_create(ctx.handle, n, native.ptr(s["mesh"]), native.ptr(s["density"]),
                                        ctypes.byref(handle)))
        native.check(lib.otm_map_inverse_mode(handle, native.ptr(points), len(points),
                                              native.INV_FIRST if case["fast"] else native.INV_DENSEST,
                                              native.ptr(face), native.ptr(hits), ctypes.byref(missing)))
        native.check(lib.otm_map_destroy(handle))
        return {"points": points, "face": face, "hits": hits, "missing": missing.value}
    if kind == "raster":
        native.check(native.lib().otm_rasterize_mode(ctx.handle, n, native.ptr(s["mesh"]), native.ptr(s["density"]),
                                                     case["rows"], case["cols"],
                                                     native.RIO_PER_VERTEX if case["per_vertex"] else
                                                     native.RIO_PER_FACE, native.ptr(s["image"])))
        return {"image": s["image"]}
    if kind == "barycenter":
        img, mesh = ot.barycenter_image(s["inverse"], s["weights"][0], s["weights"][1], s["means"], case["res"],
                                        context=ctx)
        return {"image": img, "mesh": mesh}
    d = s["density"].detach().clone().requires_grad_()
    loss = autograd.barycenter_loss(d, s["weights"], s["target"], res=case["res"], context=ctx)
    loss.backward()
    return {"loss": loss.detach(), "gradient": d.grad, "image": ctx.last_barycenter_image}


def work(case):
    """Inputs and outputs once, and per iteration of a solve the state that has to change
    (potential, direction, residual) with the transform's input and output. Iterations are
    those of a typical draw."""
    n = case["n"]
    cells, kind = n * n, case["kind"]

    def solve_work(m, iters, width):
        c = m * m
        io = 8 * c + 16 * (m + 1) ** 2
        per = 2 * 8 + 6 * width
        return io + iters * per * c, iters * c * (120 + 10 * math.log2(max(m, 2)))

    if kind == "solve":
        b, f = solve_work(n, 22, 8)
    elif kind == "batch":
        iters = 80 if case["family"] == "shapes" else 20
        side = n if case["family"] == "shapes" else 0.57 * n  # root mean square of the sizes drawn
        b, f = solve_work(side, iters, 4 if case["split"] else 8)
        b, f = case["count"] * b, case["count"] * f
    elif kind == "gradient":
        b, f = solve_work(n, 10, 8)
        # an Arnoldi step: a Poisson solve, the Jacobian, two orthogonalisations
        b, f = b + 10 * 8 * cells * 12, f + 10 * cells * (100 + 10 * math.log2(n) + 4 * 10)
    elif kind == "locate":
        b, f = 16 * (n + 1) ** 2 + 8 * cells + case["points"] * (32 + 8), 150 * case["points"]
    elif kind == "raster":
        b, f = 16 * (n + 1) ** 2 + 8 * cells + 8 * case["rows"] * case["cols"], 150 * case["rows"] * case["cols"]
    elif kind == "barycenter":
        b, f = 5 * 16 * (n + 1) ** 2 + 8 * case["res"] ** 2, 150 * case["res"] ** 2
    else:
        b, f = solve_work(n, 20, 8)
        b, f = 4 * (b + 100 * 8 * cells * 40), 4 * (f + 100 * cells * (180 + 4 * 40))
    return {"bytes": float(b), "flops": float(f)}


def exact(case, seed):
    rng = np.random.default_rng(seed)
    kind, n = case["kind"], case["n"]
    if kind == "solve":
        rho = _mixture(n, rng, case["parts"])
        _, mesh, adj, _ = solve64(rho, case["threshold"])
        return {"mesh": mesh.reshape(-1, 2).cpu().numpy(), "density": adj.reshape(-1).cpu().numpy(),
                "iterations": None}
    if kind == "batch":
        return {"mesh": [solve64(d, case["threshold"])[1].reshape(-1, 2) for d in _batch_densities(case, rng)],
                "iterations": None}
    if kind == "gradient":
        rho = _logits(n, rng, case["sigma"])
        g = torch.Generator(DEV).manual_seed(seed)
        q = torch.randn(((n + 1) ** 2, 2), dtype=F64, device=DEV, generator=g)
        psi, mesh, _, _ = solve64(rho, 1e-7)
        return {"mesh": mesh.reshape(-1, 2), "gradient": _adjoint64(psi, rho, q.reshape(n + 1, n + 1, 2)).reshape(-1)}
    if kind == "locate":
        _, mesh, _ = _map_of(case, rng)
        if _folded(mesh):
            return None
        g = torch.Generator(DEV).manual_seed(seed)
        p = torch.rand((case["points"], 2), dtype=torch.float32, device=DEV, generator=g).to(F64)
        return {"points": _locate64(mesh, p)[2] / n, "face": None, "hits": None, "missing": None}
    if kind == "raster":
        _, mesh, rho = _map_of(case, rng)
        if _folded(mesh):
            return None
        i, j = _owners(mesh, case["rows"], case["cols"])
        scale, area = float(np.float32(1.0 / (n * n))), _face_areas(mesh).abs()  # the reference keeps it in a float
        if not case["per_vertex"]:
            return {"image": (scale * rho / area)[i, j]}
        # every corner of a face takes the value of its first vertex: the mean of 1/area there
        inv = torch.nn.functional.pad(1.0 / area, (1, 1, 1, 1))
        ones = torch.nn.functional.pad(torch.ones_like(area), (1, 1, 1, 1))
        mean = [sum(t[a : a + n + 1, b : b + n + 1] for a in (0, 1) for b in (0, 1)) for t in (inv, ones)]
        return {"image": (scale * mean[0] / mean[1])[i, j]}
    if kind == "barycenter":
        inv = [_inverse_mesh(_map_of(case, rng)[1]) for _ in range(4)]
        w = ot.bilinear_weights(*_weights(rng))
        means = [float(x) for x in rng.uniform(0.5, 1.5, size=4)]
        mesh = sum(a * m for a, m in zip(w, inv)).reshape(n + 1, n + 1, 2)
        img = None
        if not _folded(mesh):
            i, j = _owners(mesh, case["res"], case["res"])
            img = (1.0 / _face_areas(mesh).abs())[i, j]
            img = (img * (sum(a * m for a, m in zip(w, means)) / img.mean())).cpu().numpy()
        return {"image": img, "mesh": mesh.reshape(-1, 2).cpu().numpy()}
    dens = [_mixture(n, rng, case["parts"]) for _ in range(4)]
    w = ot.bilinear_weights(*_weights(rng))
    target = _mixture(case["res"], rng, case["parts"])
    maps = [solve64(d, 1e-7)[:2] for d in dens]
    if any(_folded(mesh) for _, mesh in maps):
        return None
    leaves, inverse = [], []
    origin = _grid(n)
    for _, mesh in maps:
        # inverse positions as a function of the mesh: one Newton step from the located point
        i, j, s = _locate64(mesh, origin.reshape(-1, 2))
        u, v = (s[:, 0] - i)[:, None], (s[:, 1] - j)[:, None]
        leaf = mesh.clone().requires_grad_()
        p0, p1, p2, p3 = _corners(mesh, i, j)
        gu, gv = (1 - v) * (p1 - p0) + v * (p2 - p3), (1 - u) * (p3 - p0) + u * (p2 - p1)
        det = gu[:, 0] * gv[:, 1] - gu[:, 1] * gv[:, 0]
        q0, q1, q2, q3 = _corners(leaf, i, j)
        f = origin.reshape(-1, 2) - ((1 - u) * (1 - v) * q0 + u * (1 - v) * q1 + u * v * q2 + (1 - u) * v * q3)
        d = torch.stack([f[:, 0] * gv[:, 1] - f[:, 1] * gv[:, 0], gu[:, 0] * f[:, 1] - gu[:, 1] * f[:, 0]], -1)
        leaves.append(leaf)
        inverse.append((s + d / det[:, None]) / n)
    mesh = sum(a * m for a, m in zip(w, inverse)).reshape(n + 1, n + 1, 2)
    if _folded(mesh.detach()):
        return None
    i, j = _owners(mesh.detach(), case["res"], case["res"])
    img = (1.0 / _face_areas(mesh).abs())[i, j]
    means = [d.clone().requires_grad_() for d in dens]
    img = img * (sum(a * m.mean() for a, m in zip(w, means)) / img.mean())
    loss = ((img - target) ** 2).sum()
    loss.backward()
    grads = [_adjoint64(p, d, l.grad) + m.grad for (p, _), d, l, m in zip(maps, dens, leaves, means)]
    return {"loss": loss.detach(), "gradient": torch.stack(grads).reshape(4, -1), "image": img.detach()}

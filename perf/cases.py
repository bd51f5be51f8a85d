"""The work a user of this framework has it do, as cases that can be timed and compared.

Every case goes through the public entry points of the Python binding of the C ABI: whole solves on device memory
(``VoxelFEA.solve_dev``), a static study from host arrays (``solve`` and ``stresses``), load groups (``solve_batch``), the block
preconditioner of an eigensolver (``precondition_block``) and the operator product of a caller's own Krylov method
(``apply_dot_noalloc``). The models have the shapes and rules of ``parts-sim_b200/voxel_models.py`` (cantilever, L-bracket with
holes, graded SIMP grid, gyroid sheet lattice, box with spherical voids), made here on the GPU from a seed that also moves the
holes, voids, lattice phase, density field, loads and material.

Displacements come back in 32 bits where a solve or the 32-bit V-cycle made them: a solve to a relative residual of 1e-8 or 1e-10
does not determine more of them, and the post-processing that reads them is in 32 bits. The operator's product comes back in 64 bits.
``exact`` restates the element, the multigrid hierarchy and the V-cycle in plain 64-bit torch.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "parts-sim_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import psfea  # noqa: E402

# ---------------------------------------------------------------- the cases


def listed():
    return [
        # the smallest job: a textbook cantilever (a preview, a convergence check while a part is being drawn); 60 k DOF, launch-bound
        {"name": "solve_cantilever", "do": "solve", "model": "cantilever", "nx": 64, "ny": 16, "nz": 16, "precision": "fp64", "tol": 1e-10, "coarse": 1300},
        # one request of a job queue: a box with voids of odd sizes in the mixed form
        {"name": "solve_box", "do": "solve", "model": "box", "nx": 57, "ny": 41, "nz": 33, "precision": "mixed", "tol": 1e-10, "coarse": 300},
        # the drop-in static study: host arrays up, displacements and nodal stresses down, on a solid bracket of odd sizes
        {"name": "study_bracket", "do": "study", "model": "l_bracket", "nx": 97, "ny": 49, "nz": 51, "precision": "fp64", "tol": 1e-10, "coarse": 1100},
        # one load on a graded density grid in the middle of a topology run, the drop-in form
        {"name": "solve_simp", "do": "solve", "model": "simp", "nx": 96, "ny": 48, "nz": 48, "precision": "fp64", "tol": 1e-8, "coarse": 1100},
        # the same at the size of a finished topology study, FP16 coarse matrices
        {"name": "solve_simp_large", "do": "solve", "model": "simp", "nx": 192, "ny": 96, "nz": 96, "precision": "mixed", "tol": 1e-8, "coarse": 1100},
        # a thin-walled lattice in the drop-in form (25.6 M DOF)
        {"name": "solve_gyroid", "do": "solve", "model": "gyroid", "nx": 256, "ny": 256, "nz": 128, "precision": "fp64", "tol": 1e-8, "coarse": 1100},
        # the largest: the full lattice in the fastest form (85.8 M DOF)
        {"name": "solve_gyroid_large", "do": "solve", "model": "gyroid", "nx": 384, "ny": 384, "nz": 192, "precision": "fp32", "tol": 1e-8, "coarse": 1100},
        # a sizing study's load groups: 32 right-hand sides on one graded model, host arrays
        {"name": "batch_simp", "do": "batch", "model": "simp", "nx": 96, "ny": 48, "nz": 48, "nrhs": 32, "precision": "mixed", "tol": 1e-8, "coarse": 1100},
        # an eigensolver's preconditioner on a block of 8 residuals of a solid bracket (1.6 M DOF)
        {"name": "precondition_bracket", "do": "precondition", "model": "l_bracket", "nx": 128, "ny": 64, "nz": 64, "nvec": 8, "coarse": 1100},
        # the same on an odd number of vectors of a voided box
        {"name": "precondition_box", "do": "precondition", "model": "box", "nx": 75, "ny": 53, "nz": 61, "nvec": 3, "coarse": 300},
        # a caller's own Krylov step: y = K x and x . y on device vectors, a small odd grid and a large solid one
        {"name": "product_box", "do": "product", "model": "box", "nx": 57, "ny": 41, "nz": 33, "coarse": 300},
        {"name": "product_bracket", "do": "product", "model": "l_bracket", "nx": 256, "ny": 128, "nz": 128, "coarse": 1100},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


#: per model: voxel counts per axis of the smallest and the largest case of a kind, and the precision forms in use on it
_RANGE = {
    "cantilever": ((32, 8, 8), (200, 50, 50)),
    "box": ((24, 24, 24), (140, 140, 140)),
    "l_bracket": ((32, 16, 16), (160, 80, 80)),
    "simp": ((32, 16, 16), (192, 96, 96)),
    "gyroid": ((48, 48, 24), (320, 320, 160)),
}


def draw(rng):
    do = rng.choice(["solve"] * 5 + ["study", "batch", "precondition", "precondition", "product", "product"])
    model = rng.choice({"solve": ["cantilever", "box", "simp", "simp", "gyroid", "gyroid"], "study": ["cantilever", "box", "l_bracket"],
                        "batch": ["cantilever", "simp", "box"], "precondition": list(_RANGE), "product": list(_RANGE)}[do])
    lo, hi = _RANGE[model]
    if model == "box":
        dims = [_log_uniform(rng, lo[d], hi[d]) for d in range(3)]
        most = {"batch": 60, "study": 100, "precondition": 110}.get(do, 140)
        dims = [min(d, most) for d in dims]
    else:
        most = {"batch": 0.5, "study": 0.6, "precondition": 0.75}.get(do, 1.0)
        s = math.exp(rng.uniform(0.0, math.log(max(1.0, most * hi[0] / lo[0]))))
        dims = [max(4, int(round(lo[d] * s)) + rng.randint(-2, 2)) for d in range(3)]
    c = {"do": do, "model": model, "nx": dims[0], "ny": dims[1], "nz": dims[2], "coarse": 300 if model == "box" else rng.choice([1100, 1100, 1300, 300])}
    if do in ("solve", "study", "batch"):
        c["precision"] = rng.choice(["fp64", "fp64", "mixed"] if do != "solve" else ["fp64", "fp64", "mixed", "mixed", "fp32", "fp32", "half"])
        c["tol"] = 1e-8 if model in ("simp", "gyroid") or do == "batch" else 1e-10
    if do == "batch":
        c["nrhs"] = rng.choice([2, 5, 8, 12, 16, 20, 32])
    if do == "precondition":
        c["nvec"] = rng.choice([1, 2, 3, 5, 8, 12, 16])
    return c


# ---------------------------------------------------------------- inputs

_MATERIALS = ((200e9, 0.30), (70e9, 0.33), (3.5e9, 0.36), (114e9, 0.34))


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _prune(solid, held):
    """Solid voxels face-connected to one that touches a held node (both [k, j, i])."""
    touch = torch.zeros_like(solid)
    nz, ny, nx = solid.shape
    for dk in (0, 1):
        for dj in (0, 1):
            for di in (0, 1):
                touch |= held[dk:dk + nz, dj:dj + ny, di:di + nx]
    reach = solid & touch
    while True:
        before = int(reach.sum())
        for _ in range(32):
            grown = reach.clone()
            for ax in range(3):
                n = reach.shape[ax]
                grown.narrow(ax, 1, n - 1).logical_or_(reach.narrow(ax, 0, n - 1))
                grown.narrow(ax, 0, n - 1).logical_or_(reach.narrow(ax, 1, n - 1))
            reach = grown & solid
        if int(reach.sum()) == before:
            return reach


def _face_load(solid, axis, side, value):
    """Consistent nodal loads of a uniform traction on the solid voxel faces of one outer grid face; f [k, j, i, 3]."""
    nz, ny, nx = solid.shape
    f = torch.zeros(nz + 1, ny + 1, nx + 1, 3, dtype=torch.float64, device="cuda")
    ax = 2 - axis
    layer = solid.select(ax, 0 if side == 0 else solid.shape[ax] - 1).double()
    nodal = torch.zeros(layer.shape[0] + 1, layer.shape[1] + 1, dtype=torch.float64, device="cuda")
    for a in (0, 1):
        for b in (0, 1):
            nodal[a:a + layer.shape[0], b:b + layer.shape[1]] += 0.25 * layer
    f.select(ax, 0 if side == 0 else f.shape[ax] - 1).copy_(nodal[..., None] * value)
    return f


def _direction(g):
    d = _randn(g, 3)
    return d / d.norm()


def _model(case, seed):
    """density [k, j, i] (float32), bc and f [k, j, i, 3] on the GPU, nu, E [Pa] and the voxel size [m]."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    g = _generator(seed)
    E, nu = _MATERIALS[int(_rand(g, 1).item() * 4) % 4]
    h = 1e-3
    bc = torch.zeros(nz + 1, ny + 1, nx + 1, 3, dtype=torch.bool, device="cuda")
    kind = case["model"]
    centre = [(torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) for n in (nx, ny, nz)]
    X, Y, Z = centre[0][None, None, :], centre[1][None, :, None], centre[2][:, None, None]
    if kind == "cantilever":
        # one end held, a traction of random direction on the other
        density = torch.ones(nz, ny, nx, device="cuda")
        bc[:, :, 0] = True
        f = _face_load(density > 0, 0, 1, _direction(g) * 1e6 * h * h)
    elif kind == "l_bracket":
        # solid but for a quadrant and cylindrical holes along y, the y = 0 face held, a patch load on the arm
        solid = ~((X > 96 * nx / 256) & (Z > 48 * nz / 128)).expand(nz, 1, nx).clone()
        count = max(2, nx // 4)
        c = _rand(g, count, 3).cpu()
        for cx, cz, r in c.tolist():
            if cx > 0.375 and cz > 0.375:
                continue
            solid &= (X - cx * nx) ** 2 + (Z - cz * nz) ** 2 >= (3 + 5 * r) ** 2 * min(1.0, (nx / 128) ** 2)
        solid = solid.expand(nz, ny, nx).contiguous()
        bc[:, 0] = True
        solid = _prune(solid, bc[..., 0])
        density = solid.float()
        kz = min(nz - 1, int(round(48 * nz / 128)) - 1)
        w = max(2, nx // 32)
        patch = torch.zeros_like(solid)
        patch[kz, ny // 2 - w // 2:ny // 2 + (w + 1) // 2, nx - w:] = True
        patch &= solid
        if not bool(patch.any()):
            patch = solid.clone()
            patch[:, :-1] = False
        f = torch.zeros(nz + 1, ny + 1, nx + 1, 3, dtype=torch.float64, device="cuda")
        load = (_direction(g) + torch.tensor([0.0, 0.0, -2.0], dtype=torch.float64, device="cuda")) * 500.0
        p = patch.double()[..., None] * (load / patch.sum()) * 0.25
        for a in (0, 1):
            for b in (0, 1):
                f[1:, a:a + ny, b:b + nx] += p
    elif kind == "simp":
        # smoothed noise as a density field, penalised: graded over nine decades; MBB supports, unit loads on the top line
        v = _randn(g, nz, ny, nx)
        rad = 16
        t = torch.arange(-rad, rad + 1, device="cuda", dtype=torch.float64)
        w = torch.exp(-0.5 * (t / 4.0) ** 2)
        w = w / w.sum()
        for ax in range(3):
            n = v.shape[ax]
            at = (torch.arange(-rad, n + rad, device="cuda")).clamp(0, n - 1)
            pad, acc = v.index_select(ax, at), torch.zeros_like(v)
            for q in range(2 * rad + 1):
                acc += w[q] * pad.narrow(ax, q, n)
            v = acc
        v = (v - v.mean()) / v.std()
        rho = (0.5 + 0.5 * v).clamp(1e-3, 1.0)
        density = (1e-9 + rho ** 3 * (1 - 1e-9)).float()
        bc[:, :, 0, 0] = True
        bc[0, :, nx, 1:] = True
        f = torch.zeros(nz + 1, ny + 1, nx + 1, 3, dtype=torch.float64, device="cuda")
        f[nz, :, 0] = _direction(g) / (ny + 1)
        E, nu, h = 1.0, 0.3, 1.0
    elif kind == "gyroid":
        # sheet lattice of period 24 at a random phase, the bottom held, a tilted pressure on the top
        ph = (_rand(g, 3) * 24).tolist()
        x, y, z = (2 * math.pi / 24 * (a + p) for a, p in zip((X, Y, Z), ph))
        val = torch.sin(x) * torch.cos(y) + torch.sin(y) * torch.cos(z) + torch.sin(z) * torch.cos(x)
        solid = val.abs() < 0.3
        del val
        bc[0] = True
        solid = _prune(solid, bc[..., 0])
        density = solid.float()
        load = 0.2 * _direction(g) + torch.tensor([0.0, 0.0, -1.0], dtype=torch.float64, device="cuda")
        f = _face_load(solid, 2, 1, load * 5e6 * h * h)
    else:  # a box with spherical voids down to 60 % solid, one face held, a traction on the opposite one
        solid = torch.ones(nz, ny, nx, dtype=torch.bool, device="cuda")
        total, left, count = nx * ny * nz, nx * ny * nz, 0
        while left > 0.6 * total and count < 4000:
            for cx, cy, cz, cr in _rand(g, 8, 4).cpu().tolist():
                r = 2 + 8 * cr
                lo = [max(0, int(c * n - r)) for c, n in ((cx, nx), (cy, ny), (cz, nz))]
                hi = [min(n, int(c * n + r) + 1) for c, n in ((cx, nx), (cy, ny), (cz, nz))]
                sub = solid[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]]
                sub &= ((X[..., lo[0]:hi[0]] - cx * nx) ** 2 + (Y[:, lo[1]:hi[1]] - cy * ny) ** 2 + (Z[lo[2]:hi[2]] - cz * nz) ** 2) >= r * r
                count += 1
            left = int(solid.sum())
        axis, side = int(_rand(g, 1).item() * 3) % 3, int(_rand(g, 1).item() * 2) % 2
        bc.select(2 - axis, 0 if side == 0 else (nx, ny, nz)[axis]).fill_(True)
        solid = _prune(solid, bc[..., 0])
        density = solid.float()
        f = _face_load(solid, axis, 1 - side, _direction(g) * 1e6 * h * h)
    return density, bc, f, nu, E, h


def _nodal_noise(case, density, bc, seed, count):
    """`count` vectors as an eigensolver meets them: smooth waves and noise, 0 at held nodes and off the part; [count, k, j, i, 3]."""
    g = _generator(seed + 1)
    nz, ny, nx = density.shape
    active = torch.zeros(nz + 1, ny + 1, nx + 1, dtype=torch.bool, device="cuda")
    for dk in (0, 1):
        for dj in (0, 1):
            for di in (0, 1):
                active[dk:dk + nz, dj:dj + ny, di:di + nx] |= density > 0
    at = [torch.arange(n + 1, device="cuda", dtype=torch.float64) / n for n in (nx, ny, nz)]
    out = torch.empty(count, nz + 1, ny + 1, nx + 1, 3, dtype=torch.float64, device="cuda")
    for q in range(count):
        k = 1 + 5 * _rand(g, 3)
        wave = torch.sin(math.pi * (k[0] * at[0][None, None, :] + k[1] * at[1][None, :, None] + k[2] * at[2][:, None, None]))
        out[q] = wave[..., None] * _direction(g) + 0.1 * _randn(g, nz + 1, ny + 1, nx + 1, 3)
        out[q] *= (active[..., None] & ~bc)
    return out


def prepare(case, seed):
    density, bc, f, nu, E, h = _model(case, seed)
    dims = (case["nx"], case["ny"], case["nz"])
    s = {"do": case["do"], "E": E, "h": h, "tol": case.get("tol"), "precision": case.get("precision")}
    s["S"] = S = psfea.VoxelFEA(dims, density.cpu().numpy(), nu, bc.cpu().numpy().view(np.uint8), case["coarse"])
    if case["do"] == "solve":
        # vectors live on the device; the handle works on the program's stream
        s["f"], s["u"] = f.reshape(-1), torch.zeros(f.numel(), dtype=torch.float64, device="cuda")
        s["u32"] = torch.zeros(f.numel(), dtype=torch.float32, device="cuda")
        s["stream"] = torch.cuda.Stream()
        S.set_stream(s["stream"].cuda_stream)
    elif case["do"] == "study":
        s["f"] = f.reshape(-1).cpu().numpy()
    elif case["do"] == "batch":
        g = _generator(seed + 1)
        d = _randn(g, case["nrhs"], 3)
        d = d / d.norm(dim=1, keepdim=True)
        share = f.norm(dim=-1)  # where the model is loaded; every load case has a direction of its own there
        s["F"] = (share[None, ..., None] * d[:, None, None, None, :]).reshape(case["nrhs"], -1).cpu().numpy()
    else:
        n = case.get("nvec", 1)
        s["n"], s["x"] = n, _nodal_noise(case, density, bc, seed, n).reshape(n, -1)
        s["y"] = torch.zeros_like(s["x"])
        s["y32"] = torch.zeros(s["x"].shape, dtype=torch.float32, device="cuda")
        s["dot"] = torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return s


_MAX_ITER = 5000


def run(s):
    S = s["S"]
    if s["do"] == "solve":
        with torch.cuda.stream(s["stream"]):
            S.solve_dev(s["f"].data_ptr(), s["u"].data_ptr(), tol=s["tol"], max_iter=_MAX_ITER, precision=s["precision"])
            s["u32"].copy_(s["u"])
        return s["u32"]
    if s["do"] == "study":
        r = S.solve(s["f"], tol=s["tol"], max_iter=_MAX_ITER, precision=s["precision"])
        u = torch.from_numpy(r.u) / (s["E"] * s["h"])
        vm, p1, p3 = S.stresses(u.numpy(), s["E"], s["h"])
        return {"u": u.float(), "von_mises": vm, "p1": p1, "p3": p3}
    if s["do"] == "batch":
        return [torch.from_numpy(r.u).float() for r in S.solve_batch(s["F"], tol=s["tol"], max_iter=_MAX_ITER, precision=s["precision"])]
    stream = torch.cuda.current_stream().cuda_stream
    if s["do"] == "precondition":
        S.precondition_block(s["n"], s["x"].data_ptr(), s["y"].data_ptr(), stream)
        s["y32"].copy_(s["y"])
        return s["y32"]
    S.apply_dot_noalloc(s["x"].data_ptr(), s["y"].data_ptr(), s["dot"].data_ptr(), stream)
    return {"y": s["y"], "dot": s["dot"]}


def work(case):
    """Bytes: the model (a voxel's density, a node's mask), the vectors in and out, each once. Operations: one product K x per vector
    (153 multiply-adds a node, the uniform stencil's nonzeros); how many products a solve needs depends on the model."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    nodes, voxels = (nx + 1) * (ny + 1) * (nz + 1), nx * ny * nz
    vecs = case.get("nrhs", case.get("nvec", 1))
    b = 4 * voxels + nodes
    if case["do"] == "product":
        b += 3 * nodes * 16
    elif case["do"] == "precondition":
        b += vecs * 3 * nodes * 12
    else:
        b += vecs * 3 * nodes * 12 + (12 * nodes if case["do"] == "study" else 0)
    return {"bytes": b, "flops": 2 * 153 * nodes * vecs}


# ---------------------------------------------------------------- the same in plain 64 bits

_CORNER = ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))


def _element(nu):
    """Unit-cube hexahedron with Wilson's incompatible modes (E = 1): K [24, 24] and the corner stress matrices [8, 6, 24]."""
    lam, mu = nu / ((1 + nu) * (1 - 2 * nu)), 1 / (2 * (1 + nu))
    D = np.zeros((6, 6))
    D[:3, :3] = lam
    D[np.arange(3), np.arange(3)] += 2 * mu
    D[np.arange(3, 6), np.arange(3, 6)] = mu

    def strain(M, c, g):
        M[0, c], M[1, c + 1], M[2, c + 2] = g[0], g[1], g[2]
        M[3, c], M[3, c + 1] = g[1], g[0]
        M[4, c + 1], M[4, c + 2] = g[2], g[1]
        M[5, c], M[5, c + 2] = g[2], g[0]

    def rows(p):
        B, G = np.zeros((6, 24)), np.zeros((6, 9))
        for a, xyz in enumerate(_CORNER):
            sg = [2 * v - 1 for v in xyz]
            f = [1 + sg[d] * p[d] for d in range(3)]
            strain(B, 3 * a, (sg[0] * f[1] * f[2] / 4, sg[1] * f[0] * f[2] / 4, sg[2] * f[0] * f[1] / 4))
        for m in range(3):
            g = [0.0, 0.0, 0.0]
            g[m] = -4 * p[m]
            strain(G, 3 * m, g)
        return B, G

    kuu, kua, kaa = np.zeros((24, 24)), np.zeros((24, 9)), np.zeros((9, 9))
    for xyz in _CORNER:
        B, G = rows([(2 * v - 1) / math.sqrt(3.0) for v in xyz])
        kuu += B.T @ D @ B / 8
        kua += B.T @ D @ G / 8
        kaa += G.T @ D @ G / 8
    A = -np.linalg.solve(kaa, kua.T)
    K = kuu + kua @ A
    S = np.zeros((8, 6, 24))
    for a, xyz in enumerate(_CORNER):
        B, G = rows([2 * v - 1 for v in xyz])
        S[a] = D @ (B + G @ A)
    return 0.5 * (K + K.T), S


def _gather(u):
    """Corner values [k, j, i, 24] of a nodal field [k, j, i, 3]."""
    nz, ny, nx = (n - 1 for n in u.shape[:3])
    return torch.cat([u[z:z + nz, y:y + ny, x:x + nx] for x, y, z in _CORNER], dim=-1)


def _scatter(e):
    nz, ny, nx = e.shape[:3]
    y = torch.zeros(nz + 1, ny + 1, nx + 1, 3, dtype=torch.float64, device=e.device)
    for a, (cx, cy, cz) in enumerate(_CORNER):
        y[cz:cz + nz, cy:cy + ny, cx:cx + nx] += e[..., 3 * a:3 * a + 3]
    return y


class _Level:
    """One level: element matrices scale * K (K [24, 24]) or one each (K [k, j, i, 24, 24])."""

    def __init__(self, scale, K, bc):
        self.scale, self.K = scale, K
        full = K.dim() == 5
        diag = K.diagonal(dim1=-2, dim2=-1) if full else scale[..., None] * K.diagonal()
        self.diag = _scatter(diag.contiguous())
        self.bc = bc
        self.free = ~bc & (self.diag > 0)
        self.dinv = torch.where(self.free, 1 / torch.where(self.diag > 0, self.diag, torch.ones_like(self.diag)), torch.zeros_like(self.diag))

    def raw(self, u):
        e = _gather(u)
        if self.K.dim() == 5:
            return _scatter(torch.einsum("kjiab,kjib->kjia", self.K, e))
        return _scatter(self.scale[..., None] * (e @ self.K.T))

    def apply(self, u):
        return self.raw(u) * self.free

    def coarser(self):
        K = self.K
        nz, ny, nx = K.shape[:3] if K.dim() == 5 else self.scale.shape
        cz, cy, cx = (nz + 1) // 2, (ny + 1) // 2, (nx + 1) // 2
        Kc = torch.zeros(cz, cy, cx, 24, 24, dtype=torch.float64, device="cuda")
        for c in range(8):
            o = (c & 1, (c >> 1) & 1, c >> 2)
            W = np.zeros((8, 8))
            for a in range(8):
                for b in range(8):
                    t = [(o[d] + _CORNER[a][d]) * 0.5 for d in range(3)]
                    W[a, b] = np.prod([t[d] if _CORNER[b][d] else 1 - t[d] for d in range(3)])
            P = torch.from_numpy(np.kron(W, np.eye(3))).cuda()
            if K.dim() == 5:
                sub = K[o[2]::2, o[1]::2, o[0]::2]
                part = P.T @ sub @ P
            else:
                sub = self.scale[o[2]::2, o[1]::2, o[0]::2]
                part = sub[..., None, None] * (P.T @ K @ P)
            Kc[:sub.shape[0], :sub.shape[1], :sub.shape[2]] += part
        # a coarse DOF is held where a held fine one interpolates to it
        bc = self.bc
        for ax in range(3):
            n = bc.shape[ax]
            m = n // 2 + 1
            got = torch.zeros(*[m if d == ax else bc.shape[d] for d in range(3)], 3, dtype=torch.bool, device="cuda")
            for o in (-1, 0, 1):
                at = 2 * torch.arange(m, device="cuda") + o
                ok = (at >= 0) & (at < n)
                got.index_copy_(ax, torch.arange(m, device="cuda")[ok], got.index_select(ax, torch.arange(m, device="cuda")[ok]) | bc.index_select(ax, at[ok]))
            bc = got
        return _Level(None, Kc, bc)


class _Multigrid:
    """The Galerkin hierarchy and the V-cycle with its degree-2 Chebyshev smoother, in 64 bits."""

    def __init__(self, density, bc, nu, coarse):
        K, self.S = _element(nu)
        self.levels = [_Level(density.double(), torch.from_numpy(K).cuda(), bc)]
        while len(self.levels) < 12 and int(self.levels[-1].free.sum()) > coarse:
            L = self.levels[-1]
            if max(L.bc.shape[:3]) <= 2:
                break
            self.levels.append(L.coarser())
        for L in self.levels[:-1]:
            lmax = self.bound(L)
            b, a = 1.15 * lmax, 0.1 * lmax
            theta, delta = (b + a) / 2, (b - a) / 2
            sigma = theta / delta
            rho0 = 1 / sigma
            rho1 = 1 / (2 * sigma - rho0)
            L.c = (1 / theta, rho1 * rho0, 2 * rho1 / delta)
        L = self.levels[-1]
        at = L.free.reshape(-1).nonzero().reshape(-1)
        n = L.free.numel()
        index = torch.full((n,), -1, dtype=torch.long, device="cuda")
        index[at] = torch.arange(at.numel(), device="cuda")
        nodes = index.reshape(*L.free.shape)
        e = torch.cat([nodes[z:nodes.shape[0] - 1 + z, y:nodes.shape[1] - 1 + y, x:nodes.shape[2] - 1 + x] for x, y, z in _CORNER], dim=-1)
        Ke = L.K if L.K.dim() == 5 else L.scale[..., None, None] * L.K
        m = at.numel()
        A = torch.zeros(m * m, dtype=torch.float64, device="cuda")
        r, c = e[..., :, None].expand(*e.shape, 24), e[..., None, :].expand(*e.shape[:3], 24, 24)
        ok = (r >= 0) & (c >= 0)
        A.index_put_((r[ok] * m + c[ok],), Ke[ok], accumulate=True)
        self.at, self.inv = at, torch.linalg.inv(A.reshape(m, m))

    @staticmethod
    def bound(L):
        """The largest eigenvalue of D^-1 K as ten Lanczos steps from a fixed pseudo-random vector estimate it."""
        n = L.free.numel()
        i = np.arange(1, n + 1, dtype=np.uint64)
        M = np.uint64(0x7fffffff)
        A, B, ra, rb = np.uint64(1103515245), np.uint64(12345), np.ones(n, np.uint64), np.zeros(n, np.uint64)
        for bit in range(int(n).bit_length()):
            odd = (i >> np.uint64(bit)) & np.uint64(1) == 1
            rb[odd] = (A * rb[odd] + B) & M
            ra[odd] = (A * ra[odd]) & M
            B = (A * B + B) & M
            A = (A * A) & M
        s = (ra * np.uint64(12345) + rb) & M
        v = torch.from_numpy(s.astype(np.float64) / 2147483647.0 - 0.5).cuda().reshape(L.free.shape) * L.free
        v = v / v.norm()
        q, vp, al, be, b = L.dinv.sqrt(), torch.zeros_like(v), [], [], 0.0
        for _ in range(10):
            w = q * L.apply(q * v) - b * vp
            a = float((w * v).sum())
            w = w - a * v
            al.append(a)
            b = float(w.norm())
            if not b > 1e-12 * abs(a):
                break
            be.append(b)
            vp, v = v, w / b
        be = be[:len(al) - 1]
        return float(np.linalg.eigvalsh(np.diag(al) + np.diag(be, 1) + np.diag(be, -1))[-1])

    @staticmethod
    def restrict(r):
        for ax in range(3):
            n = r.shape[ax]
            m = n // 2 + 1
            out = torch.zeros(*[m if d == ax else r.shape[d] for d in range(3)], 3, dtype=torch.float64, device="cuda")
            for o, w in ((-1, 0.5), (0, 1.0), (1, 0.5)):
                at = 2 * torch.arange(m, device="cuda") + o
                ok = (at >= 0) & (at < n)
                out.index_add_(ax, torch.arange(m, device="cuda")[ok], w * r.index_select(ax, at[ok]))
            r = out
        return r

    @staticmethod
    def prolong(z, shape):
        for ax in range(3):
            at = torch.arange(shape[ax], device="cuda")
            lo, hi = at // 2, (at + 1) // 2
            z = 0.5 * (z.index_select(ax, lo) + z.index_select(ax, hi))
        return z

    def vcycle(self, r, l=0):
        L = self.levels[l]
        if l == len(self.levels) - 1:
            z = torch.zeros_like(r).reshape(-1)
            z[self.at] = self.inv @ r.reshape(-1)[self.at]
            return z.reshape(r.shape)
        c0, c1, c2 = L.c
        d = c0 * L.dinv * r
        z = d
        d = c1 * d + c2 * L.dinv * (r - L.apply(z))
        z = z + d
        rc = self.restrict(r - L.apply(z)) * self.levels[l + 1].free
        z = z + self.prolong(self.vcycle(rc, l + 1), r.shape) * L.free
        d = c0 * L.dinv * (r - L.apply(z))
        z = z + d
        d = c1 * d + c2 * L.dinv * (r - L.apply(z))
        return z + d

    def solve(self, f, tol=1e-13, most=400):
        L = self.levels[0]
        f = f * L.free
        x, r = torch.zeros_like(f), f
        z = self.vcycle(r)
        p, rz, norm = z, float((r * z).sum()), float(f.norm())
        for _ in range(most):
            q = L.apply(p)
            a = rz / float((p * q).sum())
            x, r = x + a * p, r - a * q
            if float(r.norm()) <= tol * norm:
                break
            z = self.vcycle(r)
            beta = max(0.0, -a * float((z * q).sum()) / rz)
            rz = float((r * z).sum())
            p = z + beta * p
        return x


def _stresses(S, density, u, E, h):
    """Nodal von Mises, first and third principal stress: density-weighted means over a node's voxels of their corner values."""
    e = _gather(u)
    w = density.double()
    shape = u.shape[:3]
    nz, ny, nx = density.shape
    out = [torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in range(4)]
    for a, (cx, cy, cz) in enumerate(_CORNER):
        s = e @ torch.from_numpy(S[a] * (E / h)).cuda().T
        at = (slice(cz, cz + nz), slice(cy, cy + ny), slice(cx, cx + nx))
        vm = torch.sqrt(0.5 * ((s[..., 0] - s[..., 1]) ** 2 + (s[..., 1] - s[..., 2]) ** 2 + (s[..., 2] - s[..., 0]) ** 2) + 3 * (s[..., 3:] ** 2).sum(-1))
        T = torch.stack([s[..., 0], s[..., 3], s[..., 5], s[..., 3], s[..., 1], s[..., 4], s[..., 5], s[..., 4], s[..., 2]], -1).reshape(-1, 3, 3)
        ev = torch.linalg.eigvalsh(T.cpu()).cuda().reshape(*density.shape, 3)
        for o, v in zip(out, (vm, ev[..., 2], ev[..., 0], torch.ones_like(vm))):
            o[at] += w * v
    wsum = torch.where(out[3] > 0, out[3], torch.ones_like(out[3]))
    return [(o / wsum * (out[3] > 0)).reshape(-1) for o in out[:3]]


def exact(case, seed):
    nodes = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    if case["do"] == "batch" or nodes > (5_000_000 if case["do"] == "product" else 2_200_000 if case["do"] == "precondition" else 300_000):
        return None  # tens of seconds: 64-bit solves of many load cases or millions of unknowns
    density, bc, f, nu, E, h = _model(case, seed)
    if case["do"] == "product":
        x = _nodal_noise(case, density, bc, seed, 1)[0]
        y = _Level(density.double(), torch.from_numpy(_element(nu)[0]).cuda(), bc).apply(x)
        return {"y": y.reshape(1, -1), "dot": (x * y).sum().reshape(1)}
    M = _Multigrid(density, bc, nu, case["coarse"])
    if case["do"] == "precondition":
        x = _nodal_noise(case, density, bc, seed, case["nvec"])
        return torch.stack([M.vcycle(v * M.levels[0].free) for v in x]).reshape(case["nvec"], -1)
    u = M.solve(f)
    if case["do"] == "solve":
        return u.reshape(-1)
    u = u / (E * h)
    vm, p1, p3 = _stresses(M.S, density, u, E, h)
    return {"u": u.reshape(-1), "von_mises": vm, "p1": p1, "p3": p3}

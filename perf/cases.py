"""The work that users have this framework do, as cases that can be timed and compared.

Every case goes through the package's public entry points: assembling a problem,
the operator product (host arrays, or device arrays through the C ABI), the
multigrid preconditioner, FP64 and mixed-precision solves, and the U-Net of the
learned warm start (inference and training).  Sizes are those of the
repository's own workloads (the 32x16x16 cantilever, the 128^3 porous field, the
256^3 box with voids, training fields of 64^3 and evaluation fields of 128^3, whose
node grids pad to 72^3 and 136^3) and odd sizes around them.

The geometry of a case is fixed by the case; the seed of ``prepare`` makes the
moduli, the loads, the vectors and the network's samples.

Solves run to a relative residual at which the answer does not depend on the order
of roundings any more: 1e-10 in FP64, 1e-8 to 1e-9 in mixed precision (a
residual of 1e-6 leaves the displacement of a porous field open in the ninth digit,
and more at a floppy node; sensitivities of a design loop, for instance, need the tighter one).
"""
import ctypes

import numpy as np
import torch

from vulkanfem_gb300 import api, domains, learned


def listed():
    return [
        # the smallest product: the cantilever's operator inside a user's own device-side loop
        {"name": "product_beam", "kind": "product", "shape": "beam",
         "nx": 32, "ny": 16, "nz": 16, "levels": 3, "modulus": False, "ke": "cube"},
        # a large product on an odd grid with voids and a modulus per voxel
        {"name": "product_voids", "kind": "product", "shape": "spheres", "geometry": 0,
         "nx": 191, "ny": 191, "nz": 191, "levels": 5, "modulus": True, "ke": "cube"},
        # an element matrix in another node order (as the reference's data file has it): the general product
        {"name": "product_reordered", "kind": "product", "shape": "porous", "geometry": 0, "fill": 0.5,
         "nx": 96, "ny": 80, "nz": 72, "levels": 4, "modulus": False, "ke": "reordered"},
        # K u from host arrays, for strain energies and residual checks in a Python program
        {"name": "product_host", "kind": "host_product", "shape": "porous", "geometry": 0, "fill": 0.5,
         "nx": 88, "ny": 88, "nz": 88, "levels": 4, "modulus": True, "ke": "cube"},
        # one FP64 V-cycle from host arrays, as the preconditioner of a user's own Krylov method
        {"name": "vcycle_fp64", "kind": "vcycle", "shape": "spheres", "geometry": 0,
         "nx": 96, "ny": 96, "nz": 96, "levels": 5, "modulus": True, "ke": "cube", "mode": "reference", "skip": 0},
        # the small cantilever, plain FP64 (the default solve): launches and latency
        {"name": "solve_fp64_beam", "kind": "solve", "shape": "beam",
         "nx": 32, "ny": 16, "nz": 16, "levels": 3, "modulus": False, "ke": "cube",
         "precision": "fp64", "rtol": 1e-10, "skip": 0},
        # the porous field, plain FP64
        {"name": "solve_fp64_porous", "kind": "solve", "shape": "porous", "geometry": 0, "fill": 0.5,
         "nx": 64, "ny": 64, "nz": 64, "levels": 4, "modulus": False, "ke": "cube",
         "precision": "fp64", "rtol": 1e-10, "skip": 0},
        # the 128^3 porous field, mixed precision
        {"name": "solve_mixed_porous", "kind": "solve", "shape": "porous", "geometry": 0, "fill": 0.4,
         "nx": 128, "ny": 128, "nz": 128, "levels": 4, "modulus": False, "ke": "cube",
         "precision": "mixed", "rtol": 1e-9, "skip": 0},
        # the 256^3 box with voids and lognormal moduli, mixed precision: the largest
        {"name": "solve_mixed_voids", "kind": "solve", "shape": "spheres", "geometry": 0,
         "nx": 256, "ny": 256, "nz": 256, "levels": 5, "modulus": True, "ke": "cube",
         "precision": "mixed", "rtol": 1e-8, "skip": 0},
        # one step of a design loop: new moduli, so the problem is assembled again and solved once
        {"name": "design_step", "kind": "design", "shape": "spheres", "geometry": 0,
         "nx": 96, "ny": 96, "nz": 96, "levels": 5, "modulus": True, "ke": "cube",
         "precision": "mixed", "rtol": 1e-8, "skip": 0},
        # the network's prediction for a 128^3 field
        {"name": "unet_forward", "kind": "forward", "n": 136},
        # a training step on four 64^3 fields
        {"name": "unet_train", "kind": "train", "n": 72, "batch": 4},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["product", "product", "host_product", "vcycle", "solve", "solve", "solve", "design", "forward",
                       "train"])
    if kind == "forward":
        return {"kind": kind, "n": 8 * _log(rng, 3, 17)}
    if kind == "train":
        return {"kind": kind, "n": 8 * _log(rng, 2, 9), "batch": rng.randint(1, 4)}
    shape = rng.choice(["beam", "porous", "spheres"])
    top = {"product": 180, "host_product": 112, "vcycle": 112, "solve": 160, "design": 112}[kind]
    case = {"kind": kind, "shape": shape, "modulus": rng.random() < 0.5 and shape != "beam", "ke": "cube"}
    if shape != "beam":
        case["geometry"] = rng.randrange(10)
    if shape == "porous":
        case["fill"] = round(rng.uniform(0.45, 0.6), 2)
    if kind in ("solve", "design"):
        case["precision"] = "mixed" if kind == "design" or rng.random() < 0.5 else "fp64"
        case["skip"] = 1 if rng.random() < 0.2 else 0
        case["rtol"] = 1e-10 if case["precision"] == "fp64" else 1e-9 if shape == "porous" else 1e-8
        if case["precision"] == "fp64":
            top = 72
        if shape == "porous":  # three to five times the iterations of the others
            top = 56 if case["precision"] == "fp64" else 112
    if kind == "vcycle":
        case["mode"] = rng.choice(["reference", "reference", "vcycle"])
        case["skip"] = 1 if rng.random() < 0.2 else 0
    if kind == "product" and rng.random() < 0.3:
        case["ke"], top = "reordered", 112
    low = 12 if shape == "beam" else 32
    if shape == "spheres":
        case["nx"] = case["ny"] = case["nz"] = _log(rng, low, top)
    else:
        case["nx"], case["ny"], case["nz"] = (_log(rng, low, top) for _ in range(3))
    # levels down to a coarsest grid of about 8 elements along its longest edge, as a user picks them
    longest, levels = max(case["nx"], case["ny"], case["nz"]), 1
    while longest > 12:
        longest, levels = (longest + 1) // 2, levels + 1
    case["levels"] = max(2, levels - case.get("skip", 0))
    return case


# ----------------------------------------------------------------- inputs

def _geometry(case):
    nx, ny, nz, levels = case["nx"], case["ny"], case["nz"], case["levels"]
    if case["shape"] == "beam":
        return domains.cantilever(nx, ny, nz, levels)
    if case["shape"] == "porous":
        sigma = max(3.0, 6.0 * min(nx, ny, nz) / 128.0)
        return domains.porous((nz, ny, nx), case["fill"], sigma, seed=case["geometry"], levels=levels)
    return domains.spheres(nx, 20 + (nx * 280) // 256, 3.0, max(5.0, nx / 16.0), seed=case["geometry"],
                           levels=levels, lognormal_sigma=None)


def _stiffness(case):
    ke = domains.hex8_stiffness()
    if case["ke"] == "reordered":
        dof = [3 * p + c for p in domains.KE0_NODE_PERM for c in range(3)]
        ke = ke[np.ix_(dof, dof)]
    return ke


def _inputs(case, seed):
    """Geometry, element matrix, moduli (or None) and the load vector."""
    rng = np.random.default_rng(seed)
    d = _geometry(case)
    E = rng.lognormal(0.0, 0.5, d.voxels.shape).astype(np.float32) if case["modulus"] else None
    lv = d.load_values * (1.0 + 0.3 * rng.standard_normal((len(d.load_nodes), 1)))
    lv[:, :2] = 0.2 * lv[:, 2:3] * rng.standard_normal((len(d.load_nodes), 2))
    f = np.zeros(d.num_dofs)
    f.reshape(-1, 3)[d.load_nodes] = lv
    return d, _stiffness(case), E, f


def _grid_vector(d, seed):
    """A displacement-like vector on the whole node grid: a smooth field and noise, 0 at unused nodes."""
    nz, ny, nx = (s + 1 for s in d.shape)
    g = torch.Generator().manual_seed(seed)
    w = torch.rand(3, 4, generator=g, dtype=torch.float64) * 6.0
    z, y, x = (torch.linspace(0, 1, s, dtype=torch.float64, device="cuda") for s in (nz, ny, nx))
    u = torch.stack([torch.sin(w[c, 0] * x[None, None, :] + w[c, 3]) * torch.cos(w[c, 1] * y[None, :, None])
                     + w[c, 2] * z[:, None, None] for c in range(3)], dim=-1)
    noise = torch.Generator(device="cuda").manual_seed(seed)
    u = u + 0.05 * torch.randn(u.shape, generator=noise, dtype=torch.float64, device="cuda")
    mask = torch.from_numpy(domains.used_nodes_mask(d.voxels)).cuda()
    return (u * mask[..., None]).contiguous()


def _samples(n, count, seed):
    """Features, targets and masks of `count` porous fields on the padded n^3 node grid."""
    X = np.zeros((count, n, n, n, learned.NCH), np.float32)
    T = np.zeros((count, n, n, n, 3), np.float32)
    M = np.zeros((count, n, n, n), np.float32)
    for i in range(count):
        rng = np.random.default_rng([seed, i])
        d = domains.porous(n - 8, rng.uniform(0.4, 0.6), max(3.0, n / 20.0), seed=int(rng.integers(1 << 30)))
        ids = domains.used_nodes_mask(d.voxels)
        u = np.empty(ids.shape + (3,), np.float32)
        h = np.linspace(0, 1, ids.shape[0], dtype=np.float32)
        for c in range(3):
            a = rng.uniform(1, 6, 3)
            plane = np.sin(a[0] * h)[None, :] + np.cos(a[1] * h)[:, None]
            u[..., c] = plane[None] * (a[2] * h ** 1.5)[:, None, None]
        z0 = u[ids] + 0.1 * rng.standard_normal((int(ids.sum()), 3)).astype(np.float32)
        X[i], mask, scale = learned.node_features(d.voxels, None, d.fixed, d.load_nodes, d.load_values, n, z0)
        T[i] = learned.target_grid(u[ids].astype(np.float64).reshape(-1), mask, scale, n)
        M[i] = learned.loss_mask(mask, d.fixed, n)
    return X, T, M


def prepare(case, seed):
    kind = case["kind"]
    if kind == "forward":
        X, _, _ = _samples(case["n"], 1, seed)
        return {"kind": kind, "net": learned.UNet(case["n"], learned.load(learned.CHECKPOINT)), "x": X[0]}
    if kind == "train":
        X, T, M = _samples(case["n"], case["batch"], seed)
        return {"kind": kind, "net": learned.UNet(case["n"], learned.init_params(seed)), "x": X, "t": T, "m": M}
    d, ke, E, f = _inputs(case, seed)
    s = {"kind": kind, "case": case, "d": d, "ke": ke, "E": E, "f": f}
    if kind != "design":
        s["A"] = api.assembleSystemMatrix(d.voxels, ke, d.fixed, d.num_levels, case.get("skip", 0), E=E)
    if kind == "product":
        s["x"] = _grid_vector(d, seed)
        s["y"] = torch.empty_like(s["x"])
        s["dot"] = torch.empty(1, dtype=torch.float64, device="cuda")
    elif kind == "host_product":
        x = _grid_vector(d, seed).cpu().numpy()
        s["x"] = np.ascontiguousarray(x[domains.used_nodes_mask(d.voxels)]).reshape(-1)
    elif kind == "vcycle":
        s["M"] = api.MultigridPreconditioner(s["A"], case["mode"])
        s["r"] = f + 0.01 * np.abs(f).max() * np.random.default_rng(seed + 1).standard_normal(f.size)
    elif kind == "solve":
        s["u"] = np.zeros(f.size)
    return s


def run(s):
    kind = s["kind"]
    if kind == "product":
        stream = torch.cuda.current_stream().cuda_stream
        status = api.load_library().vfem_apply_operator_device_noalloc(
            s["A"]._h, ctypes.c_void_p(s["x"].data_ptr()), ctypes.c_void_p(s["y"].data_ptr()),
            ctypes.c_void_p(s["dot"].data_ptr()), ctypes.c_void_p(stream))
        if status != api.OK:
            raise api.VfemError(status)
        return s["y"], s["dot"]
    if kind == "host_product":
        return s["A"] @ s["x"]
    if kind == "vcycle":
        return s["M"].solve(s["r"])
    if kind == "solve":
        u, _ = s["A"].solve(s["f"], out=s["u"], precision=s["case"]["precision"], rtol=s["case"]["rtol"])
        return u
    if kind == "design":
        d, case = s["d"], s["case"]
        A = api.assembleSystemMatrix(d.voxels, s["ke"], d.fixed, d.num_levels, case["skip"], E=s["E"])
        u, _ = A.solve(s["f"], precision=case["precision"], rtol=case["rtol"])
        A.close()
        return u
    if kind == "forward":
        return s["net"].forward(s["x"])
    loss, grads = s["net"].train_batch(s["x"], s["t"], s["m"], 1e-3, want_grads=True)
    return loss, grads, s["net"].get_params()


# ----------------------------------------------------------------- what a pass cannot do without

def _iterations(case):
    """About how many PCG iterations a solve of this kind takes."""
    edge = max(case["nx"], case["ny"], case["nz"])
    tight = {1e-10: 1.5, 1e-9: 1.35, 1e-8: 1.2}[case["rtol"]]
    return tight * {"beam": 20 + edge / 4, "porous": 4.5 * edge, "spheres": edge}[case["shape"]]


#: Operations of the 8 convolutions per voxel of the finest grid (a multiply and an add each).
_CONV_OPS = 2.0 * 27 * (16 * 16 + 48 * 16 + 16 * 16 + (16 * 32 + 96 * 32) / 8 + (32 * 64 + 192 * 64) / 64
                        + 64 * 128 / 512)


def work(case):
    kind = case["kind"]
    if kind == "forward":
        v = float(case["n"]) ** 3
        return {"bytes": v * 4 * (16 + 3), "flops": v * _CONV_OPS}
    if kind == "train":
        v = float(case["n"]) ** 3 * case["batch"]
        return {"bytes": v * 4 * (16 + 3 + 1), "flops": 3 * v * _CONV_OPS}
    nodes = (case["nx"] + 1.0) * (case["ny"] + 1.0) * (case["nz"] + 1.0)
    elements = float(case["nx"]) * case["ny"] * case["nz"]
    # adds and multiplies of one element's contribution: Walsh-factorised cube, or the dense 24 x 24 matrix
    product = elements * (190.0 if case["ke"] == "cube" else 2 * 576.0)
    per_element = 4.0 if case["modulus"] else 0.125
    once = nodes * 48.0 + elements * per_element
    if kind in ("product", "host_product"):
        return {"bytes": once, "flops": product}
    if kind == "vcycle":
        return {"bytes": once + nodes * 24.0, "flops": nodes * 60.0}
    # a solve: right-hand side in, displacements out; a product, a V-cycle and the vector updates per iteration
    return {"bytes": once, "flops": _iterations(case) * (product + nodes * 90.0)}


# ----------------------------------------------------------------- the same in plain 64-bit torch

_CORNERS = [(a & 1, (a >> 1) & 1, a >> 2) for a in range(8)]


class _Operator:
    """K on the dense node grid: gather of the 8 corners, the 24 x 24 matrix, scatter."""

    def __init__(self, d, ke, E):
        self.n = d.shape
        e = torch.from_numpy(d.voxels.astype(np.float64)).cuda()
        self.e = e if E is None else e * torch.from_numpy(E.astype(np.float64)).cuda()
        self.ke = torch.from_numpy(np.triu(ke) + np.triu(ke, 1).T).cuda()
        mask = domains.used_nodes_mask(d.voxels)
        ids = np.flatnonzero(mask.reshape(-1))
        live = mask.reshape(-1).copy()
        live[ids[d.fixed]] = False
        self.used = torch.from_numpy(mask).cuda()
        self.live = torch.from_numpy(live.reshape(mask.shape)).cuda()[..., None].double()

    def _at(self, v, a):
        nz, ny, nx = self.n
        dx, dy, dz = _CORNERS[a]
        return v[dz:dz + nz, dy:dy + ny, dx:dx + nx]

    def __call__(self, u):
        y = torch.zeros_like(u)
        w = torch.cat([self._at(u, a) for a in range(8)], dim=-1) @ self.ke
        w *= self.e[..., None]
        for a in range(8):
            self._at(y, a).add_(w[..., 3 * a:3 * a + 3])
        return y * self.live

    def diagonal(self):
        y = torch.zeros(self.used.shape + (3,), dtype=torch.float64, device="cuda")
        for a in range(8):
            self._at(y, a).add_(self.e[..., None] * self.ke.diagonal()[3 * a:3 * a + 3])
        return y

    def solve(self, f):
        """Jacobi-preconditioned CG to a relative residual of 1e-13."""
        b = f * self.live
        dinv = torch.where(self.live > 0, 1.0 / self.diagonal().clamp_min(1e-300), 0.0)
        x, r = torch.zeros_like(b), b.clone()
        z = dinv * r
        p, rz, stop = z.clone(), (r * z).sum(), 1e-26 * (b * b).sum()
        for it in range(20000):
            q = self(p)
            alpha = rz / (p * q).sum()
            x += alpha * p
            r -= alpha * q
            if it % 50 == 49 and bool((r * r).sum() < stop):
                break
            z = dinv * r
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
        return x


def _conv(x, w, b):
    n = x.shape[0]
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    y = b.expand(n, n, n, b.numel())
    for tap in range(27):
        dx, dy, dz = tap % 3, (tap // 3) % 3, tap // 9
        y = y + p[dz:dz + n, dy:dy + n, dx:dx + n] @ w[tap]
    return y


def _unet(x, params):
    relu, at, layers = torch.relu, 0, []
    for ci, co in zip((16, 16, 32, 64, 192, 96, 48, 16), (16, 32, 64, 128, 64, 32, 16, 16)):
        layers.append((params[at:at + 27 * ci * co].view(27, ci, co), params[at + 27 * ci * co:at + 27 * ci * co + co]))
        at += 27 * ci * co + co

    def pool(v):
        m = v.shape[0] // 2
        return v.view(m, 2, m, 2, m, 2, -1).mean(dim=(1, 3, 5))

    def up(v, skip):
        for axis in range(3):
            v = v.repeat_interleave(2, dim=axis)
        return torch.cat([v, skip], dim=-1)

    e0 = relu(_conv(x, *layers[0]))
    e1 = relu(_conv(pool(e0), *layers[1]))
    e2 = relu(_conv(pool(e1), *layers[2]))
    d = relu(_conv(pool(e2), *layers[3]))
    for skip, layer in ((e2, layers[4]), (e1, layers[5]), (e0, layers[6])):
        d = relu(_conv(up(d, skip), *layer))
    return _conv(d, *layers[7])[..., :3]


def _train_exact(case, seed):
    X, T, M = _samples(case["n"], case["batch"], seed)
    p = torch.from_numpy(learned.init_params(seed)).double().cuda().requires_grad_()
    total = 0.0
    for x, t, m in zip(X, T, M):
        x, t, m = (torch.from_numpy(v).double().cuda() for v in (x, t, m))
        loss = (m[..., None] * (_unet(x, p) - t) ** 2).sum() / (3.0 * m.sum())
        loss.backward()
        total += float(loss.detach())
    # the weights after the first Adam step: its moments are the gradient itself, bias-corrected
    g = p.grad / case["batch"]
    after = p.detach() - 1e-3 * g / (g.abs() + 1e-8)
    return total / case["batch"], g.cpu().numpy(), after.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "forward":
        with torch.no_grad():
            X, _, _ = _samples(case["n"], 1, seed)
            params = torch.from_numpy(learned.load(learned.CHECKPOINT)).double().cuda()
            return _unet(torch.from_numpy(X[0]).double().cuda(), params).cpu().numpy()
    if kind == "train":
        return _train_exact(case, seed)
    if kind == "vcycle":
        return None  # the coarsest inverse and the Galerkin diagonals would be this repository's own method again
    d, ke, E, f = _inputs(case, seed)
    K = _Operator(d, ke, E)
    if kind in ("product", "host_product"):
        x = _grid_vector(d, seed)
        y = K(x)
        return (y, (x * y).sum().reshape(1)) if kind == "product" else y[K.used].reshape(-1).cpu().numpy()
    if case["nx"] * case["ny"] * case["nz"] > 72 ** 3:
        return None  # over 20 seconds
    u = torch.zeros(K.used.shape + (3,), dtype=torch.float64, device="cuda")
    u[K.used] = torch.from_numpy(f).cuda().view(-1, 3)
    return K.solve(u)[K.used].reshape(-1).cpu().numpy()

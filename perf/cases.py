"""Performance cases: what a user of the framework has it do, each through the
public entry points (the solver classes, Batch, UNet3D, voxelize).

A pass of a solver case is one leg of a simulation: some time steps from the
state that the previous leg left, then the fields read back to the host (a
monitor or export point).  Geometries are random sphere packs of the parameters
the repository's benchmark and tests use, drawn from the seed on the GPU;
channels and cavities are the reference examples' shapes.  `exact` restates each
path in plain torch at 64 bits over the list of fluid nodes.
"""
import math

import numpy as np
import torch

# ------------------------------------------------------------------ the cases


def listed():
    return [
        # The reference's own main loop on a small lattice (step(), get_max_v()
        # now and then): launch and call latency.
        dict(name="cavity_32_single_steps", kind="sp", nx=32, ny=32, nz=32, geo="cavity", storage="f32", drive="lid",
             legs=10, steps=1, maxv=True),
        # Lid-driven cavity of the benchmark: L2-resident, short kernels.
        dict(name="cavity_64_f32", kind="sp", nx=64, ny=64, nz=64, geo="cavity", storage="f32", drive="lid", legs=1,
             steps=200, maxv=False),
        # A channel of odd sizes with a body force (the Poiseuille example), FP32
        # reference arithmetic with the forcing term.
        dict(name="channel_ragged_f32_force", kind="sp", nx=101, ny=67, nz=53, geo="channel", storage="f32",
             drive="force", legs=1, steps=200, maxv=False),
        # The headline workload: 256^3 pack, pressure drop, FP32 reference arithmetic.
        dict(name="pack_256_f32", kind="sp", nx=256, ny=256, nz=256, geo="pack", storage="f32", drive="pressure",
             legs=1, steps=300, maxv=False),
        # The same with 16-bit storage, the fast path of long permeability runs.
        dict(name="pack_256_f16", kind="sp", nx=256, ny=256, nz=256, geo="pack", storage="f16", drive="pressure",
             legs=1, steps=300, maxv=False),
        # A ragged image crop with a body force and BF16 storage.
        dict(name="pack_ragged_bf16_force", kind="sp", nx=150, ny=131, nz=97, geo="pack", storage="bf16",
             drive="force", legs=1, steps=200, maxv=False),
        # Mask in, permeability out: the whole solve of one training-size pack
        # (setup, steps, convergence checks), FP32 deviation form.
        dict(name="permeability_96_f32dev", kind="perm", nx=96, ny=96, nz=96, geo="pack", storage="f32dev",
             drive="force", steps=1000),
        # Drainage of the benchmark's 131^3 pack, two phases.
        dict(name="two_phase_131_f32", kind="tp", nx=131, ny=131, nz=131, storage="f32", drive="pressure", steps=100),
        # A small two-phase sample driven by the script's body force.
        dict(name="two_phase_small_f32", kind="tp", nx=50, ny=44, nz=37, storage="f32", drive="force", steps=50),
        # Grey-scale (partial bounce-back) rock image.
        dict(name="grey_192_f32", kind="grey", nx=192, ny=192, nz=192, storage="f32", drive="force", steps=100),
        # Many subvolumes advanced together to their permeabilities, 16-bit storage.
        dict(name="batch_8_f16", kind="batch", n=8, storage="f16", steps=400),
        # Training step of the warm-start network (forward, loss, backward, Adam).
        dict(name="unet_train_2x96", kind="unet", n=2, edge=96),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sp"] * 6 + ["perm", "tp", "tp", "grey", "batch", "unet"])
    if kind == "unet":
        return dict(kind="unet", n=rng.choice([1, 2, 3]), edge=4 * rng.randint(8, 24))
    if kind == "batch":
        return dict(kind="batch", n=rng.randint(2, 8), storage=rng.choice(["f16", "f16", "f32dev", "bf16", "f32"]),
                    steps=4 * rng.randint(25, 100))
    top = {"sp": 230, "perm": 110, "tp": 140, "grey": 200}[kind]
    # one edge scale, the three edges near it, odd and even alike
    base = _log_int(rng, 20, top)
    n = [min(top, max(16, base + rng.randint(-base // 5, base // 5))) for _ in range(3)]
    case = dict(kind=kind, nx=n[0], ny=n[1], nz=n[2])
    if kind == "tp":
        return dict(case, storage=rng.choice(["f32", "f32", "f16", "f32dev"]), drive=rng.choice(["pressure", "force"]),
                    steps=rng.randint(20, 100))
    if kind == "grey":
        return dict(case, storage=rng.choice(["f32", "f32dev", "f16"]), drive=rng.choice(["pressure", "force"]),
                    steps=rng.randint(20, 100))
    if kind == "perm":
        return dict(case, geo="pack", storage=rng.choice(["f32dev", "f16", "f32"]), drive="force",
                    steps=500 * rng.randint(1, 2))
    geo = rng.choice(["pack", "pack", "pack", "channel", "cavity"])
    if geo == "cavity":
        case.update(ny=case["nx"], nz=case["nx"])
    drive = {"pack": rng.choice(["pressure", "force"]), "channel": rng.choice(["pressure", "force"]),
             "cavity": "lid"}[geo]
    storages = ["f32", "f32", "f32dev", "f16", "bf16"] + (["f64"] if base <= 64 else [])
    case.update(geo=geo, storage=rng.choice(storages), drive=drive)
    if rng.random() < 0.2:
        return dict(case, legs=rng.randint(5, 20), steps=1, maxv=True)
    return dict(case, legs=1, steps=rng.randint(50, 300), maxv=rng.random() < 0.3)


# ------------------------------------------------------------------ inputs

RHO_IN, RHO_OUT, NIU = 1.0005, 1.0, 0.1
EDGES = (96, 48, 160, 64, 128)      # the batched workload's subvolumes
TP = dict(niu_l=0.05, niu_g=0.2, psi_solid=0.7, cap_a=0.005, rho_in=1.001, rho_out=1.0, force=5.0e-5)
# FP32 reference arithmetic needs a drive that stands clear of its rounding; the other storages resolve a slower flow
FORCE = {"f32": 1e-5, "f32dev": 1e-6, "f16": 1e-6, "bf16": 1e-6, "f64": 1e-6}
ELEM = {"f32": 4, "f32dev": 4, "f16": 2, "bf16": 2, "f64": 8}


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _pack(shape, rmin, rmax, phi, g):
    """Overlapping periodic spheres (radii uniform in [rmin, rmax]) up to an
    expected fluid fraction phi: int8 numpy mask, 1 = solid."""
    nx, ny, nz = shape
    er3 = (rmax ** 4 - rmin ** 4) / (4 * (rmax - rmin))
    count = max(1, int(round(-math.log(phi) * nx * ny * nz / (4 / 3 * math.pi * er3))))
    c = torch.rand((count, 3), generator=g, device="cuda", dtype=torch.float64)
    c = c * torch.tensor([nx, ny, nz], device="cuda", dtype=torch.float64)
    r = torch.rand((count,), generator=g, device="cuda", dtype=torch.float64) * (rmax - rmin) + rmin
    m = int(math.ceil(rmax)) + 1
    d = torch.arange(-m, m + 1, device="cuda")
    off = torch.cartesian_prod(d, d, d)
    size = torch.tensor([nx, ny, nz], device="cuda")
    solid = torch.zeros(nx * ny * nz, dtype=torch.int8, device="cuda")
    for a in range(0, count, 1024):
        p = torch.floor(c[a:a + 1024]).long()[:, None, :] + off[None]
        inside = ((p - c[a:a + 1024, None, :]) ** 2).sum(-1) <= (r[a:a + 1024] ** 2)[:, None]
        q = torch.remainder(p, size)
        cell = (q[..., 0] * ny + q[..., 1]) * nz + q[..., 2]
        solid[cell[inside]] = 1
    return solid.reshape(shape).cpu().numpy()


def _mask(case, g):
    shape = (case["nx"], case["ny"], case["nz"])
    if case["geo"] == "cavity":      # a one-cell shell on five faces, the top z face left open for the lid
        s = np.ones(shape, np.int8)
        s[1:-1, 1:-1, 1:] = 0
        return s
    if case["geo"] == "channel":     # plates on the z faces, a post at a random place
        s = np.zeros(shape, np.int8)
        s[:, :, 0] = s[:, :, -1] = 1
        at = (torch.rand(3, generator=g, device="cuda").cpu().numpy() * np.array(shape)).astype(int)
        s[at[0]:at[0] + 4, at[1]:at[1] + 4, :] = 1
        return s
    small = min(shape) < 48
    return _pack(shape, 2.0 if small else 4.0, 5.0 if small else 10.0, 0.5 if small else 0.35, g)


def _uniform(g, lo, hi):
    return lo + (hi - lo) * float(torch.rand(1, generator=g, device="cuda"))


def _sp_settings(case, g):
    """niu, force, faces of a single-phase case: (niu, force, bc, rho_bc, lid)."""
    niu = NIU * _uniform(g, 0.95, 1.05)
    force, bc, rho, lid = [0.0, 0.0, 0.0], [0] * 6, [1.0] * 6, [0.0, 0.0, 0.0]
    if case["drive"] == "force":
        force = [FORCE[case["storage"]], 0.0, 0.0]
    elif case["drive"] == "pressure":
        bc[0] = bc[1] = 1
        rho[0], rho[1] = RHO_IN, RHO_OUT
    else:
        bc[5] = 2
        lid = [_uniform(g, 0.09, 0.1), 0.0, 0.0]
    return niu, force, bc, rho, lid


def _prepare_sp(case, seed):
    from taichi_lbm3d_gb300 import LB3D_Solver_Single_Phase
    g = _gen(seed)
    solid = _mask(case, g)
    niu, force, bc, rho, lid = _sp_settings(case, g)
    perm = case["kind"] == "perm"
    conv = "standard" if perm or case["drive"] == "force" else "class"
    s = LB3D_Solver_Single_Phase(case["nx"], case["ny"], case["nz"], storage=case["storage"],
                                 viscosity_convention=conv, guo_convention=conv)
    s.solid.from_numpy(solid)
    s.set_viscosity(niu)
    s.set_force(force)
    if bc[0]:
        s.set_bc_rho_x0(rho[0])
        s.set_bc_rho_x1(rho[1])
    if bc[5]:
        s.set_bc_vel_z1(lid)
    if not perm:
        s.init_simulation()
    return dict(case=case, solver=s)


def _prepare_tp(case, seed):
    from taichi_lbm3d_gb300 import LB3D_Solver_Two_Phase
    g = _gen(seed)
    shape = (case["nx"], case["ny"], case["nz"])
    small = min(shape) < 48
    solid = _pack(shape, 2.0 if small else 3.0, 5.0 if small else 8.0, 0.5 if small else 0.40, g)
    psi = -np.ones(shape, np.float32)
    psi[:5] = 1.0
    s = LB3D_Solver_Two_Phase(*shape, storage=case["storage"])
    s.niu_l, s.niu_g = TP["niu_l"] * _uniform(g, 0.95, 1.05), TP["niu_g"]
    s.psi_solid, s.CapA = TP["psi_solid"], TP["cap_a"]
    s.bc_psi_x_left, s.psi_x_left, s.bc_psi_x_right, s.psi_x_right = 1, 1.0, 1, -1.0
    if case["drive"] == "pressure":
        s.fx = 0.0
        s.bc_x_left, s.rho_bcxl, s.bc_x_right, s.rho_bcxr = 1, TP["rho_in"], 1, TP["rho_out"]
    else:
        s.fx = TP["force"]
    s.solid.from_numpy(solid)
    s.psi.from_numpy(psi)
    s.init_simulation()
    return dict(case=case, solver=s)


def _prepare_grey(case, seed):
    from taichi_lbm3d_gb300 import LB3D_Solver_Grey_Scale
    g = _gen(seed)
    shape = (case["nx"], case["ny"], case["nz"])
    solid = _pack(shape, 4.0, 10.0, 0.35, g) if min(shape) >= 48 else _pack(shape, 2.0, 5.0, 0.5, g)
    # solid cores and a grey layer on the pore cells next to them (unresolved roughness)
    t = torch.from_numpy(solid).cuda().float()[None, None]
    near = torch.nn.functional.max_pool3d(torch.nn.functional.pad(t, (1,) * 6, mode="circular"), 3, 1)[0, 0]
    ns = near.double() * 0.25
    ns[t[0, 0] > 0] = 1.0
    ns = ns.cpu().numpy()
    s = LB3D_Solver_Grey_Scale(*shape, storage=case["storage"])
    s.niu = NIU * _uniform(g, 0.95, 1.05)
    if case["drive"] == "pressure":
        s.fx = 0.0
        s.bc_x_left, s.rho_bcxl, s.bc_x_right, s.rho_bcxr = 1, 1.0, 1, 0.995
    else:
        s.fx = FORCE[case["storage"]]
    s.ns.from_numpy(ns)
    s.solid.from_numpy(ns.astype(int))
    s.init_simulation()
    return dict(case=case, solver=s)


def _batch_masks(case, g):
    return [_pack((EDGES[q % 5],) * 3, 3.0, 8.0, _uniform(g, 0.25, 0.50), g) for q in range(case["n"])]


def _prepare_batch(case, seed):
    from taichi_lbm3d_gb300.batch import Batch
    b = Batch(_batch_masks(case, _gen(seed)), niu=NIU, force=(1e-6, 0.0, 0.0), storage=case["storage"])
    return dict(case=case, batch=b)


def _unet_inputs(case, seed):
    g = _gen(seed)
    n, e = case["n"], case["edge"]
    x = torch.zeros((n, e, e, e, 16), device="cuda")
    mask = torch.empty((n, e, e, e), device="cuda", dtype=torch.uint8)
    for q in range(n):
        solid = torch.from_numpy(_pack((e,) * 3, 3.0, 8.0, 0.4, g)).cuda().float()
        # fluid indicator and distance to solid (in cells / 8), by repeated erosion
        dist, left = torch.zeros_like(solid), 1.0 - solid
        for _ in range(8):
            dist += left
            left = -torch.nn.functional.max_pool3d(-left[None, None], 3, 1, 1)[0, 0]
        x[q, ..., 0] = 1.0 - solid
        x[q, ..., 1] = dist / 8.0
        mask[q] = (solid == 0).to(torch.uint8)
    target = torch.randn((n, e, e, e, 4), generator=g, device="cuda") * mask[..., None] + 0.5 * x[..., 1:2]
    return x.to(torch.bfloat16), target.contiguous(), mask


def _prepare_unet(case, seed):
    from taichi_lbm3d_gb300.unet import UNet3D
    x, target, mask = _unet_inputs(case, seed)
    return dict(case=case, net=UNet3D(seed=int(seed) % 1000), x=x, target=target, mask=mask,
                count=float(mask.sum().item()) * 4)


def prepare(case, seed):
    return {"sp": _prepare_sp, "perm": _prepare_sp, "tp": _prepare_tp, "grey": _prepare_grey, "batch": _prepare_batch,
            "unet": _prepare_unet}[case["kind"]](case, seed)


# ------------------------------------------------------------------ one pass


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "unet":
        m = state["net"]
        y = m.forward(state["x"])
        loss, gy = m.loss(y, state["target"], state["mask"], state["count"])
        m.backward(gy)
        m.adam_step(lr=1e-4)
        return {"y": y, "loss": loss, "gw": m.gw, "gb": m.gb, "gh": m.ghw_hb, "w": m.w}
    if kind == "batch":
        b = state["batch"]
        b.init()
        darcy, _, _ = b.run_to_convergence(tol=1e-6, check_every=case["steps"] // 2, max_steps=case["steps"])
        rho, v = b.macros(0)
        return {"darcy": darcy, "rho": rho, "v": v}
    s = state["solver"]
    if kind == "perm":
        s.init_simulation()
        r = s.run_to_convergence(tol=1e-6, check_every=500, max_steps=case["steps"])
        return {"k": r["k"], "rho": s.rho.to_numpy(), "v": s.v.to_numpy()}
    if kind == "tp":
        s.run(case["steps"])
        return {"rho": s.rho.to_numpy(), "v": s.v.to_numpy(), "psi": s.phase.to_numpy()}
    if kind == "grey":
        s.run(case["steps"])
        return {"rho": s.rho.to_numpy(), "v": s.v.to_numpy()}
    for _ in range(case["legs"]):
        if case["steps"] == 1:
            s.step()
        else:
            s.run(case["steps"])
    out = {"rho": s.rho.to_numpy(), "v": s.v.to_numpy()}
    if case["maxv"]:
        out["max_v"] = s.get_max_v()
    return out


# ------------------------------------------------------------------ what a pass cannot do without


def _fluid(case):
    """Expected number of fluid nodes."""
    if case["kind"] == "batch":
        return 0.37 * sum(EDGES[q % 5] ** 3 for q in range(case["n"]))
    n = case["nx"] * case["ny"] * case["nz"]
    small = min(case["nx"], case["ny"], case["nz"]) < 48
    if case["kind"] == "tp":
        return n * (0.5 if small else 0.4)
    return n * {"pack": 0.5 if small else 0.35, "cavity": 0.9, "channel": 0.95}[case.get("geo", "pack")]


UNET_LAYERS = [("e1", 16, 16, 0), ("e1b", 16, 16, 0), ("e2", 16, 32, 1), ("e2b", 32, 32, 1), ("b1", 32, 64, 2),
               ("b1b", 64, 64, 2), ("d2", 96, 32, 1), ("d2b", 32, 32, 1), ("d1", 48, 16, 0), ("d1b", 16, 16, 0)]


def work(case):
    """Each step reads and writes every population of a fluid node once (two
    phases: also the two densities; grey: the node's fraction); the fields go
    out once.  Network: the convolutions' multiply-adds, and the activations."""
    if case["kind"] == "unet":
        vox = case["n"] * case["edge"] ** 3
        flops = sum(3 * 2.0 * (vox >> (3 * lv)) * 27 * ci * co for _, ci, co, lv in UNET_LAYERS)
        return {"bytes": sum(2.0 * (vox >> (3 * lv)) * (2 * ci + 2 * co) for _, ci, co, lv in UNET_LAYERS),
                "flops": flops}
    nf = _fluid(case)
    steps = case["steps"] * case.get("legs", 1)
    e = ELEM[case["storage"]]
    node = 38 * e + {"tp": 6 * max(4, e), "grey": max(4, e)}.get(case["kind"], 0)
    cells = 96 ** 3 if case["kind"] == "batch" else case["nx"] * case["ny"] * case["nz"]
    return {"bytes": nf * steps * node + cells * (1 + 16 + (4 if case["kind"] == "tp" else 0)),
            "flops": nf * steps * (900 if case["kind"] == "tp" else 400)}


# ------------------------------------------------------------------ the same at 64 bits

E = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0), (1, -1, 0),
     (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1), (0, 1, -1), (0, -1, 1)]
LR = [0] + [s + 1 if s % 2 else s - 1 for s in range(1, 19)]


def _moment_rows():
    rows = []
    for x, y, z in E:
        q = x * x + y * y + z * z
        rows.append([1, q - 1, 1 - 6 * q + 3 * q * q, x, x * (3 * q - 5), y, y * (3 * q - 5), z, z * (3 * q - 5),
                     3 * x * x - q, (3 * x * x - q) * (2 * q - 3), y * y - z * z, (y * y - z * z) * (2 * q - 3),
                     x * y, y * z, x * z, x * (y * y - z * z), y * (z * z - x * x), z * (x * x - y * y)])
    return torch.tensor(rows, dtype=torch.float64, device="cuda").T.contiguous()


class _Lattice64:
    """Fluid-node list of a mask with its pull table, and the D3Q19 MRT pieces."""

    def __init__(self, solid, rest_slots=False):
        dev = "cuda"
        s = torch.from_numpy(np.ascontiguousarray(solid)).to(dev) > 0
        self.shape = nx, ny, nz = tuple(s.shape)
        self.solid = s
        self.cell = torch.nonzero(~s.reshape(-1)).reshape(-1)
        n = self.n = self.cell.numel()
        self.node = torch.full((nx * ny * nz,), -1, dtype=torch.long, device=dev)
        self.node[self.cell] = torch.arange(n, device=dev)
        self.ijk = (self.cell // (ny * nz), (self.cell // nz) % ny, self.cell % nz)
        own = torch.arange(n, device=dev)
        self.pull = torch.empty((19, n), dtype=torch.long, device=dev)      # flat slot each population comes from
        self.src = torch.empty((19, n), dtype=torch.long, device=dev) if rest_slots else None
        for k, e in enumerate(E):
            src = self.neighbour([-c for c in e])
            self.pull[k] = torch.where(src >= 0, k * n + src, LR[k] * n + own)
            if rest_slots:
                self.src[k] = src
        self.M = _moment_rows()
        self.Mi = torch.linalg.inv(self.M)
        self.e = torch.tensor(E, dtype=torch.float64, device=dev)
        self.w = torch.tensor([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12, dtype=torch.float64, device=dev)

    def neighbour(self, d, clamp=((0, 0), (0, 0), (0, 0))):
        """Node at x + d (wrapped, or clamped on the faces asked for), -1 where solid."""
        q = []
        for a in range(3):
            c = self.ijk[a] + d[a]
            top = self.shape[a] - 1
            c = torch.where(c < 0, torch.full_like(c, 0 if clamp[a][0] else top), c)
            c = torch.where(c > top, torch.full_like(c, top if clamp[a][1] else 0), c)
            q.append(c)
        return self.node[(q[0] * self.shape[1] + q[1]) * self.shape[2] + q[2]]

    def feq(self, rho, u):
        eu = self.e @ u
        return self.w[:, None] * rho * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * (u * u).sum(0))

    def rates(self, sv):
        so = 8 * (2 - sv) / (8 - sv)
        k = [0, 1, 1, 0, 2, 0, 2, 0, 2, 1, 1, 1, 1, 1, 1, 1, 2, 2, 2]
        return torch.tensor([0.0, sv, so], dtype=torch.float64, device="cuda")[torch.tensor(k, device="cuda")]

    @staticmethod
    def meq(rho, u):
        m = torch.zeros((19, rho.numel()), dtype=torch.float64, device="cuda")
        x, y, z = u
        m[0], m[3], m[5], m[7], m[1] = rho, x, y, z, (u * u).sum(0)
        m[9], m[11], m[13], m[14], m[15] = 2 * x * x - y * y - z * z, y * y - z * z, x * y, y * z, x * z
        return m

    def guo(self, u, f, a, b):
        """w (a (e - u).F + b (e.u)(e.F)) per direction."""
        ef = self.e @ f
        return self.w[:, None] * (a * (ef[:, None] - (u * f[:, None]).sum(0)) + b * (self.e @ u) * ef[:, None])

    def face(self, axis, hi):
        c = self.ijk[axis]
        return torch.nonzero(c == (self.shape[axis] - 1 if hi else 0)).reshape(-1)

    def dense(self, x, fill):
        out = torch.full((self.solid.numel(),) + tuple(x.shape[:-1]), float(fill), dtype=torch.float64, device="cuda")
        out[self.cell] = x.T if x.dim() > 1 else x
        return out.reshape(self.shape + tuple(x.shape[:-1]))


def _exact_sp(solid, steps, niu, force, bc, rho_bc, lid, conv, ns=None):
    """rho (n), v (3, n) after `steps`, and the lattice."""
    L = _Lattice64(solid, rest_slots=ns is not None)
    tau = niu / 3 + 0.5 if conv == "class" else 3 * niu + 0.5
    S = L.rates(1 / tau)[:, None]
    ga, gb = {"class": (1 / 3, 1 / 9), "standard": (3.0, 9.0), "script": (1.0, 1.0)}[conv]
    f = torch.tensor(force, dtype=torch.float64, device="cuda")
    forced = bool((f != 0).any())
    rho = torch.ones(L.n, dtype=torch.float64, device="cuda")
    u = torch.zeros((3, L.n), dtype=torch.float64, device="cuda")
    F = L.feq(rho, u)
    faces = []
    for q in range(6):
        if bc[q]:
            ids = L.face(q // 2, q % 2)
            d = [0, 0, 0]
            d[q // 2] = -1 if q % 2 else 1
            inner = L.neighbour(d)[ids] >= 0
            faces.append((bc[q], ids, inner.double(), rho_bc[q]))
    lid = torch.tensor(lid, dtype=torch.float64, device="cuda")[:, None]
    frac = None if ns is None else torch.from_numpy(ns).cuda().reshape(-1)[L.cell]
    A = torch.eye(19, dtype=torch.float64, device="cuda") - L.Mi @ (S * L.M)
    B = L.Mi * S.T
    G = L.Mi @ ((1 - 0.5 * S) * L.M)
    for _ in range(steps):
        f1 = A @ F + B @ L.meq(rho, u)
        if forced:
            f1 += G @ L.guo(u, f, ga, gb)
        if ns is None:
            F = f1.reshape(-1)[L.pull.reshape(-1)].reshape(19, L.n)
        else:
            for s in range(19):
                src = L.src[s]
                ok = src >= 0
                a = f1[s][src.clamp(min=0)]
                F[s] = torch.where(ok, a + frac[src.clamp(min=0)] * (f1[LR[s]] - a), F[s])
        for kind, ids, inner, rb in faces:
            if kind == 1:
                F[:, ids] = L.feq(torch.full((ids.numel(),), rb, dtype=torch.float64, device="cuda"), u[:, ids] * inner)
            else:
                F[:, ids] = L.feq(torch.ones(ids.numel(), dtype=torch.float64, device="cuda"),
                                  lid.expand(3, ids.numel()))
        rho = F.sum(0)
        u = (L.e.T @ F + 0.5 * f[:, None]) / rho
    return L, rho, u


def _exact_tp(case, seed):
    g = _gen(seed)
    shape = (case["nx"], case["ny"], case["nz"])
    small = min(shape) < 48
    solid = _pack(shape, 2.0 if small else 3.0, 5.0 if small else 8.0, 0.5 if small else 0.40, g)
    niu_l, niu_g = TP["niu_l"] * _uniform(g, 0.95, 1.05), TP["niu_g"]
    pressure = case["drive"] == "pressure"
    f = torch.tensor([0.0 if pressure else TP["force"], 0.0, 0.0], dtype=torch.float64, device="cuda")
    L = _Lattice64(solid)
    wl, wg = 1 / (3 * niu_l + 0.5), 1 / (3 * niu_g + 0.5)
    lg0 = 2 * wl * wg / (wl + wg)
    l1, g1 = 20 * (wl - lg0), 20 * (lg0 - wg)
    psi0 = -np.ones(shape)
    psi0[:5] = 1.0
    psi0 = torch.from_numpy(psi0).cuda()
    psi = psi0.reshape(-1)[L.cell].clone()
    rr = (psi + 1) / 2
    rb = 1 - rr
    rho = torch.ones(L.n, dtype=torch.float64, device="cuda")
    u = torch.zeros((3, L.n), dtype=torch.float64, device="cuda")
    F = L.feq(rho, u)
    clamp = ((1, 1), (0, 0), (0, 0))
    nbr = torch.stack([L.neighbour(e, clamp) for e in E])
    touch = (nbr < 0).any(0)
    ends = [(L.face(0, 0), 1.0, TP["rho_in"]), (L.face(0, 1), -1.0, TP["rho_out"])]
    inner = [(L.neighbour((1, 0, 0))[ends[0][0]] >= 0).double(), (L.neighbour((-1, 0, 0))[ends[1][0]] >= 0).double()]
    kind = torch.tensor([0, 1, 1, 0, 2, 0, 2, 0, 2, 1, 1, 1, 1, 1, 1, 1, 2, 2, 2], device="cuda")
    for _ in range(case["steps"]):
        ps = torch.where(nbr >= 0, psi[nbr.clamp(min=0)], torch.full((), TP["psi_solid"], dtype=torch.float64,
                                                                     device="cuda"))
        C = (3 * L.w[:, None] * L.e).T @ ps
        C = torch.where((rr - rb).abs().gt(0.9) & touch, torch.zeros_like(C), C)
        cc = C.square().sum(0).sqrt()
        nrm = torch.where(cc > 0, C / cc.clamp(min=1e-300), torch.zeros_like(C))
        sv = torch.where(psi > 0, torch.where(psi > 0.1, torch.full_like(psi, wl), lg0 + l1 * psi - l1 / 0.2 * psi * psi),
                         torch.where(psi < -0.1, torch.full_like(psi, wg), lg0 + g1 * psi + g1 / 0.2 * psi * psi))
        S = torch.stack([torch.zeros_like(sv), sv, 8 * (2 - sv) / (8 - sv)])[kind]
        meq = L.meq(rho, u)
        hc, (a, b, c) = 0.5 * TP["cap_a"] * cc, nrm
        meq[1] += TP["cap_a"] * cc
        meq[9] += hc * (2 * a * a - b * b - c * c)
        meq[11] += hc * (b * b - c * c)
        meq[13] += hc * a * b
        meq[14] += hc * b * c
        meq[15] += hc * a * c
        m = L.M @ F
        m = m - S * (m - meq)
        if not pressure:
            m += (1 - 0.5 * S) * (L.M @ L.guo(u, f, 1.0, 1.0))
        f1 = L.Mi @ m
        gr, gb = L.feq(rr, u), L.feq(rb, u)
        for k in range(1, 19, 2):
            ef = (L.e[k][:, None] * C).sum(0)
            cp = torch.minimum(torch.minimum(gr[k], gr[k + 1]), torch.minimum(gb[k], gb[k + 1]))
            cp = torch.where(cc > 0, cp * ef / cc.clamp(min=1e-300), torch.zeros_like(cp))
            gr[k] += cp
            gr[k + 1] -= cp
            gb[k] -= cp
            gb[k + 1] += cp
        at = L.pull.reshape(-1)
        F = f1.reshape(-1)[at].reshape(19, L.n)
        rr = gr.reshape(-1)[at].reshape(19, L.n).sum(0)
        rb = gb.reshape(-1)[at].reshape(19, L.n).sum(0)
        if pressure:
            for (ids, _, rho_f), ok in zip(ends, inner):
                F[:, ids] = L.feq(torch.full((ids.numel(),), rho_f, dtype=torch.float64, device="cuda"), u[:, ids] * ok)
        rho = F.sum(0)
        u = (L.e.T @ F + 0.5 * f[:, None]) / rho
        psi = rr - rb / (rr + rb)
        for ids, val, _ in ends:
            psi[ids], rr[ids], rb[ids] = val, (val + 1) / 2, 1 - (val + 1) / 2
    out = psi0.clone().reshape(-1)
    out[L.cell] = psi
    return {"rho": L.dense(rho, 1), "v": L.dense(u, 0), "psi": out.reshape(shape)}


def _exact_unet(case, seed):
    x, target, mask = _unet_inputs(case, seed)
    g = torch.Generator().manual_seed(int(seed) % 1000)
    w, b = {}, {}
    for name, ci, co, _ in UNET_LAYERS:
        real = 2 if name == "e1" else ci
        t = torch.zeros(co, 27, ci)
        t[:, :, :real] = torch.randn(co, 27, real, generator=g) * (2.0 / (27 * real)) ** 0.5
        w[name] = t.cuda().double().requires_grad_()
        b[name] = torch.zeros(co, device="cuda", dtype=torch.float64, requires_grad=True)
    hw = (torch.randn(4, 16, generator=g) * 0.25).cuda().double().requires_grad_()
    hb = torch.zeros(4, device="cuda", dtype=torch.float64, requires_grad=True)

    def conv(name, t):
        k = w[name]
        t = torch.nn.functional.pad(t, (1,) * 6)
        d, h, wd = (s - 2 for s in t.shape[2:])
        out = b[name][None, :, None, None, None]
        for tap in range(27):
            z, y, q = tap // 9, (tap // 3) % 3, tap % 3
            out = out + torch.einsum("ncdhw,oc->nodhw", t[:, :, z:z + d, y:y + h, q:q + wd], k[:, tap])
        return out.relu()

    t = x.double().permute(0, 4, 1, 2, 3)
    pool = torch.nn.functional.max_pool3d
    e1 = conv("e1b", conv("e1", t))
    e2 = conv("e2b", conv("e2", pool(e1, 2)))
    z = conv("b1b", conv("b1", pool(e2, 2)))
    z = conv("d2b", conv("d2", torch.cat([z.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4), e2], 1)))
    z = conv("d1b", conv("d1", torch.cat([z.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4), e1], 1)))
    y = torch.einsum("ncdhw,oc->ndhwo", z, hw) + hb
    loss = (((y - target.double()) * mask[..., None].double()) ** 2).sum() / (float(mask.sum().item()) * 4)
    loss.backward()
    return {"y": y.detach(), "loss": loss.detach().reshape(1), "gw": {k: v.grad for k, v in w.items()},
            "gb": {k: v.grad for k, v in b.items()}, "gh": torch.cat([hw.grad.reshape(-1), hb.grad]), "w": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "unet":
        return _exact_unet(case, seed) if case["n"] * case["edge"] ** 3 <= 2_000_000 else None
    if kind == "tp":
        return _exact_tp(case, seed)
    g = _gen(seed)
    if kind == "batch":
        darcy, first = [], None
        for solid in _batch_masks(case, g):
            L, rho, u = _exact_sp(solid, case["steps"], NIU, (1e-6, 0.0, 0.0), [0] * 6, [1.0] * 6, [0.0] * 3, "standard")
            darcy.append(float(u[0].sum()) / L.solid.numel())
            if first is None:
                # the batch reads its fields from the populations it has: the next step's macroscopic values
                L, rho, u = _exact_sp(solid, case["steps"] + 1, NIU, (1e-6, 0.0, 0.0), [0] * 6, [1.0] * 6, [0.0] * 3,
                                      "standard")
                first = {"rho": L.dense(rho, 1), "v": L.dense(u, 0)}
        return dict(first, darcy=np.array(darcy))
    if kind == "grey":
        shape = (case["nx"], case["ny"], case["nz"])
        solid = _pack(shape, 4.0, 10.0, 0.35, g) if min(shape) >= 48 else _pack(shape, 2.0, 5.0, 0.5, g)
        t = torch.from_numpy(solid).cuda().float()[None, None]
        near = torch.nn.functional.max_pool3d(torch.nn.functional.pad(t, (1,) * 6, mode="circular"), 3, 1)[0, 0]
        ns = near.double() * 0.25
        ns[t[0, 0] > 0] = 1.0
        niu = NIU * _uniform(g, 0.95, 1.05)
        p = case["drive"] == "pressure"
        force = (0.0 if p else FORCE[case["storage"]], 0.0, 0.0)
        L, rho, u = _exact_sp(solid, case["steps"], niu, force, [int(p)] * 2 + [0] * 4, [1.0, 0.995] + [1.0] * 4,
                              [0.0] * 3, "script", ns=ns.cpu().numpy())
        return {"rho": L.dense(rho, 1), "v": L.dense(u, 0)}
    solid = _mask(case, g)
    niu, force, bc, rho_bc, lid = _sp_settings(case, g)
    conv = "standard" if kind == "perm" or case["drive"] == "force" else "class"
    L, rho, u = _exact_sp(solid, case["steps"] * case.get("legs", 1), niu, force, bc, rho_bc, lid, conv)
    out = {"rho": L.dense(rho, 1), "v": L.dense(u, 0)}
    if kind == "perm":
        tau = 3 * niu + 0.5
        out["k"] = (tau - 0.5) / 3 * float(u[0].sum()) / L.solid.numel() / force[0]
    elif case["maxv"]:
        out["max_v"] = float(u.square().sum(0).sqrt().max())
    return out

"""Workloads of the framework for timing: what a program that solves implicit
FEM systems with it does, over the sizes it is used at.

Each case is a path through the public entry points (delfem2_gb300) at one
size. Meshes are voxel blocks of nx x ny x nz cells, six tets a cell, nodes
numbered z fastest (the benchmark's meshes), and square cloth sheets; moduli,
loads and vectors come from the seed.

  step      a design loop's step: per-tet moduli on the device -> assembly,
            clamp, ILU(fill), FP64 Solve_PCG to 1e-10
  solve     Solve_PCG / Solve_PCG_Mixed on an assembled and factored system:
            many right-hand sides for one matrix
  precond   SolvePrecond alone, as a caller's own Krylov loop applies it
  setup     CopyValue + Decompose of a new matrix and its first application
  assemble  setZero, assembly, clamp, and the residual product of the result
  gradient  the differentiable solve, forward and backward (moduli and load)
  cloth     one implicit cloth step (StepTime_InternalDynamicsILU)
  poisson   the scalar problem on the tets (1x1 blocks), assembly to solution
  warp      a stiffness-warped backward-Euler step (not symmetric): assembly,
            ILU(0), Solve_PBiCGStab

exact() restates each path in 64-bit torch on the block's 15-point stencil.
"""
import itertools
import math

import numpy as np
import torch

import delfem2_gb300 as D
from delfem2_gb300 import cloth as DC
from delfem2_gb300.autograd import linear_elastic_solve

NU, RHO, GRAV = 0.3, 1.0, (0.0, 0.0, -1e-3)
TOL = 1e-10
WARP = dict(myu=1.0, lam=2.0, rho=1.5, g=(0.0, 0.0, -9.8), dt=0.01)
CLOTH = dict(nu=0.3, bend=1e-3, g=(0.0, 0.0, -10.0), dt=0.01)


def listed():
    return [
        # an interactive toy block: the smallest calls, where launches and waits count
        dict(name="step_8x7x9", path="step", nx=8, ny=7, nz=9, fill=0),
        # an ordinary ragged part with level-1 fill, whole step
        dict(name="step_fill1_25x27x23", path="step", nx=25, ny=27, nz=23, fill=1),
        # the FP64 drop-in at scale (823,875 DOF): many loads on one factored matrix
        dict(name="solve_f64_64x64x64", path="solve", nx=64, ny=64, nz=64, precision="f64"),
        # the headline: 3,244,995 DOF, FP32 iteration with FP64 reliable updates
        dict(name="solve_mixed_128x128x64", path="solve", nx=128, ny=128, nz=64, precision="mixed"),
        # the preconditioner inside a caller's own FP32 Krylov loop, large and ragged
        dict(name="precond_f32_101x97x67", path="precond", nx=101, ny=97, nz=67, precision="f32"),
        # the same in FP64 at an ordinary size
        dict(name="precond_f64_40x37x43", path="precond", nx=40, ny=37, nz=43, precision="f64"),
        # a new matrix on a kept pattern: factorisation and first application
        dict(name="setup_63x64x61", path="setup", nx=63, ny=64, nz=61, fill=0),
        # a load step's assembly and residual, large
        dict(name="assemble_96x95x64", path="assemble", nx=96, ny=95, nz=64),
        # material identification: gradient of a misfit w.r.t. moduli and load
        dict(name="gradient_48x48x48", path="gradient", nx=48, ny=48, nz=48, precision="mixed"),
        # one frame of an implicit cloth sheet
        dict(name="cloth_44", path="cloth", ndiv=44),
        # heat / potential problem on the tets, assembly to solution
        dict(name="poisson_64x64x64", path="poisson", nx=64, ny=64, nz=64),
        # one frame of a stiffness-warped solid
        dict(name="warp_21x20x19", path="warp", nx=21, ny=20, nz=19),
    ]


# cells of the smallest and largest drawn block of each path
_RANGE = dict(step=(300, 30_000), solve=(2_000, 300_000), precond=(2_000, 800_000), setup=(1_000, 300_000),
              assemble=(1_000, 700_000), gradient=(2_000, 120_000), poisson=(2_000, 300_000), warp=(500, 30_000))


def draw(rng):
    path = rng.choice(["step", "solve", "precond", "setup", "assemble", "gradient", "cloth", "poisson", "warp"])
    if path == "cloth":
        return dict(path=path, ndiv=rng.randint(8, 46))
    lo, hi = _RANGE[path]
    cells = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    ax, ay = (math.exp(rng.uniform(-0.5, 0.5)) for _ in range(2))
    side = (cells / (ax * ay)) ** (1.0 / 3.0)
    case = dict(path=path, nx=max(3, round(side * ax)), ny=max(3, round(side * ay)), nz=max(3, round(side)))
    if path == "step":
        case["fill"] = rng.choice([0, 0, 1])
    if path == "setup":
        case["fill"] = rng.choice([0, 0, 1])
    if path == "solve":
        case["precision"] = rng.choice(["f64", "mixed"])
    if path == "precond":
        case["precision"] = rng.choice(["f64", "f32"])
    if path == "gradient":
        case["precision"] = rng.choice(["fp64", "mixed"])
    return case


# ---- inputs ---------------------------------------------------------------------
_CORNER = ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))
_SIX = ((0, 1, 2, 6), (0, 1, 6, 5), (0, 4, 5, 6), (0, 2, 3, 6), (0, 3, 7, 6), (0, 4, 6, 7))


def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _mesh(case):
    """(xyz, tet) of the block: spacing 1/nx, z fastest, six tets a cell."""
    nx, ny, nz = _dims(case)
    h = 1.0 / nx
    g = np.indices((nx + 1, ny + 1, nz + 1)).reshape(3, -1).T * h
    base = np.arange((nx + 1) * (ny + 1) * (nz + 1), dtype=np.uint32).reshape(nx + 1, ny + 1, nz + 1)[:nx, :ny, :nz]
    off = [(x * (ny + 1) + y) * (nz + 1) + z for x, y, z in _CORNER]
    six = np.array([[off[c] for c in t] for t in _SIX], np.uint32).reshape(-1)
    tet = base.reshape(-1, 1) + six
    return np.ascontiguousarray(g).reshape(-1), np.ascontiguousarray(tet).reshape(-1)


def _nodes(case):
    nx, ny, nz = _dims(case)
    return (nx + 1) * (ny + 1) * (nz + 1)


def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 16 + salt)


def _young(case, seed, lo=0.1, hi=10.0):
    """Per-tet modulus, log-uniform in [lo, hi]."""
    nx, ny, nz = _dims(case)
    u = torch.rand(6 * nx * ny * nz, dtype=torch.float64, device="cuda", generator=_gen(seed, 1))
    return torch.exp(math.log(lo) + u * math.log(hi / lo))


def _normal(n, seed, salt):
    return torch.randn(n, dtype=torch.float64, device="cuda", generator=_gen(seed, salt))


def _top(case, seed):
    """Prescribed values of the scalar problem: 0 on z = 0, uniform in [0.5, 1.5] on the top face."""
    nx, ny, nz = _dims(case)
    v = torch.zeros(nx + 1, ny + 1, nz + 1, dtype=torch.float64, device="cuda")
    v[:, :, nz] = 0.5 + torch.rand(nx + 1, ny + 1, dtype=torch.float64, device="cuda", generator=_gen(seed, 2))
    return v.reshape(-1)


def _motion(case, seed):
    """Displacement, velocity and a per-node rotation about z (up to 0.6 rad) of the warped solid."""
    n = _nodes(case)
    u, v = 0.01 * _normal(3 * n, seed, 3), 0.1 * _normal(3 * n, seed, 4)
    th = 0.6 * torch.rand(n, dtype=torch.float64, device="cuda", generator=_gen(seed, 5))
    R = torch.zeros(n, 3, 3, dtype=torch.float64, device="cuda")
    R[:, 0, 0], R[:, 0, 1], R[:, 1, 0], R[:, 1, 1], R[:, 2, 2] = th.cos(), -th.sin(), th.sin(), th.cos(), 1.0
    return u, v, R.reshape(-1)


def _arrays(case):
    xyz, tet = _mesh(case)
    n = xyz.size // 3
    ind, psup = D.JArray_PSuP_MeshElem(tet, 4, n)
    bc = np.repeat((xyz[2::3] == 0.0).astype(np.int32), 3)
    return dict(xyz=xyz, tet=tet, psup_ind=ind, psup=psup, bc=bc, young=np.ones(tet.size // 4), np=n,
                ntet=tet.size // 4)


def _system(a, ndim):
    K = D.CMatrixSparse()
    K.Initialize(a["np"], ndim, True)
    K.SetPattern(a["psup_ind"], a["psup"])
    ilu = D.CPreconditionerILU()
    ilu.SetPattern0(K)
    return K, ilu, D.TetMesh(K, a["xyz"], a["tet"])


def _zeros(n):
    return torch.zeros(n, dtype=torch.float64, device="cuda")


def prepare(case, seed):
    s = dict(case=case)
    path = case["path"]
    if path == "cloth":
        xyz0, _, tri, quad = DC.SetClothShape_Square(case["ndiv"], 1.0)
        c = s["cloth"] = DC.Cloth(xyz0, tri, quad)
        s["bc"] = torch.from_numpy(DC.pin_two_corners(case["ndiv"])).cuda()
        s["E"] = 500.0 + 1500.0 * torch.rand(c.ntri, dtype=torch.float64, device="cuda", generator=_gen(seed, 1))
        s["x"] = torch.from_numpy(xyz0).cuda()
        s["v"] = 0.05 * _normal(xyz0.size, seed, 2)
        s["v"] *= (s["bc"] == 0)
        return s
    a = _arrays(case)
    n3 = 3 * a["np"]
    if path in ("step", "solve", "precond", "setup", "gradient"):
        P = s["P"] = D.StaticElasticProblem(a, NU, RHO, GRAV)
        if case.get("fill", 0):
            P.ilu.Initialize_ILUk(P.K, case["fill"])
        s["E"] = _young(case, seed) if path != "gradient" else _young(case, seed, 0.5, 2.0)
    if path == "step":
        s["b"], s["x"], s["r"] = _zeros(n3), _zeros(n3), _zeros(n3)
    elif path in ("solve", "precond", "setup"):
        s["b"] = P.assemble(s["E"], _zeros(n3))
        if path == "solve":
            # the body force and a smooth traction-like load of random strength
            s["b"] *= 1.0 + 0.5 * math.sin(seed)
        else:
            s["b"] = _normal(n3, seed, 6)
        if path != "setup":
            assert P.factor()
        if case.get("precision") == "f32":
            s["b"] = s["b"].float()
        s["x"] = torch.zeros_like(s["b"])
        s["r"] = torch.zeros_like(s["b"])
    elif path == "assemble":
        s["K"], _, s["mesh"] = _system(a, 3)
        s["E"] = _young(case, seed)
        s["u"] = _normal(n3, seed, 6)
        s["bc"] = torch.from_numpy(a["bc"]).cuda()
        s["b"], s["y"] = _zeros(n3), _zeros(n3)
    elif path == "gradient":
        s["f"] = 1e-3 * _normal(n3, seed, 6)
        s["target"] = 1e-2 * _normal(n3, seed, 7)
    elif path == "poisson":
        s["K"], s["ilu"], s["mesh"] = _system(a, 1)
        z = a["xyz"][2::3]
        s["bc"] = torch.from_numpy(((z == 0.0) | (z > z.max() - 1e-9)).astype(np.int32)).cuda()
        s["val"] = _top(case, seed)
        s["b"], s["x"], s["r"] = _zeros(a["np"]), _zeros(a["np"]), _zeros(a["np"])
    elif path == "warp":
        s["K"], s["ilu"], s["mesh"] = _system(a, 3)
        s["bc"] = torch.from_numpy(a["bc"]).cuda()
        s["u"], s["v"], s["rot"] = _motion(case, seed)
        s["b"], s["x"], s["r"] = _zeros(n3), _zeros(n3), _zeros(n3)
    return s


# ---- one pass -------------------------------------------------------------------
def run(s):
    case = s["case"]
    path = case["path"]
    if path == "step":
        P = s["P"]
        P.assemble(s["E"], s["b"])
        P.factor()
        s["r"].copy_(s["b"])
        D.Solve_PCG(s["r"], s["x"], TOL, 20000, P.K, P.ilu)
        return [s["x"], s["b"]]
    if path == "solve":
        P = s["P"]
        if case["precision"] == "f64":
            s["r"].copy_(s["b"])
            D.Solve_PCG(s["r"], s["x"], TOL, 20000, P.K, P.ilu)
        else:
            D.Solve_PCG_Mixed(s["b"], s["x"], TOL, P.K, P.ilu, method="reliable")
        return s["x"]
    if path == "precond":
        s["x"].copy_(s["b"])
        s["P"].ilu.SolvePrecond(s["x"])
        return s["x"]
    if path == "setup":
        s["P"].factor()
        s["x"].copy_(s["b"])
        s["P"].ilu.SolvePrecond(s["x"])
        return s["x"]
    if path == "assemble":
        s["b"].zero_()
        s["K"].setZero()
        s["mesh"].assemble_linear(s["E"], NU, RHO, GRAV, s["b"], s["u"])
        s["K"].SetFixedBC(s["bc"])
        D.setRHS_Zero(s["b"], s["bc"])
        s["K"].MatVec(s["y"], 1.0, s["u"], 0.0)
        return [s["b"], s["y"]]
    if path == "gradient":
        E, f = s["E"].detach().requires_grad_(True), s["f"].detach().requires_grad_(True)
        u = linear_elastic_solve(E, f, s["P"], case["precision"], 0.2 * TOL)
        loss = 0.5 * torch.sum((u - s["target"]) ** 2)
        gE, gf = torch.autograd.grad(loss, (E, f))
        return [u.detach(), gE, gf]
    if path == "cloth":
        x, v = s["x"].clone(), s["v"].clone()
        s["cloth"].StepTime_InternalDynamicsILU(x, v, s["bc"], s["E"], CLOTH["nu"], CLOTH["bend"], CLOTH["g"],
                                                1.0 / s["cloth"].np, CLOTH["dt"], TOL, 1000)
        return [x, v]
    s["b"].zero_()
    s["K"].setZero()
    if path == "poisson":
        s["mesh"].assemble_poisson(1.0, 1.0, s["b"], s["val"])
    else:
        s["mesh"].assemble_beuler(WARP["myu"], WARP["lam"], WARP["rho"], WARP["g"], WARP["dt"], s["u"], s["v"],
                                  s["b"], s["rot"])
    s["K"].SetFixedBC(s["bc"])
    D.setRHS_Zero(s["b"], s["bc"])
    s["ilu"].CopyValue(s["K"])
    s["ilu"].Decompose()
    s["r"].copy_(s["b"])
    if path == "poisson":
        D.Solve_PCG(s["r"], s["x"], 0.1 * TOL, 20000, s["K"], s["ilu"])
    else:
        D.Solve_PBiCGStab(s["r"], s["x"], 0.1 * TOL, 20000, s["K"], s["ilu"])
    return [s["x"], s["b"]]


# ---- what a pass cannot do without ------------------------------------------------
def _iterations(case):
    """Krylov iterations of the path at this size, as it needs about that many."""
    if case["path"] == "cloth":
        return 40
    if case["path"] == "warp":
        return 10
    big = max(_dims(case))
    if case["path"] == "poisson":
        return 2.4 * big
    it = 60.0 * math.sqrt(big)
    return it * (0.6 if case.get("fill", 0) else 1.0)


def work(case):
    if case["path"] == "cloth":
        n = (case["ndiv"] + 1) ** 2
        nnz, B, tets = 12 * n, 3, 2 * case["ndiv"] ** 2
    else:
        n, B = _nodes(case), 1 if case["path"] == "poisson" else 3
        nnz, tets = 14 * n, 6 * case["nx"] * case["ny"] * case["nz"]
    path, f32 = case["path"], case.get("precision") in ("f32", "mixed")
    S = 4 if f32 else 8
    blocks = nnz + n
    fac = blocks * (2.4 if case.get("fill", 0) else 1.0)
    mat = B * B * 8 * blocks + 4 * (nnz + n)  # the FP64 matrix once
    assembly = mat + tets * (16 + 8) + 3 * 8 * n + 2 * 8 * B * n
    factor = mat + 2 * B * B * 8 * fac
    sweep = (B * B * S + 4) * fac + 4 * B * S * n
    spmv = (B * B * S + 4) * blocks + 2 * B * S * n
    it = _iterations(case) if path not in ("precond", "setup", "assemble") else 0
    per_it = sweep + spmv + 10 * B * S * n
    fl_sweep, fl_spmv = 2 * B * B * fac, 2 * B * B * blocks
    fl_asm, fl_fac = tets * 16 * B * B * 8, fac * 12 * 2 * B ** 3
    solves = dict(step=1, solve=1, gradient=2, cloth=1, poisson=1, warp=2).get(path, 0)
    b, f = solves * it * per_it, solves * it * (fl_sweep + fl_spmv + 10 * B * n)
    if path in ("step", "gradient", "cloth", "poisson", "warp", "assemble"):
        b, f = b + assembly, f + fl_asm
    if path in ("step", "gradient", "cloth", "poisson", "warp", "setup"):
        b, f = b + factor, f + fl_fac
    if path in ("precond", "setup"):
        b, f = b + sweep, f + fl_sweep
    if path == "assemble":
        b, f = b + spmv, f + fl_spmv
    return {"bytes": float(b), "flops": float(f)}


# ---- 64-bit restatement -------------------------------------------------------------
def _tet_gradients(case):
    """(6, 4, 3) shape-function gradients of the cell's tets and the tets' volume."""
    h = 1.0 / case["nx"]
    P = torch.tensor([[_CORNER[c] for c in t] for t in _SIX], dtype=torch.float64) * h
    J = torch.cat([torch.ones(6, 4, 1, dtype=torch.float64), P], 2)  # rows (1, p_k); its inverse's rows 1..3: dN
    return torch.linalg.inv(J)[:, 1:, :].transpose(1, 2).contiguous().cuda(), h ** 3 / 6.0


def _element_matrices(case, scalar, lam, myu):
    """(6, 4, 4, B, B) element matrices of the cell's tets."""
    G, vol = _tet_gradients(case)
    dot = torch.einsum("sad,sbd->sab", G, G)
    if scalar:
        return (vol * dot)[..., None, None]
    eye = torch.eye(3, dtype=torch.float64, device="cuda")
    return vol * (lam * torch.einsum("sar,sbc->sabrc", G, G) + myu * torch.einsum("sbr,sac->sabrc", G, G)
                  + myu * dot[..., None, None] * eye)


def _lame():
    return NU / ((1 + NU) * (1 - 2 * NU)), 1.0 / (2 * (1 + NU))


_LOWER = [tuple(-c for c in o) for o in sorted(itertools.product((0, 1), repeat=3), reverse=True) if any(o)]
_OFFSETS = [(0, 0, 0)] + _LOWER + [tuple(-c for c in o) for o in reversed(_LOWER)]


class _Stencil:
    """Block matrix on the block's nodes: 15 blocks a node, kept on a grid padded by one node all round."""

    def __init__(self, case, ke, scale=None):
        self.N = tuple(d + 1 for d in _dims(case))
        self.B = B = ke.shape[-1]
        self.at = {o: k for k, o in enumerate(_OFFSETS)}
        self.A = torch.zeros((15,) + tuple(n + 2 for n in self.N) + (B, B), dtype=torch.float64, device="cuda")
        cells = _dims(case)
        w = None if scale is None else scale.reshape(cells + (6,))
        for s, t in enumerate(_SIX):
            for a, b in itertools.product(range(4), range(4)):
                ca, cb = _CORNER[t[a]], _CORNER[t[b]]
                o = self.at[tuple(y - x for x, y in zip(ca, cb))]
                to = self.A[(o,) + tuple(slice(1 + c, 1 + c + n) for c, n in zip(ca, cells))]
                to += ke[s, a, b] if w is None else w[..., s, None, None] * ke[s, a, b]

    def inner(self, k):
        return self.A[(k,) + tuple(slice(1, 1 + n) for n in self.N)]

    def shifted(self, x):
        """x at each node's 15 neighbours (zero outside), one after another."""
        p = torch.zeros(tuple(n + 2 for n in self.N) + x.shape[3:], dtype=x.dtype, device=x.device)
        p[1:-1, 1:-1, 1:-1] = x
        for k, o in enumerate(_OFFSETS):
            yield k, p[tuple(slice(1 + d, 1 + d + n) for d, n in zip(o, self.N))]

    def matvec(self, x):
        x = x.reshape(self.N + (self.B,))
        y = torch.zeros_like(x)
        for k, xs in self.shifted(x):
            y += (self.inner(k) * xs.unsqueeze(-2)).sum(-1)
        return y.reshape(-1)

    def clamp(self, free):
        """Rows and columns of the fixed DOFs become the identity's."""
        m = free.reshape(self.N + (self.B,))
        for k, ms in self.shifted(m):
            self.inner(k).mul_(m.unsqueeze(-1)).mul_(ms.unsqueeze(-2))
        d = torch.diagonal(self.inner(0), dim1=-2, dim2=-1)
        d += 1.0 - m

    def jacobi(self):
        inv = torch.linalg.inv(self.inner(0).reshape(-1, self.B, self.B))
        return lambda r: torch.bmm(inv, r.reshape(-1, self.B, 1)).reshape(-1)

    def solve(self, b, passes=3):
        """Conjugate gradients to working accuracy, refined on the true residual."""
        M, x = self.jacobi(), torch.zeros_like(b)
        for _ in range(passes):
            r = b - self.matvec(x)
            stop = 1e-9 * float(r.norm())
            if float(r.norm()) <= 1e-15 * float(b.norm()):
                break
            d, z = torch.zeros_like(b), M(r)
            p, rz = z.clone(), torch.dot(r, z)
            for it in range(40000):
                Ap = self.matvec(p)
                alpha = rz / torch.dot(p, Ap)
                d += alpha * p
                r -= alpha * Ap
                if it % 25 == 24 and float(r.norm()) < stop:
                    break
                z = M(r)
                rz, old = torch.dot(r, z), rz
                p = z + (rz / old) * p
            x += d
        return x

    def solve_general(self, b, passes=4):
        """BiCGStab (the matrix need not be symmetric), refined on the true residual."""
        M, x = self.jacobi(), torch.zeros_like(b)
        for _ in range(passes):
            r = b - self.matvec(x)
            if float(r.norm()) <= 1e-15 * float(b.norm()):
                break
            d, r0, stop = torch.zeros_like(b), r.clone(), 1e-6 * float(r.norm())
            p = r.clone()
            for _ in range(2000):
                ph = M(p)
                v = self.matvec(ph)
                rr = torch.dot(r0, r)
                alpha = rr / torch.dot(r0, v)
                s = r - alpha * v
                sh = M(s)
                t = self.matvec(sh)
                om = torch.dot(t, s) / torch.dot(t, t)
                d += alpha * ph + om * sh
                r = s - om * t
                if float(r.norm()) < stop:
                    break
                p = r + (torch.dot(r0, r) / rr) * (alpha / om) * (p - om * v)
            x += d
        return x

    def ilu0_solve(self, v):
        """(LU)^-1 v of the incomplete factorisation on the stencil's own pattern, by levels x + y + z."""
        B, dims = self.B, tuple(n + 2 for n in self.N)
        A = self.A.reshape(15, -1, B, B)
        flat = torch.arange(A.shape[1], device="cuda").reshape(dims)[1:-1, 1:-1, 1:-1]
        g = torch.meshgrid(*(torch.arange(n, device="cuda") for n in self.N), indexing="ij")
        level = (g[0] + g[1] + g[2]).reshape(-1)
        order = torch.argsort(level, stable=True)
        counts = torch.bincount(level).tolist()
        rows = torch.split(flat.reshape(-1)[order], counts)
        lin = {o: (o[0] * dims[1] + o[1]) * dims[2] + o[2] for o in _OFFSETS}
        upper = [o for o in _OFFSETS if o != (0, 0, 0) and o not in _LOWER]
        Dinv = torch.zeros_like(A[0])
        z = torch.zeros(A.shape[1], B, 1, dtype=torch.float64, device="cuda")
        rhs = torch.zeros_like(z)
        rhs[flat.reshape(-1)] = v.double().reshape(-1, B, 1)
        for I in rows:
            for k in _LOWER:
                L = A[self.at[k]][I]
                for u in upper:
                    t = tuple(p + q for p, q in zip(k, u))
                    if t in self.at:
                        A[self.at[t]][I] -= torch.bmm(L, A[self.at[u]][I + lin[k]])
            Dinv[I] = torch.linalg.inv(A[0][I])
            for u in upper:
                A[self.at[u]][I] = torch.bmm(Dinv[I], A[self.at[u]][I])
            acc = rhs[I]
            for k in _LOWER:
                acc = acc - torch.bmm(A[self.at[k]][I], z[I + lin[k]])
            z[I] = torch.bmm(Dinv[I], acc)
        for I in reversed(rows):
            acc = z[I]
            for u in upper:
                acc = acc - torch.bmm(A[self.at[u]][I], z[I + lin[u]])
            z[I] = acc
        return z[flat.reshape(-1)].reshape(-1)


def _free(case, B, top=False):
    N = tuple(d + 1 for d in _dims(case))
    m = torch.ones(N + (B,), dtype=torch.float64, device="cuda")
    m[:, :, 0] = 0.0
    if top:
        m[:, :, -1] = 0.0
    return m.reshape(-1)


def _node_volume(case):
    """Volume share of each node: a quarter of every tet it belongs to."""
    cells = _dims(case)
    out = torch.zeros(tuple(d + 1 for d in cells), dtype=torch.float64, device="cuda")
    q = (1.0 / case["nx"]) ** 3 / 24.0
    for t in _SIX:
        for c in t:
            out[tuple(slice(d, d + n) for d, n in zip(_CORNER[c], cells))] += q
    return out.reshape(-1)


def _body_force(case, rho, g):
    return (rho * _node_volume(case)[:, None] * torch.tensor(g, dtype=torch.float64, device="cuda")).reshape(-1)


def exact(case, seed):
    path = case["path"]
    if path == "cloth":
        return None
    if path == "poisson":
        free, val = _free(case, 1, True), _top(case, seed)
        S = _Stencil(case, _element_matrices(case, True, 0, 0))
        b = (_node_volume(case) - S.matvec(val)) * free
        S.clamp(free)
        return [S.solve(b), b]
    free = _free(case, 3)
    if path == "warp":
        w = WARP
        S = _Stencil(case, _element_matrices(case, False, w["lam"], w["myu"]))
        u, v, R = _motion(case, seed)
        R = R.reshape(S.N + (3, 3))
        P = torch.from_numpy(_mesh(case)[0]).cuda()
        KP = S.matvec(P).reshape(S.N + (3, 1))
        Rt = R.transpose(-1, -2)
        for k in range(15):
            S.inner(k).copy_(R @ S.inner(k) @ Rt)
        elastic = S.matvec(P + u + w["dt"] * v) - (R @ KP).reshape(-1)
        b = (_body_force(case, w["rho"], w["g"]) - elastic) / w["dt"] * free
        mass = (w["rho"] * _node_volume(case) / w["dt"] ** 2).reshape(S.N + (1,))
        d = torch.diagonal(S.inner(0), dim1=-2, dim2=-1)
        d += mass
        S.clamp(free)
        return [S.solve_general(b), b]
    lo, hi = (0.5, 2.0) if path == "gradient" else (0.1, 10.0)
    E = _young(case, seed, lo, hi)
    ke = _element_matrices(case, False, *_lame())
    S = _Stencil(case, ke, E)
    if path == "assemble":
        u = _normal(3 * _nodes(case), seed, 6)
        b = (_body_force(case, RHO, GRAV) - S.matvec(u)) * free
        S.clamp(free)
        return [b, S.matvec(u)]
    S.clamp(free)
    if path in ("precond", "setup"):
        if case.get("fill", 0):
            return None
        v = _normal(3 * _nodes(case), seed, 6)
        return S.ilu0_solve(v.float() if case.get("precision") == "f32" else v)
    if path == "gradient":
        f = 1e-3 * _normal(3 * _nodes(case), seed, 6)
        u = S.solve(f * free)
        lam = S.solve(u - 1e-2 * _normal(3 * _nodes(case), seed, 7)) * free
        cells = _dims(case)
        gE = torch.zeros(cells + (6,), dtype=torch.float64, device="cuda")
        for s, t in enumerate(_SIX):
            at = [tuple(slice(d, d + n) for d, n in zip(_CORNER[c], cells)) for c in t]
            ue = [u.reshape(S.N + (3,))[k] for k in at]
            le = [lam.reshape(S.N + (3,))[k] for k in at]
            for a, c in itertools.product(range(4), range(4)):
                gE[..., s] -= (le[a] * (ue[c] @ ke[s, a, c].T)).sum(-1)
        return [u, gE.reshape(-1), lam]
    b = _body_force(case, RHO, GRAV) * free
    if path == "solve":
        return S.solve(b * (1.0 + 0.5 * math.sin(seed)))
    return [S.solve(b), b]

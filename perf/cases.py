"""Performance cases of the MPM step: what a program that uses this package has it do.

A `rollout` case is the step in use: the caller holds a particle (and cloth) state in
its own device arrays in the C-ABI's FP64 layouts, uploads it, runs `steps` time steps
and reads the whole state back.  `solve` is the same with the adaptive loop
(HybridSolver::solve) in the place of the steps, `train` and `forward` are the learned
return map's two own calls.  Everything goes through the C-ABI of include/aep.h (capi),
whose pointers may be device memory.

Inputs come from a seed alone: particles in a box at about eight per cell that touches
the ground, a smooth velocity field with noise, rotated and strained deformation
gradients (about +-1%, both sides of the yield surfaces), all of them FP32 numbers, so
that the FP64 evaluation in `exact` starts from the same state.  `exact` is the step in
plain torch, written from its equations.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from anisotropicelastoplasticity_gb300 import LagrangianMesh, LevelSet, RegularGrid, capi, make_params
from anisotropicelastoplasticity_gb300.learned import ReturnMapMLP

SNOW, SAND = capi.AEP_SNOW, capi.AEP_SAND
GROUND = 0.05
SNOW_DENSITY, SAND_DENSITY = 400.0, 2200.0


# ---------------------------------------------------------------------------------------
# the cases

def _rollout(name, n, res, *, material="sand", steps=8, dt=5e-5, cloth=0, learned=False, track_fp=False,
             walls=False, coulomb=False, friction=0.5, rz=0):
    """rz: the resolution along z where it differs (0: cubic); cloth: vertices per side
    of a square sheet over the particles (0: none)."""
    return {"name": name, "kind": "rollout", "n": n, "res": res, "rz": rz or res, "material": material,
            "steps": steps, "dt": dt, "cloth": cloth, "learned": learned, "track_fp": track_fp, "walls": walls,
            "coulomb": coulomb, "friction": friction}


def listed():
    return [
        # the smallest scene in use (the golden fixtures' size): launches and latency only
        _rollout("snow 512", 512, 32, material="snow", steps=16, dt=1e-4, friction=0.2),
        # the snow block drop at its stated size
        _rollout("snow block 32k", 32768, 64, material="snow", steps=16, dt=1e-4, friction=0.2),
        # an odd count on a grid that is no cube, full plastic gradient, walls and a sphere, Coulomb friction
        _rollout("mixed 100k F_P", 100003, 75, rz=61, material="mixed", track_fp=True, walls=True, coulomb=True),
        # coupled to another solver: the state is exchanged around every single step
        _rollout("exchange 262k", 262144, 128, material="mixed", steps=1),
        # the sand column at its stated size
        _rollout("sand column 524k", 524288, 128),
        # the snow + sand collision at its stated size
        _rollout("collision 2M", 2097152, 256, material="mixed"),
        # the cloth drape at its stated size: a sheet without particles
        _rollout("cloth drape 196k", 0, 128, cloth=256, dt=2e-5),
        # sand and cloth with the learned return map, the quarter-resolution scene
        _rollout("sand cloth learned 1.1M", 950000, 256, cloth=256, dt=2e-5, learned=True),
        # sand and cloth at its stated size, the largest
        _rollout("sand cloth 8.4M", 7604222, 512, cloth=512, dt=2e-5, steps=4),
        # the adaptive loop: volumes, then steps whose time step follows the velocities (slow
        # enough here that the loop's own floor decides, not a single nearly massless node)
        {"name": "solve 131k", "kind": "solve", "n": 131072, "res": 64, "rz": 64, "material": "mixed", "steps": 24,
         "cfl": 0.024, "friction": 0.2},
        # training of the learned map: Adam steps over the batch size of the benchmark
        {"name": "train 16k", "kind": "train", "n": 262144, "batch": 16384, "steps": 32},
        # batched inference over harvested records
        {"name": "forward 1M", "kind": "forward", "n": 1000003},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["rollout", "solve", "train", "forward"], [8, 1, 1, 1])[0]
    if kind == "train":
        return {"kind": kind, "n": _log_int(rng, 20000, 1000000), "batch": _log_int(rng, 1000, 32768),
                "steps": rng.randint(8, 32)}
    if kind == "forward":
        return {"kind": kind, "n": _log_int(rng, 100, 2000000)}
    n = _log_int(rng, 512, 2200000)
    side_cells = (n / 8.0) ** (1.0 / 3.0)
    res = max(20, math.ceil(side_cells / rng.uniform(0.3, 0.55)))
    rz = max(res, res + rng.randint(-2, 9))
    material = rng.choice(["snow", "sand", "mixed"])
    if kind == "solve":
        n = min(n, 200000)
        res = rz = min(64, max(20, math.ceil((n / 8.0) ** (1.0 / 3.0) / 0.5)))
        return {"kind": kind, "n": n, "res": res, "rz": rz, "material": material, "steps": rng.randint(8, 32),
                "cfl": 300.0 * min(1e-4, 0.0075 / max(res, rz)), "friction": rng.uniform(0.1, 0.6)}
    cloth = rng.choice([0, 0, _log_int(rng, 9, 300)])
    dt = rng.uniform(0.6, 1.0) * min(1e-4 if not cloth else 2e-5, 0.0125 / max(res, rz))
    return {"kind": kind, "n": n, "res": res, "rz": rz, "material": material,
            "steps": rng.choice([1, 3, 4, 8, 8, 13]), "dt": dt, "cloth": cloth,
            "learned": rng.random() < 0.25, "track_fp": rng.random() < 0.25, "walls": rng.random() < 0.4,
            "coulomb": rng.random() < 0.4, "friction": rng.uniform(0.1, 0.6)}


def _cloth_items(case):
    k = case.get("cloth", 0)
    return (k * k, 2 * (k - 1) * (k - 1)) if k else (0, 0)


def work(case):
    if case["kind"] == "forward":
        return {"bytes": case["n"] * (32 + 12), "flops": case["n"] * 2 * (7 * 64 + 2 * 64 * 64 + 64 * 3)}
    if case["kind"] == "train":
        rows = case["steps"] * case["batch"]
        return {"bytes": rows * 32, "flops": rows * 6 * (7 * 64 + 2 * 64 * 64 + 64 * 3)}
    nv, nf = _cloth_items(case)
    items = case["n"] + nv + nf
    fp = 9 if case.get("track_fp") else 0
    # one step: x, v, B, F, plastic scalar (25 numbers) read and written, m and the volume
    # read, in FP32; the exchange: those numbers in and out in FP64, the outputs in FP32
    step = items * 4 * (2 * (25 + fp) + 2)
    exchange = items * (27 + fp) * (8 + 8 + 4)
    # per item and step: two scatters and two gathers over 64 nodes, the 3x3 algebra
    return {"bytes": case["steps"] * step + exchange, "flops": case["steps"] * items * 5000}


# ---------------------------------------------------------------------------------------
# inputs

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _f32(t):
    """Rounded to FP32 values, in FP64."""
    return t.to(torch.float32).to(torch.float64)


def _rotations(rn, n, size):
    """Rotation matrices (n, 3, 3) about random axes (Rodrigues)."""
    w = size * rn(n, 3)
    th = w.norm(dim=1).clamp_min(1e-12)
    k = w / th[:, None]
    K = torch.zeros(n, 3, 3, dtype=torch.float64, device=w.device)
    K[:, 0, 1], K[:, 0, 2], K[:, 1, 2] = -k[:, 2], k[:, 1], -k[:, 0]
    K[:, 1, 0], K[:, 2, 0], K[:, 2, 1] = k[:, 2], -k[:, 1], k[:, 0]
    eye = torch.eye(3, dtype=torch.float64, device=w.device)
    return eye + torch.sin(th)[:, None, None] * K + (1 - torch.cos(th))[:, None, None] * (K @ K)


def _smooth_velocity(x):
    """A velocity field that varies over a fraction of the domain."""
    X, Y, Z = (x[:, a] for a in range(3))
    return torch.stack([0.4 * torch.sin(9 * Y) - 1.5 * (Z - 0.25), 0.3 * torch.cos(11 * X + 2 * Z),
                        -0.6 + 0.4 * torch.sin(8 * X) * torch.cos(7 * Y)], dim=1)


def _box_particles(case, h, gen, dev):
    n = case["n"]
    rn = lambda *s: torch.randn(*s, generator=gen, dtype=torch.float64, device=dev)  # noqa: E731
    side = [(n / 8.0) ** (1.0 / 3.0) * v for v in h]  # eight particles per cell
    lo = [0.5 - side[0] / 2, 0.5 - side[1] / 2, GROUND + 0.6 * h[2]]
    u = torch.rand(n, 3, generator=gen, dtype=torch.float64, device=dev)
    x = torch.stack([lo[a] + side[a] * u[:, a] for a in range(3)], dim=1)
    if case["material"] == "mixed":  # two blocks face to face along x, in the caller's order
        mat = torch.where(u[:, 0] < 0.5, SNOW, SAND).to(torch.uint8)
    else:
        mat = torch.full((n,), SNOW if case["material"] == "snow" else SAND, dtype=torch.uint8, device=dev)
    snow = mat == SNOW
    vol = side[0] * side[1] * side[2] / n
    v = _smooth_velocity(x) + 0.1 * rn(n, 3)
    if case["material"] == "mixed":
        v[:, 0] += torch.where(snow, 0.8, -0.8)
    strain = torch.where(snow, 0.006, 0.01)[:, None, None].to(torch.float64) * rn(n, 3, 3)
    eye = torch.eye(3, dtype=torch.float64, device=dev)
    F = _rotations(rn, n, 0.2) @ (eye + strain)
    plastic = torch.where(snow, 1 + 0.01 * rn(n).clamp(-3, 3), 0.02 * torch.rand(n, generator=gen,
                                                                                 dtype=torch.float64, device=dev))
    out = {"x": x, "v": v, "B": 0.02 * min(h) * rn(n, 3, 3), "F": F,
           "m": vol * torch.where(snow, SNOW_DENSITY, SAND_DENSITY).to(torch.float64),
           "vol": torch.full((n,), vol, dtype=torch.float64, device=dev), "q": plastic}
    if case.get("track_fp"):
        out["Fp"] = eye + 0.01 * rn(n, 3, 3)
    out = {k: _f32(t) for k, t in out.items()}
    out["mat"] = mat
    return out


def _sheet(case, h, gen, dev):
    """A square sheet above the particles (or in the middle of an empty domain): rest
    state flat, current state stretched and sheared a little, moving."""
    k = case["cloth"]
    n = case["n"]
    height = GROUND + h[2] * (0.6 + (n / 8.0) ** (1.0 / 3.0) + 0.3) if n else 0.6
    t = torch.linspace(-0.3, 0.3, k, dtype=torch.float64, device=dev)
    X, Y = torch.meshgrid(0.5 + t, 0.5 + t, indexing="ij")
    rest = torch.stack([X.reshape(-1), Y.reshape(-1), torch.full((k * k,), height, dtype=torch.float64, device=dev)], 1)
    i = torch.arange(k * k, device=dev).reshape(k, k)
    a, b, c, d = i[:-1, :-1].reshape(-1), i[1:, :-1].reshape(-1), i[1:, 1:].reshape(-1), i[:-1, 1:].reshape(-1)
    faces = torch.cat([torch.stack([a, b, c], 1), torch.stack([a, c, d], 1)])
    rn = lambda *s: torch.randn(*s, generator=gen, dtype=torch.float64, device=dev)  # noqa: E731
    edge = 0.6 / (k - 1)
    xv = _f32(rest + 0.01 * edge * rn(k * k, 3) + 0.1 * h[2] * torch.sin(20 * rest[:, :1]) * torch.tensor(
        [0.0, 0.0, 1.0], dtype=torch.float64, device=dev))
    nf = len(faces)
    p0, p1, p2 = xv[faces[:, 0]], xv[faces[:, 1]], xv[faces[:, 2]]
    nrm = torch.linalg.cross(p1 - p0, p2 - p0)
    nrm = nrm / nrm.norm(dim=1, keepdim=True)
    d3 = nrm * (1 + 0.02 * rn(nf, 1)) + 0.01 * rn(nf, 3)
    return {"rest": rest, "faces": faces, "xv": xv, "vv": _f32(_smooth_velocity(xv) + 0.05 * rn(k * k, 3)),
            "Bv": _f32(0.01 * min(h) * rn(k * k, 3, 3)), "xe": _f32((p0 + p1 + p2) / 3),
            "ve": _f32(_smooth_velocity((p0 + p1 + p2) / 3)), "Be": _f32(0.01 * min(h) * rn(nf, 3, 3)),
            "D": _f32(torch.stack([p1 - p0, p2 - p0, d3], dim=2))}


CLOTH = dict(youngs_modulus=1e4, poisson_ratio=0.3, shear_stiffness=1e3, stiffness=1e3, friction_coeff=0.3)


def _grid(case):
    """The unit square times a height that makes the cells cubes where rz differs."""
    res = [case["res"], case["res"], case["rz"]]
    return RegularGrid([0, 0, 0], [1, 1, case["rz"] / case["res"]], res)


def _inputs(case, seed):
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(1000003 * seed + 17)
    h = [float(v) for v in _grid(case).h]
    s = {"parts": _box_particles(case, h, gen, dev) if case["n"] else None}
    s["mesh"] = _sheet(case, h, gen, dev) if case.get("cloth") else None
    return s


def _level_set(case):
    ls = LevelSet.ground(GROUND)
    if case.get("walls"):
        ls = ls | LevelSet.wall2ground(0.9, 0.88, 0.03) | LevelSet.sphere([0.45, 0.55, 0.02], 0.07)
    return ls


def _params(case):
    return make_params(friction=case["friction"], track_plastic_F=int(case.get("track_fp", False)),
                       friction_bug=int(not case.get("coulomb", False)), cloth_volume_weighting=1)


def _weights(gen):
    """He-normal parameters of the 7 -> 64 -> 64 -> 64 -> 3 network in the packed layout
    (W^T blocks of 64x16, 64x64, 64x64, 8x64, then the biases), bfloat16 values."""
    rn = lambda *s: torch.randn(*s, generator=gen, dtype=torch.float32)  # noqa: E731
    w1 = torch.zeros(64, 16)
    w1[:, :7] = rn(64, 7) * math.sqrt(2 / 7)
    w4 = torch.zeros(8, 64)
    w4[:3] = 0.3 * rn(3, 64) * math.sqrt(2 / 64)
    w = [w1, rn(64, 64) * math.sqrt(2 / 64), rn(64, 64) * math.sqrt(2 / 64), w4]
    b = [0.05 * rn(200 - 8), torch.zeros(8)]
    return torch.cat([t.to(torch.bfloat16).float().reshape(-1) for t in w] + [t.reshape(-1) for t in b])


def _records(n, gen, dev):
    """Plastic states and their exact projections, as the step harvests them: snow clamps
    and sand cone projections of log singular values of about 1e-4 to 3e-2."""
    prm = capi.default_params()
    u = lambda *s: torch.rand(*s, generator=gen, dtype=torch.float64, device=dev)  # noqa: E731
    rn = lambda *s: torch.randn(*s, generator=gen, dtype=torch.float64, device=dev)  # noqa: E731
    sand = u(n) < 0.6
    ln = torch.where(sand[:, None], torch.exp(math.log(3e-4) + u(n, 1) * math.log(100.0)) * rn(n, 3), 0.03 * rn(n, 3))
    tr = ln.sum(1, keepdim=True)
    ln = torch.where((sand[:, None]) & (tr > 0), -ln, ln)  # sand in compression: the cone, not its apex
    ln = _f32(torch.sort(ln, dim=1, descending=True).values)
    q = _f32(torch.where(sand, 0.05 * u(n), torch.zeros_like(u(n))))
    cone, _ = _drucker_prager(ln, q, prm)
    lo, hi = math.log(1 - prm.snow.theta_c), math.log(1 + prm.snow.theta_s)
    new = torch.where(sand[:, None], cone, ln.clamp(lo, hi))
    rec = torch.cat([ln, q[:, None], torch.where(sand, SAND, SNOW)[:, None].double(), new - ln], dim=1)
    return rec.float().contiguous()


# ---------------------------------------------------------------------------------------
# the state a program keeps, and one pass

def _ptr(t, kind=C.c_double):
    return C.cast(C.c_void_p(t.data_ptr()), C.POINTER(kind)) if t is not None else None


def _rows(B):
    """(N, 3, 3) affine momenta in the C-ABI's layout (row, component, item)."""
    return B.permute(1, 2, 0).contiguous()


class _Solver:
    """A C-ABI handle, the caller's device arrays of its state, and where it reads back."""

    def __init__(self, case, seed):
        self.case = case
        self.lib = capi.load()
        self.h = C.c_void_p()
        self.stream = torch.cuda.Stream()
        grid = _grid(case)
        prm = _params(case)
        self._ok(self.lib.aep_solver_create(C.byref(grid.desc()), C.byref(prm), C.byref(self.h)))
        self._ok(self.lib.aep_set_stream(self.h, C.c_void_p(self.stream.cuda_stream)))
        shapes, count = _level_set(case).to_c()
        self._ok(self.lib.aep_set_levelset(self.h, shapes, count))
        s = _inputs(case, seed)
        p, m = s["parts"], s["mesh"]
        self.n = case["n"]
        self.fp = bool(case.get("track_fp"))
        if p is not None:
            self.part = [p["x"].T.contiguous(), p["v"].T.contiguous(), _rows(p["B"]),
                         p["F"].transpose(1, 2).contiguous(), p["Fp"].transpose(1, 2).contiguous() if self.fp else None,
                         p["m"], p["vol"], p["q"]]
            self.mat = p["mat"]
            sizes = [3, 3, 9, 9, 9 if self.fp else 0, 1, 1]
            self.out = torch.empty(sum(sizes) * self.n, dtype=torch.float64, device="cuda")
            self.fields = self._split(self.out, [k * self.n for k in sizes])
        self.nv, self.nf = _cloth_items(case)
        if m is not None:
            h = 1.0 / case["res"]
            mesh = LagrangianMesh.from_triangles(m["rest"].cpu().numpy(), m["faces"].cpu().numpy(), density=0.2 / h,
                                                 thickness=h, **CLOTH)
            self.mesh_args = m
            self.mesh_in = [m["xv"].T.contiguous(), m["vv"].T.contiguous(), _rows(m["Bv"]), m["xe"].T.contiguous(),
                            m["ve"].T.contiguous(), _rows(m["Be"]), m["D"].permute(2, 1, 0).contiguous()]
            sizes = [3 * self.nv, 3 * self.nv, 9 * self.nv, 3 * self.nf, 3 * self.nf, 9 * self.nf, 9 * self.nf]
            self.mesh_out = torch.empty(sum(sizes), dtype=torch.float64, device="cuda")
            self.mesh_fields = self._split(self.mesh_out, sizes)
        torch.cuda.synchronize()
        self._upload_particles()
        if m is not None:
            self._attach(mesh)
        self.mlp = None
        if case.get("learned"):
            gen = torch.Generator(device="cuda")
            gen.manual_seed(5 * seed + 3)
            cpu = torch.Generator()
            cpu.manual_seed(5 * seed + 4)
            rec = _records(400000, gen, "cuda")
            torch.cuda.synchronize()
            self.mlp = ReturnMapMLP(seed=0)
            self.mlp.set_params(_weights(cpu).numpy())
            self.mlp.train(rec.data_ptr(), len(rec), steps=2000, batch=16384, lr=1e-3, lr_final=1e-5)
            # the residual bound that the learned map's configuration states
            self._ok(self.lib.aep_set_return_map(self.h, self.mlp.handle, 0.0))
            self._ok(self.lib.aep_set_return_map_bounds(self.h, 0.0, 1e-4))

    @staticmethod
    def _split(flat, sizes):
        return [flat[sum(sizes[:i]):sum(sizes[:i + 1])] if k else None for i, k in enumerate(sizes)]

    def _ok(self, status):
        if status != capi.AEP_OK:
            raise capi.AepError(status, self.lib.aep_last_error(self.h).decode() if self.h else "")

    def _attach(self, mesh):
        d = lambda a: np.ascontiguousarray(a, np.float64)  # noqa: E731
        p = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
        xv, faces = d(mesh.vertex_positions.T), np.ascontiguousarray(mesh.faces.T, np.int32)
        mv, vv, me, ve = (d(a) for a in (mesh.vertex_masses, mesh.vertex_volumes, mesh.element_masses,
                                         mesh.element_volumes))
        dirs = d(mesh.element_directions.transpose(2, 1, 0))
        self._ok(self.lib.aep_set_mesh(self.h, self.nv, self.nf, p(xv), faces.ctypes.data_as(C.POINTER(C.c_int32)), None,
                                       None, p(mv), p(vv), p(me), p(ve), p(dirs), p(dirs), mesh.mu, mesh.lambda_,
                                       mesh.shear_stiffness, mesh.stiffness, mesh.friction_coeff))

    def _upload_particles(self):
        if self.n:
            self._ok(self.lib.aep_set_particles(self.h, self.n, *(_ptr(t) for t in self.part),
                                                _ptr(self.mat, C.c_uint8)))

    def upload(self):
        self._upload_particles()
        if self.nf:
            self._ok(self.lib.aep_set_mesh_state(self.h, self.nv, self.nf, *(_ptr(t) for t in self.mesh_in)))

    def step(self, dt):
        self._ok(self.lib.aep_step(self.h, dt))

    def solve(self, cfl, max_steps):
        self._ok(self.lib.aep_set_max_steps(self.h, max_steps))
        self._ok(self.lib.aep_solve(self.h, cfl, 1e9, 0.0))

    def read(self):
        out = {}
        with torch.cuda.stream(self.stream):
            if self.n:
                self._ok(self.lib.aep_get_particles(self.h, self.n, *(_ptr(t) for t in self.fields)))
                f = self._split(self.out.float(), [0 if t is None else t.numel() for t in self.fields])
                out = {k: t for k, t in zip(("x", "v", "B", "F", "Fp", "vol", "q"), f) if t is not None}
            if self.nf:
                self._ok(self.lib.aep_get_mesh(self.h, *(_ptr(t) for t in self.mesh_fields)))
                f = self._split(self.mesh_out.float(), [t.numel() for t in self.mesh_fields])
                out.update(zip(("xv", "vv", "Bv", "xe", "ve", "Be", "D"), f))
        return out

    def __del__(self):
        if getattr(self, "h", None):
            self.lib.aep_solver_destroy(self.h)
            self.h = None


def prepare(case, seed):
    if case["kind"] in ("rollout", "solve"):
        return _Solver(case, seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1000003 * seed + 29)
    cpu = torch.Generator()
    cpu.manual_seed(1000003 * seed + 31)
    rec = _records(case["n"], gen, "cuda")
    mlp = ReturnMapMLP(seed=0)
    mlp.set_params(_weights(cpu).numpy())
    out = torch.empty(case["n"], 3, device="cuda") if case["kind"] == "forward" else None
    torch.cuda.synchronize()
    return {"case": case, "mlp": mlp, "rec": rec, "out": out}


def run(state):
    if isinstance(state, _Solver):
        case = state.case
        state.upload()
        if case["kind"] == "solve":
            state.solve(case["cfl"], case["steps"])
        else:
            for _ in range(case["steps"]):
                state.step(case["dt"])
        return state.read()
    case, mlp, rec = state["case"], state["mlp"], state["rec"]
    if case["kind"] == "forward":
        mlp.forward(rec.data_ptr(), len(rec), state["out"].data_ptr())
        return state["out"]
    mlp.train(rec.data_ptr(), len(rec), steps=case["steps"], batch=case["batch"], lr=1e-3, lr_final=5e-4)
    return mlp.get_params()


# ---------------------------------------------------------------------------------------
# the same in 64 bits

MOST_ITEM_STEPS = 20_000_000  # about 20 seconds


def _eig3(S):
    """Eigenvalues (N, 3) and eigenvectors (N, 3, 3) of symmetric S, cyclic Jacobi."""
    a = {(i, j): S[:, i, j].clone() for i in range(3) for j in range(i, 3)}
    V = torch.eye(3, dtype=S.dtype, device=S.device).repeat(len(S), 1, 1)
    for _ in range(7):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            r = 3 - p - q
            g = a[p, q]
            tiny = g.abs() < 1e-300
            z = (a[q, q] - a[p, p]) / (2 * torch.where(tiny, torch.ones_like(g), g))
            t = torch.where(z >= 0, 1.0, -1.0) / (z.abs() + torch.sqrt(1 + z * z))
            t = torch.where(tiny, torch.zeros_like(t), t)
            c = torch.rsqrt(1 + t * t)
            s = c * t
            a[p, p], a[q, q] = a[p, p] - t * g, a[q, q] + t * g
            kp, kq = tuple(sorted((p, r))), tuple(sorted((q, r)))
            a[kp], a[kq] = c * a[kp] - s * a[kq], s * a[kp] + c * a[kq]
            a[p, q] = torch.zeros_like(g)
            vp, vq = V[:, :, p].clone(), V[:, :, q].clone()
            V[:, :, p], V[:, :, q] = c[:, None] * vp - s[:, None] * vq, s[:, None] * vp + c[:, None] * vq
    return torch.stack([a[i, i] for i in range(3)], 1), V


def _stretch(F):
    """F = U diag(s) V^T: (ln s, V) from the eigen-decomposition of F^T F - I."""
    E = F.transpose(1, 2) @ F - torch.eye(3, dtype=F.dtype, device=F.device)
    lam, V = _eig3(E)
    return 0.5 * torch.log1p(lam), V


def _with(F, V, f):
    """F V diag(f) V^T."""
    return F @ (V * f[:, None, :]) @ V.transpose(1, 2)


def _cof(A):
    c = lambda i, j: (A[:, (i + 1) % 3, (j + 1) % 3] * A[:, (i + 2) % 3, (j + 2) % 3]  # noqa: E731
                      - A[:, (i + 1) % 3, (j + 2) % 3] * A[:, (i + 2) % 3, (j + 1) % 3])
    return torch.stack([torch.stack([c(i, j) for j in range(3)], 1) for i in range(3)], 1)


def _lame(E, nu):
    return E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))


def _drucker_prager(ln, q, prm):
    lam, mu = _lame(prm.sand.E, prm.sand.nu)
    k = (3 * lam + 2 * mu) / (2 * mu)
    phi = torch.deg2rad(prm.sand.h0 + (prm.sand.h1 * q - prm.sand.h3) * torch.exp(-prm.sand.h2 * q))
    alpha = math.sqrt(2 / 3) * 2 * torch.sin(phi) / (3 - torch.sin(phi))
    tr = ln.sum(1)
    dev = ln - tr[:, None] / 3
    nd = dev.norm(dim=1)
    dg = nd + k * tr * alpha
    elastic = dg <= 0
    apex = ~elastic & ((nd == 0) | (tr > 0))
    cone = ln - (dg / nd.clamp_min(1e-300))[:, None] * dev
    new = torch.where(elastic[:, None], ln, torch.where(apex[:, None], torch.zeros_like(ln), cone))
    return new, q + torch.where(elastic, torch.zeros_like(q), torch.where(apex, ln.norm(dim=1), dg))


class _Exact:
    """The step in FP64: items are particles, then cloth vertices, then cloth elements."""

    def __init__(self, case, s):
        self.case, self.prm = case, _params(case)
        dev = _device()
        g = _grid(case)
        t = lambda a: torch.tensor(np.asarray(a, np.float64), device=dev)  # noqa: E731
        self.h, self.res = t(g.h), torch.tensor([int(r) for r in g.resolution], device=dev)
        self.ng = int(np.prod(g.resolution))
        self.dinv = 3.0 / float(g.h.min()) ** 2
        p, m = s["parts"], s["mesh"]
        self.n = case["n"]
        self.nv, self.nf = _cloth_items(case)
        z = lambda *k: torch.zeros(*k, dtype=torch.float64, device=dev)  # noqa: E731
        cat = lambda key, *more: torch.cat(([p[key]] if p is not None else []) + [a for a in more if a is not None])  # noqa: E731
        if m is not None:
            self._mesh(m)
            self.x, self.v = cat("x", m["xv"], m["xe"]), cat("v", m["vv"], m["ve"])
            self.B = cat("B", m["Bv"], m["Be"])
            self.m = cat("m", _f32(self.mv), _f32(self.me))
            self.D = m["D"].clone()
        else:
            self.x, self.v, self.B, self.m = (p[k].clone() for k in ("x", "v", "B", "m"))
        if p is not None:
            self.F, self.vol, self.q, self.mat = p["F"].clone(), p["vol"].clone(), p["q"].clone(), p["mat"]
            self.Fp = p["Fp"].clone() if "Fp" in p else None
        self.gravity = t([self.prm.gravity[a] for a in range(3)])
        k = torch.arange(self.ng, device=dev)
        rx, ry = int(self.res[0]), int(self.res[1])
        self.node_x = torch.stack([k % rx, (k // rx) % ry, k // (rx * ry)], 1) * self.h
        self._zero = z

    def _mesh(self, m):
        f, V = m["faces"], m["rest"]
        h = 1.0 / self.case["res"]
        e1, e2 = V[f[:, 1]] - V[f[:, 0]], V[f[:, 2]] - V[f[:, 0]]
        nrm = torch.linalg.cross(e1, e2)
        area = 0.5 * nrm.norm(dim=1)
        self.faces, self.evol = f, _f32(0.25 * area * h)
        self.me = 0.2 / h * 0.25 * area * h
        vvol = torch.zeros(self.nv, dtype=torch.float64, device=V.device)
        for c in range(3):
            vvol.index_add_(0, f[:, c], 0.25 * area * h)
        self.mv = 0.2 / h * vvol
        rest = torch.stack([e1, e2, nrm / nrm.norm(dim=1, keepdim=True)], 2)
        r11 = e1.norm(dim=1)
        r12 = (e2 * e1).sum(1) / r11
        r22 = (e2 - (r12 / r11)[:, None] * e1).norm(dim=1)
        self.inv_rest = (1 / r11, -r12 / r11 / r22, 1 / r22)
        self.w2 = rest[:, 2, :]

    def _stencil(self):
        u = self.x / self.h
        cell = torch.minimum(u.floor().clamp_min(0).long(), self.res - 1)
        f = (u - cell).clamp(0, 1)
        g = 1 - f
        w = torch.stack([g ** 3 / 6, f ** 3 / 2 - f * f + 2 / 3, g ** 3 / 2 - g * g + 2 / 3, f ** 3 / 6], 2)
        dw = torch.stack([-g * g / 2, 1.5 * f * f - 2 * f, 2 * g - 1.5 * g * g, f * f / 2], 2) / self.h[:, None]
        node = cell[:, :, None] - 1 + torch.arange(4, device=f.device)
        out = (node < 0) | (node >= self.res[:, None])
        w, dw = w.masked_fill(out, 0.0), dw.masked_fill(out, 0.0)
        self.w, self.dw, self.node = w, dw, node.clamp_min(0).minimum(self.res[:, None] - 1)
        self.xi = (torch.arange(4, device=f.device) - 1 - f[:, :, None]) * self.h[:, None]

    def _each_node(self, rows=slice(None), grad=False):
        """Over the 64 stencil nodes: node index, weight, weight gradient, x_i - x_p."""
        w, dw, node, xi = (a[rows] for a in (self.w, self.dw, self.node, self.xi))
        rx, ry = int(self.res[0]), int(self.res[1])
        for o in range(64):
            a, b, c = o & 3, (o >> 2) & 3, o >> 4
            idx = (node[:, 2, c] * ry + node[:, 1, b]) * rx + node[:, 0, a]
            wa, wb, wc = w[:, 0, a], w[:, 1, b], w[:, 2, c]
            g = torch.stack([dw[:, 0, a] * wb * wc, wa * dw[:, 1, b] * wc, wa * wb * dw[:, 2, c]], 1) if grad else None
            yield idx, wa * wb * wc, g, torch.stack([xi[:, 0, a], xi[:, 1, b], xi[:, 2, c]], 1)

    def p2g(self):
        self._stencil()
        acc = self._zero(self.ng, 4)
        for idx, w, _, xi in self._each_node():
            vel = self.v + self.dinv * (self.B @ xi[:, :, None])[:, :, 0]
            acc.index_add_(0, idx, (w * self.m)[:, None] * torch.cat([torch.ones_like(vel[:, :1]), vel], 1))
        self.gm = acc[:, 0]
        # nodes lighter than half a unit of the grid's fixed-point mass hold nothing
        self.live = self.gm > 0.5 * float(self.m.max()) * 2.0 ** -self.prm.mass_bits
        self.gv = torch.where(self.live[:, None], acc[:, 1:] / self.gm.clamp_min(1e-300)[:, None], torch.zeros_like(acc[:, 1:]))

    def volumes(self):
        rho = self._zero(len(self.m))
        for idx, w, _, _ in self._each_node():
            rho += w * self.gm[idx]
        self.vol = self.m[:self.n] * float(self.h.prod()) / rho[:self.n]

    def _cloth_forces(self, dt):
        """In-plane vertex forces (volume weighted) and element normal stresses."""
        D = self.D
        d1, d2, d3 = D[:, :, 0], D[:, :, 1], D[:, :, 2]
        dot = lambda a, b: (a * b).sum(1)  # noqa: E731
        r11 = d1.norm(dim=1)
        q1 = d1 / r11[:, None]
        r12 = dot(d2, q1)
        t = d2 - r12[:, None] * q1
        r22 = t.norm(dim=1)
        q2 = t / r22[:, None]
        r13, r23 = dot(d3, q1), dot(d3, q2)
        t = d3 - r13[:, None] * q1 - r23[:, None] * q2
        r33 = t.norm(dim=1)
        q3 = t / r33[:, None]
        lam, mu = _lame(CLOTH["youngs_modulus"], CLOTH["poisson_ratio"])
        i11, i12, i22 = self.inv_rest
        # T = inverse rest factor x current factor (both upper triangular), P its fixed corotated stress
        t00, t01, t11 = i11 * r11, i11 * r12 + i12 * r22, i22 * r22
        a, c = t00 + t11, -t01
        rn = torch.rsqrt(a * a + c * c)
        cs, sn = a * rn, c * rn
        lj = lam * (t00 * t11 - 1)
        P00, P01 = 2 * mu * (t00 - cs) + lj * t11, 2 * mu * (t01 + sn)
        P10, P11 = -2 * mu * sn - lj * t01, 2 * mu * (t11 - cs) + lj * t00
        ip0, ip1, ip2 = i11 * P00 + i12 * P10, i11 * P01 + i12 * P11, i22 * P11
        f1 = -(P00 * i11 + P01 * i12)[:, None] * q1
        f2 = (-P01 * i22)[:, None] * q1 + (-P11 * i22)[:, None] * q2
        fv = self._zero(self.nv, 3)
        for k, f in enumerate((-(f1 + f2), f1, f2)):
            fv.index_add_(0, self.faces[:, k], self.evol[:, None] * f)
        shear, stiff = CLOTH["shear_stiffness"], CLOTH["stiffness"]
        e13, e23 = shear * r13, shear * r23
        e33 = torch.where(r33 > 1, torch.zeros_like(r33), -stiff * (1 - r33) ** 2)
        # K = dR R^T, its upper triangle mirrored
        K00, K01, K02 = ip0 * r11 + ip1 * r12 + e13 * r13, ip1 * r22 + e13 * r23, e13 * r33
        K11, K12, K22 = ip2 * r22 + e23 * r23, e23 * r33, e33 * r33
        w2 = self.w2
        y0 = w2[:, 0] / r11
        y1 = (w2[:, 1] - r12 * y0) / r22
        y2 = (w2[:, 2] - r13 * y0 - r23 * y1) / r33
        z = (K00 * y0 + K01 * y1 + K02 * y2, K01 * y0 + K11 * y1 + K12 * y2, K02 * y0 + K12 * y1 + K22 * y2)
        dF3 = z[0][:, None] * q1 + z[1][:, None] * q2 + z[2][:, None] * q3
        return dt * fv, -dt * self.evol[:, None, None] * dF3[:, :, None] * d3[:, None, :]

    def forces(self, dt):
        imp = self._zero(self.ng, 3)
        S = self._zero(len(self.m), 3, 3)
        if self.n:
            G = self._zero(self.n, 3, 3)
            for idx, _, g, _ in self._each_node(slice(0, self.n), grad=True):
                G += self.gv[idx][:, :, None] * g[:, None, :]
            Fh = self.F + dt * (G @ self.F)
            ln, V = _stretch(Fh)
            # sand: U diag((2 mu ln s + lambda tr) / s) V^T = Fh V diag(. / s^2) V^T
            lam, mu = _lame(self.prm.sand.E, self.prm.sand.nu)
            P = _with(Fh, V, (2 * mu * ln + lam * ln.sum(1, keepdim=True)) * torch.exp(-2 * ln))
            snow = self.mat == SNOW
            if snow.any():
                lam, mu = _lame(self.prm.snow.E, self.prm.snow.nu)
                jp = torch.linalg.det(self.Fp) if self.Fp is not None else self.q
                hard = torch.exp(self.prm.snow.xi * (1 - jp))[:, None, None]
                J = torch.exp(ln.sum(1))[:, None, None]
                fixed = 2 * mu * hard * (Fh - _with(Fh, V, torch.exp(-ln))) + lam * hard * (J - 1) * _cof(Fh)
                P = torch.where(snow[:, None, None], fixed, P)
            S[:self.n] = -dt * self.vol[:, None, None] * (P @ self.F.transpose(1, 2))
        fv = None
        if self.nf:
            fv, S[self.n + self.nv:] = self._cloth_forces(dt)
        for idx, w, g, _ in self._each_node(grad=True):
            f = (S @ g[:, :, None])[:, :, 0]
            if fv is not None:
                f[self.n:self.n + self.nv] = w[self.n:self.n + self.nv, None] * fv
            imp.index_add_(0, idx, f)
        return imp

    def _phi(self):
        x = self.node_x
        phi, nrm = x[:, 2] - GROUND, torch.zeros_like(x)
        nrm[:, 2] = 1
        if self.case.get("walls"):
            ax, ay, az = 0.9 - x[:, 0], 0.88 - x[:, 1], x[:, 2] - 0.03
            ph = torch.minimum(torch.minimum(az, ax), ay)
            zz = (az.abs() <= ax.abs()) & (az.abs() <= ay.abs())
            yy = ~zz & (ay.abs() <= ax.abs())
            wn = torch.stack([torch.where(zz | yy, 0.0, -1.0), torch.where(yy, -1.0, 0.0), torch.where(zz, 1.0, 0.0)], 1)
            less = ph < phi
            phi, nrm = torch.where(less, ph, phi), torch.where(less[:, None], wn.double(), nrm)
            d = x - torch.tensor([0.45, 0.55, 0.02], dtype=torch.float64, device=x.device)
            r = d.norm(dim=1)
            less = r - 0.07 < phi
            phi, nrm = torch.where(less, r - 0.07, phi), torch.where(less[:, None], d / r.clamp_min(1e-30)[:, None], nrm)
        return phi, nrm

    def grid(self, imp, dt):
        v = self.gv + torch.where(self.live[:, None], imp / self.gm.clamp_min(1e-300)[:, None] + dt * self.gravity,
                                  torch.zeros_like(imp))
        self.vmax = float(v.norm(dim=1).max())
        phi, nrm = self._phi()
        vn = (v * nrm).sum(1)
        hit = self.live & (phi <= 0) & (vn < 0)
        tan = v - vn[:, None] * nrm
        nt = tan.norm(dim=1)
        mu = self.case["friction"]
        slide = tan * (1 + mu * vn / nt.clamp_min(1e-300))[:, None] if self.case.get("coulomb") else tan
        after = torch.where((nt < -mu * vn)[:, None], torch.zeros_like(tan), slide)
        self.vbf = torch.where(hit[:, None], tan, v)
        self.gv = torch.where(hit[:, None], after, v)

    def g2p(self, dt):
        N = len(self.m)
        vp, xn, Cm, G = self._zero(N, 3), self._zero(N, 3), self._zero(N, 3, 3), self._zero(N, 3, 3)
        for idx, w, g, xi in self._each_node(grad=True):
            v, b = self.gv[idx], self.vbf[idx]
            vp += w[:, None] * v
            Cm += (w[:, None] * v)[:, :, None] * xi[:, None, :]
            xn += w[:, None] * (self.x + xi + dt * b)
            G += b[:, :, None] * g[:, None, :]
        n, nv = self.n, self.nv
        damp = torch.zeros(N, 1, 1, dtype=torch.float64, device=vp.device)
        damp[n:] = self.prm.mesh_damp
        sym = 0.5 * (Cm + Cm.transpose(1, 2))
        self.B = Cm - damp * sym
        self.x, self.v = xn, vp
        if n:
            self._return_map(dt * (G[:n] @ self.F))
        if self.nf:
            xv, vv, f = xn[n:n + nv], vp[n:n + nv], self.faces
            self.x[n + nv:] = (xv[f[:, 0]] + xv[f[:, 1]] + xv[f[:, 2]]) / 3
            self.v[n + nv:] = (vv[f[:, 0]] + vv[f[:, 1]] + vv[f[:, 2]]) / 3
            d3 = self.D[:, :, 2] + dt * (G[n + nv:] @ self.D[:, :, 2:])[:, :, 0]
            d1, d2 = xv[f[:, 1]] - xv[f[:, 0]], xv[f[:, 2]] - xv[f[:, 0]]
            q1 = d1 / d1.norm(dim=1, keepdim=True)
            q2 = d2 - (d2 * q1).sum(1, keepdim=True) * q1
            q2 = q2 / q2.norm(dim=1, keepdim=True)
            r13, r23 = (d3 * q1).sum(1, keepdim=True), (d3 * q2).sum(1, keepdim=True)
            q3 = d3 - r13 * q1 - r23 * q2
            r33 = q3.norm(dim=1, keepdim=True)
            q3 = q3 / r33
            cap = CLOTH["friction_coeff"] * CLOTH["stiffness"] * (r33 - 1) ** 2
            shear = CLOTH["shear_stiffness"] * torch.sqrt(r13 * r13 + r23 * r23)
            sc = torch.where(shear > cap, cap / shear.clamp_min(1e-300), torch.ones_like(cap))
            tension = r33 > 1
            sc = torch.where(tension, torch.zeros_like(sc), sc)
            r33 = torch.where(tension, torch.ones_like(r33), r33)
            self.D = torch.stack([d1, d2, sc * (r13 * q1 + r23 * q2) + r33 * q3], 2)

    def _return_map(self, D):
        Ftr = self.F + D
        ln, V = _stretch(Ftr)
        snow = self.mat == SNOW
        cone, q = _drucker_prager(ln, self.q, self.prm)
        lo, hi = math.log(1 - self.prm.snow.theta_c), math.log(1 + self.prm.snow.theta_s)
        new = torch.where(snow[:, None], ln.clamp(lo, hi), cone)
        self.F = _with(Ftr, V, torch.exp(new - ln))
        self.q = torch.where(snow, self.q * torch.exp((ln - new).sum(1)), q)
        if self.Fp is not None:
            self.Fp = (V * torch.exp(ln - new)[:, None, :]) @ V.transpose(1, 2) @ self.Fp
            self.q = torch.where(snow, torch.linalg.det(self.Fp), self.q)

    def step(self, dt_force, dt=None):
        self.p2g()
        self.grid(self.forces(dt_force), dt_force)
        self.g2p(dt_force if dt is None else dt)

    def solve(self, cfl, steps):
        self.p2g()
        self.volumes()
        hmin = float(self.h.min())
        dt = cfl / max(300.0, float(self.gv.norm(dim=1).max()) / hmin)
        inner = 0.0
        for _ in range(steps):
            self.p2g()
            self.grid(self.forces(dt), dt)
            dt = cfl / max(300.0, self.vmax / hmin)
            if inner + dt >= 1 / 60:
                dt, inner = 1 / 60 - inner, 0.0
            else:
                inner += dt
            self.g2p(dt)

    def outputs(self):
        n, nv = self.n, self.nv
        flat = lambda t: t.contiguous().reshape(-1)  # noqa: E731
        out = {}
        if n:
            out = {"x": flat(self.x[:n].T), "v": flat(self.v[:n].T), "B": flat(self.B[:n].permute(1, 2, 0)),
                   "F": flat(self.F.transpose(1, 2)), "vol": self.vol, "q": self.q}
            if self.Fp is not None:
                out["Fp"] = flat(self.Fp.transpose(1, 2))
        if self.nf:
            a, b = slice(n, n + nv), slice(n + nv, None)
            out.update(xv=flat(self.x[a].T), vv=flat(self.v[a].T), Bv=flat(self.B[a].permute(1, 2, 0)),
                       xe=flat(self.x[b].T), ve=flat(self.v[b].T), Be=flat(self.B[b].permute(1, 2, 0)),
                       D=flat(self.D.permute(2, 1, 0)))
        return out


def _features(rec):
    """Network inputs of the records and the scale of its outputs."""
    rec = rec.double()
    ln, q, mat = rec[:, :3], rec[:, 3], rec[:, 4]
    snow = mat == SNOW
    sc = torch.where(snow, 50.0, 1 / ln.norm(dim=1).clamp_min(1e-30))
    one = [(mat == k).double() for k in (SNOW, SAND, 2)]
    return torch.stack([*(ln * sc[:, None]).T, torch.where(snow, 0.0, 100.0 * q), *one], 1), sc


def _network(p, x):
    """The packed parameters' network on rows x (7 inputs)."""
    cut = [64 * 16, 64 * 64, 64 * 64, 8 * 64, 64, 64, 64, 8]
    w1, w2, w3, w4, b1, b2, b3, b4 = torch.split(p, cut)
    act = torch.nn.functional.silu
    x = act(x @ w1.reshape(64, 16)[:, :7].T + b1)
    x = act(x @ w2.reshape(64, 64).T + b2)
    x = act(x @ w3.reshape(64, 64).T + b3)
    return (x @ w4.reshape(8, 64).T + b4)[:, :3]


def _exact_mlp(case, seed):
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(1000003 * seed + 29)
    cpu = torch.Generator()
    cpu.manual_seed(1000003 * seed + 31)
    rec = _records(case["n"], gen, dev)
    p = _weights(cpu).double().to(dev)
    x, sc = _features(rec)
    if case["kind"] == "forward":
        return torch.cat([_network(p, c) for c in x.split(1 << 18)]) / sc[:, None]
    target = rec[:, 5:8].double() * sc[:, None]
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    for it in range(case["steps"]):
        frac = it / (case["steps"] - 1) if case["steps"] > 1 else 1.0
        lr = 5e-4 + 0.5 * 5e-4 * (1 + math.cos(math.pi * frac))
        rows = (it * case["batch"] + torch.arange(case["batch"], device=dev)) % case["n"]
        q = p.detach().requires_grad_(True)
        loss = ((_network(q, x[rows]) - target[rows]) ** 2).sum() / (3 * case["batch"])
        (g,) = torch.autograd.grad(loss, q)
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p - lr * (m / (1 - 0.9 ** (it + 1))) / (torch.sqrt(v / (1 - 0.999 ** (it + 1))) + 1e-8)
    return p


def exact(case, seed):
    if case["kind"] in ("train", "forward"):
        return _exact_mlp(case, seed)
    items = case["n"] + sum(_cloth_items(case))
    if items * case["steps"] > MOST_ITEM_STEPS:
        return None
    e = _Exact(case, _inputs(case, seed))
    if case["kind"] == "solve":
        e.solve(case["cfl"], case["steps"])
    else:
        for _ in range(case["steps"]):
            e.step(case["dt"])
    return e.outputs()

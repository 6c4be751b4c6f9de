"""Performance cases of the blob-step engine: what is timed when its speed is measured.

Each case is one call pattern of a user's program through the package's public classes (``lib.Blob``, ``lib.Batch``,
``lib.Adjoint``): a simulation in progress is advanced by a number of steps and its positions (and velocities) are
read back. The meshes are the seeded Kuhn boxes of ``mesh.py`` with the cell sizes, materials, solvers, time steps and
tolerances that the tests and the benchmark use.

``exact`` restates the step in plain torch, FP64: linear tetrahedra, the MRG32k3a stream, Stokes terms, the three
solvers and, by automatic differentiation, the gradients of a step window.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from ffea_ci_demo_gb300 import lib
from ffea_ci_demo_gb300.mesh import Mesh, apply_shear, kuhn_box, relinearise

KT = 4.11e-21
# mesoscopic units (include/dimensions.h of the reference)
M_LEN, M_ENERGY, M_MASS, M_VOL = 1.7e-10, 4.141945559999999e-21, 1.994307387553024e-26, 4.913e-30
M_TIME, M_PRES = 3.7302915560886126e-13, 8.4305832688784826e8


# -- the cases -----------------------------------------------------------------------------------------------------

def _dt(n):
    """Inertia-free steps: the reference's default for protein-sized blobs, ten times that for coarser ones (the
    equipartition scan's middle)."""
    return 1e-14 if n < 10 else 1e-13


def _blob(name, solver, precision, cells, steps, cell=5.0, stokes=0, pins=0, vel=1):
    """`cells`: cells along x, y and z; `cell`: their edge (nm); `vel`: velocities are read back beside positions."""
    dt = _dt(min(cells)) if solver == "CG_nomass" else 1e-14
    return {"name": name, "kind": "blob", "solver": solver, "precision": precision, "nx": cells[0], "ny": cells[1],
            "nz": cells[2], "cell": cell, "steps": steps, "dt": dt, "stokes": stokes, "pins": pins, "vel": vel}


def listed():
    return [
        # the reference's own physics tests: a protein-sized blob of some 60 nodes in a solvent, stepped between two
        # measurement frames; consistent mass and the default (FP64) arithmetic
        _blob("protein CG fp64", "CG", "fp64", (3, 3, 3), 100, cell=3.0, stokes=1),
        # the parity tests' cube (343 nodes), default solver and arithmetic
        _blob("cube6 nomass fp64", "CG_nomass", "fp64", (6, 6, 6), 20, cell=10 / 3),
        # the same blob, explicit solver: launches and latency
        _blob("cube6 lumped fp64", "masslumped", "fp64", (6, 6, 6), 200, cell=10 / 3),
        # a clamped bar of the mesh sizes FFEA users build from density maps, ragged in every direction, in a solvent
        _blob("bar nomass mixed", "CG_nomass", "mixed", (33, 9, 7), 10, cell=5.0, stokes=1, pins=1),
        # the gradient window's mesh (20^3 cells)
        _blob("cube20 nomass mixed", "CG_nomass", "mixed", (20, 20, 20), 5),
        # the same mesh, consistent mass in a solvent, default arithmetic
        _blob("cube20 CG fp64", "CG", "fp64", (20, 20, 20), 10, stokes=1),
        # the benchmark's headline blob, 384,000 elements, in both arithmetics
        _blob("cube40 nomass mixed", "CG_nomass", "mixed", (40, 40, 40), 5, vel=0),
        _blob("cube40 nomass fp64", "CG_nomass", "fp64", (40, 40, 40), 1, vel=0),
        # the benchmark's largest blob: its matrix does not fit in the L2 cache
        _blob("cube64 nomass mixed", "CG_nomass", "mixed", (64, 64, 64), 1, vel=0),
        # a large blob with the explicit solver, FP32 bulk
        _blob("cube56 lumped mixed", "masslumped", "mixed", (56, 56, 56), 50, vel=0),
        # a replica ensemble of uneven blobs (cells per side log-uniform in [8, 32], as the benchmark draws them)
        {"name": "ensemble 32", "kind": "batch", "blobs": 32, "nmin": 8, "nmax": 32, "cell": 5.0, "steps": 2,
         "dt": 1e-13},
        # the gradient of a loss on final positions with respect to the material and the initial positions
        {"name": "gradient window", "kind": "adjoint", "precision": "mixed", "nx": 10, "ny": 10, "nz": 10,
         "cell": 5.0, "steps": 4, "every": 2, "dt": _dt(10)},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["nomass", "nomass", "nomass", "mass", "mass", "batch", "adjoint"])
    if kind == "batch":
        nmax = _log_int(rng, 4, 32)
        return {"kind": "batch", "blobs": _log_int(rng, 2, 40 if nmax < 24 else 24), "nmin": max(2, nmax // 4),
                "nmax": nmax, "cell": rng.choice([3.0, 4.0, 5.0]), "steps": rng.randint(1, 4),
                "dt": _dt(max(2, nmax // 4) + 2)}
    cells = []
    top = 10 if kind == "adjoint" else 48
    n = math.exp(rng.uniform(math.log(2), math.log(top)))
    for _ in range(3):
        cells.append(max(2, min(top, int(round(n * rng.uniform(0.7, 1.4))))))
    volume = cells[0] * cells[1] * cells[2]
    if kind == "adjoint":
        steps = rng.randint(2, 6)
        return {"kind": "adjoint", "precision": rng.choice(["fp64", "mixed"]), "nx": cells[0], "ny": cells[1],
                "nz": cells[2], "cell": 5.0, "steps": steps, "every": rng.randint(1, steps),
                "dt": _dt(min(cells))}
    precision = rng.choice(["fp64", "mixed"])
    solver = "CG_nomass" if kind == "nomass" else rng.choice(["CG", "masslumped"])
    most = {"CG_nomass": 15, "CG": 60, "masslumped": 200}[solver]
    steps = max(1, min(most, int(most * 500 / volume) + 1))
    c = _blob("", solver, precision, cells, steps, cell=rng.choice([10 / 3, 5.0]), stokes=rng.randint(0, 1),
              pins=int(rng.random() < 0.3), vel=int(volume < 10000))
    del c["name"]
    return c


# -- what a user's program has in hand -----------------------------------------------------------------------------

@functools.lru_cache(maxsize=64)
def _box(nx, ny, nz, cell):
    return kuhn_box(nx, ny, nz, cell, seed=12345, stokes_radius=0.25 * cell)


def _mesh(case) -> Mesh:
    m = _box(case["nx"], case["ny"], case["nz"], case["cell"])
    m = Mesh(**{**m.__dict__})
    if case.get("pins"):
        m.pinned = np.nonzero(m.pos[:m.n_linear, 0] == 0.0)[0].astype(np.int32)
    return m


def _ensemble(case):
    """Uneven cubes with their own shear moduli (the softer part of the benchmark's range); the mesh of a blob depends on its size alone."""
    rng = np.random.default_rng(2024)
    cells = np.rint(np.exp(rng.uniform(np.log(case["nmin"]), np.log(case["nmax"]), size=case["blobs"]))).astype(int)
    out = []
    for n, g in zip(cells, rng.uniform(1e8, 4e8, size=case["blobs"])):
        m = Mesh(**{**_box(int(n), int(n), int(n), case["cell"]).__dict__})
        m.material = m.material.copy()
        m.material[:, 3], m.material[:, 4] = g, 3.9 * g
        out.append(m)
    return out


def _stream(seed, k=0):
    return np.random.default_rng([seed, k]).integers(1, 4294944443, size=6).astype(np.uint32)


def _start(mesh, seed):
    """Positions (meso units) off the rest state: a simple shear of 0.05 to 0.1 % with every vertex moved by up to
    1 % of the shortest edge, as in a blob in thermal motion; pinned vertices stay."""
    rng = np.random.default_rng([seed, 3])
    p = apply_shear(mesh, rng.uniform(0.0005, 0.001))
    h = np.sqrt(((mesh.pos[mesh.tets[:, 1]] - mesh.pos[mesh.tets[:, 0]]) ** 2).sum(1).min())
    p[:mesh.n_linear] += rng.uniform(-0.01 * h, 0.01 * h, size=(mesh.n_linear, 3))
    if len(mesh.pinned):
        p[mesh.pinned] = mesh.pos[mesh.pinned]
    return relinearise(p, mesh.tets) * (mesh.scale / M_LEN)


def _window(case, seed):
    """The gradient window's inputs: lognormal material, start positions and a target."""
    m = _mesh(case)
    rng = np.random.default_rng([seed, 7])
    m.material = m.material.copy()
    m.material[:, 3] = 3e8 * np.exp(0.2 * rng.standard_normal(m.n_elem))
    m.material[:, 4] = 1.2e9 * np.exp(0.2 * rng.standard_normal(m.n_elem))
    return m, _start(m, seed), m.pos * (m.scale / M_LEN)


def _pinned(n):
    return torch.empty((n, 3), dtype=torch.float64, pin_memory=True).numpy()


def prepare(case, seed):
    s = {"case": case}
    if case["kind"] == "batch":
        meshes = _ensemble(case)
        b = lib.Batch(meshes, dt=case["dt"], kT=KT, calc_noise=1)
        b.set_positions(np.concatenate([_start(m, seed + i) for i, m in enumerate(meshes)]))
        for i in range(len(meshes)):
            b.set_rng_state(i, _stream(seed, i))
        s.update(batch=b, pos=_pinned(sum(m.n_nodes for m in meshes)))
        return s
    if case["kind"] == "adjoint":
        m, start, target = _window(case, seed)
        b = lib.Blob(m, precision=case["precision"], dt=case["dt"], kT=KT, calc_noise=1,
                     rng_state=_stream(seed))
        s.update(blob=b, start=start, target=target, stream=_stream(seed), pos=_pinned(m.n_nodes),
                 adjoint=lib.Adjoint(b, case["steps"], case["every"]))
        return s
    m = _mesh(case)
    b = lib.Blob(m, solver=case["solver"], precision=case["precision"], dt=case["dt"], kT=KT, calc_noise=1,
                 calc_stokes=case["stokes"], rng_state=_stream(seed))
    b.set_state(pos=_start(m, seed))
    s.update(blob=b, pos=_pinned(m.n_nodes), vel=_pinned(m.n_nodes))
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "batch":
        s["batch"].update(case["steps"])
        return s["batch"].positions(s["pos"])
    b = s["blob"]
    if case["kind"] == "adjoint":
        b.set_state(pos=s["start"])
        b.set_rng_state(s["stream"])
        s["adjoint"].forward()
        x = b.pos(s["pos"])
        g = s["adjoint"].backward(x - s["target"])
        return [x] + [_as_computed(g[k], case) for k in ("G", "E", "A", "B", "x0")]
    b.update(case["steps"])
    x = b.pos(s["pos"])
    return [x, _as_computed(b.vel(s["vel"]), case)] if case["vel"] else [x]


def _as_computed(v, case):
    """The mixed arithmetic holds velocities, forces and adjoint vectors in FP32 (positions accumulate in FP64)."""
    return torch.from_numpy(v).to(torch.float32) if case["precision"] == "mixed" else v


def work(case):
    """Bytes: the state and every element's data once per step. Operations: the element phase, and one application
    of the matrix per iteration of a Jacobi-preconditioned CG, whose count grows with the longest side."""
    if case["kind"] == "batch":
        rng = np.random.default_rng(2024)
        cells = np.rint(np.exp(rng.uniform(np.log(case["nmin"]), np.log(case["nmax"]), size=case["blobs"])))
        each = [_work_one(int(n), int(n), int(n), "CG_nomass", "mixed") for n in cells]
    else:
        each = [_work_one(case["nx"], case["ny"], case["nz"], case.get("solver", "CG_nomass"), case["precision"])]
    k = case["steps"] * (3 if case["kind"] == "adjoint" else 1)
    return {"bytes": k * sum(b for b, _ in each), "flops": k * sum(f for _, f in each)}


def _work_one(nx, ny, nz, solver, precision):
    T, N = 6 * nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)
    blocks = 15 * N
    iters = {"CG_nomass": 12.5 * max(nx, ny, nz), "CG": 25.0, "masslumped": 0.0}[solver]
    p = 4 if precision == "mixed" else 8
    return T * (16 + 14 * p) + N * 96, 450.0 * T + iters * blocks * (18 if solver == "CG_nomass" else 6)


# -- the same in 64 bits -------------------------------------------------------------------------------------------

MRG_M1, MRG_M2 = 4294967087, 4294944443
_A1, _A2 = ((0, 1, 0), (0, 0, 1), (-810728, 1403580, 0)), ((0, 1, 0), (0, 0, 1), (-1370589, 0, 527612))


def _mat_pow(a, e, m):
    r = np.eye(3, dtype=object)
    a = np.array(a, dtype=object) % m
    while e:
        if e & 1:
            r = r.dot(a) % m
        a = a.dot(a) % m
        e >>= 1
    return r


def _jump(states, e):
    """(6, n) int64 stream states advanced by e draws each."""
    out = torch.empty_like(states)
    for o, a, m in ((0, _A1, MRG_M1), (3, _A2, MRG_M2)):
        p = _mat_pow(a, e, m)
        for i in range(3):
            acc = torch.zeros_like(states[0])
            for k in range(3):
                s, c = states[o + k], int(p[i, k])
                acc += ((s * (c >> 16)) % m * 65536 + s * (c & 65535)) % m  # c < 2^32, s < 2^32: no overflow
            out[o + i] = acc % m
    return out


def _draws(state, n, per, dev):
    """(n, per) draws of RAND(-1/2, 1/2): row i holds draws per i .. per i + per - 1 of the stream at `state`."""
    s = torch.tensor([int(v) for v in state], dtype=torch.int64, device=dev).reshape(6, 1)
    while s.shape[1] < n:
        s = torch.cat([s, _jump(s, per * s.shape[1])], 1)
    s = list(s[:, :n])
    out = torch.empty((n, per), dtype=torch.float64, device=dev)
    for k in range(per):
        p1 = (1403580 * s[1] - 810728 * s[0]) % MRG_M1
        p2 = (527612 * s[5] - 1370589 * s[3]) % MRG_M2
        s = [s[1], s[2], p1, s[4], s[5], p2]
        d = torch.where(p1 > p2, p1 - p2, p1 - p2 + MRG_M1)
        out[:, k] = d.double() / (MRG_M1 + 1.0) - 0.5
    return out


class _Exact:
    """One blob's step in FP64 torch."""

    def __init__(self, mesh, state, solver, dt, stokes, material=None):
        self.dev = dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        t = lambda v: torch.as_tensor(np.asarray(v), dtype=torch.float64, device=dev)  # noqa: E731
        s = mesh.scale / M_LEN
        self.N, self.n_all = mesh.n_linear, mesh.n_nodes
        self.tet = torch.as_tensor(mesh.tets[:, :4].astype(np.int64), device=dev)
        self.solver, self.dt, self.kT = solver, dt / M_TIME, KT / M_ENERGY
        mat = t(mesh.material)
        self.rho, self.A = mat[:, 0] * M_VOL / M_MASS, mat[:, 1] / (M_PRES * M_TIME)
        self.B = mat[:, 2] / (M_PRES * M_TIME) - (2.0 / 3.0) * mat[:, 1]
        self.G, self.E = mat[:, 3] / M_PRES, mat[:, 4] / M_PRES
        x = t(mesh.pos * s)[:self.N]
        J0 = self.edges(x)
        self.vol0, self.J0inv = torch.linalg.det(J0).abs() / 6.0, torch.linalg.inv(J0)
        self.stream = [int(v) for v in state]
        self.free = torch.ones(self.N, 1, dtype=torch.float64, device=dev)
        if len(mesh.pinned):
            self.free[torch.as_tensor(mesh.pinned.astype(np.int64), device=dev)] = 0.0
        self.drag = None
        if stokes:
            self.drag_all = 6.0 * math.pi * (1e-3 / (M_PRES * M_TIME)) * t(mesh.stokes_radius * s)
            self.drag = self.drag_all[:self.N, None]
        # each midpoint node's edge ends
        ends = np.zeros((self.n_all, 2), np.int64)
        ends[:self.N] = np.arange(self.N)[:, None]
        for k, (a, b) in enumerate(((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3))):
            ends[mesh.tets[:, 4 + k], 0], ends[mesh.tets[:, 4 + k], 1] = mesh.tets[:, a], mesh.tets[:, b]
        self.ends = torch.as_tensor(ends, device=dev)
        self.v = torch.zeros(self.N, 3, dtype=torch.float64, device=dev)

    def edges(self, x):
        q = x[self.tet]
        return q[:, 1:] - q[:, :1]

    def scatter(self, fe):
        out = torch.zeros(self.N, fe.shape[-1], dtype=torch.float64, device=self.dev)
        return out.index_add(0, self.tet.reshape(-1), fe.reshape(-1, fe.shape[-1]))

    def geometry(self, x):
        """Volumes and the four shape functions' gradients (T, 4, 3)."""
        J = self.edges(x)
        g = torch.linalg.inv(J).transpose(1, 2)  # rows: gradients of nodes 1, 2, 3
        return J, torch.linalg.det(J).abs() / 6.0, torch.cat([-g.sum(1, keepdim=True), g], 1)

    def viscous(self, grad, vol, v):
        """V v by elements: forces of the stress B tr(L) I + A (L + L^T)."""
        L = torch.einsum("eai,eaj->eij", v[self.tet], grad)  # L_ij = dv_i/dx_j
        S = self.A[:, None, None] * (L + L.transpose(1, 2))
        tr = self.B * (L[:, 0, 0] + L[:, 1, 1] + L[:, 2, 2])
        S = S + tr[:, None, None] * torch.eye(3, dtype=torch.float64, device=self.dev)
        return self.scatter(vol[:, None, None] * torch.einsum("eij,eaj->eai", S, grad))

    def force(self, x):
        J, vol, grad = self.geometry(x)
        eye = torch.eye(3, dtype=torch.float64, device=self.dev)
        F = torch.einsum("eki,ejk->eij", J, self.J0inv)  # deformation gradient: J = rows of edges
        G, E = self.G, self.E
        S = (G * self.vol0 / vol)[:, None, None] * (F @ F.transpose(1, 2)) - G[:, None, None] * eye
        c = G * (1 - self.vol0 / vol) + 0.5 * (E - G * 2 / 3) * (vol / self.vol0 - self.vol0 / vol)
        S = S + c[:, None, None] * eye
        T = self.tet.shape[0]
        d = _draws(self.stream, T, 7, self.dev)
        used = 7 * T
        a = torch.sqrt(self.A)
        n = torch.sqrt(24 * self.kT / (vol * self.dt))
        diag = math.sqrt(2.0) * a[:, None] * d[:, 1:4] + (torch.sqrt(self.B) * d[:, 0])[:, None]
        o = a[:, None] * d[:, 4:7]
        noise = torch.stack([torch.stack([diag[:, 0], o[:, 0], o[:, 1]], 1),
                             torch.stack([o[:, 0], diag[:, 1], o[:, 2]], 1),
                             torch.stack([o[:, 1], o[:, 2], diag[:, 2]], 1)], 1)
        S = S + n[:, None, None] * noise
        f = -self.scatter(vol[:, None, None] * torch.einsum("eij,eaj->eai", S, grad))
        if self.solver != "CG_nomass":
            f = f - self.viscous(grad, vol, self.v)
        if self.drag is not None:
            if self.solver != "CG_nomass":
                f = f - self.v * self.drag
            st = [int(v) for v in _jump(torch.tensor(self.stream, device=self.dev).reshape(6, 1), used)[:, 0]]
            r = -_draws(st, self.n_all, 3, self.dev) * torch.sqrt(24 * self.kT * self.drag_all / self.dt)[:, None]
            used += 3 * self.n_all
            # a vertex keeps its own, a midpoint's goes half to each end
            w = torch.full((self.n_all, 1), 0.5, dtype=torch.float64, device=self.dev)
            f = f.index_add(0, self.ends[:, 0], w * r).index_add(0, self.ends[:, 1], w * r)
        self.stream = [int(v) for v in _jump(torch.tensor(self.stream, device=self.dev).reshape(6, 1), used)[:, 0]]
        return f * self.free, grad, vol

    def diagonal(self, grad, vol):
        g2 = grad * grad
        d = vol[:, None, None] * ((self.A + self.B)[:, None, None] * g2 + self.A[:, None, None] *
                                  g2.sum(2, keepdim=True))
        return self.scatter(d)

    def solve(self, apply, diag, f):
        """Jacobi-preconditioned CG from 0 (where the matrix is singular: the solution D-orthogonal to its kernel)."""
        x, r = torch.zeros_like(f), f.clone()
        p = z = r / diag
        rz, f2 = (r * z).sum(), float((f * f).sum())
        for k in range(6000):
            q = apply(p)
            a = rz / (p * q).sum()
            x = x + a * p
            r = r - a * q
            if k % 8 == 7 and float((r * r).sum()) < 1e-25 * f2:
                break
            z = r / diag
            rz, old = (r * z).sum(), rz
            p = z + (rz / old) * p
        return x

    def step(self, x):
        f, grad, vol = self.force(x)
        pin = 1 - self.free
        if self.solver == "masslumped":
            m = self.scatter((0.25 * self.rho * self.vol0)[:, None, None].expand(-1, 4, 1))
            a = f / (m * self.free + pin)
        elif self.solver == "CG":
            w = (0.05 * self.rho * self.vol0)[:, None, None]
            diag = self.scatter((2 * w).expand(-1, 4, 1)) * self.free + pin

            def apply(p):
                q = (p * self.free)[self.tet]
                return self.scatter(w * (q + q.sum(1, keepdim=True))) * self.free + p * pin
            a = self.solve(apply, diag.expand(-1, 3), f)
        else:
            d = self.diagonal(grad, vol)
            if self.drag is not None:
                d = d + self.drag
            d = d * self.free + pin

            def apply(p):
                q = self.viscous(grad, vol, p * self.free)
                if self.drag is not None:
                    q = q + self.drag * p
                return q * self.free + p * pin
            self.v = self.solve(apply, d, f)
            return x + self.v * self.dt
        self.v = self.v + a * self.dt
        return x + self.v * self.dt

    def dense_step(self, x):
        """A CG_nomass step without drag or pins that autograd follows: the same solution from the dense matrix
        V + D Z (Z^T D Z)^-1 Z^T D, Z the six rigid motions, applied to the force projected off D Z."""
        f, grad, vol = self.force(x)
        N, dev = self.N, self.dev
        gd = torch.einsum("eai,ebi->eab", grad, grad)
        K = torch.einsum("eai,ebj->eaibj", grad, grad) * self.B[:, None, None, None, None]
        K = K + torch.einsum("eaj,ebi->eaibj", grad, grad) * self.A[:, None, None, None, None]
        eye = torch.eye(3, dtype=torch.float64, device=dev)
        K = K + torch.einsum("eab,ij->eaibj", gd, eye) * self.A[:, None, None, None, None]
        K = K * vol[:, None, None, None, None]
        dof = (3 * self.tet[:, :, None] + torch.arange(3, device=dev)).reshape(-1, 12)
        at = (dof[:, :, None] * (3 * N) + dof[:, None, :]).reshape(-1)
        V = torch.zeros(9 * N * N, dtype=torch.float64, device=dev).index_add(0, at, K.reshape(-1)).reshape(3 * N, 3 * N)
        D = self.diagonal(grad, vol).reshape(-1, 1)
        c = x - x.detach().mean(0)
        o = torch.zeros(N, dtype=torch.float64, device=dev)
        Z = torch.cat([eye.repeat(N, 1),
                       torch.stack([torch.stack([o, -c[:, 2], c[:, 1]], 1), torch.stack([c[:, 2], o, -c[:, 0]], 1),
                                    torch.stack([-c[:, 1], c[:, 0], o], 1)], 2).reshape(3 * N, 3)], 1)
        DZ = D * Z
        R = torch.linalg.solve(Z.T @ DZ, DZ.T)
        b = f.reshape(-1, 1)
        b = b - DZ @ torch.linalg.solve(Z.T @ DZ, Z.T @ b)
        self.v = torch.linalg.solve(V + DZ @ R, b).reshape(N, 3)
        return x + self.v * self.dt

    def everywhere(self, x, mids=True):
        """All nodes of the reference numbering: midpoints at their edges' middles (velocities: zero)."""
        q = 0.5 * (x[self.ends[:, 0]] + x[self.ends[:, 1]])
        if not mids:
            q = torch.cat([x, torch.zeros_like(q[self.N:])])
        return q


def exact(case, seed):
    if case["kind"] == "batch":
        meshes = _ensemble(case)
        if sum(m.n_elem for m in meshes) * case["steps"] > 3_000_000:
            return None  # one blob after another: too long
        out = []
        for i, m in enumerate(meshes):
            e = _Exact(m, _stream(seed, i), "CG_nomass", case["dt"], 0)
            x = torch.as_tensor(_start(m, seed + i)[:m.n_linear], device=e.dev)
            for _ in range(case["steps"]):
                x = e.step(x)
            out.append(e.everywhere(x))
        return torch.cat(out)
    if case["kind"] == "adjoint":
        m, start, target = _window(case, seed)
        if m.n_linear > 2000:
            return None  # dense matrices
        e = _Exact(m, _stream(seed), "CG_nomass", case["dt"], 0)
        leaves = {}
        for k in ("G", "E", "A", "B"):
            leaves[k] = getattr(e, k).clone().requires_grad_(True)
            setattr(e, k, leaves[k])
        x0 = torch.as_tensor(start[:m.n_linear], device=e.dev).clone().requires_grad_(True)
        x = x0
        for _ in range(case["steps"]):
            x = e.dense_step(x)
        p = e.everywhere(x)
        loss = 0.5 * ((p - torch.as_tensor(target, device=e.dev)) ** 2).sum()
        g = torch.autograd.grad(loss, [*leaves.values(), x0])
        return [p.detach(), *g[:4], e.everywhere(g[4], mids=False)]
    m = _mesh(case)
    iters = {"CG_nomass": 15 * max(case["nx"], case["ny"], case["nz"]), "CG": 60, "masslumped": 1}[case["solver"]]
    if case["steps"] * (iters * (1e-3 + 4e-9 * m.n_elem) + 0.05 + 1e-7 * m.n_elem) > 20:
        return None  # over about 20 seconds
    e = _Exact(m, _stream(seed), case["solver"], case["dt"], case["stokes"])
    x = torch.as_tensor(_start(m, seed)[:m.n_linear], device=e.dev)
    for _ in range(case["steps"]):
        x = e.step(x)
    return [e.everywhere(x), e.everywhere(e.v, mids=False)] if case["vel"] else [e.everywhere(x)]

"""What this framework is used for, as cases that can be timed and compared.

A case is a dict of plain values.  Its `kind` says which public path it runs:

  step     one RK4 step of one block (Engine.step): the inner loop of every run
  amr      one Berger-Oliger coarse step of a hierarchy (Engine.coarse_step)
  adjoint  loss and gradient of a short evolution (Adjoint.forward / backward)
  rhs      the drop-in right-hand side on host arrays (dropin.compute_rhs_bssn)
  monitor  the constraint norms of a level (Engine.constraint_norms)

The states are what an evolution of puncture black holes holds: the conformal
factor and pre-collapsed lapse of Brill-Lindquist punctures, with smooth
perturbations of every other field (each with its parity), so that every term
of the right-hand sides is non-zero and the shift takes both signs.

exact() restates the equations in index notation with torch in 64 bits (the
BSSN system of bssn_rhs.f90 with 1+log slicing and the Gamma driver, its Z4c
form, RK4, Sommerfeld faces, the constraints); it shares no code with the
framework.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nr-amssncku_b200"))

EPS = 0.1          # Kreiss-Oliger strength of every run here
CHITINY = 1e-5     # floor of chi
PAIRS = [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)]
# directions (bit d) in which a field changes sign under reflection
ANTI = [0, 0] + [0, 3, 5, 0, 6, 0] * 2 + [1, 2, 4, 0, 1, 2, 4, 1, 2, 4, 0]
# most points of a drawn block: the listed 198^3 block has 7.8 M
MOST_POINTS = 4_000_000


def step(name, n, precision="fp64", formulation="bssn", symmetry=0, h=0.25):
    return dict(name=name, kind="step", nx=n[0], ny=n[1], nz=n[2], precision=precision, formulation=formulation,
                symmetry=symmetry, h=h)


def listed():
    return [
        # the smallest block a refined level is cut into (24^3 points): launches count
        step("step_24", (24, 24, 24)),
        # an uneven block as the splitter makes them, odd extents, a spacing that is no power of two
        step("step_ragged", (47, 61, 38), h=0.2),
        # the 64^3 block with 3 ghost cells a side of the single-block runs, FP64 and mixed
        step("step_70", (70, 70, 70)),
        step("step_70_mixed", (70, 70, 70), precision="mixed"),
        # an octant run: mirrored stencils at three planes
        step("step_octant", (57, 64, 51), symmetry=2, h=0.3),
        # a Z4c block of 128^3 cells, and a large mixed-precision block
        step("step_134_z4c", (134, 134, 134), formulation="z4c"),
        step("step_198_mixed", (198, 198, 198), precision="mixed"),
        # the benchmark's binary hierarchy: 96^3 coarse and 6 refined levels of 48^3 boxes, in both precisions
        dict(name="amr_binary", kind="amr", coarse=96, levels=7, box=48, two=True, precision="fp64", formulation="bssn"),
        dict(name="amr_binary_mixed", kind="amr", coarse=96, levels=7, box=48, two=True, precision="mixed",
             formulation="bssn"),
        # gradient of the constraint loss through a short evolution, checkpointed
        dict(name="adjoint", kind="adjoint", nx=46, ny=40, nz=42, steps=4, ck=2),
        # the reference's driver calling the right-hand side of one block through the drop-in symbol
        dict(name="rhs_dropin", kind="rhs", nx=54, ny=54, nz=54, symmetry=0, h=0.25),
        # the constraint monitor of a run's level
        dict(name="monitor", kind="monitor", nx=102, ny=102, nz=102, symmetry=0, h=0.25),
    ]


def _sizes(rng, lo, hi, most):
    while True:
        n = [int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(3)]
        if n[0] * n[1] * n[2] <= most:
            return n


def draw(rng):
    u = rng.random()
    if u < 0.6:
        n = _sizes(rng, 18, 200, MOST_POINTS)
        c = step("", n, precision=rng.choice(["fp64", "mixed"]), formulation=rng.choice(["bssn", "bssn", "z4c"]),
                 symmetry=rng.choice([0, 0, 0, 1, 2]), h=rng.choice([0.25, 0.125, 0.2, 0.3]))
        del c["name"]
        return c
    if u < 0.75:
        return dict(kind="amr", coarse=rng.choice([64, 72, 80, 96]), levels=rng.randint(2, 5),
                    box=rng.choice([32, 36, 40, 44, 48, 52]), two=False, precision=rng.choice(["fp64", "mixed"]),
                    formulation=rng.choice(["bssn", "z4c"]))
    if u < 0.85:
        n = _sizes(rng, 20, 64, 120_000)
        steps = rng.randint(2, 5)
        return dict(kind="adjoint", nx=n[0], ny=n[1], nz=n[2], steps=steps, ck=rng.randint(1, steps))
    n = _sizes(rng, 18, 110, 1_100_000)
    return dict(kind="rhs" if u < 0.93 else "monitor", nx=n[0], ny=n[1], nz=n[2], symmetry=rng.choice([0, 0, 1, 2]),
                h=rng.choice([0.25, 0.2]))


# ---- inputs ------------------------------------------------------------------

def _nf(case):
    return 25 if case.get("formulation") == "z4c" else 24


def _grid(case):
    """bbox and cell centres of a block: centred on the origin, or from 0 up
    where its symmetry has a reflection plane."""
    h, sym = case.get("h", 0.25), case.get("symmetry", 0)
    n = (case["nx"], case["ny"], case["nz"])
    lo = [0.0 if sym == 2 or (sym == 1 and d == 2) else -0.5 * n[d] * h for d in range(3)]
    bbox = tuple(lo) + tuple(lo[d] + n[d] * h for d in range(3))
    X = [np.array([bbox[d] + (j + 0.5) * ((bbox[3 + d] - bbox[d]) / n[d]) for j in range(n[d])]) for d in range(3)]
    return bbox, X


def _state(X, masses, pos, nf, seed, amp, scale, noise=0.0):
    """Puncture data plus smooth perturbations of size `amp` on every field,
    over the length `scale`; (nf, ez, ey, ex) on the GPU."""
    dev = "cuda"
    z, y, x = torch.meshgrid(*[torch.as_tensor(v, dtype=torch.float64, device=dev) for v in X[::-1]], indexing="ij")
    xyz = (x, y, z)
    rng = np.random.default_rng(seed)
    psi = torch.ones_like(x)
    for m, p in zip(masses, pos):
        r = torch.sqrt(sum((xyz[d] - p[d]) ** 2 for d in range(3)))
        psi += 0.5 * m / torch.clamp(r, min=1e-6)
    size = [1.0, 0.1] + [1.0, 0.5, 0.5, 1.0, 0.5, 1.0] + [0.5] * 6 + [1.0] * 3 + [1.0] + [3.0] * 3 + [1.0] * 3 + [0.1]
    st = torch.empty((nf,) + tuple(x.shape), dtype=torch.float64, device=dev)
    for f in range(nf):
        c = rng.uniform(0.6, 1.4, 3)
        s = float(rng.choice([-1.0, 1.0]) * rng.uniform(0.5, 1.0))
        q = sum((c[d] * xyz[d] / scale) ** 2 for d in range(3))
        v = amp * size[f] * s * torch.exp(-q)
        for d in range(3):
            if (ANTI[f] >> d) & 1:
                v = v * (xyz[d] / scale)
        st[f] = v
    st[0] += psi ** -4 - 1.0
    st[17] += psi ** -2 - 1.0
    if noise:
        g = torch.Generator(device=dev).manual_seed(int(seed))
        st += noise * (2.0 * torch.rand(st.shape, dtype=torch.float64, device=dev, generator=g) - 1.0)
    return st


def _inputs(case, seed):
    """(bbox, X, state on the GPU) of a single-block case."""
    bbox, X = _grid(case)
    rng = np.random.default_rng([int(seed), 7])
    extent = min(bbox[3 + d] for d in range(3))
    if case.get("symmetry", 0):
        pos = [[0.0, 0.0, 0.0]]          # on the reflection planes
    else:
        pos = [list(rng.uniform(-0.15, 0.15, 3) * extent)]
    masses = [float(rng.uniform(0.3, 0.6)) * min(1.0, extent / 4.0)]
    return bbox, X, _state(X, masses, pos, _nf(case), int(seed), 0.01, 0.4 * extent, noise=1e-8)


def _amr_inputs(case, seed):
    from amss_b200 import hierarchy
    ext = case["coarse"] / 2.0
    centres = [(-3.0, 0.0, 0.0), (3.0, 0.0, 0.0)] if case["two"] else [(0.0, 0.0, 0.0)]
    H = hierarchy.box_in_box(case["coarse"], ext, centres, case["levels"], box_cells=case["box"], seed=1, block_min=18,
                             block_max=74)
    rng = np.random.default_rng([int(seed), 7])
    pos = [[float(c[d] + rng.uniform(0.02, 0.1)) for d in range(3)] for c in centres]
    masses = [float(rng.uniform(0.4, 0.6)) for _ in centres]
    return H, masses, pos


class _Held:
    """Closes an engine (or adjoint) when the last thing that uses it goes."""

    def __init__(self, handle):
        self.handle = handle

    def __del__(self):
        self.handle.close()


class _View:
    """Device memory of an engine as torch takes it; keeps the engine open."""

    def __init__(self, held, ptr, shape, strides):
        self.held = held
        self.__cuda_array_interface__ = dict(shape=shape, strides=strides, typestr="<f8", data=(ptr, False), version=3)


def _outputs(held, blocks, views):
    """The current states of the blocks, where they are: one tensor per block,
    or for a single block one per field."""
    eng, out = held.handle, []
    for b in blocks:
        ptr, fs = eng.state_device(b)
        if (b, ptr) not in views:
            ex = eng.blocks[b]
            t = torch.as_tensor(_View(held, ptr, (eng.nf, ex[2], ex[1], ex[0]),
                                      (8 * fs, 8 * ex[0] * ex[1], 8 * ex[0], 8)), device="cuda")
            views[(b, ptr)] = t if len(blocks) > 1 else list(t.unbind(0))
        out.append(views[(b, ptr)])
    return out


class _Run:
    """What a program keeps between calls."""

    def __init__(self, case):
        self.case, self.views, self.held = case, {}, None

    def keep(self, handle):
        self.held = _Held(handle)
        return handle


def prepare(case, seed):
    import amss_b200
    from amss_b200 import adjoint
    s = _Run(dict(case))
    kind = case["kind"]
    if kind == "amr":
        H, masses, pos = _amr_inputs(case, seed)
        eng = s.keep(amss_b200.Engine.from_hierarchy(H, precision=case["precision"], eps=EPS,
                                                     formulation=case["formulation"]))
        for i, b in enumerate(H.blocks):
            st = _state(H.coords(b), masses, pos, _nf(case), int(seed), 1e-3, 6.0)
            eng.set_state(i, st.cpu().numpy())
        eng.set_punctures(pos)
        s.dt = 0.25 * H.h0
        s.blocks = range(len(H.blocks))
        return s
    bbox, X, st = _inputs(case, seed)
    h = case.get("h", 0.25)
    if kind in ("step", "monitor"):
        eng = s.keep(amss_b200.Engine(precision=case.get("precision", "fp64"), symmetry=case["symmetry"], eps=EPS,
                                      formulation=case.get("formulation", "bssn")))
        b = eng.add_block(0, (case["nx"], case["ny"], case["nz"]), bbox, bbox)
        eng.commit()
        eng.set_state(b, st.cpu().numpy())
        s.dt, s.blocks = 0.25 * h, [b]
    elif kind == "adjoint":
        s.keep(adjoint.Adjoint((case["nx"], case["ny"], case["nz"]), bbox, eps=EPS))
        s.state = st.cpu().numpy()
        s.dt = 0.25 * h
    else:
        s.X, s.state = X, st.cpu().numpy()
    return s


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "step":
        s.held.handle.step(0, s.dt)
        return _outputs(s.held, s.blocks, s.views)[0]
    if kind == "amr":
        s.held.handle.coarse_step(s.dt)
        return _outputs(s.held, s.blocks, s.views)
    if kind == "monitor":
        return s.held.handle.constraint_norms(0)[:7]
    if kind == "adjoint":
        adj = s.held.handle
        adj.set_state(s.state)
        loss = adj.forward(s.dt, case["steps"], case["ck"])
        return {"loss": loss, "gradient": adj.backward()}
    from amss_b200 import dropin
    _, rhs, gamma, ricci, cons = dropin.compute_rhs_bssn(s.X[0], s.X[1], s.X[2], s.state, symmetry=case["symmetry"],
                                                         eps=EPS, co=0)
    return {"rhs": rhs, "gamma": gamma, "ricci": ricci, "cons": cons}


# ---- cost and tolerance ------------------------------------------------------

# operations of one right-hand side at one point: the pointwise algebra about
# 2700, the stencils about 3200
RHS_FLOPS = 5900


def work(case):
    kind, nf = case["kind"], _nf(case)
    if kind == "amr":
        H, _, _ = _amr_inputs(case, 0)
        pts = sum(H.interior_zones(lev) * 2 ** lev for lev in range(len(H.levels)))
        return {"bytes": 2.0 * 8 * nf * pts, "flops": 4.0 * RHS_FLOPS * pts}
    pts = float(case["nx"] * case["ny"] * case["nz"])
    if kind == "step":        # the state in and out
        return {"bytes": 2 * 8 * nf * pts, "flops": 4 * RHS_FLOPS * pts}
    if kind == "adjoint":     # the state in, the gradient out; the reverse is about twice the forward
        return {"bytes": 2 * 8 * 24 * pts, "flops": 3 * 4 * RHS_FLOPS * pts * case["steps"]}
    if kind == "rhs":         # 24 fields and 10 matter fields in, 55 out
        return {"bytes": 8 * (24 + 10 + 55) * pts, "flops": RHS_FLOPS * pts}
    return {"bytes": 8 * 24 * pts, "flops": RHS_FLOPS * pts}


def tolerance(case):
    """About four times the largest difference seen between the framework and
    exact() over listed and drawn cases (single blocks: 1.3e-12 in FP64, 7e-7
    in mixed precision; the gradient 2e-13, the right-hand side 1e-13, the
    norms 6e-16).  amr has no exact(): its two kernel forms differ by 1e-14
    (FP64) and 6e-9 (mixed), and share most of their operation order."""
    kind = case["kind"]
    mixed = case.get("precision") == "mixed"
    if kind == "amr":
        return {"rel": 1e-7 if mixed else 1e-12, "max": 1e-5 if mixed else 1e-9}
    if kind == "step":
        return {"rel": 3e-6 if mixed else 6e-12, "max": 1e-4 if mixed else 1e-8}
    if kind == "adjoint":
        return {"rel": 4e-12, "max": 4e-9}
    if kind == "rhs":
        return {"rel": 1e-12, "max": 1e-9}
    return {"rel": 1e-13, "max": 1e-12}


# ---- the equations in 64 bits ------------------------------------------------

class _Exact:
    """Finite differences and equations of one block with its patch's faces."""

    def __init__(self, bbox, X, symmetry, nf, dev):
        self.nf, self.dev = nf, dev
        self.n = [len(v) for v in X]
        self.h = [float(v[1] - v[0]) for v in X]
        self.ls = [symmetry == 2, symmetry == 2, symmetry > 0]
        self.xyz = [self._along(torch.as_tensor(X[d], dtype=torch.float64, device=dev), d) for d in range(3)]

        def fits(lo, hi):   # index ranges that stay in the block, over all directions
            g = None
            for d in range(3):
                i = torch.arange(self.n[d], device=dev)
                ok = (i + hi <= self.n[d] - 1) & (i - lo >= (-3 if self.ls[d] else 0))
                ok = self._along(ok, d)
                g = ok if g is None else g & ok
            return g
        self.o4, self.o2, self.ko, self.lop = fits(2, 2), fits(1, 1), fits(3, 3), fits(-10 ** 6, 1)
        face = torch.zeros(self.n[::-1], dtype=torch.bool, device=dev)
        for d in range(3):
            i = torch.arange(self.n[d], device=dev)
            face = face | self._along((i == self.n[d] - 1) | ((i == 0) & (not self.ls[d])), d)
        self.face = face

    @staticmethod
    def _along(v, d):
        return v.reshape([-1 if 2 - a == d else 1 for a in range(3)])

    def pad(self, f, F):
        """Three mirrored cells (with the field's parity) below, zeros above."""
        for d in range(3):
            a = 2 - d
            low = torch.flip(f.narrow(a, 0, 3), [a])
            if (ANTI[F] >> d) & 1:
                low = -low
            f = torch.cat([low, f, torch.zeros_like(low)], dim=a)
        return f

    def at(self, P, o):
        return P[3 + o[2]:3 + o[2] + self.n[2], 3 + o[1]:3 + o[1] + self.n[1], 3 + o[0]:3 + o[0] + self.n[0]]

    def line(self, P, d, m):
        return self.at(P, [m if a == d else 0 for a in range(3)])

    def gate(self, a4, a2):
        return torch.where(self.o4, a4, torch.where(self.o2, a2, torch.zeros_like(a2)))

    def grad(self, P):
        out = []
        for d in range(3):
            f = [self.line(P, d, m) for m in (-2, -1, 1, 2)]
            out.append(self.gate((f[0] - 8 * f[1] + 8 * f[2] - f[3]) / (12 * self.h[d]),
                                 (f[2] - f[1]) / (2 * self.h[d])))
        return out

    def hess(self, P):
        w4, out = {-2: 1.0, -1: -8.0, 1: 8.0, 2: -1.0}, []
        for a, b in PAIRS:
            if a == b:
                f = {m: self.line(P, a, m) for m in range(-2, 3)}
                a4 = (-f[-2] + 16 * f[-1] - 30 * f[0] + 16 * f[1] - f[2]) / (12 * self.h[a] ** 2)
                a2 = (f[-1] - 2 * f[0] + f[1]) / self.h[a] ** 2
            else:
                def cell(i, j):
                    o = [0, 0, 0]
                    o[a], o[b] = i, j
                    return self.at(P, o)
                a4 = sum(w4[i] * w4[j] * cell(i, j) for i in w4 for j in w4) / (144 * self.h[a] * self.h[b])
                a2 = (cell(-1, -1) - cell(1, -1) - cell(-1, 1) + cell(1, 1)) / (4 * self.h[a] * self.h[b])
            out.append(self.gate(a4, a2))
        return out

    def advect(self, P, beta):
        """Upwinded advection and Kreiss-Oliger dissipation of one field."""
        r = torch.zeros_like(beta[0])
        ko = torch.zeros_like(r)
        for d in range(3):
            f = {m: self.line(P, d, m) for m in range(-3, 4)}
            up = -3 * f[-1] - 10 * f[0] + 18 * f[1] - 6 * f[2] + f[3]
            dn = 3 * f[1] + 10 * f[0] - 18 * f[-1] + 6 * f[-2] - f[-3]
            ce = f[-2] - 8 * f[-1] + 8 * f[1] - f[2]
            i = self._along(torch.arange(self.n[d], device=self.dev), d)
            hi, lo = self.n[d] - 1, (-3 if self.ls[d] else 0)
            z = torch.zeros_like(r)
            pos = torch.where(i + 3 <= hi, up, torch.where(i + 2 <= hi, ce, torch.where(i + 1 <= hi, dn, z)))
            neg = torch.where(i - 3 >= lo, dn, torch.where(i - 2 >= lo, ce, torch.where(i - 1 >= lo, up, z)))
            r = r + beta[d] * torch.where(beta[d] > 0, pos, neg) / (12 * self.h[d])
            ko = ko + ((f[-3] + f[3]) - 6 * (f[-2] + f[2]) + 15 * (f[-1] + f[1]) - 20 * f[0]) / self.h[d]
        return torch.where(self.lop, r, torch.zeros_like(r)) + torch.where(self.ko, EPS / 64 * ko, torch.zeros_like(r))

    def rhs(self, u, constraints=False):
        """Right-hand sides (nf fields); with constraints also the physical
        Christoffel symbols, the Ricci tensor and the 7 constraints."""
        R3, S3 = range(3), range(3)
        z4c = self.nf == 25
        P = [self.pad(u[f], f) for f in range(self.nf)]
        chi, K, al = u[0] + 1, u[1], u[17] + 1
        full = lambda v: [[v[PAIRS.index((min(i, j), max(i, j)))] for j in R3] for i in R3]  # noqa: E731
        eye = [[1.0 if i == j else 0.0 for j in R3] for i in R3]
        g = [[u[2 + PAIRS.index((min(i, j), max(i, j)))] + eye[i][j] for j in R3] for i in R3]
        A = full([u[8 + m] for m in range(6)])
        Gam, be, B = [u[14 + i] for i in R3], [u[18 + i] for i in R3], [u[21 + i] for i in R3]
        Th = u[24] if z4c else torch.zeros_like(K)
        Kd = K + 2 * Th
        dchi, dK, dal = self.grad(P[0]), self.grad(P[1]), self.grad(P[17])
        db = [self.grad(P[18 + i]) for i in R3]              # db[i][j] = d_j beta^i
        dg6 = [self.grad(P[2 + m]) for m in range(6)]
        dg = [[[dg6[PAIRS.index((min(i, j), max(i, j)))][k] for k in R3] for j in R3] for i in R3]
        div = db[0][0] + db[1][1] + db[2][2]
        cof = lambda i, j: (g[(i + 1) % 3][(j + 1) % 3] * g[(i + 2) % 3][(j + 2) % 3]  # noqa: E731
                            - g[(i + 1) % 3][(j + 2) % 3] * g[(i + 2) % 3][(j + 1) % 3])
        det = sum(g[0][j] * cof(0, j) for j in R3)
        gu = full([cof(i, j) / det for i, j in PAIRS])
        low = [full([0.5 * (dg[l][i][j] + dg[l][j][i] - dg[i][j][l]) for i, j in PAIRS]) for l in R3]   # Gamma_{l,ij}
        G = [full([sum(gu[k][l] * low[l][i][j] for l in S3) for i, j in PAIRS]) for k in R3]
        Ga = [sum(gu[j][k] * G[i][j][k] for j in R3 for k in R3) for i in R3]
        Au = full([sum(gu[i][k] * gu[j][l] * A[k][l] for k in R3 for l in R3) for i, j in PAIRS])
        out = [None] * self.nf
        out[0] = 2 / 3 * chi * (al * Kd - div)
        out[17] = -2 * al * K
        for m, (i, j) in enumerate(PAIRS):
            out[2 + m] = (-2 * al * A[i][j] - 2 / 3 * g[i][j] * div
                          + sum(g[i][k] * db[k][j] + g[j][k] * db[k][i] for k in R3))
        hb = [full(self.hess(P[18 + i])) for i in R3]
        Kg = [dK[j] + (self.grad(P[24])[j] / 2 if z4c else 0) for j in R3]
        for i in R3:
            r = sum(-2 * dal[j] * Au[i][j] - 3 * al / chi * dchi[j] * Au[i][j] - 4 / 3 * al * gu[i][j] * Kg[j] for j in R3)
            r = r + 2 * al * sum(G[i][j][k] * Au[j][k] for j in R3 for k in R3)
            r = r + 2 / 3 * Ga[i] * div - sum(Ga[j] * db[i][j] for j in R3)
            r = r + sum(gu[i][j] * hb[k][j][k] for j in R3 for k in R3) / 3
            r = r + sum(gu[j][k] * hb[i][j][k] for j in R3 for k in R3)
            out[14 + i] = r - (2 * al * 0.02 * (Gam[i] - Ga[i]) if z4c else 0)
            out[18 + i] = 0.75 * B[i]
            out[21 + i] = r - 2 * B[i]
        dGam = [self.grad(P[14 + i]) for i in R3]
        Ric = []
        for m, (i, j) in enumerate(PAIRS):
            hg = full(self.hess(P[2 + m]))
            r = -0.5 * sum(gu[k][l] * hg[k][l] for k in R3 for l in R3)
            r = r + 0.5 * sum(g[k][i] * dGam[k][j] + g[k][j] * dGam[k][i] + Ga[k] * (low[i][j][k] + low[j][i][k])
                              for k in R3)
            for l in R3:
                for n in R3:
                    r = r + gu[l][n] * sum(G[k][l][i] * low[j][k][n] + G[k][l][j] * low[i][k][n]
                                           + G[k][i][n] * low[k][l][j] for k in R3)
            Ric.append(r)
        hc = self.hess(P[0])
        cc = [hc[m] - sum(G[k][i][j] * dchi[k] for k in R3) for m, (i, j) in enumerate(PAIRS)]
        cf = full(cc)
        tr = sum(gu[i][j] * (cf[i][j] - 1.5 / chi * dchi[i] * dchi[j]) for i in R3 for j in R3)
        Ric = [Ric[m] + (cc[m] - dchi[i] * dchi[j] / chi / 2 + g[i][j] * tr) / chi / 2 for m, (i, j) in enumerate(PAIRS)]
        cu = [sum(gu[k][l] * dchi[l] for l in R3) / chi for k in R3]
        Gp = [full([G[k][i][j] - 0.5 * (eye[k][i] * dchi[j] / chi + eye[k][j] * dchi[i] / chi - g[i][j] * cu[k])
                    for i, j in PAIRS]) for k in R3]
        ha = self.hess(P[17])
        La = [ha[m] - sum(Gp[k][i][j] * dal[k] for k in R3) for m, (i, j) in enumerate(PAIRS)]
        Rf, Lf = full(Ric), full(La)
        AA = [sum(gu[k][l] * A[i][k] * A[j][l] for k in R3 for l in R3) for i, j in PAIRS]
        AAf = full(AA)
        trace = lambda t: sum(gu[i][j] * t[i][j] for i in R3 for j in R3)  # noqa: E731
        A2, trL, trR = trace(AAf), trace(Lf), trace(Rf)
        if z4c:
            f = (trR * al - trL) / 3
        else:
            f = -(trL + al / chi * (2 / 3 * K * K - A2)) / 3
        for m, (i, j) in enumerate(PAIRS):
            out[8 + m] = (chi * (al * Ric[m] - La[m] - g[i][j] * f) + al * (Kd * A[i][j] - 2 * AA[m])
                          + sum(A[i][k] * db[k][j] + A[j][k] * db[k][i] for k in R3) - 2 / 3 * A[i][j] * div)
        out[1] = -chi * trL + al * (Kd * Kd / 3 + A2)
        if z4c:
            out[1] = out[1] + al * 0.02 * Th
            out[24] = al * (chi * trR + 2 / 3 * Kd * Kd - A2) / 2 - al * 2 * 0.02 * Th
        out = [out[f] + self.advect(P[f], be) for f in range(self.nf)]
        if not constraints:
            return out
        cons = [chi * trR + 2 / 3 * K * K - A2]
        dA6 = [self.grad(P[8 + m]) for m in range(6)]
        for i in R3:
            r = -2 / 3 * dK[i]
            for j in R3:
                for k in R3:
                    d = dA6[PAIRS.index((min(i, k), max(i, k)))][j]
                    d = d - sum(Gp[l][j][k] * A[l][i] + Gp[l][j][i] * A[l][k] for l in R3) - dchi[j] * A[i][k] / chi
                    r = r + gu[j][k] * d
            cons.append(r)
        for i in R3:
            cons.append(Gam[i] - sum(gu[i][k] * gu[j][l] * dg[k][l][j] for j in R3 for k in R3 for l in R3))
        return out, [Gp[k][i][j] for k in R3 for i, j in PAIRS], Ric, cons

    def sommerfeld(self, u):
        R = torch.sqrt(sum(x * x for x in self.xyz))
        out = []
        for F in range(self.nf):
            P = self.pad(u[F], F)
            v = math.sqrt(2.0) if F in (0, 1, 17) else 1.0
            s = u[F]
            for d in range(3):
                f = {m: self.line(P, d, m) for m in range(-2, 3)}
                i = self._along(torch.arange(self.n[d], device=self.dev), d)
                hi, lo, x = self.n[d] - 1, (-1 if self.ls[d] else 0), self.xyz[d]
                back, mid, fwd = 3 * f[0] - 4 * f[-1] + f[-2], f[1] - f[-1], -f[2] + 4 * f[1] - 3 * f[0]
                a = torch.where(i - 2 >= lo, back, torch.where(i - 1 >= lo, mid, fwd))
                b = torch.where(i + 2 <= hi, fwd, torch.where(i + 1 <= hi, mid, back))
                s = s + x * torch.where(x > 0, a, torch.where(x < 0, b, torch.zeros_like(a))) / (2 * self.h[d])
            out.append(-v * s / R)
        return out

    def enforce(self, u):
        u = list(u)
        eye = [1.0, 0.0, 0.0, 1.0, 0.0, 1.0]
        g6 = [u[2 + m] + eye[m] for m in range(6)]
        full = lambda v: [[v[PAIRS.index((min(i, j), max(i, j)))] for j in range(3)] for i in range(3)]  # noqa: E731

        def cofs(g):
            return [g[(i + 1) % 3][(j + 1) % 3] * g[(i + 2) % 3][(j + 2) % 3]
                    - g[(i + 1) % 3][(j + 2) % 3] * g[(i + 2) % 3][(j + 1) % 3] for i, j in PAIRS]
        g = full(g6)
        c = full(cofs(g))
        s = sum(g[0][j] * c[0][j] for j in range(3)) ** (-1.0 / 3.0)
        g6 = [v * s for v in g6]
        c = full(cofs(full(g6)))
        A = full([u[8 + m] for m in range(6)])
        tr = sum(c[i][j] * A[i][j] for i in range(3) for j in range(3))
        for m, (i, j) in enumerate(PAIRS):
            u[2 + m] = g6[m] - eye[m]
            u[8 + m] = A[i][j] - g6[m] * tr / 3
        return u

    def full_rhs(self, u):
        k, s = self.rhs(u), self.sommerfeld(u)
        return [torch.where(self.face, s[f], k[f]) for f in range(self.nf)]

    def step(self, u, dt):
        u0 = self.enforce(u)
        x, acc = u0, None
        for sub in range(4):
            k = self.full_rhs(x)
            if sub < 3:
                x = [u0[f] + (0.5 * dt if sub < 2 else dt) * k[f] for f in range(self.nf)]
                acc = k if sub == 0 else [acc[f] + 2 * k[f] for f in range(self.nf)]
            else:
                x = [u0[f] + dt / 6 * (k[f] + acc[f]) for f in range(self.nf)]
            x[0] = torch.clamp(x[0], min=CHITINY - 1.0)
            if sub < 3:
                x = self.enforce(x)
        return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "amr":
        return None          # minutes: hundreds of level steps and their transfers
    bbox, X, st = _inputs(case, seed)
    E = _Exact(bbox, X, case.get("symmetry", 0), _nf(case), st.device)
    dt = 0.25 * case.get("h", 0.25)
    u = [st[f] for f in range(_nf(case))]
    if kind == "adjoint":
        leaf = st.clone().requires_grad_(True)
        u = [leaf[f] for f in range(24)]
        from torch.utils.checkpoint import checkpoint
        for _ in range(case["steps"]):
            u = list(checkpoint(lambda *a: tuple(E.step(list(a), dt)), *u, use_reentrant=False))
        ham = E.rhs(u, constraints=True)[3][0]
        inner = tuple(slice(3, -3) for _ in range(3))
        loss = (ham[inner] ** 2).sum() * E.h[0] * E.h[1] * E.h[2]
        loss.backward()
        return {"loss": float(loss), "gradient": leaf.grad}
    with torch.no_grad():
        if kind == "step":
            return E.step(u, dt)
        rhs, gamma, ricci, cons = E.rhs(u, constraints=True)
        if kind == "rhs":
            return {"rhs": torch.stack(rhs), "gamma": torch.stack(gamma), "ricci": torch.stack(ricci),
                    "cons": torch.stack(cons)}
        return np.array([math.sqrt(float((c ** 2).sum()) * E.h[0] * E.h[1] * E.h[2]) for c in cons])

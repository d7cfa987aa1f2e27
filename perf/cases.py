"""Performance cases: the work a user's program has this framework do, through its public entry points.

Every case is one model (a structured block or beam of C3D8 or Kuhn-split C3D4 elements with jittered nodes, one end
plane held, a follower pressure on the other) and one call on it:

  assemble   Assembly.assemble_Stiffness_Matrix      residual and tangent, once per Newton iteration
  force      Assembly.assemble_force                 residual alone: loaded explicit dynamics, residual checks
  energy     StaticImplicitSolver.get_total_energy   once or more per Newton iteration
  pcg        DevicePlan.pcg / pcg_mixed              the tangent solve to a relative residual of 1e-8
  explicit   DynamicExplicitSolver.solve             central-difference steps
  vjp        adjoint.residual_vjp                    sensitivities to all nodal coordinates and the shear modulus
  newton     StaticImplicitSolver.solve              a whole static solve
  batch      serving.BatchedPCG                      the tangent solves of several served requests at once

The meshes and ``exact`` below use numpy and torch alone.
"""
import itertools
import math

import numpy as np
import torch

import fea_b200 as F
from fea_b200 import adjoint, serving
from fea_b200.solver import LinearSolve

DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64
NN = {"C3D8": 8, "C3D4": 4}
FACES = {"C3D4": [[0, 2, 1], [0, 1, 3], [1, 2, 3], [0, 3, 2]],
         "C3D8": [[0, 3, 2, 1], [4, 5, 6, 7], [0, 1, 5, 4], [1, 2, 6, 5], [2, 3, 7, 6], [0, 4, 7, 3]]}
SIGNS = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]])
PCG_TOL = 1e-16          # squared relative residual, in the Jacobi-scaled norm


# -- the cases ---------------------------------------------------------------------------------------------------------
def case(name, call, elem, nx, ny, nz, size=1.0, bc="clamp", numbering="grid", load=0.02, **more):
    return dict(name=name, call=call, elem=elem, nx=nx, ny=ny, nz=nz, size=size, bc=bc, numbering=numbering, load=load,
                **more)


def listed():
    return [
        # the smallest models of the tests and of a first try: launches and latency
        case("assemble_hex_5x7x6", "assemble", "C3D8", 5, 7, 6, bc="roller", numbering="runs"),
        # the headline benchmark's block
        case("assemble_hex_64", "assemble", "C3D8", 64, 64, 64),
        # a large cantilever of the serving stream (C3D4, 2,000 to 200,000 elements), numbered as a mesher would
        case("assemble_tet_beam_190k", "assemble", "C3D4", 132, 16, 15, size=11.0, numbering="runs"),
        # residual alone on the block of the implicit dynamics benchmark
        case("force_hex_48", "force", "C3D8", 48, 48, 48),
        # the total potential the line search and the Newton loop evaluate
        case("energy_hex_48", "energy", "C3D8", 48, 48, 48),
        # the tangent solve in FP64, and with FP32 inner iterations on the headline block
        case("pcg_hex_40", "pcg", "C3D8", 40, 40, 40, solve="fp64"),
        case("pcg_mixed_hex_64", "pcg", "C3D8", 64, 64, 64, solve="mixed"),
        # the explicit benchmark's free cube (2.06 million C3D4), and an implicit-sized C3D8 block run explicitly
        case("explicit_tet_70", "explicit", "C3D4", 70, 70, 70, bc="free", load=0.0, steps=20, fp32=False),
        case("explicit_hex_40", "explicit", "C3D8", 40, 40, 40, load=0.0, steps=20, fp32=False),
        # the compliance benchmark's sensitivities
        case("vjp_hex_40", "vjp", "C3D8", 40, 40, 40),
        # one served request of moderate size, solved whole: assembly, PCG, line search, host control
        case("newton_tet_beam_30k", "newton", "C3D4", 56, 10, 9, size=9.0),
        # the tangent solves of eight requests resident at once
        case("batch_tet_8", "batch", "C3D4", 70, 11, 10, size=9.0, slots=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["assemble", "assemble", "force", "energy", "pcg", "explicit", "vjp", "newton", "batch"])
    elem = "C3D4" if call in ("newton", "batch") else rng.choice(["C3D8", "C3D4"])
    more, size = {}, 1.0
    numbering = rng.choice(["grid", "grid", "runs"])
    bc = rng.choice(["clamp", "clamp", "roller"])
    load = 0.02
    if call in ("newton", "batch"):
        ny, nz = rng.randint(3, 9), rng.randint(3, 9)
        nx, size, bc = rng.randint(4, 6) * max(ny, nz) + rng.randint(0, 5), 8.0, "clamp"
        if call == "batch":
            more = {"slots": rng.randint(2, 8)}
    elif call == "pcg":
        n = _log(rng, 4, 40 if elem == "C3D8" else 28)
        nx, ny, nz = n, max(3, n - rng.randint(0, n // 4)), max(3, n - rng.randint(0, n // 4))
        bc, more = "clamp", {"solve": rng.choice(["fp64", "mixed", "csr"])}
    else:
        top = {"assemble": 56, "force": 48, "energy": 48, "explicit": 40, "vjp": 40}[call]
        nx, ny, nz = (_log(rng, 3, top if elem == "C3D8" else top * 3 // 4) for _ in range(3))
        if call == "explicit":
            load, more = 0.0, {"steps": rng.randint(3, 20), "fp32": rng.random() < 0.4}
            bc = rng.choice(["free", "clamp", "roller"])
    c = case("", call, elem, nx, ny, nz, size, bc, numbering, load, **more)
    del c["name"]
    return c


# -- meshes and inputs -------------------------------------------------------------------------------------------------
class Model:
    """Nodes, elements, free DOFs, loaded faces, material and a displacement, all from (case, seed)."""

    def __init__(self, c, seed, which=0):
        rng = np.random.default_rng([seed, which])
        dims = [c["nx"], c["ny"], c["nz"]]
        if which:                                    # further requests of a batch: shorter beams
            dims = [max(4, dims[0] * (12 - which) // 12), max(2, dims[1] - which // 3), max(2, dims[2] - which // 2)]
        self.kind = kind = c["elem"]
        h = self.h = c["size"] / max(dims)
        ax = [np.arange(d + 1) for d in dims]
        ijk = np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
        X = ijk * h + rng.uniform(-0.1, 0.1, ijk.shape) * h
        X[:, 0] += 1.0 - dims[0] * h                 # the loaded plane lies near x = 1, off the origin
        ids = lambda a: (a[..., 0] * (dims[1] + 1) + a[..., 1]) * (dims[2] + 1) + a[..., 2]  # noqa: E731
        cell = np.stack(np.meshgrid(*[a[:-1] for a in ax], indexing="ij"), -1).reshape(-1, 1, 3)
        if kind == "C3D8":
            el = ids(cell + (SIGNS[None] + 1) // 2)
        else:
            paths = []
            for p in itertools.permutations(range(3)):
                at = np.zeros((4, 3), np.int64)
                for s, axis in enumerate(p):
                    at[s + 1:, axis] = 1
                odd = np.linalg.det(at[1:].astype(float)) < 0
                paths.append(at[[0, 2, 1, 3]] if odd else at)
            el = ids(cell[:, :, None] + np.stack(paths)[None]).reshape(-1, 4)
        first, last = ijk[:, 0] == 0, ijk[:, 0] == dims[0]
        faces = []                                   # (element, face id) on the loaded plane
        for f, loc in enumerate(FACES[kind]):
            e = np.nonzero(last[el[:, loc]].all(1))[0]
            if e.size:
                faces.append((e, f))
        if c["numbering"] == "runs":                 # runs of neighbouring nodes in another order, as meshers leave them
            N = len(X)
            order = np.concatenate([np.arange(N)[k * 48:(k + 1) * 48] for k in rng.permutation((N + 47) // 48)])
            new = np.empty(N, np.int64)
            new[order] = np.arange(N)
            X, el, first, last = X[order], new[el], first[order], last[order]
        self.X, self.el, self.faces, self.dims = X, el.astype(np.int64), faces, dims
        self.face_nodes = np.concatenate([self.el[e][:, FACES[kind][f]] for e, f in faces])
        self.mu = float(rng.uniform(0.9, 1.1))
        self.kappa = 20.0 * self.mu if kind == "C3D4" else 50.0 * self.mu
        self.p = c["load"] * float(rng.uniform(0.9, 1.1))
        self.held = {"clamp": (0, 1, 2), "roller": (0, 2), "free": ()}[c["bc"]]
        self.nodes_held = np.nonzero(first)[0]
        self.free = np.ones((len(X), 3), bool)
        for d in self.held:
            self.free[self.nodes_held, d] = False
        # a smooth bend and stretch of the block with nodal noise of a hundredth of an element
        s = ijk / np.array(dims)
        s = s[order] if c["numbering"] == "runs" else s
        a = rng.uniform(0.5, 1.0, 3)
        u = 0.03 * c["size"] * np.stack([a[0] * s[:, 0], a[1] * s[:, 0] ** 2, a[2] * np.sin(2 * s[:, 0]) * s[:, 1]], 1)
        u = u * min(1.0, 2.0 / c["size"]) + rng.normal(0, 0.01 * h, u.shape)
        self.gc = u[self.free]
        self.noise = rng.normal(0, 1.0, self.gc.shape)

    def assembly(self):
        X = self.X
        part = F.Part(X)
        e = getattr(F.elements, self.kind)(elems=self.el, elems_index=np.arange(len(self.el)), part=part)
        e.set_materials(F.materials.NeoHookean(self.mu, self.kappa))
        e.set_density(1.0)
        part.add_element(e)
        part.set_nodes["held"] = self.nodes_held
        part.add_surface_set("loaded", self.faces)
        asm = F.Assembly()
        asm.add_part(part, "body")
        asm.add_instance(F.Instance(part), "body")
        if self.p:
            asm.add_load(F.loads.Pressure("body", "loaded", self.p), "pressure")
        if self.held:
            asm.add_boundary(F.boundarys.Boundary_Condition("body", "held", indexDoF=self.held), "held")
        asm.initialize()
        return asm

    def dt(self):
        """Half the time a pressure wave takes through the smallest cell's shortest height (Kuhn tets: h / 2)."""
        c = math.sqrt(self.kappa + 4 * self.mu / 3)
        return 0.2 * self.h / c


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=DEV)


def prepare(c, seed):
    call = c["call"]
    if call == "batch":
        return _prepare_batch(c, seed)
    m = Model(c, seed)
    asm = m.assembly()
    s = dict(case=c, asm=asm, gc=_dev(m.gc))
    if call == "energy":
        s["solver"] = F.solver.StaticImplicitSolver()
        s["solver"].initialize(asm)
    elif call == "pcg":
        R, s["K"] = asm.assemble_csr(torch.zeros_like(s["gc"]))
        s["b"] = -R
    elif call == "explicit":
        s["dt"] = m.dt()
        s["v0"] = _dev(0.01 * m.noise)
        s["gc"] = 0.1 * s["gc"]
        s["solver"] = F.solver.DynamicExplicitSolver(time_end=(c["steps"] - 0.5) * s["dt"], time_per_storage=1e9,
                                                     fp32=c["fp32"])
        s["solver"].initialize(asm)
        s["solver"]._deltaT = s["dt"]
    elif call == "vjp":
        s["lam"] = _dev(m.gc + 0.1 * m.h * m.noise)
    elif call == "newton":
        s["solver"] = F.solver.StaticImplicitSolver(rtol=1e-8, maximum_iteration=100)
        s["solver"].initialize(asm)
        s["gc"] = torch.zeros_like(s["gc"])
    return s


def _prepare_batch(c, seed):
    systems = []
    for k in range(c["slots"]):
        asm = Model(c, seed, k).assembly()
        gc = torch.zeros(asm.plan.ndof, dtype=F64, device=DEV)
        R, K = asm.assemble_csr(gc)
        lin = LinearSolve(K, (-R).contiguous(), gc, PCG_TOL, 20000, True)
        work = torch.empty(serving.BatchedPCG.work_len(asm.plan), dtype=F64, device=DEV)
        systems.append((asm, lin, work))
    items = c["slots"] * max((a.plan.n_nodes + 15) // 16 + 1 for a, _, _ in systems)
    return dict(case=c, systems=systems, eng=serving.BatchedPCG(c["slots"], items))


# -- one pass ----------------------------------------------------------------------------------------------------------
def run(s):
    c = s["case"]
    call, asm = c["call"], s.get("asm")
    if call == "assemble":
        R, _, K = asm.assemble_Stiffness_Matrix(GC=s["gc"])      # (the pattern is the plan's, constant)
        return {"R": R, "K": K}
    if call == "force":
        return {"R": asm.assemble_force(GC=s["gc"])}
    if call == "energy":
        return {"E": s["solver"].get_total_energy(s["gc"])}
    if call == "pcg":
        x, P = torch.zeros_like(s["b"]), asm.plan
        if c["solve"] == "mixed":
            P.pcg_mixed(s["K"], None, s["b"], x, PCG_TOL, 0.0, 20000, check_every=50)
        else:
            P.pcg(s["K"], s["b"], x, PCG_TOL, 20000, check_every=50, generic=c["solve"] == "csr")
        return {"x": x}
    if call == "explicit":
        sol = s["solver"]
        sol._GC_list, sol._GV_list, sol._GA_list, sol._time_list = [], [], [], []   # a new history, the mass kept
        sol._next_storage_time = 0.0
        sol.solve(GC0=s["gc"], GV0=s["v0"])
        return {"u": sol.GC, "v": sol.GV, "a": sol.GA}
    if call == "vjp":
        dX, dmu = adjoint.residual_vjp(asm, s["gc"], s["lam"])
        return {"dX": dX, "dmu": dmu[0]}
    if call == "newton":
        return {"gc": s["solver"].solve(GC0=s["gc"])}
    eng = s["eng"]                                               # batch
    for k, (a, lin, work) in enumerate(s["systems"]):
        lin.x.zero_()
        eng.assign(k, a.plan, lin, work)
    eng.sync()
    for k in range(c["slots"]):
        eng.start(k)
    while True:
        eng.run_round()
        eng.poll_async()
        if (eng.wait()[:, 0] != 0).all():
            break
    return [lin.x for _, lin, _ in s["systems"]]


# -- what a pass cannot do without -------------------------------------------------------------------------------------
def _counts(c):
    """Elements, nodes, free DOFs, node pairs sharing an element (both ordered), loaded faces."""
    d = [c["nx"], c["ny"], c["nz"]]
    if c["call"] == "batch":
        d[0] = d[0] * 5 // 6
    N = math.prod(x + 1 for x in d)
    if c["elem"] == "C3D8":
        E, pairs = math.prod(d), math.prod(3 * x + 1 for x in d)
    else:
        E = 6 * math.prod(d)
        offs = {o for o in itertools.product((0, 1), repeat=3)}
        offs |= {tuple(-x for x in o) for o in offs}
        pairs = sum(math.prod(x + 1 - abs(y) for x, y in zip(d, o)) for o in offs)
    held = {"clamp": 3, "roller": 2, "free": 0}[c["bc"]] * (d[1] + 1) * (d[2] + 1)
    faces = d[1] * d[2] * (1 if c["elem"] == "C3D8" else 2)
    return E, N, 3 * N - held, pairs, faces


def work(c):
    E, N, n, pairs, faces = _counts(c)
    nn, ng = (8, 8) if c["elem"] == "C3D8" else (4, 1)
    mesh = 4 * nn * E + 24 * N                          # connectivity and coordinates
    nnz = 9 * pairs * n / (3 * N)
    kin = E * ng * (36 * nn + 150)                      # displacement gradient, F, its inverse and determinant
    call = c["call"]
    if call == "assemble":
        # the upper node blocks: 3 multiply-adds an entry, 9 entries a block
        return {"bytes": mesh + 16 * n + 8 * nnz, "flops": kin + E * ng * (nn * (nn + 1) // 2 * 66 + 30 * nn)}
    if call == "force":
        return {"bytes": mesh + 16 * n, "flops": kin + E * ng * 30 * nn}
    if call == "energy":
        return {"bytes": mesh + 8 * n, "flops": kin}
    if call == "vjp":
        return {"bytes": mesh + 16 * n + 24 * N, "flops": 2 * kin + E * ng * 300}
    if call == "explicit":
        return {"bytes": (c["steps"] + 1) * (mesh + 56 * n), "flops": (c["steps"] + 1) * (kin + E * ng * 30 * nn)}
    # iterations of the Jacobi-PCG to 1e-8 grow with the cells along the body
    its = (62 if c["elem"] == "C3D8" else 45) * max(c["nx"], c["ny"], c["nz"]) ** (1.0 if c["size"] == 1.0 else 0.9)
    value = 4 if c.get("solve") == "mixed" else 8
    per_it = value * nnz + 4 * pairs + 10 * value * n
    if call == "newton":
        its, per_it = 6 * its, per_it
    slots = c.get("slots", 1)
    return {"bytes": slots * its * per_it, "flops": slots * its * (2 * nnz + 12 * n)}


def tolerance(c):
    if c["call"] in ("pcg", "batch", "newton"):
        # both sides stop at a relative residual of 1e-8 in the scaled norm, at iterates of their own (up to 1.1e-7
        # off the exact solution)
        return {"rel": 5e-7}
    if c["call"] == "explicit":
        return {"rel": 1.4e-4 if c["fp32"] else 4e-13}
    return {"rel": 1e-13}                               # at most 1.4e-14 off in 64 bits


# -- the same in 64 bits, by numpy and torch ---------------------------------------------------------------------------
def _tables(kind):
    """dN/dxi [g, nn, 3], weights [g], N [g, nn]."""
    if kind == "C3D4":
        d = np.array([[[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]]], float)
        return _dev(d), _dev(np.array([1 / 6])), _dev(np.full((1, 4), 0.25))
    g, d, N = SIGNS / math.sqrt(3), np.empty((8, 8, 3)), np.empty((8, 8))
    for k in range(8):
        f = 1 + SIGNS * g[k]
        N[k] = f.prod(1) / 8
        for m in range(3):
            d[k, :, m] = SIGNS[:, m] * f[:, [i for i in range(3) if i != m]].prod(1) / 8
    return _dev(d), _dev(np.ones(8)), _dev(N)


def _gauss(X, U, dxi, w):
    """F, g_a = dN_a/dX and w detJ0 of elements at one Gauss point."""
    J0 = torch.einsum("eai,am->eim", X, dxi)
    det = torch.linalg.det(J0)
    g = torch.einsum("am,emi->eai", dxi, torch.linalg.inv(J0))
    return torch.eye(3, dtype=F64, device=X.device) + torch.einsum("eai,eaj->eij", U, g), g, w * det


def _element(X, U, kind, mu, kappa, want):
    """Energy [e], residual [e, nn, 3] or (residual, tangent [e, nn, 3, nn, 3]) of elements."""
    dxi, w, _ = _tables(kind)
    E = R = K = 0
    for k in range(len(w)):
        Fg, g, wk = _gauss(X, U, dxi[k], w[k])
        J = torch.linalg.det(Fg)
        Jm, IC = J ** (-2.0 / 3.0), (Fg * Fg).sum((1, 2))
        if want == "energy":
            E = E + wk * (mu / 2 * (Jm * IC - 3) + kappa / 2 * (J - 1) ** 2)
            continue
        q = torch.einsum("eai,eij->eaj", g, torch.linalg.inv(Fg))     # F^-T g
        f = torch.einsum("eij,eaj->eai", Fg, g)
        m, b = wk * mu * Jm, wk * kappa * J
        R = R + m[:, None, None] * (f - IC[:, None, None] / 3 * q) + (b * (J - 1))[:, None, None] * q
        if want == "tangent":
            z = lambda s: s[:, None, None, None, None]  # noqa: E731
            qq = torch.einsum("eai,ebj->eaibj", q, q)
            fq = torch.einsum("eai,ebj->eaibj", q, f) + torch.einsum("eai,ebj->eaibj", f, q)
            gg = torch.einsum("eak,ebk,ij->eaibj", g, g, torch.eye(3, dtype=F64, device=g.device))
            K = K + (z(m) * (gg - 2 / 3 * fq) + z(m * IC * 2 / 9 + b * (2 * J - 1)) * qq
                     + z(m * IC / 3 - b * (J - 1)) * qq.permute(0, 1, 4, 3, 2))
    return E if want == "energy" else R if want == "force" else (R, K)


def _volume(x):
    """Enclosed-volume integral of one face [nf, 3]: 1/3 int x . n dA."""
    if x.shape[0] == 3:
        pts, w = [(1 / 6, 1 / 6), (2 / 3, 1 / 6), (1 / 6, 2 / 3)], 1 / 6
        tab = [([1 - a - b, a, b], [-1, 1, 0], [-1, 0, 1]) for a, b in pts]
    else:
        s, w = [(-1, -1), (1, -1), (1, 1), (-1, 1)], 1.0
        tab = [([(1 + p * a) * (1 + q * b) / 4 for p, q in s], [p * (1 + q * b) / 4 for p, q in s],
                [q * (1 + p * a) / 4 for p, q in s]) for a, b in ((u / math.sqrt(3), v / math.sqrt(3)) for u, v in s)]
    v = 0
    for rows in tab:
        r = torch.tensor(rows, dtype=F64, device=x.device) @ x
        v = v + w / 3 * torch.dot(r[0], torch.linalg.cross(r[1], r[2]))
    return v


class Exact:
    def __init__(self, c, seed, which=0):
        self.m = m = Model(c, seed, which)
        self.X, self.el, self.fn = _dev(m.X), _dev(m.el), _dev(m.face_nodes)
        self.free = _dev(m.free).reshape(-1)
        self.num = torch.cumsum(self.free.long(), 0) - 1
        self.n = int(self.free.sum())
        self.gc = _dev(m.gc)
        self.step = 20000 if m.kind == "C3D8" else 200000

    def full(self, v):
        out = torch.zeros(self.X.numel(), dtype=F64, device=DEV)
        out[self.free] = v
        return out.view(-1, 3)

    def dofs(self, nodes):
        return (3 * nodes[:, :, None] + torch.arange(3, device=DEV)).reshape(nodes.shape[0], -1)

    def chunks(self):
        return self.el.split(self.step)

    def energy(self, gc):
        U = self.full(gc)
        e = sum(_element(self.X[k], U[k], self.m.kind, self.m.mu, self.m.kappa, "energy").sum() for k in self.chunks())
        if self.m.p:
            e = e + self.m.p * torch.func.vmap(_volume)((self.X + U)[self.fn]).sum()
        return e

    def force(self, gc, X=None, mu=None):
        X, mu, U = self.X if X is None else X, self.m.mu if mu is None else mu, self.full(gc)
        R = torch.zeros_like(X)
        for k in self.chunks():
            R = R.index_add(0, k.reshape(-1), _element(X[k], U[k], self.m.kind, mu, self.m.kappa, "force").reshape(-1, 3))
        if self.m.p:
            f = torch.func.vmap(torch.func.grad(_volume))((X + U)[self.fn])
            R = R.index_add(0, self.fn.reshape(-1), self.m.p * f.reshape(-1, 3))
        return R.reshape(-1)[self.free]

    def tangent(self, gc):
        """(indptr, columns, values) of the reduced tangent, columns sorted."""
        U, keys, vals = self.full(gc), [], []

        def add(dofs, blocks):
            r = dofs[:, :, None].expand(-1, -1, dofs.shape[1]).reshape(-1)
            q = dofs[:, None, :].expand(-1, dofs.shape[1], -1).reshape(-1)
            ok = self.free[r] & self.free[q]
            k, at = torch.unique(self.num[r[ok]] * self.n + self.num[q[ok]], return_inverse=True)
            keys.append(k)
            vals.append(torch.zeros(len(k), dtype=F64, device=DEV).index_add(0, at, blocks.reshape(-1)[ok]))
        for k in self.chunks():
            add(self.dofs(k), _element(self.X[k], U[k], self.m.kind, self.m.mu, self.m.kappa, "tangent")[1])
        if self.m.p:
            add(self.dofs(self.fn), self.m.p * torch.func.vmap(torch.func.hessian(_volume))((self.X + U)[self.fn]))
        k, at = torch.unique(torch.cat(keys), return_inverse=True)
        v = torch.zeros(len(k), dtype=F64, device=DEV).index_add(0, at, torch.cat(vals))
        ptr = torch.searchsorted(k, torch.arange(self.n + 1, device=DEV) * self.n)
        return ptr, k % self.n, v

    def solve(self, K, b, tol=1e-26, cap=60000):
        ptr, col, v = K
        A = torch.sparse_csr_tensor(ptr, col, v, (self.n, self.n), check_invariants=False)
        rows = torch.repeat_interleave(torch.arange(self.n, device=DEV), ptr[1:] - ptr[:-1])
        dinv = 1 / v[rows == col].abs()
        x, r = torch.zeros_like(b), b.clone()
        z = r * dinv
        p, rz = z.clone(), torch.dot(r, z)
        stop = tol * float(rz)
        for it in range(cap):
            if it % 50 == 0 and float(rz) <= stop:
                break
            q = A @ p
            a = rz / torch.dot(p, q)
            x += a * p
            r -= a * q
            z = r * dinv
            new = torch.dot(r, z)
            p, rz = z + new / rz * p, new
        return x

    def newton(self):
        gc = torch.zeros(self.n, dtype=F64, device=DEV)
        first, best = None, None
        for _ in range(60):
            R = self.force(gc)
            rn = float(R.norm())
            first = rn if first is None else first
            if best is not None and rn > 0.5 * best and best < 1e-9 * first:
                break
            best = rn if best is None else min(best, rn)
            d, a, E = -self.solve(self.tangent(gc), R), 1.0, float(self.energy(gc))
            slope = float(torch.dot(d, R))
            while float(self.energy(gc + a * d)) > E + 0.3 * a * slope + 1e-10 * abs(E) and a > 1e-9:
                a /= 2
            gc = gc + a * d
        return gc

    def explicit(self, steps, dt):
        m = self.m
        dxi, w, N = _tables(m.kind)
        mass = torch.zeros_like(self.X)
        free = self.free.view(-1, 3).double()
        for k in self.chunks():
            me = 0
            for g in range(len(w)):
                wk = w[g] * torch.linalg.det(torch.einsum("eai,am->eim", self.X[k], dxi[g]))
                me = me + wk[:, None, None] * N[g][None, :, None] * torch.einsum("b,ebd->ed", N[g], free[k])[:, None]
            mass = mass.index_add(0, k.reshape(-1), me.reshape(-1, 3))
        mass = mass.reshape(-1)[self.free]
        u, v = 0.1 * self.gc, 0.01 * _dev(m.noise)
        a = -self.force(u) / mass
        vh = v - 0.5 * dt * a
        for _ in range(steps):
            old = vh
            vh = vh + dt * a
            u = u + dt * vh
            a = -self.force(u) / mass
            v = 0.5 * (vh + old)
        return u, v, a


def exact(c, seed):
    if c["call"] == "batch":
        out = []
        for k in range(c["slots"]):
            e = Exact(c, seed, k)
            z = torch.zeros(e.n, dtype=F64, device=DEV)
            out.append(e.solve(e.tangent(z), -e.force(z)))
        return out
    e = Exact(c, seed)
    if c["call"] == "assemble":
        return {"R": e.force(e.gc), "K": e.tangent(e.gc)[2]}
    if c["call"] == "force":
        return {"R": e.force(e.gc)}
    if c["call"] == "energy":
        return {"E": e.energy(e.gc)}
    if c["call"] == "pcg":
        z = torch.zeros(e.n, dtype=F64, device=DEV)
        return {"x": e.solve(e.tangent(z), -e.force(z))}
    if c["call"] == "explicit":
        return dict(zip("uva", e.explicit(c["steps"], e.m.dt())))
    if c["call"] == "newton":
        return {"gc": e.newton()}
    lam = _dev(e.m.gc + 0.1 * e.m.h * e.m.noise)                 # vjp
    X, mu = e.X.clone(), torch.tensor(e.m.mu, dtype=F64, device=DEV)
    dX, dmu, U, lf = torch.zeros_like(X), torch.zeros_like(mu), e.full(e.gc), e.full(lam)
    for k in e.chunks():
        Xe, me = X[k].requires_grad_(True), mu.clone().requires_grad_(True)
        # dkappa/dmu is not part of it: the two are separate parameters
        phi = (_element(Xe, U[k], e.m.kind, me, e.m.kappa, "force") * lf[k]).sum()
        gX, gm = torch.autograd.grad(phi, (Xe, me))
        dX.index_add_(0, k.reshape(-1), gX.reshape(-1, 3))
        dmu += gm
    if e.m.p:
        H = torch.func.vmap(torch.func.hessian(_volume))((X + U)[e.fn])
        hv = e.m.p * torch.einsum("faibj,fbj->fai", H, lf[e.fn])
        dX.index_add_(0, e.fn.reshape(-1), hv.reshape(-1, 3))
    return {"dX": dX, "dmu": dmu}

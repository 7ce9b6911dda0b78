"""Workloads of the elastic DG solver: what a program has it do, over the
orders, sizes, mesh forms and options it is used with.

A case is one of
  step      a domain stepped by its LSRK integrator (state on the device),
            with or without a read of the discrete energy
  solve     initial fields from host memory, steps, fields back to the host
  shot      a point-source solve on a domain that is kept: zero state, a new
            source and new receivers, steps, seismograms back to the host
  ensemble  independent adapted domains of mixed orders stepped in one batch
  serve     a chunk of the solve server: conforming bricks with sources and
            receivers, stepped in one batch
  glued     two halves of a brick, each of its own order, stepped together

The inputs (mesh, material law, pulse, time step) are those of
bfam_b200.configs and bfam_b200.serving.  exact() evaluates the same
semi-discretisation and time integrator in 64 bits with torch.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import bfam_b200 as bf
from bfam_b200 import configs

METHODS = {"kc54": bf.LSRK_KC54, "w33": bf.LSRK_W33, "heun": bf.LSRK_HEUN}
PRECISIONS = {"fp64": bf.PRECISION_FP64, "fp32": bf.PRECISION_FP32}


def _case(kind, dim, N, n, steps, **more):
    c = {"kind": kind, "dim": dim, "N": N, "nx": n[0], "ny": n[1],
         "nz": n[2] if dim == 3 else 1, "steps": steps, "refine": 0.3,
         "precision": "fp64", "flux": "upwind", "bounded": False,
         "method": "kc54", "graph": True, "energy": False, "count": 1, "N2": N}
    c.update(more)
    return c


def listed():
    return [
        # a 2D conforming brick with a plane wave, stepped as the library
        # does by default (eager launches): the smallest problem, where the
        # latency of a launch counts (configs.cfg0)
        _case("step", 2, 4, (16, 16), 20, refine=0.0, graph=False, name="wave-2d-n4"),
        # a 2D plate with absorbing sides and a free surface, adapted
        _case("step", 2, 3, (200, 150), 5, bounded=True, name="plate-2d-n3"),
        # low order on a ragged adapted brick
        _case("step", 3, 2, (37, 29, 23), 4, name="brick-3d-n2"),
        # one shot of a survey: the request of the solve server, solved alone
        _case("shot", 3, 3, (12, 12, 12), 100, refine=0.0, name="shot-3d-n3"),
        # an adapted bounded basin with its energy watched
        _case("step", 3, 4, (22, 19, 13), 5, bounded=True, energy=True,
              name="basin-3d-n4"),
        # the headline problem (configs.cfg1)
        _case("step", 3, 5, (32, 32, 32), 1, name="adapted-3d-n5"),
        # the precision form at the highest order (configs.cfg2's mesh family)
        _case("step", 3, 7, (24, 24, 24), 1, precision="fp32", name="adapted-3d-n7-fp32"),
        # the plain form at the highest order, mid-sized
        _case("step", 3, 7, (11, 12, 9), 2, name="adapted-3d-n7"),
        # a whole small solve from and to host memory
        _case("solve", 3, 5, (7, 6, 5), 60, precision="fp32", name="solve-3d-n5-fp32"),
        # an ensemble of instances of orders 3, 5, 7 (configs.cfg3)
        _case("ensemble", 3, 0, (5, 14, 0), 2, refine=0.2, precision="fp32", count=14,
              name="ensemble-3d-fp32"),
        # the server's batch between two arrivals (bfam_b200.serving)
        _case("serve", 3, 0, (8, 24, 0), 10, refine=0.0, precision="fp32", count=9,
              name="serve-3d-fp32"),
        # two orders joined along x
        _case("glued", 3, 3, (8, 16, 16), 2, refine=0.0, N2=5, name="glued-3d-n3-n5"),
    ]


def draw(rng: random.Random):
    kind = rng.choice(["step"] * 7 + ["solve", "shot", "ensemble", "serve", "glued"])
    precision = rng.choice(["fp64", "fp64", "fp32"])
    if kind == "ensemble":
        lo = rng.randint(3, 6)
        return _case(kind, 3, 0, (lo, lo + rng.randint(2, 8), 0), rng.randint(1, 4),
                     refine=0.2, precision=precision, count=rng.randint(3, 12))
    if kind == "serve":
        return _case(kind, 3, 0, (8, rng.randint(10, 24), 0), rng.randint(2, 12),
                     refine=0.0, precision="fp32", count=rng.randint(2, 9))
    dim = 3 if kind in ("shot", "glued") else rng.choice([2, 3, 3])
    if kind == "shot":
        N = rng.choice([3, 5])
    else:
        N = rng.randint(1, 8 if dim == 2 else 7)
    refine = rng.choice([0.0, 0.2, 0.3, 0.5]) if kind in ("step", "solve") else 0.0
    # base cells for a number of degrees of freedom spread over its logarithm
    top = {"step": 1e8, "solve": 4e6, "shot": 8e6, "glued": 3e7}[kind]
    dofs = math.exp(rng.uniform(math.log(2e4), math.log(top)))
    per_cell = (9 if dim == 3 else 5) * (N + 1) ** dim * (1 + (2 ** dim - 1) * refine)
    side = (dofs / per_cell) ** (1.0 / dim)
    n = [max(2, int(side * rng.uniform(0.8, 1.25))) for _ in range(dim)]
    steps = max(1, min(40, int(3e7 / dofs)))
    return _case(kind, dim, N, n, steps, refine=refine, precision=precision,
                 flux=rng.choice(["upwind", "upwind", "upwind", "central"]),
                 bounded=kind in ("step", "solve") and rng.random() < 0.4,
                 method=rng.choice(["kc54", "kc54", "w33", "heun"]) if kind == "step" else "kc54",
                 graph=kind != "step" or rng.random() < 0.7,
                 energy=kind == "step" and rng.random() < 0.2,
                 N2=rng.choice([3, 5, 7]) if kind == "glued" else N)


# ------------------------------------------------------------------- inputs

def _bc(dim):
    """absorbing sides, a free surface on the last axis's top"""
    return (bf.BC_ABSORBING,) * (2 * dim - 1) + (bf.BC_FREE_SURFACE,)


def _domain(dim, N, n, refine, mesh_seed, seed, bounded=False, bc=None, periodic=None,
            L=(1.0, 1.0, 1.0)):
    """mesh, material, initial fields and time step of one domain"""
    periodic = periodic or ((not bounded,) * 3)
    mesh = bf.Mesh(dim, N, n[:dim], L=L, refine_prob=refine, seed=mesh_seed, periodic=periodic)
    rho, lam, mu = bf.material_random(mesh.K, seed)
    r = bf.lgl_operators(N)[0]
    g = np.random.default_rng(seed)
    q0 = mesh.gaussian_pulse(r, g.uniform(0.3, 0.7, 3) * np.array(L), 0.12)
    return {"mesh": mesh, "rho": rho, "lam": lam, "mu": mu, "q0": q0,
            "bc": bc if bc is not None else _bc(dim),
            "dt": configs.stable_dt(mesh, rho, lam, mu, 0.4)}


def _shot(dims, seed, d):
    """a Ricker point source and 16 receivers (the server's request law)"""
    g = np.random.default_rng(seed + 77)
    f0 = g.uniform(5.0, 15.0)
    force = g.standard_normal(3)
    d.update(x=g.uniform(0, 1, 3), force=force / np.linalg.norm(force), f0=f0, t0=1.2 / f0,
             recv=g.uniform(0, 1, (16, 3)))
    return d


def _inputs(case, seed):
    dim, N, kind = case["dim"], case["N"], case["kind"]
    n = (case["nx"], case["ny"], case["nz"])
    if kind in ("step", "solve"):
        d = _domain(dim, N, n, case["refine"], 0, seed, case["bounded"])
        if case["refine"] == 0.0 and not case["bounded"]:
            # a homogeneous medium and a plane wave
            g = np.random.default_rng(seed)
            for k, v in (("rho", 1.0), ("lam", 2.0), ("mu", 1.0)):
                d[k] = np.full(d["mesh"].K, v)
            wave = 2 * math.pi * g.integers(1, 3, dim)
            d["q0"] = d["mesh"].plane_wave(bf.lgl_operators(N)[0], wave, g.uniform(0.5, 2.0),
                                           1.0, 2.0, 1.0, 0.0)
            d["dt"] = configs.stable_dt(d["mesh"], 1.0, 2.0, 1.0, 0.4)
        return [d]
    if kind == "shot":
        d = _shot(dim, seed, _domain(dim, N, n, case["refine"], 0, seed))
        d["q0"] = np.zeros_like(d["q0"])
        return [d]
    g = random.Random(case["count"])  # the domains' sizes belong to the case
    if kind == "ensemble":
        out = []
        for i in range(case["count"]):
            side = [g.randint(case["nx"], case["ny"]) for _ in range(2)]
            out.append(_domain(3, (3, 5, 7)[i % 3], (side[0], side[0], side[1]),
                               case["refine"], i, seed + 1000 * i))
        return out
    if kind == "serve":
        out = []
        for i in range(case["count"]):
            m = g.randint(case["nx"], case["ny"])
            d = _domain(3, (3, 5)[i % 2], (m, m, m), 0.0, 0, seed + 1000 * i)
            out.append(_shot(3, seed + 1000 * i, d))
        return out
    # glued along x, free surfaces on the other sides
    bc = (bf.BC_GLUED,) * 2 + (bf.BC_FREE_SURFACE,) * 4
    out = []
    for i, order in enumerate((N, case["N2"])):
        out.append(_domain(3, order, n, case["refine"], 0, seed + 1000 * i, bc=bc,
                           periodic=(False, True, True), L=(0.5, 1.0, 1.0)))
    dt = min(d["dt"] for d in out)
    for d in out:
        d["dt"] = dt
    return out


class _DeviceArray:
    """a domain's stacked fields as a CUDA array (keeps the domain)"""

    def __init__(self, dom, ptr):
        self.dom = dom
        shape = (dom.nfields, dom.field_length)
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape,
                                         "typestr": "<f8", "version": 3}


class _Fields:
    """the domain's current state as a tensor on the device"""

    def __init__(self, dom):
        self.dom, self.views = dom, {}

    def __call__(self):
        ptr = self.dom.field_device_ptr(0)
        if ptr not in self.views:
            self.views[ptr] = torch.as_tensor(_DeviceArray(self.dom, ptr), device="cuda")
        return self.views[ptr]


def prepare(case, seed):
    inputs = _inputs(case, seed)
    flux = bf.FLUX_CENTRAL if case["flux"] == "central" else bf.FLUX_UPWIND
    doms = []
    for d in inputs:
        dom = bf.GpuDomain(d["mesh"], d["rho"], d["lam"], d["mu"], flux=flux,
                           precision=PRECISIONS[case["precision"]], bc=d["bc"])
        dom.set_fields(d["q0"])
        doms.append(dom)
    state = {"case": case, "inputs": inputs, "doms": doms,
             "fields": [_Fields(dom) for dom in doms]}
    if case["kind"] in ("step", "solve"):
        state["ts"] = bf.LSRK(doms[0], METHODS[case["method"]])
        state["out"] = np.empty((doms[0].nfields, doms[0].field_length))
    elif case["kind"] != "shot":
        if case["kind"] == "serve":
            for dom, d in zip(doms, inputs):
                dom.set_source(d["x"], d["force"], d["f0"], d["t0"])
                dom.set_receivers(d["recv"], 20000)
        batch = bf.Batch(doms, t0=0.0)
        if case["kind"] == "glued":
            pairs = bf.glued_x_pairs(inputs[0]["mesh"], inputs[1]["mesh"])
            state["glue"] = bf.PGlue(doms[0], doms[1], *pairs)
            batch.add_pglue(state["glue"])
        state["batch"] = batch
        state["dts"] = np.array([d["dt"] for d in inputs])
    return state


def run(state):
    case, d, dom = state["case"], state["inputs"][0], state["doms"][0]
    kind = case["kind"]
    if kind == "step":
        state["ts"].step(d["dt"], case["steps"], use_graph=case["graph"])
        q = state["fields"][0]()
        return (q, dom.energy()) if case["energy"] else q
    if kind == "solve":
        dom.set_fields(d["q0"])
        state["ts"].step(d["dt"], case["steps"], use_graph=True)
        return dom.get_fields(state["out"])
    if kind == "shot":
        dom.set_fields(d["q0"])
        dom.set_source(d["x"], d["force"], d["f0"], d["t0"])
        dom.set_receivers(d["recv"], case["steps"])
        ts = bf.LSRK(dom)
        ts.step(d["dt"], case["steps"], use_graph=True)
        seismograms = dom.seismograms()
        ts.free()
        return seismograms, state["fields"][0]()
    state["batch"].step(state["dts"], case["steps"])
    return [f() for f in state["fields"]]


def _elements(dim, n, refine):
    return np.prod(n[:dim]) * (1 + (2 ** dim - 1) * refine)


def work(case):
    """Bytes: per stage the state and the increment, each read once and
    written once (the increment is not read by the first stage); per energy a
    read of the state; per host transfer the fields.  Operations: the
    one-dimensional derivatives, two per coefficient."""
    dim = case["dim"]
    stages = {"kc54": 5, "w33": 3, "heun": 2}[case["method"]]
    if case["kind"] in ("ensemble", "serve"):
        g = random.Random(case["count"])
        parts = []
        for i in range(case["count"]):
            if case["kind"] == "ensemble":
                side = [g.randint(case["nx"], case["ny"]) for _ in range(2)]
                parts.append(((3, 5, 7)[i % 3], (side[0], side[0], side[1]), case["refine"]))
            else:
                m = g.randint(case["nx"], case["ny"])
                parts.append(((3, 5)[i % 2], (m, m, m), 0.0))
    else:
        n = (case["nx"], case["ny"], case["nz"])
        parts = [(case["N"], n, case["refine"])]
        if case["kind"] == "glued":
            parts.append((case["N2"], n, case["refine"]))
    nbytes = flops = 0.0
    for N, n, refine in parts:
        nodes = _elements(dim, n, refine) * (N + 1) ** dim
        dofs = nodes * (9 if dim == 3 else 5)
        nbytes += case["steps"] * dofs * (32.0 * stages - 8.0)
        flops += case["steps"] * stages * nodes * (18 if dim == 3 else 8) * 2 * (N + 1)
        if case["energy"]:
            nbytes += 8.0 * dofs
        if case["kind"] == "solve":
            nbytes += 16.0 * dofs
        if case["kind"] == "shot":
            nbytes += 8.0 * dofs
    return {"bytes": float(nbytes), "flops": float(flops)}


# ---------------------------------------------------- the answer in 64 bits

KC54_A = (0.0, -567301805773 / 1357537059087, -2404267990393 / 2016746695238,
          -3550918686646 / 2091501179385, -1275806237668 / 842570457699)
KC54_B = (1432997174477 / 9575080441755, 5161836677717 / 13612068292357,
          1720146321549 / 2090206949498, 3134564353537 / 4481467310338,
          2277821191437 / 14882151754819)
KC54_C = (0.0, 1432997174477 / 9575080441755, 2526269341429 / 6820363962896,
          2006345519317 / 3224310063776, 2802321613138 / 2924317926251)
TABLES = {"kc54": (KC54_A, KC54_B, KC54_C),
          "w33": ((0.0, -5 / 9, -153 / 128), (1 / 3, 15 / 16, 8 / 15), (0.0, 1 / 3, 3 / 4)),
          "heun": ((0.0, -1.0), (1.0, 0.5), (0.0, 1.0))}


def _lgl(N):
    """Legendre-Gauss-Lobatto nodes and weights"""
    leg = np.polynomial.legendre.Legendre.basis(N)
    x = np.concatenate([[-1.0], np.sort(leg.deriv().roots().real), [1.0]]) if N > 1 \
        else np.array([-1.0, 1.0])
    for _ in range(3):  # polish the interior nodes
        if N > 1:
            x[1:-1] -= leg.deriv()(x[1:-1]) / leg.deriv(2)(x[1:-1])
    return x, 2.0 / (N * (N + 1) * leg(x) ** 2)


def _lagrange(nodes, at):
    """[at, nodes] values of the Lagrange basis"""
    out = np.ones((len(at), len(nodes)))
    for i in range(len(nodes)):
        for m in range(len(nodes)):
            if m != i:
                out[:, i] *= (at - nodes[m]) / (nodes[i] - nodes[m])
    return out


def _derivative(nodes):
    c = np.array([np.prod([a - b for b in nodes if b != a]) for a in nodes])
    D = np.zeros((len(nodes),) * 2)
    for i in range(len(nodes)):
        for j in range(len(nodes)):
            if i != j:
                D[i, j] = c[i] / (c[j] * (nodes[i] - nodes[j]))
        D[i, i] = -D[i].sum()
    return D


def _projection(src, dst, at, jac):
    """L2 projection to the basis on `dst` of a function on `src` whose
    nodes lie at at(src nodes) with Jacobian jac"""
    x, w = np.polynomial.legendre.leggauss(max(len(src), len(dst)) + 1)
    Ld = _lagrange(dst, x)
    M = Ld.T @ (w[:, None] * Ld)
    return np.linalg.solve(M, jac * _lagrange(dst, at(x)).T @ (w[:, None] * _lagrange(src, x)))


class _Exact:
    """The semi-discrete operator of one domain in float64: tensor-product
    LGL derivatives, upwind or central flux, lumped lift, L2 mortars."""

    def __init__(self, d, central, device):
        m = d["mesh"]
        self.d, self.m, self.dim, self.N, self.Nq = d, m, m.dim, m.N, m.Nq
        self.K, self.central, self.dev = m.K, central, device
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=device)  # noqa: E731
        self.t = t
        self.r, self.w = _lgl(m.N)
        self.D = t(_derivative(self.r))
        halves = [lambda x: 0.5 * (x - 1), lambda x: 0.5 * (x + 1)]
        self.I = [t(_lagrange(self.r, h(self.r))) for h in halves]
        self.P = [t(_projection(self.r, self.r, h, 0.5)) for h in halves]
        self.rho, self.lam, self.mu = t(d["rho"]), t(d["lam"]), t(d["mu"])
        self.Zp = torch.sqrt(self.rho * (self.lam + 2 * self.mu))
        self.Zs = torch.sqrt(self.rho * self.mu)
        self.rx = t(2.0 / m.h[:, :m.dim])
        NF, Nfp = m.Nfaces, m.Nfp
        vP = m.vmapP.reshape(m.K, NF, Nfp)
        vM = m.vmapM.reshape(m.K, NF, Nfp)
        self.gmask = [t(vM[0, f].astype(np.int64)) for f in range(NF)]
        joined = (vP != vM).any(axis=2)
        for e, f in zip(m.EToEb, m.EToFb):
            joined[e, f] = False
        self.conf = []
        for f in range(NF):
            e = np.flatnonzero(joined[:, f])
            self.conf.append((t(e), t(vP[e, f, 0].astype(np.int64) // m.Np)))
        self.bnd = []
        bc = d["bc"]
        for f in range(NF):
            self.bnd.append((t(m.EToEb[m.EToFb == f].astype(np.int64)), bc[f]))
        # hanging faces by face and piece: (coarse, fine, face of the coarse)
        h = m.EToHm
        self.hang = []
        for f in range(NF):
            for p in range(1, (4 if m.dim == 3 else 2) + 1):
                g = np.flatnonzero((m.EToFm == f) & (h == p))
                if len(g):
                    self.hang.append((f, p, t(m.EToEm[g].astype(np.int64)),
                                      t(m.EToEm[m.EToEp[g]].astype(np.int64))))

    def trace_fields(self, ax):
        if self.dim == 3:
            return [0, 1, 2] + [[3, 6, 7], [6, 4, 8], [7, 8, 5]][ax]
        return [0, 1] + [[2, 4], [4, 3]][ax]

    def traces(self, q, e, f):
        """[2 dim, faces, Nfp] velocity and stress row normal to face f"""
        idx = (e * self.m.Np)[:, None] + self.gmask[f][None]
        return torch.stack([q[c].reshape(-1)[idx] for c in self.trace_fields(f // 2)])

    def on_face(self, op0, op1, x):
        """tensor product of 1-D operators on the faces' nodes"""
        if self.dim == 2:
            return x @ op0.T
        n = int(round(math.sqrt(x.shape[-1])))
        y = torch.einsum("ai,bj,...ji->...ba", op0, op1, x.reshape(*x.shape[:-1], n, n))
        return y.reshape(*x.shape[:-1], -1)

    def jumps(self, jump, ax, sg, Zpm, Zsm, Zpp, Zsp):
        """(T* - T-, v* - v-) from the trace jumps"""
        dim = self.dim
        dv, dT = jump[:dim], sg * jump[dim:]
        if self.central:
            return torch.cat([0.5 * dT, 0.5 * dv])
        J = torch.empty_like(jump)
        for a in range(dim):
            Zm, Zq = (Zpm, Zpp) if a == ax else (Zsm, Zsp)
            u = (Zq[:, None] * dv[a] + dT[a]) / (Zm + Zq)[:, None]
            J[dim + a] = u
            J[a] = Zm[:, None] * u
        return J

    def lift(self, out, e, f, J):
        dim, ax, sg = self.dim, f // 2, 1.0 if f & 1 else -1.0
        L = (self.rx[e, ax] / float(self.w[0]))[:, None]
        idx = (e * self.m.Np)[:, None] + self.gmask[f][None]
        add = lambda c, v: out[c].view(-1).index_add_(0, idx.reshape(-1), v.reshape(-1))  # noqa: E731
        dv = J[dim:]
        for a in range(dim):
            add(a, L / self.rho[e][:, None] * J[a])
        ll = L * self.lam[e][:, None] * sg * dv[ax]
        lm = L * self.mu[e][:, None] * sg
        for a in range(dim):
            add(dim + a, ll + (2 * lm * dv[a] if a == ax else 0.0))
        shear = {(0, 1): 6, (0, 2): 7, (1, 2): 8} if dim == 3 else {(0, 1): 4}
        for (a, b), c in shear.items():
            if ax == a:
                add(c, lm * dv[b])
            elif ax == b:
                add(c, lm * dv[a])

    def rhs(self, q):
        dim, Nq, K = self.dim, self.Nq, self.K
        shape = (K,) + (Nq,) * dim
        out = torch.zeros_like(q)

        def dx(c, a):
            v = torch.movedim(q[c].reshape(shape), dim - a, -1) @ self.D.T
            return (torch.movedim(v, -1, dim - a).reshape(K, -1)) * self.rx[:, a:a + 1]

        stress = [[3, 6, 7], [6, 4, 8], [7, 8, 5]] if dim == 3 else [[2, 4], [4, 3]]
        o = out.view(q.shape[0], K, -1)
        lam, mu = self.lam[:, None], self.mu[:, None]
        for a in range(dim):
            for b in range(dim):
                o[a] += dx(stress[a][b], b) / self.rho[:, None]
                g = dx(a, b)
                if a == b:
                    for c in range(dim):
                        o[dim + c] += (lam + 2 * mu if c == a else lam) * g
                else:
                    o[stress[a][b]] += mu * g
        for f in range(2 * dim):
            e, nb = self.conf[f]
            if len(e):
                jump = self.traces(q, nb, f ^ 1) - self.traces(q, e, f)
                self.lift(out, e, f, self.jumps(jump, f // 2, 1.0 if f & 1 else -1.0,
                                                self.Zp[e], self.Zs[e], self.Zp[nb], self.Zs[nb]))
            e, bc = self.bnd[f]
            if len(e) and bc != bf.BC_GLUED:
                tr = self.traces(q, e, f)
                jump = -tr if bc == bf.BC_ABSORBING else torch.cat([0 * tr[:dim], -2 * tr[dim:]])
                self.lift(out, e, f, self.jumps(jump, f // 2, 1.0 if f & 1 else -1.0,
                                                self.Zp[e], self.Zs[e], self.Zp[e], self.Zs[e]))
        for f, p, coarse, fine in self.hang:
            a, b = (p - 1) & 1, (p - 1) >> 1
            jump = self.traces(q, fine, f ^ 1) - self.on_face(self.I[a], self.I[b],
                                                              self.traces(q, coarse, f))
            sg = 1.0 if f & 1 else -1.0
            Z = (self.Zp[coarse], self.Zs[coarse]), (self.Zp[fine], self.Zs[fine])
            J = self.jumps(jump, f // 2, sg, *Z[0], *Z[1])
            self.lift(out, coarse, f, self.on_face(self.P[a], self.P[b], J))
            self.lift(out, fine, f ^ 1, self.jumps(-jump, f // 2, -sg, *Z[1], *Z[0]))
        return out

    def weights(self, x):
        """element holding x and the Lagrange weights of its nodes there"""
        m = self.m
        inside = ((x[:m.dim] >= m.x0[:, :m.dim])
                  & (x[:m.dim] < m.x0[:, :m.dim] + m.h[:, :m.dim])).all(axis=1)
        e = int(np.flatnonzero(inside)[0])
        xi = 2 * (x[:m.dim] - m.x0[e, :m.dim]) / m.h[e, :m.dim] - 1
        v = np.ones(1)
        for a in range(m.dim):
            v = (_lagrange(self.r, xi[a:a + 1])[0][:, None] * v[None]).reshape(-1)
        return e, v

    def point_force(self):
        """nodes, their weights and the force over density"""
        e, v = self.weights(self.d["x"])
        w = np.ones(1)
        for _ in range(self.dim):
            w = (self.w[:, None] * w[None]).reshape(-1)
        J = np.prod(0.5 * self.m.h[e, :self.dim])
        nodes = torch.arange(e * self.m.Np, (e + 1) * self.m.Np, device=self.dev)
        return nodes, self.t(v / (w * J)) / self.rho[e], self.d["force"]

    def energy(self, q):
        w = np.ones(1)
        for _ in range(self.dim):
            w = (self.w[:, None] * w[None]).reshape(-1)
        o = q.view(q.shape[0], self.K, -1)
        dim, lam, mu = self.dim, self.lam[:, None], self.mu[:, None]
        e = self.rho[:, None] * (o[:dim] ** 2).sum(0)
        tr = o[dim:2 * dim].sum(0)
        e = e + ((o[dim:2 * dim] ** 2).sum(0) - lam / (dim * lam + 2 * mu) * tr ** 2) / (2 * mu)
        e = e + (o[2 * dim:] ** 2).sum(0) / mu
        J = torch.prod(1.0 / self.rx, dim=1)
        return float(0.5 * (J * (e @ self.t(w))).sum())


def _glue(case, exact):
    """adds the jumps of the two halves' joined faces to their operators"""
    pairs = bf.glued_x_pairs(exact[0].m, exact[1].m)
    g, _ = _lgl(max(x.N for x in exact))
    same = lambda x: x  # noqa: E731
    I = [x.t(_lagrange(x.r, g)) for x in exact]
    P = [x.t(_projection(g, x.r, same, 1.0)) for x in exact]
    elems, faces = [], []
    for x, b in zip(exact, pairs):
        elems.append(x.t(x.m.EToEb[b].astype(np.int64)))
        faces.append(x.m.EToFb[b])

    def add(qs, outs):
        for f in (0, 1):
            s = np.flatnonzero(faces[0] == f)
            e = [el[exact[0].t(s)] for el in elems]
            tr = [x.on_face(i, i, x.traces(q, el, f ^ k))
                  for k, (x, i, q, el) in enumerate(zip(exact, I, qs, e))]
            for k, x in enumerate(exact):
                y, fk = exact[1 - k], f ^ k
                J = x.jumps(tr[1 - k] - tr[k], 0, 1.0 if fk & 1 else -1.0, x.Zp[e[k]],
                            x.Zs[e[k]], y.Zp[e[1 - k]], y.Zs[e[1 - k]])
                x.lift(outs[k], e[k], fk, x.on_face(P[k], P[k], J))
    return add


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    inputs = _inputs(case, seed)
    ops = [_Exact(d, case["flux"] == "central", device) for d in inputs]
    glue = _glue(case, ops) if case["kind"] == "glued" else None
    qs = [torch.as_tensor(d["q0"].copy(), device=device) for d in inputs]
    dqs = [torch.zeros_like(q) for q in qs]
    A, B, C = TABLES[case["method"]]
    shots = case["kind"] in ("shot", "serve")
    forces = [x.point_force() for x in ops] if shots else []
    seis = []
    if case["kind"] == "shot":
        held = [ops[0].weights(x) for x in inputs[0]["recv"]]
    for step in range(case["steps"]):
        for a, b, c in zip(A, B, C):
            outs = [x.rhs(q) for x, q in zip(ops, qs)]
            if glue:
                glue(qs, outs)
            for k, d in enumerate(inputs):
                if shots:
                    nodes, w, force = forces[k]
                    s = (math.pi * d["f0"] * (step * d["dt"] + c * d["dt"] - d["t0"])) ** 2
                    for i in range(3):
                        outs[k][i][nodes] += (1 - 2 * s) * math.exp(-s) * force[i] * w
                dqs[k].mul_(a).add_(outs[k], alpha=d["dt"])
            del outs
            for q, dq in zip(qs, dqs):
                q.add_(dq, alpha=b)
        if case["kind"] == "shot":
            o = qs[0].view(9, ops[0].K, -1)
            seis.append(torch.stack([o[:, e] @ ops[0].t(w) for e, w in held]))
    if case["kind"] == "shot":
        return torch.stack(seis), qs[0]
    if case["kind"] == "solve":
        return qs[0]
    if case["kind"] == "step":
        return (qs[0], ops[0].energy(qs[0])) if case["energy"] else qs[0]
    return qs

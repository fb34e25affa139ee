"""Performance cases of the particle path, through its public entry points.

A case names a mesh, particle parameters, a form (fp32 or fp64) and an
operation.  A simulation is restarted from a developed particle set: 1 to
max + 1 particles at random places in every cell part (a run seeded with one
per part settles near 1.9 per part at max 2 within a few hundred steps, and
stays there), their velocities the nodal field's plus N(0, 0.01), so that
every pass has face crossers, emptied and over-full parts.  Operations:

  step    one time step on device vectors (ParticleHandler.step_device, Vold
          = the last projection): the solver loop with its vectors on the GPU
  host    the same step with the solver's vectors on the host (step_solver)
  output  a step followed by the packed particle output (pack_output_device)
  window  the differentiated window of K steps and its adjoint
  fem     the solver step's three Q1 systems on device vectors
  noalloc the stateless projection of caller-owned particle arrays

`exact` restates the operations in plain torch, in 64 bits, from the
published algorithm (Q1 shape functions, Euler or midpoint sub-steps, Newton
inverse map, vertex-patch search, per-part counts), without this package's
kernels.
"""
from __future__ import annotations

import functools
import math
import os

import numpy as np
import torch

from pfem2dealii_b200 import _lib
from pfem2dealii_b200 import mesh as M
from pfem2dealii_b200.handler import ParticleHandler, ParticleParams, project_noalloc

MESH3 = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests", "golden", "Mesh3.tgz")
NOISE = 0.01  # standard deviation of the restarted particles' velocity noise
RHO, MU, FEM_DT = 1.0, 0.01, 1e-3


def _case(name, op, mesh, nx, ny, nz, q, maxpp, S, dt, form, **more):
    d = {"name": name, "op": op, "mesh": mesh, "nx": nx, "ny": ny, "nz": nz, "q0": q[0], "q1": q[1],
         "q2": q[2] if len(q) > 2 else 1, "maxpp": maxpp, "S": S, "dt": dt, "form": form, "rk2": False, "K": 0, "C": 0}
    d.update(more)
    return d


def listed():
    return [
        # the 2D channel at its configured size: the smallest problem a user runs, where launches count
        _case("channel_fp32", "step", "channel", 64, 16, 0, (4, 4), 2, 4, 0.01, "fp32"),
        # a small channel with odd counts, an uneven part grid and the midpoint integrator, plain form
        _case("channel_odd_rk2_fp64", "step", "channel", 61, 17, 0, (3, 5), 2, 5, 0.01, "fp64", rk2=True),
        # the 3D duct, the benchmark's headline workload, in both forms
        _case("duct_fp32", "step", "duct", 128, 32, 32, (3, 3, 3), 2, 3, 2e-3, "fp32"),
        _case("duct_fp64", "step", "duct", 128, 32, 32, (3, 3, 3), 2, 3, 2e-3, "fp64"),
        # the Turek obstacle on the reference's own unstructured mesh, both forms
        _case("turek_fp32", "step", "turek", 0, 0, 0, (4, 4), 2, 3, 5e-4, "fp32"),
        _case("turek_fp64", "step", "turek", 0, 0, 0, (4, 4), 2, 3, 5e-4, "fp64"),
        # the perturbed (non-affine) cube: the largest workload (33 million particles) in FP32, a ragged
        # smaller one in FP64
        _case("cube_fp32", "step", "cube", 64, 64, 64, (4, 4, 4), 2, 3, 1e-3, "fp32"),
        _case("cube_odd_fp64", "step", "cube", 37, 37, 37, (4, 4, 4), 2, 3, 1e-3, "fp64"),
        # the duct for a solver that keeps its vectors on the host
        _case("duct_host_fp32", "host", "duct", 128, 32, 32, (3, 3, 3), 2, 3, 2e-3, "fp32"),
        # a time step that also writes particle output, ragged duct, plain form
        _case("duct_output_fp64", "output", "duct", 97, 31, 29, (2, 2, 2), 2, 3, 2e-3, "fp64"),
        # the differentiated window and its adjoint on the Turek mesh
        _case("turek_window_fp32", "window", "turek", 0, 0, 0, (4, 4), 2, 3, 5e-4, "fp32", K=20, C=5),
        # the three Q1 systems of a solver step on the duct
        _case("duct_fem", "fem", "duct", 128, 32, 32, (2, 2, 2), 2, 3, 2e-3, "fp64"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["step"] * 6 + ["host", "output", "window", "fem", "noalloc"])
    form = "fp64" if op in ("fem", "noalloc", "output") else rng.choice(["fp32", "fp32", "fp64"])
    kind = rng.choice(["channel", "duct", "duct", "cylinder", "cube"])
    S, maxpp = rng.choice([1, 2, 3, 3, 4, 5]), rng.choice([1, 2, 2, 2, 3])
    n = nx = ny = nz = 0
    if kind == "channel":
        ny = _log(rng, 12, 300)
        nx, q, dt = ny * 4 + rng.randrange(-3, 4), (rng.choice([2, 3, 4, 5]), rng.choice([2, 3, 4])), 0.16 / ny
    elif kind == "duct":
        ny = _log(rng, 6, 24)
        nz, nx = max(4, ny + rng.randrange(-3, 4)), ny * rng.choice([2, 3, 4]) + rng.randrange(-3, 4)
        q = tuple(rng.choice([2, 3, 3, 4]) for _ in range(3))
        dt = 0.064 / ny
    elif kind == "cylinder":
        nx = _log(rng, 12, 96)
        ny, nz, q, dt = nx // 2 + rng.randrange(0, 3), nx * 5 + rng.randrange(-3, 4), (rng.choice([3, 4]), 4), 0.048 / nx
    else:
        n = _log(rng, 7, 40)
        nx = ny = nz = n
        q, dt = tuple(rng.choice([2, 3, 4, 4]) for _ in range(3)), 0.08 / n
    d = _case("", op, kind, nx, ny, nz, q, maxpp, S, round(dt, 9), form)
    del d["name"]
    if op == "window":
        d["K"], d["C"] = rng.choice([(4, 2), (10, 5), (11, 3), (16, 4)])
    elif op in ("step", "host", "output"):
        d["rk2"] = rng.random() < 0.15
    return d


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

@functools.lru_cache(maxsize=64)
def _mesh(kind, nx, ny, nz):
    """Mesh and nodal velocity field of unit amplitude, as the benchmark configurations have them."""
    if kind == "channel":
        m = M.hyper_rectangle((0.0, 0.0), (4.0, 1.0), (nx, ny), kind)
        return m, M.field_at_dofs(m, M.channel_profile(1.0, 1.0))
    if kind == "duct":
        m = M.hyper_rectangle((0.0, 0.0, 0.0), (8.0, 1.0, 1.0), (nx, ny, nz), kind)
        return m, M.field_at_dofs(m, M.duct_profile(1.0))
    if kind == "cube":
        m = M.perturbed_cube(nx, amplitude=0.1, seed=0)
        return m, M.field_at_dofs(m, M.taylor_green_3d())
    m = M.read_unv_native(MESH3) if kind == "turek" else M.turek_channel(nx, ny, nz)
    return m, M.field_at_dofs(m, M.cylinder_inflow(1.5))


def _setup(case):
    return _mesh(case["mesh"], case["nx"], case["ny"], case["nz"])


def _q(case, dim):
    return (case["q0"], case["q1"], case["q2"])[:dim]


def _params(case, dim):
    m, q = _setup(case)[0], _q(case, dim)
    # slots for max + 1 particles in every part and one step's new ones, so that a long run without
    # host synchronisation never meets the limit
    return ParticleParams(particles_per_cell=q, max_particles_per_cell_part=case["maxpp"],
                          particle_integration_steps=case["S"], time_step=case["dt"], integrator=int(case["rk2"]),
                          capacity=(case["maxpp"] + 2) * m.n_cells * int(np.prod(q)))


def _shape(xi):
    """Q1 shape functions in lexicographic vertex order: (n, dim) -> (n, 2^dim)."""
    N = None
    for d in range(xi.shape[1]):
        f = torch.stack([1.0 - xi[:, d], xi[:, d]], 1)
        N = f if N is None else (f[:, :, None] * N[:, None, :]).flatten(1)
    return N


def _start(case, seed):
    """The inputs of a case, on the GPU, from its seed: the nodal field and
    the particle set (cell, xi, x, v) in (cell, part) order."""
    m, V0 = _setup(case)
    g = torch.Generator("cuda").manual_seed(seed)

    def rand(*shape):
        return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)

    V = torch.from_numpy(V0).cuda() * (1.0 + 0.05 * (2.0 * rand(m.dim, 1) - 1.0))
    q = _q(case, m.dim)
    part = torch.cartesian_prod(*[torch.arange(k, device="cuda") for k in q]).reshape(-1, m.dim)
    nparts = m.n_cells * part.shape[0]  # 1 .. max + 1 particles, equally many parts of each, in a random order
    count = 1 + torch.randperm(nparts, generator=g, device="cuda") % (case["maxpp"] + 1)
    cp = torch.repeat_interleave(torch.arange(nparts, device="cuda"), count)  # (cell, part) of each particle
    n, cell = cp.shape[0], cp // part.shape[0]
    xi = (part[cp % part.shape[0]] + rand(n, m.dim)) / torch.tensor(q, device="cuda", dtype=torch.float64)
    del cp
    X = torch.from_numpy(m.vertices).cuda()
    cv, cd = torch.from_numpy(m.cells).cuda().long(), torch.from_numpy(m.cell_dofs).cuda().long()
    x, v = torch.empty_like(xi), torch.empty_like(xi)
    for a in range(0, n, 1 << 21):
        s = slice(a, min(n, a + (1 << 21)))
        N = _shape(xi[s])
        for d in range(m.dim):
            x[s, d] = (N * X[:, d][cv[cell[s]]]).sum(1)
            v[s, d] = (N * V[d][cd[cell[s]]]).sum(1)
    v += NOISE * torch.randn(n, m.dim, generator=g, device="cuda", dtype=torch.float64)
    return m, V, cell, xi, x, v, g


def prepare(case, seed):
    op = case["op"]
    m, V, cell, xi, x, v, gen = _start(case, seed)
    st = {"op": op, "V": V, "m": m}
    if op == "noalloc":
        st.update(cd=torch.from_numpy(m.cell_dofs).cuda(), cell=cell.int(), xi=xi.t().contiguous(),
                  v=v.t().contiguous(), out=torch.zeros_like(V))
        return st
    g = ParticleHandler(m.dim, _params(case, m.dim), case["form"])
    g.initialize_maps(m)
    st["g"] = g
    if op == "fem":
        nnz, nd = len(g.fem_pattern()[1]), m.n_dofs
        st["U2"] = V + 0.01 * torch.randn(V.shape, generator=gen, device="cuda", dtype=torch.float64)
        st["P"] = torch.randn(nd, generator=gen, device="cuda", dtype=torch.float64)

        def new(*shape):
            return torch.empty(shape, dtype=torch.float64, device="cuda")

        st["A"] = [new(m.dim, nnz), new(1, nnz), new(1, nnz)]
        st["rhs"] = [new(m.dim, nd), new(1, nd), new(m.dim, nd)]
        torch.cuda.synchronize()
        return st
    n = cell.shape[0]
    P = {"id": np.arange(1, n + 1, dtype=np.uint32), "cell": cell.int().cpu().numpy(), "xi": xi.cpu().numpy(),
         "v": v.cpu().numpy(), "x": x.cpu().numpy() if case["form"] == "fp64" else np.empty((0, m.dim))}
    g.seed_particles_device(V)  # takes the capacity; the restart replaces the particles
    g.set_particles(P, n)
    st["out"] = torch.empty_like(V)
    g.project_particle_fields_device(st["out"])
    if op == "host":
        st["hV"] = V.cpu().numpy()
    elif op == "output":  # room for every particle the handle can hold: n x 3 positions, then n x 3 velocities
        st["packed"] = torch.zeros(6 * g.params.capacity, device="cuda")
    elif op == "window":
        st.update(K=case["K"], C=case["C"], Vold=st["out"].clone(), U=torch.empty_like(V),
                  gU=torch.randn(V.shape, generator=gen, device="cuda", dtype=torch.float64),
                  gv0=torch.empty(n, m.dim, dtype=torch.float64, device="cuda"), gV=torch.empty_like(V),
                  gVold=torch.empty_like(V))
    torch.cuda.synchronize()
    return st


def run(st):
    op = st["op"]
    if op == "noalloc":
        empty = project_noalloc(st["cd"], st["cell"], st["xi"], st["v"], st["out"])
        return {"V": st["out"], "empty": empty}
    g = st["g"]
    if op == "host":
        return {"V": g.step_solver(st["hV"])}
    if op == "window":
        g.window_forward_device(st["K"], st["C"], st["V"], st["Vold"], None, st["U"])
        g.window_backward_device(st["gU"], st["gv0"], st["gV"], st["gVold"])
        return {k: st[k] for k in ("U", "gv0", "gV", "gVold")}
    if op == "fem":
        for k in range(3):  # the C ABI's device form, on the handle's stream
            _lib.check(g.L.pfem2gpu_fem_assemble_device(
                g.h, k, RHO, MU, FEM_DT, st["V"].data_ptr(), st["U2"].data_ptr(), st["P"].data_ptr(),
                st["A"][k].data_ptr(), st["rhs"][k].data_ptr()), g.h)
        return {"A": st["A"], "rhs": st["rhs"]}
    g.step_device(st["V"], None, st["out"])
    if op == "output":
        return {"V": st["out"], "packed": st["packed"], "n": g.pack_output_device(st["packed"])[1]}
    return {"V": st["out"]}


def work(case):
    """Bytes: the particle state and the nodal vectors read once and written
    once, the cell tables read once.  Flops: interpolations and maps of every
    particle (window: also the adjoint's), or the quadrature loops."""
    m, _ = _setup(case)
    dim, nv, op = m.dim, m.nv, case["op"]
    w = 8 if case["form"] == "fp64" else 4
    n = m.n_cells * int(np.prod(_q(case, dim))) * (case["maxpp"] + 2) / 2
    mesh = m.n_cells * nv * 4 + m.n_verts * dim * 8  # DoF ids, vertex coordinates
    nodal = m.n_dofs * dim * 8
    if op == "fem":
        nnz = _nnz(case["mesh"], case["nx"], case["ny"], case["nz"])
        out = (dim + 2) * nnz * 8 + (2 * dim + 1) * m.n_dofs * 8
        return {"bytes": 3 * mesh + 5 * nodal + out, "flops": m.n_cells * nv ** 3 * (14 * dim + 12)}
    state = 8 + dim * w * (3 if w == 8 else 2)  # cell, id, xi, v (and x)
    per = nv * dim * 2 + nv * (dim - 1)         # one interpolation
    if op == "noalloc":
        return {"bytes": n * (4 + 16 * dim) + mesh + nodal, "flops": n * 2 * per}
    sub = case["S"] * (2 if case["rk2"] else 1)
    flops = n * per * (2 + 2 * sub)
    if op == "window":  # the states once in and the gradients out; K steps and their adjoints
        return {"bytes": n * (state + 8 * dim) + mesh + 7 * nodal, "flops": 3 * case["K"] * flops}
    b = 2 * n * state + mesh + 3 * nodal
    return {"bytes": b + (n * 24 if op == "output" else 0), "flops": flops}


# ---------------------------------------------------------------------------
# The same in plain torch, 64 bits
# ---------------------------------------------------------------------------

class _Exact:
    def __init__(self, case, m, V):
        self.case, self.m, self.V, self.dim = case, m, V, m.dim
        self.X = torch.from_numpy(m.vertices).cuda()
        self.cv, self.cd = torch.from_numpy(m.cells).cuda().long(), torch.from_numpy(m.cell_dofs).cuda().long()
        self.q = torch.tensor(_q(case, m.dim), device="cuda")
        self.h = case["dt"] / case["S"]
        # cells around each vertex, ascending, padded with -1
        vert, cell = self.cv.flatten(), torch.arange(m.n_cells, device="cuda").repeat_interleave(m.nv)
        o = torch.argsort(vert, stable=True)
        vert, cell = vert[o], cell[o]
        cnt = torch.bincount(vert, minlength=m.n_verts)
        k = torch.arange(vert.shape[0], device="cuda") - (torch.cumsum(cnt, 0) - cnt)[vert]
        self.around = torch.full((m.n_verts, int(cnt.max())), -1, device="cuda")
        self.around[vert, k] = cell
        self.centre = self.X[self.cv].mean(1)

    def field(self, F, c, N):
        """sum_i N_i F_i of a component-major nodal field."""
        d = self.cd[c]
        return torch.stack([(N * F[k][d]).sum(1) for k in range(self.dim)], 1)

    def place(self, c, N):
        return torch.einsum("nv,nvd->nd", N, self.X[self.cv[c]])

    def jac(self, c, xi):
        """J[n, a, b] = d x_a / d xi_b."""
        X = self.X[self.cv[c]]
        cols = []
        for b in range(self.dim):
            hi, lo = xi.clone(), xi.clone()
            hi[:, b], lo[:, b] = 1.0, 0.0
            cols.append(torch.einsum("nv,nvd->nd", _shape(hi) - _shape(lo), X))
        return torch.stack(cols, 2)

    def inverse(self, c, x, xi, iters):
        """Newton on F_c(xi) = x from xi; NaN where it fails to converge."""
        for _ in range(iters):
            r = x - self.place(c, _shape(xi))
            xi = xi + torch.linalg.solve(self.jac(c, xi), r)
        bad = ~((x - self.place(c, _shape(xi))).abs().amax(1) < 1e-9) | ~(torch.linalg.det(self.jac(c, xi)) > 0)
        return torch.where(bad[:, None], torch.full_like(xi, math.nan), xi)

    @staticmethod
    def inside(xi):
        return ((xi >= 0.0) & (xi <= 1.0)).all(1)

    def substep(self, c, xi, x):
        """One sub-step: new (c, xi, x, alive) (the vertex-patch search for particles that leave their cell)."""
        u = self.field(self.V, c, _shape(xi))
        if self.case["rk2"]:
            dl = torch.linalg.solve(self.jac(c, xi), u)
            u = self.field(self.V, c, _shape(xi + 0.5 * self.h * dl))
        xd = x.detach() + u.detach() * self.h
        with torch.no_grad():
            new, cn = self.inverse(c, xd, xi, 6), c.clone()
            out = torch.nonzero(~self.inside(new)).flatten()
            alive = torch.ones_like(c, dtype=torch.bool)
            if out.numel():
                co, xo, uo = c[out], xd[out], u[out]
                old, Xo = self.place(co, _shape(xi[out])), self.X[self.cv[co]]
                to = Xo - old[:, None, :]
                near = ((to * uo[:, None, :]).sum(2) / to.norm(dim=2)).argmax(1)
                vid = self.cv[co, near]
                cand = self.around[vid]
                dirs = self.centre[cand.clamp(min=0)] - self.X[vid][:, None, :]
                dirs = dirs / dirs.norm(dim=2, keepdim=True)
                dot = (dirs * (xo - self.X[vid])[:, None, :]).sum(2)
                dot[(cand < 0) | (cand == co[:, None])] = -math.inf
                order = torch.argsort(dot, dim=1, descending=True, stable=True)
                left = torch.arange(out.numel(), device="cuda")
                for t in range(cand.shape[1]):
                    pick = order[left, t]
                    k, real = cand[left, pick], dot[left, pick] > -math.inf
                    y = self.inverse(k.clamp(min=0), xo[left], torch.full_like(xo[left], 0.5), 12)
                    ok = real & self.inside(y)
                    new[out[left[ok]]], cn[out[left[ok]]] = y[ok], k[ok]
                    left = left[~ok]
                alive[out[left]] = False
        if u.requires_grad or xi.requires_grad:  # d xi' = J(xi')^-1 d x', the cells held fixed
            xt = self.place(c, _shape(xi)) + u * self.h
            J = self.jac(cn, new)
            eye = torch.eye(self.dim, device="cuda", dtype=torch.float64)
            Ji = torch.linalg.inv(torch.where(alive[:, None, None], J, eye))
            new = new + torch.einsum("nab,nb->na", Ji, xt - xt.detach())
        return cn, new, xd, alive

    def project(self, c, xi, v):
        N = _shape(xi)
        d = self.cd[c].flatten()
        den = torch.zeros(self.m.n_dofs, device="cuda", dtype=torch.float64).index_add(0, d, N.flatten())
        num = [torch.zeros_like(den).index_add(0, d, (N * v[:, k:k + 1]).flatten()) for k in range(self.dim)]
        return torch.stack(num), den

    def step(self, cell, xi, x, v):
        """Correct, move, count correction, project; the projection and (x, v) in the output's order."""
        n, npart = cell.shape[0], int(self.q.prod())
        num, den = self.chunked(lambda s: self.project(cell[s], xi[s], v[s]), n)
        dV = self.V - num / den
        parts = []
        for a in range(0, n, 1 << 20):
            s = slice(a, min(n, a + (1 << 20)))
            c, y, z = cell[s], xi[s], x[s]
            w = v[s] + self.field(dV, c, _shape(y))
            pid = torch.arange(s.start, s.stop, device="cuda")
            keep = torch.ones_like(c, dtype=torch.bool)
            for _ in range(self.case["S"]):
                c2, y2, z2, alive = self.substep(c[keep], y[keep], z[keep])
                idx = torch.nonzero(keep).flatten()
                c, y, z = c.clone(), y.clone(), z.clone()
                c[idx], y[idx], z[idx] = c2, y2, z2
                keep[idx] = alive
            parts.append((c[keep], y[keep], z[keep], w[keep], pid[keep], cell[s][keep]))
        c, y, z, w, pid, c0 = (torch.cat(t) for t in zip(*parts))
        part = torch.zeros_like(c)
        for d in range(self.dim):
            part = part * self.q[d] + (y[:, d] * self.q[d]).long().clamp(max=int(self.q[d]) - 1)
        group = c * npart + part
        o = torch.argsort(group, stable=True)  # ids ascend within a group
        cnt = torch.bincount(group, minlength=self.m.n_cells * npart)
        rank = torch.empty_like(group)
        rank[o] = torch.arange(group.shape[0], device="cuda") - (torch.cumsum(cnt, 0) - cnt)[group[o]]
        s = rank <= self.case["maxpp"]
        empty = (cnt == 0).view(-1, npart) & (cnt.view(-1, npart).sum(1) > 0)[:, None]
        sc, sp = torch.nonzero(empty, as_tuple=True)
        digits, r = [], sp
        for d in reversed(range(self.dim)):
            digits.append(r % self.q[d])
            r = r // self.q[d]
        sy = (torch.stack(digits[::-1], 1).double() + 0.5) / self.q
        N = _shape(sy)
        moved = (c != c0).long()
        c, y, z, w = (torch.cat(t) for t in ((c[s], sc), (y[s], sy), (z[s], self.place(sc, N)),
                                             (w[s], self.field(self.V, sc, N))))
        kind = torch.cat([moved[s], torch.full_like(sc, 2)])
        tie = torch.cat([pid[s], sp])
        num, den = self.chunked(lambda s: self.project(c[s], y[s], w[s]), c.shape[0])
        order = torch.argsort((c * 3 + kind) * (n + npart) + tie)
        return num / den, z[order], w[order]

    @staticmethod
    def chunked(f, n):
        total = None
        for a in range(0, max(n, 1), 1 << 21):
            t = f(slice(a, min(n, a + (1 << 21))))
            total = t if total is None else tuple(p + q for p, q in zip(total, t))
        return total


def _csr(m):
    """Row-major (row, col) keys of the Q1 pattern, and each local entry's place among them."""
    cd = torch.from_numpy(m.cell_dofs).cuda().long()
    key = (cd[:, :, None] * m.n_dofs + cd[:, None, :]).flatten()
    return torch.unique(key, return_inverse=True)


@functools.lru_cache(maxsize=16)
def _nnz(*mesh):
    return int(_csr(_mesh(*mesh)[0])[0].shape[0])


def _exact_fem(m, U, U2, P):
    """The volume terms of the three systems (src/pfem2fem.cpp:247-510), QGauss(2)."""
    dim, nv, nd = m.dim, m.nv, m.n_dofs
    X = torch.from_numpy(m.vertices).cuda()[torch.from_numpy(m.cells).cuda().long()]
    cd = torch.from_numpy(m.cell_dofs).cuda().long()
    keys, at = _csr(m)
    g1 = 0.5 + np.array([-1.0, 1.0]) / (2.0 * math.sqrt(3.0))
    A = [torch.zeros(k, m.n_cells, nv, nv, device="cuda", dtype=torch.float64) for k in (dim, 1, 1)]
    r = [torch.zeros(k, m.n_cells, nv, device="cuda", dtype=torch.float64) for k in (dim, 1, dim)]
    Uc, U2c, Pc = U[:, cd], U2[:, cd], P[cd]
    for qi in range(1 << dim):
        xi = torch.tensor([[g1[(qi >> d) & 1] for d in range(dim)]], device="cuda", dtype=torch.float64)
        N = _shape(xi)[0]
        G = []
        for b in range(dim):
            hi, lo = xi.clone(), xi.clone()
            hi[:, b], lo[:, b] = 1.0, 0.0
            G.append((_shape(hi) - _shape(lo))[0])
        G = torch.stack(G, 1)                                     # (nv, dim) reference gradients
        J = torch.einsum("cva,vb->cab", X, G)
        g = torch.einsum("cba,vb->cva", torch.linalg.inv(J), G)   # physical gradients
        w = torch.linalg.det(J) / (1 << dim)
        mass = RHO * torch.outer(N, N)[None] * w[:, None, None]
        gg = torch.einsum("cia,cjb->ijabc", g, g).permute(4, 0, 1, 2, 3) * (w * MU * FEM_DT)[:, None, None, None, None]
        lap = sum(gg[..., a, a] for a in range(dim))
        for k in range(dim):
            A[0][k] += mass + lap + gg[..., k, k] / 3.0
            r[0][k] += torch.einsum("cij,cj->ci", mass, U2c[k])
            for b in range(dim):
                if b != k:
                    r[0][k] -= torch.einsum("cij,cj->ci", gg[..., b, k] - 2.0 / 3.0 * gg[..., k, b], Uc[b])
        A[1][0] += lap / (MU * FEM_DT)
        uq = torch.einsum("j,kcj->kc", N, Uc)
        r[1][0] += RHO / FEM_DT * torch.einsum("kc,cik->ci", uq, g) * w[:, None]
        A[2][0] += mass
        gp = torch.einsum("cja,cj->ac", g, Pc)
        for k in range(dim):
            r[2][k] += torch.einsum("cij,cj->ci", mass, Uc[k]) - FEM_DT * N[None] * (w * gp[k])[:, None]

    def total(v, where, size):
        return torch.stack([torch.zeros(size, device="cuda", dtype=torch.float64).index_add(0, where, t.flatten())
                            for t in v])

    return {"A": [total(a, at, keys.shape[0]) for a in A], "rhs": [total(b, cd.flatten(), nd) for b in r]}


def exact(case, seed):
    op = case["op"]
    m, V, cell, xi, x, v, gen = _start(case, seed)
    if op == "fem":
        U2 = V + 0.01 * torch.randn(V.shape, generator=gen, device="cuda", dtype=torch.float64)
        return _exact_fem(m, V, U2, torch.randn(m.n_dofs, generator=gen, device="cuda", dtype=torch.float64))
    E = _Exact(case, m, V)
    if op == "noalloc":
        num, den = E.chunked(lambda s: E.project(cell[s], xi[s], v[s]), cell.shape[0])
        return {"V": num / den, "empty": int((den == 0).sum())}
    if op == "window":
        if cell.shape[0] * case["K"] * case["S"] * m.nv > 6e8:
            return None  # the recorded sub-steps would not fit, nor end in time
        num, den = E.project(cell, xi, v)
        gU = torch.randn(V.shape, generator=gen, device="cuda", dtype=torch.float64)
        Vold = (num / den).requires_grad_()
        E.V = V.clone().requires_grad_()
        v0 = v.clone().requires_grad_()
        c, y, z, w = cell, xi, x, v0
        for _ in range(case["K"]):
            w = w + E.field(E.V - Vold, c, _shape(y))
            for _ in range(case["S"]):
                c, y, z, alive = E.substep(c, y, z)
                c, y, z, w = c[alive], y[alive], z[alive], w[alive]
        num, den = E.project(c, y, w)
        reached = den.detach() > 0
        U = torch.where(reached, num / torch.where(reached, den, torch.ones_like(den)), torch.zeros_like(num))
        gv0, gV, gVold = torch.autograd.grad((U * gU).sum(), (v0, E.V, Vold))
        return {"U": torch.where(reached, U.detach(), torch.full_like(V, math.nan)), "gv0": gv0, "gV": gV,
                "gVold": gVold}
    out, px, pv = E.step(cell, xi, x, v)
    if op == "output":
        n = px.shape[0]
        packed = torch.zeros(6 * _params(case, m.dim).capacity, device="cuda", dtype=torch.float64)
        packed[:3 * n].view(n, 3)[:, :m.dim], packed[3 * n:6 * n].view(n, 3)[:, :m.dim] = px, pv
        return {"V": out, "packed": packed, "n": n}
    return {"V": out}

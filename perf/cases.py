"""The calls a user of this library makes, as timed cases.

Every case is one run of a deck: the initial state goes in from host arrays, the
cycles run, and the final state (or the gradients) comes back to host arrays, so
a pass can be repeated on the same inputs.  ``kind`` says through which entry
points:

  solve     ``setup`` and the one-shot ``sgh_solve``: what replaces the
            reference's own driver sequence (a handle is made on each call)
  handle    a persistent ``SGHSolver``: ``set_state``, ``run``, ``get_state``;
            with ``chunk`` the cycles run that many at a time with the energy
            tallies read after each (a monitored run)
  batch     a ``Batch`` of decks of different sizes and problems, made for the run
  adjoint   ``adj_forward`` and ``adj_backward``: the gradient of a function of
            the final density and energy

``exact`` computes the same runs with plain torch operations in 64 bits, written
from the scheme's equations.
"""
import math
import random

import numpy as np
import torch

from fierro_gb300 import mesh as meshes
from fierro_gb300 import problems, sgh

MODES = {"exact": sgh.FP_EXACT, "fma": sgh.FP_FMA}


def listed():
    return [
        # the smallest deck of the tests, watched by a driver that reads the energies
        # every ten cycles: launch and call latency
        dict(name="noh8_monitored", kind="handle", deck="noh", n=8, mode="exact", cycles=50, chunk=10),
        # the 12^3 Sedov deck the reference ships a mesh for, through the one-shot call
        dict(name="sedov12_solve", kind="solve", deck="sedov", n=12, mode="exact", cycles=200, chunk=0),
        # the 32^3 Noh deck the reference ships a mesh for
        dict(name="noh32", kind="handle", deck="noh", n=32, mode="fma", cycles=100, chunk=0),
        # three materials' worth of fills on an odd-sided box, the size of the shipped
        # unstructured meshes times a few
        dict(name="triple_71x31x17", kind="handle", deck="triple", n=71, mode="exact", cycles=50, chunk=0),
        # a strength model in every element
        dict(name="sedov40_hypo", kind="handle", deck="hypo", n=40, mode="fma", cycles=40, chunk=0),
        # mid-size production run, device-resident
        dict(name="sedov64", kind="handle", deck="sedov", n=64, mode="fma", cycles=40, chunk=0),
        # the parity deck's size in the reference's arithmetic
        dict(name="sedov120_exact", kind="handle", deck="sedov", n=120, mode="exact", cycles=8, chunk=0),
        # the largest: a state far above the L2
        dict(name="sedov144", kind="handle", deck="sedov", n=144, mode="fma", cycles=16, chunk=0),
        # axisymmetric decks: the reference's 64^2 test size, and a large one
        dict(name="sedov_rz64", kind="handle", deck="sedov_rz", n=64, mode="exact", cycles=200, chunk=0),
        dict(name="noh_rz768", kind="handle", deck="noh_rz", n=768, mode="fma", cycles=40, chunk=0),
        # a parameter study: decks of different sizes and problems advanced together
        dict(name="ensemble12", kind="batch", deck="mixed", n=32, mode="fma", cycles=100, chunk=0, members=12),
        # a gradient with checkpoints, recomputation and the reverse sweep
        dict(name="adjoint32", kind="adjoint", deck="sedov", n=32, mode="exact", cycles=40, chunk=20),
    ]


# kind, deck, modes, smallest and largest side, element cycles one pass may take,
# and the longest run (short of the decks' final times: dt is at most 1e-2)
_RANGES = [
    ("handle", "noh", ("exact", "fma"), 8, 96, 24e6, 100),
    ("handle", "sedov", ("exact", "fma"), 8, 128, 24e6, 140),
    ("handle", "triple", ("exact", "fma"), 14, 140, 16e6, 200),
    ("solve", "sedov", ("exact", "fma"), 8, 48, 4e6, 140),
    ("handle", "hypo", ("exact", "fma"), 8, 64, 8e6, 100),
    ("handle", "sedov_rz", ("exact", "fma"), 16, 768, 24e6, 100),
    ("handle", "noh_rz", ("exact", "fma"), 16, 768, 24e6, 100),
    ("batch", "mixed", ("exact", "fma"), 12, 40, 16e6, 100),
    ("adjoint", "sedov", ("exact",), 8, 40, 1.5e6, 60),
]


def draw(rng: random.Random):
    kind, deck, modes, lo, hi, budget, longest = rng.choice(_RANGES)
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))
    n = min(max(n, lo), hi)
    members = rng.randint(4, 12) if kind == "batch" else 0
    ne = max(members, 1) * int(np.prod(_shape(deck, n)))
    cycles = max(4, min(longest, int(budget / ne * rng.uniform(0.3, 1.0))))
    case = dict(kind=kind, deck=deck, n=n, mode=rng.choice(modes), cycles=cycles, chunk=0)
    if kind == "batch":
        case["members"] = members
    elif kind == "adjoint":
        case["chunk"] = rng.randint(5, 20)
    elif kind == "handle" and n <= 32:
        case["chunk"] = rng.choice([0, 10])
    return case


def _shape(deck, n):
    if deck in ("sedov_rz", "noh_rz"):
        return (n, n)
    if deck == "triple":
        return (n, max(2, round(n * 3 / 7)), max(2, round(n * 1.7 / 7)))
    return (n, n, n)


def _problem(deck, n, cycles, seed):
    seed = seed % 99991  # the mesh builder's hash takes small seeds
    if deck == "sedov":
        return problems.sedov(n, jitter=0.1, seed=seed, permute=True, cycles=cycles)
    if deck == "noh":
        return problems.noh(n, jitter=0.1, seed=seed, permute=True, cycles=cycles)
    if deck == "triple":
        nx, ny, nz = _shape(deck, n)
        m = meshes.box_mesh(nx, ny, nz, length=(7.0, 3.0, 1.7), jitter=0.1, seed=seed, permute=True)
        return problems.triple_point(m, cycles=cycles)
    if deck == "hypo":
        return problems.with_strength(_problem("sedov", n, cycles, seed), "hypo", 1.0)
    if deck == "sedov_rz":
        return problems.sedov_rz(n, jitter=0.1, seed=seed, permute=True, cycles=cycles,
                                 source_radius=max(1.2 / n, 1.2 / 64))
    if deck == "noh_rz":
        return problems.noh_rz(n, jitter=0.1, seed=seed, permute=True, cycles=cycles)
    raise ValueError(deck)


def _sides(case):
    """The sides of an ensemble's decks: from 8 up to the case's, which comes first."""
    r = np.random.RandomState(1000 * case["n"] + case["members"])
    return [case["n"]] + [int(v) for v in r.randint(8, case["n"] + 1, case["members"] - 1)]


def _members(case, seed):
    """The decks of an ensemble: Sedov and Noh in turn, each with a gamma of its own."""
    r, out = np.random.RandomState(seed % (1 << 31)), []
    for i, n in enumerate(_sides(case)):
        out.append(_problem("sedov" if i % 2 == 0 else "noh", n, case["cycles"], seed + i))
        out[-1].materials[0].gamma = float(r.uniform(1.3, 1.7))
    return out


def _seeds(case, problem, seed):
    """The objective's weights on the final density and energy."""
    r = np.random.RandomState((seed + 77) % (1 << 31))
    ne = problem.mesh.num_elems
    return r.uniform(0.5, 1.5, ne), r.uniform(0.5, 1.5, ne)


# ---------------------------------------------------------------- the framework
def prepare(case, seed):
    mode = MODES[case["mode"]]
    if case["kind"] == "batch":
        decks = _members(case, seed)
        return {"case": case, "decks": decks, "mode": mode, "states": [sgh.setup(p) for p in decks]}
    p = _problem(case["deck"], case["n"], case["cycles"], seed)
    s = {"case": case, "problem": p, "mode": mode}
    if case["kind"] == "solve":
        return s
    s["initial"] = sgh.setup(p)
    s["solver"] = sgh.SGHSolver(p, fp_mode=mode)
    s["final"] = sgh.empty_state(p.mesh.num_nodes, p.mesh.num_elems, p.num_state_vars, dims=p.mesh.dims)
    if case["kind"] == "adjoint":
        s["sie0"] = s["initial"]["elem_sie"][1].copy()
        s["gamma"] = s["initial"]["elem_statev"][:, 0].copy()
        s["wden"], s["wsie"] = _seeds(case, p, seed)
    return s


_STATE = ("node_coords", "node_vel", "node_mass", "elem_den", "elem_pres", "elem_sspd", "elem_sie", "elem_vol",
          "elem_div", "corner_force")


def run(state):
    case = state["case"]
    if case["kind"] == "solve":
        st = sgh.setup(state["problem"])
        r = sgh.sgh_solve(state["problem"], st, fp_mode=state["mode"])
        return {"time": r["time_value"], "cycles": r["cycles"], **{k: st[k] for k in _STATE}}
    if case["kind"] == "batch":
        # a batch takes its states once, so an ensemble run makes its own
        out = []
        with sgh.Batch(state["decks"], fp_mode=state["mode"]) as b:
            for i, st in enumerate(state["states"]):
                b.set_state(i, st)
            b.run(case["cycles"])
            for i in range(len(b)):
                st = b.get_state(i)
                out.append([st[k] for k in ("node_coords", "node_vel", "elem_den", "elem_pres", "elem_sie")])
        return out
    s = state["solver"]
    s.set_state(state["initial"])
    if case["kind"] == "adjoint":
        ran = s.adj_forward(state["sie0"], state["gamma"], case["cycles"], case["chunk"])
        st = s.get_state(state["final"])
        dsie, dgamma, dvel = s.adj_backward(den=state["wden"], sie=state["wsie"])
        return {"cycles": ran, "den": st["elem_den"], "sie": st["elem_sie"], "dsie": dsie, "dgamma": dgamma,
                "dvel": dvel}
    out = {}
    if case["chunk"]:
        ran, tallies = 0, []
        for done in range(0, case["cycles"], case["chunk"]):
            ran += s.run(min(case["chunk"], case["cycles"] - done))
            tallies.append(s.energy())
        out["tallies"] = np.array(tallies)
    else:
        ran = s.run(case["cycles"])
    st = s.get_state(state["final"])
    out.update({k: st[k] for k in _STATE})
    if case["deck"] == "hypo":
        out["elem_stress"] = st["elem_stress"]
    return {"cycles": ran, "time": s.time()[0], **out}


def _work_of(shape, cycles, adjoint=False):
    dims = len(shape)
    ne = int(np.prod(shape))
    nn = int(np.prod([v + 1 for v in shape]))
    npe = 2 ** dims
    # state in: two bins of positions and velocities, node mass, nine element fields
    # and two energies, ids; out: the same and the corner forces
    state = 8 * (nn * (4 * dims + 1) + ne * 12)
    out = state + 8 * ne * npe * dims
    # an RK2 cycle of the scheme: two stages of geometry, viscosity, gather, update
    flops = 2 * (1000 if dims == 3 else 300)
    if adjoint:
        return 2 * state, 4.0 * flops * ne * cycles
    return state + out, float(flops) * ne * cycles


def work(case):
    if case["kind"] == "batch":
        parts = [_work_of((n, n, n), case["cycles"]) for n in _sides(case)]
    else:
        parts = [_work_of(_shape(case["deck"], case["n"]), case["cycles"], case["kind"] == "adjoint")]
    return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}


# ---------------------------------------------------------------- 64-bit torch
def _trilinear_tensor():
    """C[i,j,k] with V = sum C x_i y_j z_k the exact volume of a trilinear hex: the
    integral of det(grad N_i, grad N_j, grad N_k), by 2-point Gauss quadrature."""
    signs = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                      [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], dtype=np.float64)
    g = 1.0 / math.sqrt(3.0)
    C = np.zeros((8, 8, 8))
    for a in (-g, g):
        for b in (-g, g):
            for c in (-g, g):
                f = 1.0 + signs * np.array([a, b, c])
                d = 0.125 * signs * np.stack([f[:, 1] * f[:, 2], f[:, 0] * f[:, 2], f[:, 0] * f[:, 1]], axis=1)
                cr = np.cross(d[:, None, :], d[None, :, :])
                C += np.einsum("id,jkd->ijk", d, cr)
    return np.round(C * 48.0) / 48.0


class _Run:
    """The scheme on one deck: plain torch, 64 bits."""

    def __init__(self, p, device):
        self.p, self.dev = p, device
        self.f = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=device)
        self.nie = torch.as_tensor(p.mesh.nodes_in_elem.astype(np.int64), device=device)
        self.ne, self.npe = self.nie.shape
        self.dims = p.mesh.dims
        x = self.f(p.mesh.coords)
        self.nn = x.shape[0]
        if self.dims == 3:
            C = self.f(_trilinear_tensor())
            self.Cx = C.permute(1, 2, 0).reshape(64, 8).contiguous()  # (y_j z_k) -> node i
            self.Cy = C.permute(2, 0, 1).reshape(64, 8).contiguous()  # (z_k x_i) -> node j
            self.Cz = C.permute(0, 1, 2).reshape(64, 8).contiguous()  # (x_i y_j) -> node k
        self._neighbours()
        self._initial(x)

    def _neighbours(self):
        flat = self.nie.reshape(-1)
        order = torch.argsort(flat, stable=True)
        counts = torch.bincount(flat, minlength=self.nn)
        start = torch.cumsum(counts, 0) - counts
        nodes = flat[order]
        slot = torch.arange(flat.numel(), device=self.dev) - start[nodes]
        table = torch.full((self.nn, int(counts.max())), -1, dtype=torch.int64, device=self.dev)
        table[nodes, slot] = order // self.npe
        nb = table[self.nie].reshape(self.ne, -1)
        own = torch.arange(self.ne, device=self.dev)[:, None]
        self.no_nb = (nb < 0) | (nb == own)
        self.nb = nb.clamp(min=0).to(torch.int32)

    def geometry(self, x):
        """Corner normals (the volume's gradient) and volume; for quads also the area."""
        X = x[self.nie]
        if self.dims == 3:
            X = X - X.mean(dim=1, keepdim=True)
            a, b, c = X[..., 0], X[..., 1], X[..., 2]
            pair = lambda s, t: (s[:, :, None] * t[:, None, :]).reshape(self.ne, 64)
            B = torch.stack([pair(b, c) @ self.Cx, pair(c, a) @ self.Cy, pair(a, b) @ self.Cz], dim=2)
            return B, (a * B[..., 0]).sum(1), None
        a, r = X[..., 0], X[..., 1]
        i, k = [1, 2, 3, 0], [3, 0, 1, 2]
        B = torch.stack([0.5 * (r[:, i] - r[:, k]), 0.5 * (a[:, k] - a[:, i])], dim=2)
        area = 0.5 * ((a[:, 0] - a[:, 2]) * (r[:, 1] - r[:, 3]) + (a[:, 3] - a[:, 1]) * (r[:, 0] - r[:, 2]))

        def third(l, m, n):  # area of a triangle times the sum of its radii
            tri = (a[:, m] - a[:, l]) * (r[:, n] - r[:, l]) - (r[:, m] - r[:, l]) * (a[:, n] - a[:, l])
            return 0.5 * tri * (r[:, l] + r[:, m] + r[:, n])

        return B, (third(0, 1, 2) + third(0, 2, 3)) / 3.0, area

    def _initial(self, x):
        p = self.p
        B, vol, area = self.geometry(x)
        cen = x[self.nie].mean(dim=1)
        den, sie = torch.zeros(self.ne, device=self.dev, dtype=torch.float64), torch.zeros_like(vol)
        mat = torch.zeros(self.ne, dtype=torch.int64, device=self.dev)
        v = torch.zeros_like(x)
        for f in p.fills:
            if f.volume == "global":
                on = torch.ones(self.ne, dtype=torch.bool, device=self.dev)
            elif f.volume == "box":
                lo, hi = (f.x1, f.y1, f.z1), (f.x2, f.y2, f.z2)
                on = torch.ones(self.ne, dtype=torch.bool, device=self.dev)
                for d in range(self.dims):
                    on &= (cen[:, d] >= lo[d]) & (cen[:, d] <= hi[d])
            else:
                r = cen.norm(dim=1)
                on = (r >= f.radius1) & (r <= f.radius2)
            den = torch.where(on, torch.full_like(den, f.den), den)
            sie = torch.where(on, torch.full_like(sie, f.sie), sie)
            mat[on] = f.mat_id
            nodes = self.nie[on].reshape(-1).unique()
            if f.velocity == "cartesian":
                v[nodes] = self.f([f.u, f.v, f.w][: self.dims])
            else:
                r = x[nodes].norm(dim=1, keepdim=True)
                v[nodes] = torch.where(r > 1e-14, f.speed * x[nodes] / r.clamp(min=1e-300), torch.zeros_like(x[nodes]))
        self.free = torch.ones_like(x)
        for b in p.boundaries:
            d = "xyz".index(b.surface[0])
            at = (x[:, d] - b.value).abs() <= 1e-7
            self.free[at, d] = 0.0
        sv = self.f(p.state_vars())[mat]
        self.gamma, self.csmin, self.shear = sv[:, 0], sv[:, 1], sv[:, 3]
        m = [(q.q1, q.q1ex, q.q2, q.q2ex) for q in p.materials]
        self.q = self.f(m)[mat]
        self.mass = den * vol
        nm = torch.zeros(self.nn, dtype=torch.float64, device=self.dev)
        if self.dims == 3:
            corner = (self.mass / 8.0)[:, None].expand(-1, 8)
        else:
            # Barlow's corner areas from the four triangles around the centroid
            X = x[self.nie]
            c = X.mean(dim=1, keepdim=True)
            n = X[:, [1, 2, 3, 0]]
            t = 0.5 * ((X - c)[..., 0] * (n - c)[..., 1] - (X - c)[..., 1] * (n - c)[..., 0]).abs()
            prev = t[:, [3, 0, 1, 2]]
            corner = (t.sum(1, keepdim=True) + 4.0 * t + 4.0 * prev) / 12.0 * den[:, None]
        self.node_mass = nm.index_add(0, self.nie.reshape(-1), corner.reshape(-1))
        self.ext = self.node_mass * x[:, 1] if self.dims == 2 else None
        if self.dims == 2:
            pairs = torch.cat([self.nie[:, [i, (i + 1) % 4]] for i in range(4)])
            self.edges = torch.cat([pairs, pairs.flip(1)])
        self.x, self.v, self.vol, self.sie, self.den = x, v * self.free, vol, sie, den
        self.B, self.area = B, area
        self.stress = torch.zeros((self.ne, 3, 3), dtype=torch.float64, device=self.dev)

    def eos(self):
        g = self.gamma
        self.pres = (g - 1.0) * self.sie * self.den
        c2 = g * (g - 1.0) * self.sie
        low = c2 < self.csmin ** 2
        self.c = torch.where(low, self.csmin, torch.where(low, torch.ones_like(c2), c2).sqrt())

    def divergence(self):
        V = self.v[self.nie]
        flux = (V * self.B).sum(dim=(1, 2))
        if self.dims == 3:
            return flux / self.vol
        return flux / self.area + V[..., 1].mean(1) / (self.vol / self.area)

    def step(self, dt, t):
        """get_timestep: growth, CFL, clamps, final time (no dump falls in these runs)."""
        q = self.p.params
        X = self.x[self.nie]
        d2 = None
        for i in range(self.npe):
            for j in range(i + 1, self.npe):
                s = ((X[:, i] - X[:, j]) ** 2).sum(1)
                d2 = s if d2 is None else torch.minimum(d2, s)
        cfl = (q.dt_cfl * d2.sqrt() / (self.c + q.fuzz)).min()
        cfl = cfl.clamp(min=q.dt_min, max=q.dt_max)
        dt = torch.minimum(dt * 1.1, cfl)
        return torch.minimum(dt, q.time_final - t)

    def force(self):
        q = self.p.params
        V = self.v[self.nie]
        dv = V - V.mean(dim=1, keepdim=True)
        s2 = (dv * dv).sum(2)
        still = s2 == 0
        speed = torch.where(still, torch.zeros_like(s2), torch.where(still, torch.ones_like(s2), s2).sqrt())
        comp = self.div < 0
        qa, qb = torch.where(comp, self.q[:, 0], self.q[:, 1]), torch.where(comp, self.q[:, 2], self.q[:, 3])
        mu = self.den[:, None] * ((qa * self.c)[:, None] + qb[:, None] * speed) * self.B.norm(dim=2)
        tot = mu.sum(1)
        on = tot > q.fuzz
        # v* - v_l from velocity differences: free of the sums' cancellation
        rel = torch.where(on[:, None], (mu[..., None] * dv).sum(1) / torch.where(on, tot, torch.ones_like(tot))[:, None],
                          -V.mean(dim=1))
        D = self.div + q.small
        nb = self.div[self.nb]
        far = torch.where(self.no_nb, torch.full_like(nb, math.inf), nb).min(dim=1).values
        near = torch.where(self.no_nb, torch.full_like(nb, -math.inf), nb).max(dim=1).values
        pick = torch.where(D > 0, far, near)
        lone = self.no_nb.all(dim=1)
        r = torch.where(lone, torch.ones_like(pick), 0.9 * (torch.where(lone, D, pick) + q.small) / D)
        phi = 1.0 - r.clamp(min=0.0, max=1.0)
        length = self.vol ** (1.0 / 3.0) if self.dims == 3 else self.area.sqrt()
        phi = phi * (20.0 * length * self.div.abs() / (self.c + q.fuzz)).clamp(max=1.0)
        F = self.B * self.pres[:, None, None] + (phi[:, None] * mu)[..., None] * (rel[:, None, :] - dv)
        if self.strength:
            F = F - torch.einsum("elk,ekd->eld", self.B, self.stress)
        return F

    def cycle(self, dt):
        S = self.p.params.rk_num_stages
        x0, v0, e0, s0 = self.x, self.v, self.sie, self.stress
        self.start = (x0, v0, e0, s0)
        for k in range(S):
            a = dt / (S - k)
            self.div_used, F = self.div, self.force()
            self.F = F
            if self.strength:
                L = torch.einsum("eli,elj->eij", self.v[self.nie], self.B) / self.vol[:, None, None]
                E = 0.5 * (L + L.transpose(1, 2))
                E = E - torch.eye(3, dtype=E.dtype, device=E.device) * (E.diagonal(dim1=1, dim2=2).sum(1) / 3.0)[:, None, None]
                self.stress = s0 + (a * 2.0 * self.shear)[:, None, None] * E
            total = torch.zeros_like(x0).index_add(0, self.nie.reshape(-1), F.reshape(-1, self.dims))
            v1 = (v0 + a * total / self.node_mass[:, None]) * self.free
            half = 0.5 * (v0 + v1)
            r_in = self.x[:, 1]
            x1 = x0 + a * half
            H = half[self.nie]
            if self.dims == 2:
                H = H * r_in[self.nie][..., None]
            self.sie = e0 - a / self.mass * (F * H).sum(dim=(1, 2))
            self.x, self.v = x1, v1
            self.B, self.vol, self.area = self.geometry(x1)
            self.den = self.mass / self.vol
            self.eos()
            self.div = self.divergence()
            if self.dims == 2:
                y = x1[:, 1]
                off = y > self.p.params.tiny
                m = torch.where(off, self.ext / torch.where(off, y, torch.ones_like(y)), torch.zeros_like(y))
                a_, b_ = self.edges[:, 0], self.edges[:, 1]
                take = (y[a_] < self.p.params.tiny) & off[b_]
                best = torch.zeros_like(m).scatter_reduce(0, a_[take], m[b_[take]] / 2.0, "amax")
                self.node_mass = torch.where(y < self.p.params.tiny, torch.maximum(m, best), m)

    def go(self, cycles, chunk=0, checkpoint=False):
        q = self.p.params
        self.strength = any(m.strength != "none" for m in self.p.materials)
        self.eos()
        self.div = self.divergence()
        dt, t = self.f(q.dt_start), self.f(0.0)
        ran, tallies = 0, []
        names = ("x", "v", "sie", "vol", "den", "pres", "c", "div", "B")

        def one(dt, t, *held):
            for k, h in zip(names, held):
                setattr(self, k, h)
            dt = self.step(dt, t)
            self.cycle(dt)
            return (dt, t + dt) + tuple(getattr(self, k) for k in names)

        for _ in range(cycles):
            held = tuple(getattr(self, k) for k in names)
            if checkpoint:
                from torch.utils.checkpoint import checkpoint as ck
                res = ck(one, dt, t, *held, use_reentrant=False)
            else:
                res = one(dt, t, *held)
            dt, t = res[0], res[1]
            for k, h in zip(names, res[2:]):
                setattr(self, k, h)
            ran += 1
            if chunk and (ran % chunk == 0 or ran == cycles):
                w = self.node_mass * (self.x[:, 1] if self.dims == 2 else 1.0)
                tallies.append([float((self.mass * self.sie).sum()), float(0.5 * (w * (self.v ** 2).sum(1)).sum())])
        self.t, self.ran, self.tallies = t, ran, tallies
        return self

    def state(self):
        x0, v0, e0, s0 = self.start
        return {"node_coords": torch.stack([x0, self.x]), "node_vel": torch.stack([v0, self.v]),
                "node_mass": self.node_mass, "elem_den": self.den, "elem_pres": self.pres, "elem_sspd": self.c,
                "elem_sie": torch.stack([e0, self.sie]), "elem_vol": self.vol, "elem_div": self.div_used,
                "corner_force": self.F.reshape(-1, self.dims)}


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "batch":
        out = []
        for p in _members(case, seed):
            st = _Run(p, device).go(case["cycles"]).state()
            out.append([st[k] for k in ("node_coords", "node_vel", "elem_den", "elem_pres", "elem_sie")])
        return out
    p = _problem(case["deck"], case["n"], case["cycles"], seed)
    r = _Run(p, device)
    if case["kind"] == "adjoint":
        wden, wsie = (r.f(w) for w in _seeds(case, p, seed))
        r.sie.requires_grad_(True)
        r.gamma = r.gamma.clone().requires_grad_(True)
        r.v.requires_grad_(True)
        leaves = (r.sie, r.gamma, r.v)
        r.go(case["cycles"], checkpoint=True)
        J = (wden * r.den).sum() + (wsie * r.sie).sum()
        # taken before the backward pass, whose recomputation runs the cycles again
        out = {"cycles": r.ran, "den": r.den.detach(), "sie": torch.stack([r.start[2], r.sie]).detach()}
        out["dsie"], out["dgamma"], out["dvel"] = torch.autograd.grad(J, leaves)
        return out
    r.go(case["cycles"], chunk=case["chunk"])
    out = {"time": float(r.t), "cycles": r.ran, **r.state()}
    if case["chunk"]:
        out["tallies"] = np.array(r.tallies)
    if case["deck"] == "hypo":
        out["elem_stress"] = torch.stack([r.start[3], r.stress])
    return out

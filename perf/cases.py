"""The calls whose time matters to a user of this package, and what they give.

Each case is one call (or one time step) through the public entry points of
`dgv0d3v_direct_collision_b200`: the collision integral Q(f,f) in its three
arithmetics, Runge-Kutta steps, the Jacobian products that gradients and the
linearised operator need, and the mixed-grid batch.  Grids, batches, initial
data and time steps are those of the repository's own benchmark, tests and
training-data writer; the operator is the seeded synthetic A (the stand-in for
A-arrays that take hours to precompute), made once per grid as a program makes
or reads its operator once and then applies it to many distributions.

`exact` evaluates the same operator in plain torch in 64 bits: per cell c1 of
the first velocity one dense product over all second velocities, from its own
grid, weights and records.
"""
import math

import numpy as np
import torch

import dgv0d3v_direct_collision_b200 as dgv
from dgv0d3v_direct_collision_b200.autograd import collision

SEED_A = 20260101  # the benchmark's operator


def listed():
    return [
        # one Q of one VDF on the smallest production grid (15^3): what a
        # relaxation run or a parameter study calls over and over; latency
        {"name": "q15_f64", "op": "collide", "s": 3, "M": 5, "nb": 1, "precision": "f64", "projection": True,
         "host": False},
        # the Fortran driver's time step: RK2 on host arrays, advanced in place
        {"name": "rk2_15_f64_host", "op": "step", "s": 3, "M": 5, "nb": 1, "precision": "f64", "projection": False,
         "host": True, "order": 2, "dt": 0.01},
        # the relaxation run on 21^3 in the FP32-compensated arithmetic (RK4)
        {"name": "rk4_21_f32c", "op": "step", "s": 3, "M": 7, "nb": 1, "precision": "f32c", "projection": True,
         "host": False, "order": 4, "dt": 0.005},
        # the plain FP64 operator on the benchmark's grid, a small batch
        {"name": "q27_f64_b4", "op": "collide", "s": 3, "M": 9, "nb": 4, "precision": "f64", "projection": False,
         "host": False},
        # the benchmark: 256 VDFs on 27^3 on the tensor cores, projected
        {"name": "q27_tc_b256", "op": "collide", "s": 3, "M": 9, "nb": 256, "precision": "tc", "projection": True,
         "host": False},
        # a shard of training data from host arrays; a batch that fills no tile
        {"name": "q21_tc_b37_host", "op": "collide", "s": 3, "M": 7, "nb": 37, "precision": "tc", "projection": True,
         "host": True},
        # eight nodes per cell, a batch of more than one tile and not a multiple
        {"name": "q14_tc_b150", "op": "collide", "s": 2, "M": 7, "nb": 150, "precision": "tc", "projection": True,
         "host": False},
        # one training step's forward and backward through the autograd op, FP64
        {"name": "grad21_f64", "op": "grad", "s": 3, "M": 7, "nb": 1, "precision": "f64", "projection": False,
         "host": False},
        # the adjoint of a batch on the tensor cores
        {"name": "vjp21_tc_b150", "op": "vjp", "s": 3, "M": 7, "nb": 150, "precision": "tc", "projection": False,
         "host": False},
        # the linearised operator (mixed terms at a Maxwellian) on a perturbation
        {"name": "lin21_f64", "op": "linear", "s": 3, "M": 7, "nb": 1, "precision": "f64", "projection": False,
         "host": False},
        # the mixed batch: 21^3 and 15^3 grids in one call, perturbed mixtures
        {"name": "mixed_tc", "op": "group", "s": 3, "M": 7, "nb": 96, "s2": 3, "M2": 5, "nb2": 32, "precision": "tc",
         "projection": True, "host": False},
    ]


def _cost(c):
    """Rough cost of a case, in FP64 evaluations of one 27^3 VDF (FP64 and
    FP32-compensated: per VDF; tensor cores: per started 32 VDFs)."""
    def q(s, M, nb):
        return (s * M / 27.0) ** 8 * (nb if c["precision"] != "tc" else 0.6 * math.ceil(nb / 32))
    n = q(c["s"], c["M"], c["nb"])
    if c["op"] == "group":
        n += q(c["s2"], c["M2"], c["nb2"])
    return n * {"collide": 1, "group": 1, "linear": 1.3, "vjp": 2.2, "grad": 3.2, "step": c.get("order", 1)}[c["op"]]


def draw(rng):
    """One more case: any of the calls on grids of 2 or 3 nodes and 3 to 10
    cells per axis, batches of 1 to 256 of any size between."""
    while True:
        op = rng.choice(["collide", "collide", "collide", "step", "step", "vjp", "grad", "linear", "group"])
        prec = rng.choice(["f64", "f32c", "tc"]) if op in ("collide", "step") else (
            "f64" if op == "linear" else "tc" if op == "group" else rng.choice(["f64", "tc"]))
        s = rng.choice([2, 3, 3])
        c = {"op": op, "s": s, "M": rng.randint(3, 9 if s == 3 else 10), "precision": prec,
             "projection": rng.random() < 0.5, "host": op in ("collide", "step") and rng.random() < 0.25}
        most = 256 if prec == "tc" else 1 if op == "linear" else 32
        c["nb"] = min(most, int(round(math.exp(rng.uniform(0.0, math.log(most + 0.5))))))
        if op == "step":
            c["order"], c["dt"] = rng.choice([2, 4]), rng.choice([0.005, 0.01])
        if op in ("grad", "vjp", "linear"):
            c["projection"] = False
        if op == "group":
            c["s2"] = s
            c["M2"] = rng.choice([m for m in range(3, 8) if m != c["M"]])
            c["nb2"] = int(round(math.exp(rng.uniform(0.0, math.log(256.5)))))
        if s * c["M"] >= 9 and _cost(c) <= 4.0:  # no more than the largest of the list
            return c


# ---------------------------------------------------------------- inputs
def _extent(s, M):
    return 7.0 if s * M >= 27 else 6.0


_solvers = {}  # the operators a program keeps: those of the case at hand


def _solver(s, M):
    key = (s, M)
    if key not in _solvers:
        sol = dgv.DGVSolver(s, M, _extent(s, M))
        sol.generate_synthetic_A(seed=SEED_A, support=1)
        _solvers[key] = sol
    return _solvers[key]


def _grids(case):
    g = [(case["s"], case["M"], case["nb"])]
    if case["op"] == "group":
        g.append((case["s2"], case["M2"], case["nb2"]))
    return g


def _keep(case):
    want = {(s, M) for s, M, _ in _grids(case)}
    for key in [k for k in _solvers if k not in want]:
        del _solvers[key]  # a state that still holds one keeps it alive


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Nodes:
    """Nodes, weights and cells of the uniform grid, in the node order u, v, w
    with the cells outermost."""

    def __init__(self, s, M, L, device):
        # Gauss-Legendre rules of 2 and 3 points, the outer node by Newton's
        # method on P_s (to the last bit: pairs on the edge of the records'
        # support are decided by it)
        z = math.cos(math.pi * 0.75 / (s + 0.5))
        for _ in range(8):
            p = {2: (3.0 * z * z - 1.0) / 2, 3: (5.0 * z * ((3.0 * z * z - 1.0) / 2) - 2.0 * z) / 3}[s]
            below = {2: z, 3: (3.0 * z * z - 1.0) / 2}[s]
            z -= p / (s * (z * p - below) / (z * z - 1.0))
        x1 = {2: [-z, z], 3: [-z, 0.0, z]}[s]
        w1 = {2: [1.0, 1.0], 3: [5 / 9.0, 8 / 9.0, 5 / 9.0]}[s]
        g = -L + (2 * L) / float(M) * np.arange(M + 1)
        self.s, self.M, self.P, self.Nc = s, M, s ** 3, M ** 3
        self.N, self.cc, self.edges = self.P * self.Nc, M // 2, g
        n1 = np.array([[x * (g[c + 1] - g[c]) / 2.0 + (g[c + 1] + g[c]) / 2.0 for x in x1] for c in range(M)])
        full = (M, M, M, s, s, s)
        u = np.broadcast_to(n1[:, None, None, :, None, None], full).reshape(-1)
        v = np.broadcast_to(n1[None, :, None, None, :, None], full).reshape(-1)
        w = np.broadcast_to(n1[None, None, :, None, None, :], full).reshape(-1)
        h = g[1:] - g[:-1]
        q = np.array(w1)
        wt = (q[:, None, None] * q[None, :, None] * q[None, None, :])[None, None, None] * \
            h[:, None, None, None, None, None] * h[None, :, None, None, None, None] * h[None, None, :, None, None, None] / 8.0
        t = lambda a: torch.from_numpy(np.array(a)).to(device)  # noqa: E731
        self.u, self.v, self.w, self.wt = t(u), t(v), t(w), t(np.broadcast_to(wt, full).reshape(-1))


_nodes_of = {}


def _nodes(s, M):
    key = (s, M, str(_device()))
    if key not in _nodes_of:
        _nodes_of.clear()
        _nodes_of[key] = _Nodes(s, M, _extent(s, M), _device())
    return _nodes_of[key]


def _mixtures(n, nb, rng, perturb=0.0):
    """nb mixtures of 1-4 Maxwellians (weights ~ Dirichlet(1), bulk velocities
    ~ U[-2,2]^3, temperatures ~ U[0.5,2]), density 1; with `perturb` each
    node times 1 + perturb N(0,1), clipped at 0."""
    par = np.zeros((nb, 4, 5))
    par[:, :, 4] = 1.0
    for b in range(nb):
        k = int(rng.integers(1, 5))
        par[b, :k, 0] = rng.dirichlet(np.ones(k))
        par[b, :k, 1:4] = rng.uniform(-2, 2, (k, 3))
        par[b, :k, 4] = rng.uniform(0.5, 2.0, k)
    par = torch.from_numpy(par).to(n.u.device)
    f = torch.zeros((nb, n.N), dtype=torch.float64, device=n.u.device)
    for j in range(4):
        wt, a, b, c, T = (par[:, j, i:i + 1] for i in range(5))
        f += wt * torch.exp(-((n.u - a) ** 2 + (n.v - b) ** 2 + (n.w - c) ** 2) / T) / (math.pi * T) ** 1.5
    if perturb:
        f *= (1.0 + perturb * _normal(n, nb, rng)).clamp_min(0.0)
    return f / (f * n.wt).sum(1, keepdim=True)


def _normal(n, nb, rng):
    gen = torch.Generator(device=n.u.device).manual_seed(int(rng.integers(1 << 60)))
    return torch.randn((nb, n.N), dtype=torch.float64, device=n.u.device, generator=gen)


def _inputs(case, seed):
    """Per grid of the case: the arrays the call takes, [nb, N] (one VDF: [N])."""
    out = []
    for i, (s, M, nb) in enumerate(_grids(case)):
        rng = np.random.default_rng([int(seed), i])
        n = _nodes(s, M)
        a = {"f": _mixtures(n, nb, rng, 0.1 if case["op"] == "group" else 0.0)}
        if case["op"] in ("vjp", "grad"):
            a["v"] = _normal(n, nb, rng)  # the cotangent
        if case["op"] == "linear":  # a Maxwellian and a perturbation of it
            T, u0 = rng.uniform(0.5, 2.0), rng.uniform(-0.5, 0.5, 3)
            r2 = (n.u - u0[0]) ** 2 + (n.v - u0[1]) ** 2 + (n.w - u0[2]) ** 2
            a["f"] = (torch.exp(-r2 / T) / (math.pi * T) ** 1.5)[None]
            a["v"] = a["f"] * 0.01 * _normal(n, 1, rng)
        out.append({k: (x[0] if nb == 1 else x).contiguous() for k, x in a.items()})
    return out


def prepare(case, seed):
    """The operator (kept from call to call) and this seed's arrays."""
    _keep(case)
    arrays = _inputs(case, seed)
    if case["host"]:
        arrays = [{k: x.cpu().numpy().copy() for k, x in a.items()} for a in arrays]
    elif torch.cuda.is_available():
        torch.cuda.synchronize()  # the library works on a stream of its own
    members = []
    for (s, M, nb), a in zip(_grids(case), arrays):
        sol = _solver(s, M)
        sol.set_projection(case["projection"])
        like = np.zeros_like if case["host"] else torch.zeros_like
        members.append(dict(a, solver=sol, q=like(a["f"]), r=like(a["f"])))
    if not case["host"] and torch.cuda.is_available():
        torch.cuda.synchronize()
    return {"case": case, "members": members}


def run(state):
    case, m = state["case"], state["members"][0]
    sol, op, prec = m["solver"], case["op"], case["precision"]
    if op == "collide":
        return sol.EvalCollisionPeriodicAPlus_DGV(m["f"], m["q"], precision=prec)
    if op == "step":  # f is advanced in place
        sol.TimeIntegratorORK_SH_DGV(m["f"], case["dt"], m["r"], order=case["order"], precision=prec)
        return [m["f"], m["r"]]
    if op == "vjp":
        return sol.vjp(m["f"], m["v"], m["q"], precision=prec)
    if op == "grad":
        f = m["f"].detach().requires_grad_(True)
        q = collision(f, sol, precision=prec)
        return [q.detach(), torch.autograd.grad(q, f, m["v"])[0]]
    if op == "linear":
        return sol.EvalCollisionPeriodicMixedTermsA_DGV(m["v"], m["f"], m["q"])
    if op == "group":
        return dgv.collide_group([(x["solver"], x["f"], x["q"]) for x in state["members"]], precision=prec)
    raise ValueError(op)


def work(case):
    """Reads of A (its values once in the arithmetic's width, one pair of node
    indices per unordered pair), f and the results; per record and shift one
    multiply-add, per pair and shift the product of the two f (the adjoint: the
    two scattered products)."""
    byts = flops = 0.0
    for s, M, nb in _grids(case):
        info = _solver(s, M).A_info()
        P, N = s ** 3, (s * M) ** 3
        word = 8 if case["precision"] == "f64" else 4
        a_bytes = info["records"] * word + info["pairs"] * 8
        shifts = info["record_shifts"]
        fwd, adj = shifts * (2 + 1 / P), shifts * (2 + 4 / P)
        nq = {"collide": 1, "group": 1, "linear": 1, "step": case.get("order", 1), "vjp": 0, "grad": 1}[case["op"]]
        na = {"vjp": 1, "grad": 1}.get(case["op"], 0)
        flops += nb * (nq * fwd * (1.5 if case["op"] == "linear" else 1.0) + na * adj)
        byts += (nq + na) * a_bytes + nb * N * 8 * {"collide": 2, "group": 2, "linear": 3, "step": 3, "vjp": 3,
                                                    "grad": 4}[case["op"]]
    return {"bytes": byts, "flops": flops}


# ---------------------------------------------------------------- 64 bits
def _signed(x):
    return x - (1 << 64) if x >= 1 << 63 else x


def _splitmix(x):
    """splitmix64 of an int64 tensor (the bits of unsigned 64-bit words)."""
    def shr(a, k):
        return (a >> k) & ((1 << (64 - k)) - 1)
    x = x + _signed(0x9E3779B97F4A7C15)
    x = (x ^ shr(x, 30)) * _signed(0xBF58476D1CE4E5B9)
    x = (x ^ shr(x, 27)) * _signed(0x94D049BB133111EB)
    return x ^ shr(x, 31)


class _Operator:
    """Q, its mixed terms and its adjoint over the synthetic records."""

    def __init__(self, n):
        self.n = n
        M, dev = n.M, n.u.device
        g, c = n.edges, n.cc
        self.lo, self.hi = float(g[c]), float(g[c + 1])
        e = self.hi - self.lo
        self.dphi = math.sqrt((e * e + e * e) + e * e)
        cell = torch.arange(n.Nc, device=dev)
        self.xyz = torch.stack([cell // (M * M), cell // M % M, cell % M], 1)
        self.key = _splitmix(torch.tensor(_signed(SEED_A), dtype=torch.int64, device=dev))

    def records(self, c1):
        """Values [nodes of the cells >= c1, P (l1), P (p)] of the pairs whose
        first velocity lies in c1."""
        n, P = self.n, self.n.P
        a, b = torch.arange(c1 * P, (c1 + 1) * P, device=n.u.device), torch.arange(c1 * P, n.N, device=n.u.device)
        ax = [x[a][None, :] for x in (n.u, n.v, n.w)]
        bx = [x[b][:, None] for x in (n.u, n.v, n.w)]
        d = [p - q for p, q in zip(ax, bx)]
        dsph = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
        m = [p + q - self.lo - self.hi for p, q in zip(ax, bx)]
        dist = torch.sqrt(m[0] * m[0] + m[1] * m[1] + m[2] * m[2])
        ok = ~((dist > dsph + self.dphi) | (dist + self.dphi < dsph))
        near, far = torch.zeros_like(dsph), torch.zeros_like(dsph)
        for p, q in zip(ax, bx):  # the collision sphere has to meet the canonical cell
            x = (p + q) / 2.0
            t = torch.maximum(torch.clamp(self.lo - x, min=0.0), torch.clamp(x - self.hi, min=0.0))
            near = near + t * t
            t = torch.maximum((x - self.lo).abs(), (x - self.hi).abs())
            far = far + t * t
        r2 = (dsph / 2.0) * (dsph / 2.0)
        ok &= (r2 >= near) & (r2 <= far) & (b[:, None] > a[None, :])
        ab = ((a[None, :] << 24) ^ b[:, None])[:, :, None]
        h = _splitmix((ab ^ (torch.arange(P, device=n.u.device) << 48)) ^ self.key)
        u = ((h >> 11) & ((1 << 53) - 1)).double() * (2.0 / 9007199254740992.0) - 1.0
        scale = torch.where(ok, n.wt[a][None, :] * n.wt[b][:, None] * (dsph / 8.0), torch.zeros_like(dsph))
        return u * scale[:, :, None]

    def cells(self, c1):
        """The output cells D whose first cell c1 + D - cc lies in the grid:
        (D, that cell, the second cells of every c2 >= c1 with Nc for those
        outside)."""
        n, M = self.n, self.n.M
        s1 = self.xyz + self.xyz[c1] - n.cc
        D = torch.nonzero(((s1 >= 0) & (s1 < M)).all(1))[:, 0]
        first = (s1[D, 0] * M + s1[D, 1]) * M + s1[D, 2]
        s2 = self.xyz[None, c1:] + self.xyz[D][:, None] - n.cc
        second = (s2[..., 0] * M + s2[..., 1]) * M + s2[..., 2]
        return D, first, torch.where(((s2 >= 0) & (s2 < M)).all(2), second, torch.full_like(second, n.Nc))

    def _fold(self, f):
        z = torch.zeros((f.shape[0], 1, self.n.P), dtype=f.dtype, device=f.device)
        return torch.cat([f.reshape(f.shape[0], self.n.Nc, self.n.P), z], 1)

    def bilinear(self, f, g=None):
        """2/w sum A f f, or with g the mixed terms 2/w sum A (f g + g f)."""
        n, P = self.n, self.n.P
        F, G = self._fold(f), None if g is None else self._fold(g)
        out = torch.zeros((f.shape[0], n.Nc, P), dtype=f.dtype, device=f.device)
        for c1 in range(n.Nc):
            W = self.records(c1).reshape(-1, P * P)
            D, first, second = self.cells(c1)
            if not len(D):
                continue
            def term(x, y):  # noqa: E306
                prod = (y[:, second].reshape(-1, W.shape[0]) @ W).reshape(f.shape[0], len(D), P, P)
                return torch.einsum("bdi,bdip->bdp", x[:, first], prod)
            out[:, D] += term(F, F) if G is None else term(F, G) + term(G, F)
        return 2.0 * out.reshape(f.shape[0], n.N) / n.wt

    def adjoint(self, f, v):
        n, P = self.n, self.n.P
        F, c = self._fold(f), (2.0 * v / n.wt).reshape(f.shape[0], n.Nc, P)
        out = torch.zeros_like(F)
        for c1 in range(n.Nc):
            W = self.records(c1).reshape(-1, P * P)
            D, first, second = self.cells(c1)
            if not len(D):
                continue
            prod = (F[:, second].reshape(-1, W.shape[0]) @ W).reshape(f.shape[0], len(D), P, P)
            out[:, first] += torch.einsum("bdp,bdip->bdi", c[:, D], prod)
            h = (F[:, first][..., None] * c[:, D][:, :, None, :]).reshape(-1, P * P)
            back = (h @ W.T).reshape(f.shape[0], -1, P)
            out.index_add_(1, second.reshape(-1), back)
        return out[:, :-1].reshape(f.shape[0], n.N)

    def project(self, q):
        """q without its components along 1, u, v, w, |v|^2."""
        n = self.n
        psi = torch.stack([torch.ones_like(n.u), n.u, n.v, n.w, n.u ** 2 + n.v ** 2 + n.w ** 2])
        lam = torch.linalg.solve((psi * n.wt) @ psi.T, ((q * n.wt) @ psi.T).T).T
        return q - lam @ psi


def _exact_seconds(case):
    """Rough time of the dense products below: FP64 operations over a rate."""
    t = 0.0
    for s, M, nb in _grids(case):
        dense = M ** 3 * (0.35 * M ** 3) * (0.5 * (s * M) ** 3) * s ** 6 * 2 * nb
        t += (dense / 2e13 + M ** 3 * (2e-3 + (s * M) ** 3 * s ** 6 * 2e-10)) * {
            "step": case.get("order", 1), "grad": 3, "vjp": 2, "linear": 2}.get(case["op"], 1)
    return t


def exact(case, seed):
    if _exact_seconds(case) > 15.0 or not torch.cuda.is_available():
        return None
    outs = []
    for (s, M, nb), a in zip(_grids(case), _inputs(case, seed)):
        op = _Operator(_nodes(s, M))
        f = a["f"].reshape(nb, -1)

        def q_of(x):
            q = op.bilinear(x)
            return op.project(q) if case["projection"] else q

        def shaped(x):
            return x.reshape(a["f"].shape)

        if case["op"] in ("collide", "group"):
            outs.append(shaped(q_of(f)))
        elif case["op"] == "vjp":
            return shaped(op.adjoint(f, a["v"].reshape(nb, -1)))
        elif case["op"] == "grad":
            return [shaped(q_of(f)), shaped(op.adjoint(f, a["v"].reshape(nb, -1)))]
        elif case["op"] == "linear":
            return shaped(op.bilinear(f, a["v"].reshape(nb, -1)))
        else:  # the stages of the two- and four-stage schemes
            dt = case["dt"]
            k1 = q_of(f)
            if case["order"] == 2:
                new = f + dt * (k1 / 4.0 + q_of(f + dt * k1 * (2.0 / 3.0)) * 0.75)
            else:
                k2 = q_of(f + dt * k1 / 2.0)
                k3 = q_of(f + dt * (k1 / 4.0 + k2 / 4.0))
                new = f + dt * (k1 / 6.0 + k3 * (2.0 / 3.0) + q_of(f - dt * k2 + dt * k3 * 2.0) / 6.0)
            return [shaped(new), shaped(k1)]
    return outs if case["op"] == "group" else outs[0]

"""Performance cases of the UGKS time step.

Each case is one call that a user's program makes again and again: some steps
of one cavity or channel (``FusedSolver.step``), one step of a batch of
cavities, a tick of a serving pool (``SolvePool.tick``), or one step of the
per-kernel driver (``UGKSim.one_step``).  The sizes are those of ``configs``
(the 32x32 cavity, the 2x2-block cavity, the 256x64 channel, the batched
cavities with n in 24..128 and 16..48 velocities per axis), of the serving
stream, and odd ones between them.

The state starts from smooth random fields of density, velocity and
temperature made from the seed; ``exact`` is the same scheme written in plain
torch in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

# flux_method names of the case descriptions: vanLeer, WENO5, minmod
_CFL = 0.2


def listed():
    return [
        # the smallest solves a user submits (serving requests, parameter
        # sweeps): launches and latency decide
        dict(name="cavity24_fp64", kind="cavity", n=24, nj=24, m=16, vlim=5.0, scheme="vanLeer", precision="fp64",
             Kn=0.1, steps=8),
        dict(name="cavity24_mixed", kind="cavity", n=24, nj=24, m=16, vlim=5.0, scheme="WENO5", precision="mixed",
             Kn=0.3, steps=8),
        # the 32x32 cavity with 25x25 velocities that users start from
        dict(name="cavity32_fp64", kind="cavity", n=32, nj=32, m=24, vlim=4.0, scheme="vanLeer", precision="fp64",
             Kn=0.075, steps=4),
        # an odd, curvilinear grid with the minmod limiter
        dict(name="warped61x45_mixed", kind="warped", n=61, nj=45, m=20, vlim=5.0, scheme="minmod", precision="mixed",
             Kn=0.05, steps=2),
        # the 2x2-block WENO5 cavity, the workload quoted for the framework,
        # in both storage precisions
        dict(name="blocks128_fp64", kind="blocks", nb=2, n=64, m=32, vlim=5.0, scheme="WENO5", precision="fp64",
             Kn=0.01, steps=1),
        dict(name="blocks128_mixed", kind="blocks", nb=2, n=64, m=32, vlim=5.0, scheme="WENO5", precision="mixed",
             Kn=0.01, steps=1),
        # the pressure-driven channel with an adsorbing wall
        dict(name="channel256x64_fp64", kind="channel", nb=4, n=64, nj=64, m=32, vlim=5.0, scheme="WENO5",
             precision="fp64", Kn=0.05, steps=1),
        # a wide velocity grid (rarefied flow)
        dict(name="cavity96_wide_fp64", kind="cavity", n=96, nj=96, m=48, vlim=5.0, scheme="vanLeer",
             precision="fp64", Kn=0.5, steps=1),
        # batches of independent cavities of mixed sizes and limiters
        dict(name="batch16_mixed", kind="batch", count=16, sizes=1, precision="mixed", steps=1),
        dict(name="batch16_fp64", kind="batch", count=16, sizes=1, precision="fp64", steps=1),
        # a tick of the continuous-batching server
        dict(name="serve6_mixed", kind="serve", count=6, sizes=7, precision="mixed", steps=10),
        # the per-kernel path that replaces pyUGKS's OpenCL program
        dict(name="dropin64_fp64", kind="dropin", nb=2, n=32, m=24, vlim=4.0, scheme="vanLeer", precision="fp64",
             Kn=0.075, steps=1),
    ]


def draw(rng):
    """A case of the listed kinds with sizes spread over the same ranges."""
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["cavity", "cavity", "cavity", "warped", "blocks", "blocks", "channel", "batch", "batch",
                       "serve", "dropin"])
    precision = "fp64" if kind == "dropin" else rng.choice(["fp64", "mixed"])
    if kind == "batch":
        case = dict(kind=kind, count=rng.randint(3, 14), sizes=rng.randint(100, 100000), precision=precision, steps=1)
        while _units(case) > 100e6:  # no larger than the listed batch
            case["count"] -= 1
        return case
    if kind == "serve":
        return dict(kind=kind, count=rng.randint(2, 8), sizes=rng.randint(100, 100000), precision=precision,
                    steps=rng.randint(4, 12))
    scheme = rng.choice(["vanLeer", "WENO5", "WENO5", "minmod"])
    # the velocity count is rounded to 4k + 1 per axis
    case = dict(kind=kind, m=4 * rng.randint(4, 12), vlim=5.0, scheme=scheme, precision=precision,
                Kn=round(math.exp(rng.uniform(math.log(0.05), math.log(1.0))), 4), steps=1)
    if kind in ("cavity", "warped"):
        case["n"], case["nj"] = spread(24, 112), spread(24, 112)
        case["steps"] = 4 if case["n"] * case["nj"] < 1600 else 1
    elif kind == "blocks":
        case["nb"] = rng.choice([2, 2, 3])
        case["n"] = spread(14, 64 if case["nb"] == 2 else 40)
    elif kind == "channel":
        case.update(nb=rng.randint(2, 4), n=spread(16, 64), nj=spread(16, 64))
    else:
        case.update(nb=rng.choice([1, 2]), n=spread(16, 32), m=4 * rng.randint(4, 8))
    return case


# ---------------------------------------------------------------------------
# problems: plain descriptions, used by prepare (as configs' case dicts) and
# by exact (as they are)
# ---------------------------------------------------------------------------
def _smooth(rng, ni, nj, amp):
    """amp times a smooth random field of unit size on ni x nj cells."""
    x = (np.arange(ni) + 0.5)[:, None] / ni
    y = (np.arange(nj) + 0.5)[None, :] / nj
    f = np.zeros((ni, nj))
    for _ in range(6):
        kx, ky = rng.integers(0, 4, 2)
        px, py = rng.uniform(0, 2 * np.pi, 2)
        f += rng.standard_normal() * np.cos(np.pi * kx * x + px) * np.cos(np.pi * ky * y + py)
    return amp * f / math.sqrt(6.0)


def _fields(rng, ni, nj):
    """Start-up density, velocities and temperature of a low-speed gas."""
    return dict(D=1.0 + _smooth(rng, ni, nj, 0.02), U=_smooth(rng, ni, nj, 0.03), V=_smooth(rng, ni, nj, 0.03),
                T=1.0 + _smooth(rng, ni, nj, 0.02))


def _batch_shapes(count, sizes):
    """(n, m, scheme, Kn, lid, T_wall) of the cavities of a batch, drawn as
    the batched-cavity workload draws them."""
    rng = np.random.default_rng(sizes)
    out = []
    for _ in range(count):
        n = int(rng.choice((24, 32, 48, 64, 96, 128)))
        m = int(rng.choice((16, 24, 32, 48)))
        Kn = float(10 ** rng.uniform(np.log10(0.005), 0.0))
        lid = float(rng.uniform(0.05, 0.3))
        Tw = float(rng.uniform(0.8, 1.2))
        out.append((n, m, "WENO5" if rng.random() < 0.5 else "vanLeer", Kn, lid, Tw))
    return out


def _shapes(case):
    if case["kind"] == "batch":
        return _batch_shapes(case["count"], case["sizes"])
    # serving requests of the small end
    return [(min(n, 48), min(m, 24), s, Kn, lid, Tw)
            for n, m, s, Kn, lid, Tw in _batch_shapes(case["count"], case["sizes"])]


def _problems(case, seed):
    """The solves of a case: dicts of scheme, m, vlim, Kn and blocks; a block
    has ni, nj, its corner coordinates, four faces (north, east, south, west)
    and start-up fields."""
    rng = np.random.default_rng([seed, 20])
    wall = lambda T=1.0, U=0.0: ("diffuse", T, U)
    kind = case["kind"]

    def cavity(n, nj, m, vlim, scheme, Kn, lid, Tw, warp=0.0):
        return dict(scheme=scheme, m=m, vlim=vlim, Kn=Kn, warp=warp, blocks=[
            dict(ni=n, nj=nj, box=(0.0, 1.0, 0.0, 1.0), bc=[wall(Tw, lid), wall(Tw), wall(Tw), wall(Tw)],
                 fill=_fields(rng, n, nj))])

    if kind in ("batch", "serve"):
        return [cavity(n, n, m, 5.0, s, Kn, lid, Tw) for n, m, s, Kn, lid, Tw in _shapes(case)]
    if kind in ("cavity", "warped"):
        return [cavity(case["n"], case["nj"], case["m"], case["vlim"], case["scheme"], case["Kn"], 0.15, 1.0,
                       0.04 if kind == "warped" else 0.0)]
    nb, n = case["nb"], case["n"]
    head = dict(scheme=case["scheme"], m=case["m"], vlim=case["vlim"], Kn=case["Kn"], warp=0.0)
    blocks = []
    if kind == "channel":
        nj, length = case["nj"], 4.0
        f = _fields(rng, nb * n, nj)
        f["D"] = f["D"] + 0.2 * (1.0 - (np.arange(nb * n) + 0.5)[:, None] / (nb * n))
        for b in range(nb):
            blocks.append(dict(
                ni=n, nj=nj, box=(length * b / nb, length * (b + 1) / nb, 0.0, 1.0),
                bc=[wall(), ("adjacent", b + 1) if b + 1 < nb else ("inflow", 1.0), ("adsorbing", 1.0),
                    ("adjacent", b - 1) if b > 0 else ("inflow", 1.2)],
                fill={k: np.ascontiguousarray(x[b * n:(b + 1) * n]) for k, x in f.items()}))
    else:  # nb x nb blocks of a cavity
        f = _fields(rng, nb * n, nb * n)
        for bi in range(nb):
            for bj in range(nb):
                blocks.append(dict(
                    ni=n, nj=n, box=(bi / nb, (bi + 1) / nb, bj / nb, (bj + 1) / nb),
                    bc=[("adjacent", bi * nb + bj + 1) if bj + 1 < nb else wall(1.0, 0.15),
                        ("adjacent", (bi + 1) * nb + bj) if bi + 1 < nb else wall(),
                        ("adjacent", bi * nb + bj - 1) if bj > 0 else wall(),
                        ("adjacent", (bi - 1) * nb + bj) if bi > 0 else wall()],
                    fill={k: np.ascontiguousarray(x[bi * n:(bi + 1) * n, bj * n:(bj + 1) * n])
                          for k, x in f.items()}))
    return [dict(head, blocks=blocks)]


def _vertices(b, warp):
    """Vertex coordinates (ni + 1, nj + 1) of a block."""
    x0, x1, y0, y1 = b["box"]
    i = np.arange(b["ni"] + 1, dtype=np.float64)[:, None]
    j = np.arange(b["nj"] + 1, dtype=np.float64)[None, :]
    x = x0 + (x1 - x0) * (i / b["ni"]) + 0.0 * j
    y = y0 + (y1 - y0) * (j / b["nj"]) + 0.0 * i
    if warp:
        x, y = (x + warp * np.sin(2 * np.pi * x) * np.sin(np.pi * y),
                y + warp * np.sin(np.pi * x) * np.sin(2 * np.pi * y))
    return np.ascontiguousarray(x), np.ascontiguousarray(y)


def _config(p):
    """A problem as the case dict of ``configs``."""
    from pyugks_b200 import configs
    case = configs.base_case(p["scheme"], p["Kn"], p["m"], p["vlim"], CFL=_CFL)
    opposite = [2, 3, 0, 1]
    for b in p["blocks"]:
        x, y = _vertices(b, p["warp"])
        bc = []
        for face, c in enumerate(b["bc"]):
            if c[0] == "diffuse":
                bc.append(configs.diffuse(c[1], U=c[2]))
            elif c[0] == "adjacent":
                bc.append(configs.adjacent(c[1], opposite[face]))
            elif c[0] == "inflow":
                bc.append(configs.inflow(c[1], 1.0))
            else:
                bc.append(configs.adsorbing(c[1]))
        case["blocks"].append(dict(ni=b["ni"], nj=b["nj"], x=x, y=y, bc=bc, fill=dict(b["fill"], qx=0.0, qy=0.0)))
    return case


# ---------------------------------------------------------------------------
# the measured calls
# ---------------------------------------------------------------------------
def prepare(case, seed):
    cases = [_config(p) for p in _problems(case, seed)]
    if case["kind"] == "dropin":
        from pyugks_b200.ugks_sim import UGKSim
        sim = UGKSim(cases[0])
        return dict(case=case, sim=sim, out=[dict(f=b.f_D, macro=b.macro_D) for b in sim.blocks])
    if case["kind"] == "serve":
        from pyugks_b200.serving import SolvePool
        pool = SolvePool(precision=case["precision"])
        ids = [pool.admit(c) for c in cases]
        return dict(case=case, pool=pool, ids=ids,
                    out=[dict(f=b.f, macro=b.macro) for i in ids for b in pool.solves[i].solver.blocks])
    from pyugks_b200.fused import FusedSolver
    solver = FusedSolver(cases if case["kind"] == "batch" else cases[0], precision=case["precision"])
    out = []
    for k in range(len(cases)):
        for i in solver.solve_block_ids(k):
            b = solver.blocks[i]
            out.append(dict(f=b.f, macro=b.macro))
            if case["kind"] == "channel":
                out[-1]["cover"] = b.wall_cover
    return dict(case=case, solver=solver, out=out)


def run(state):
    case = state["case"]
    if case["kind"] == "dropin":
        for _ in range(case["steps"]):
            if state["sim"].one_step():
                raise RuntimeError("the step flagged an error")
        return state["out"]
    if case["kind"] == "serve":
        # the server reads the solve records after each tick
        pool = state["pool"]
        pool.tick(case["steps"])
        records = pool.states(rebuild=False)
        return dict(solves=state["out"], steps=np.array([records[i]["steps"] for i in state["ids"]]),
                    residual=np.array([records[i]["residual"] for i in state["ids"]], dtype=np.float32))
    state["solver"].step(case["steps"])
    return state["out"]


def work(case):
    """f is read and written once per step; operations of the reconstruction,
    moments and fluxes of two faces and of the update per cell and velocity."""
    size = 8 if case["precision"] == "fp64" else 4
    units, weno = 0, 0
    for cells, m, scheme in _sizes(case):
        nv = (m // 4 * 4 + 1) ** 2
        units += cells * nv
        weno += cells * nv * (scheme == "WENO5")
    return dict(bytes=float(case["steps"] * units * 4 * size),
                flops=float(case["steps"] * (units * (2 * (2 * 12 + 60) + 50) + weno * 2 * 2 * 40)))


def _sizes(case):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        return [(s[0] * s[0], s[1], s[2]) for s in _shapes(case)]
    n = case["n"]
    cells = n * case["nj"] if kind in ("cavity", "warped") else \
        case["nb"] * n * case["nj"] if kind == "channel" else (case["nb"] * n) ** 2
    return [(cells, case["m"], case["scheme"])]


def _units(case):
    """Cell-velocity points of one step."""
    return sum(cells * (m // 4 * 4 + 1) ** 2 for cells, m, _ in _sizes(case))


# ---------------------------------------------------------------------------
# the same steps in plain torch, 64 bits
# ---------------------------------------------------------------------------
_PI = float("%0.15e" % math.pi)
_PR, _GAM, _K, _OMEGA = float("%.12g" % (2.0 / 3.0)), float("%.12g" % (5.0 / 3.0)), 1.0, 0.81


def _newton(n):
    w = np.full(n, 64.0 / 45.0)
    k = np.arange(1, n + 1)
    w[(k - 5) % 4 == 0] = 28.0 / 45.0
    w[(k - 3) % 4 == 0] = 24.0 / 45.0
    w[0] = w[-1] = 14.0 / 15.0
    return w


def _velocities(m, vlim):
    n = m // 4 * 4 + 1
    d = (2 * vlim) / float(n - 1)
    u = np.array([-vlim + i * d for i in range(n)])
    w = _newton(n) * d
    round15 = lambda a: np.array([float("%0.15e" % x) for x in a.ravel()])
    return n, round15(u), round15(w[:, None] * w[None, :]), w


def _conserved(p):
    r, U, V, lam = p.unbind(-1)
    return torch.stack([r, r * U, r * V, 0.5 * r / lam / (_GAM - 1.0) + 0.5 * r * (U * U + V * V)], -1)


def _primary(w):
    r, a, b, e = w.unbind(-1)
    return torch.stack([r, a / r, b / r, 0.5 * r / (_GAM - 1.0) / (e - 0.5 * (a * a + b * b) / r)], -1)


def _maxwellian(p, u, v, wt):
    r, U, V, lam = (x.unsqueeze(-1) for x in p.unbind(-1))
    h = wt * (r * (lam / _PI) * torch.exp(-lam * ((u - U) ** 2 + (v - V) ** 2)))
    return h, h * _K / (2.0 * lam)


def _shakhov(p, q, u, v, h, b):
    r, U, V, lam = (x.unsqueeze(-1) for x in p.unbind(-1))
    cx, cy = u - U, v - V
    s = 0.8 * (1 - _PR) * lam * lam / r * (cx * q[..., 0:1] + cy * q[..., 1:2])
    part = 2 * lam * (cx * cx + cy * cy)
    return s * (part - 4) * h, s * (part - 2) * b


def _equilibrium(p, q, u, v, wt):
    h, b = _maxwellian(p, u, v, wt)
    sh, sb = _shakhov(p, q, u, v, h, b)
    return torch.stack([h + sh, b + sb], -1)


def _moments(f, u, v):
    h, b = f[..., 0], f[..., 1]
    return torch.stack([h.sum(-1), (u * h).sum(-1), (v * h).sum(-1),
                        0.5 * ((u * u + v * v) * h + b).sum(-1)], -1)


def _heat_flux(f, p, u, v):
    cx, cy = u - p[..., 1:2], v - p[..., 2:3]
    t = (cx * cx + cy * cy) * f[..., 0] + f[..., 1] / _K
    return torch.stack([0.5 * (cx * t).sum(-1), 0.5 * (cy * t).sum(-1)], -1)


def _tau(p, Kn):
    return Kn / p[..., 0] * p[..., 3] ** (1.0 - _OMEGA)


def _micro_slope(p, sw):
    r, U, V, lam = p.unbind(-1)
    s0, s1, s2, s3 = sw.unbind(-1)
    c = 0.5 * (_K + 2) / lam
    a3 = 4.0 * lam * lam / (_K + 2) / r * (2.0 * s3 - 2.0 * U * s1 - 2.0 * V * s2 + s0 * (U * U + V * V - c))
    a2 = 2.0 * lam / r * (s2 - V * s0) - V * a3
    a1 = 2.0 * lam / r * (s1 - U * s0) - U * a3
    a0 = s0 / r - U * a1 - V * a2 - 0.5 * (U * U + V * V + c) * a3
    return a0, a1, a2, a3


def _moment_uv(mu, mv, mx, a, b, d):
    return torch.stack([mu[a] * mv[b] * mx[d // 2], mu[a + 1] * mv[b] * mx[d // 2], mu[a] * mv[b + 1] * mx[d // 2],
                        0.5 * (mu[a + 2] * mv[b] * mx[d // 2] + mu[a] * mv[b + 2] * mx[d // 2] +
                               mu[a] * mv[b] * mx[(d + 2) // 2])], -1)


def _moment_au(a, mu, mv, mx, i, j):
    e = lambda x: x.unsqueeze(-1)
    return (e(a[0]) * _moment_uv(mu, mv, mx, i, j, 0) + e(a[1]) * _moment_uv(mu, mv, mx, i + 1, j, 0) +
            e(a[2]) * _moment_uv(mu, mv, mx, i, j + 1, 0) +
            e(0.5 * a[3]) * (_moment_uv(mu, mv, mx, i + 2, j, 0) + _moment_uv(mu, mv, mx, i, j + 2, 0) +
                             _moment_uv(mu, mv, mx, i, j, 2)))


def _slope(scheme, S, inv_l, ds):
    """Limited slope from the stencil cells S (upwind to downwind)."""
    if scheme == "WENO5":
        b = []
        for k, (c0, c1, c2) in enumerate(((1.0, -4.0, 3.0), (1.0, 0.0, -1.0), (3.0, -4.0, 1.0))):
            t1 = S[k] - 2.0 * S[k + 1] + S[k + 2]
            t2 = c0 * S[k] + c1 * S[k + 1] + c2 * S[k + 2]
            b.append((13.0 / 12.0) * t1 * t1 + 0.25 * t2 * t2)
        a = [c / (1e-16 + x) ** 2 for c, x in zip((0.1, 0.6, 0.3), b)]
        s = a[0] + a[1] + a[2]
        # the three candidate face values, less the middle cell
        f0 = (1.0 / 3.0) * (S[0] - S[1]) - (5.0 / 6.0) * (S[1] - S[2])
        f1 = (1.0 / 6.0) * (S[2] - S[1]) + (1.0 / 3.0) * (S[3] - S[2])
        f2 = (2.0 / 3.0) * (S[3] - S[2]) - (1.0 / 6.0) * (S[4] - S[3])
        return (a[0] / s * f0 + a[1] / s * f1 + a[2] / s * f2) / ds
    d1, d2 = S[1] - S[0], S[2] - S[1]
    if scheme == "vanLeer":
        s1, s2 = d1 * inv_l, d2 * inv_l
        return (torch.sign(s1) + torch.sign(s2)) * (s1.abs() * s2.abs()) / (s1.abs() + s2.abs() + 1e-16)
    m = torch.where((d2.abs() < d1.abs()) & (d1 * d2 > 0), d2,
                    torch.where((d1.abs() < d2.abs()) & (d1 * d2 > 0), d1,
                                torch.where(d1 == d2, d2, torch.zeros_like(d1))))
    return 0.5 * m / ds


class _Block:
    """One block of a problem in 64 bits."""

    def __init__(self, b, p, dev):
        self.ni, self.nj, self.bc = b["ni"], b["nj"], b["bc"]
        self.scheme, self.Kn, self.dev = p["scheme"], float("%0.15e" % p["Kn"]), dev
        self.G = 3 if p["scheme"] == "WENO5" else 2
        n, ax, wt, _ = _velocities(p["m"], p["vlim"])
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
        self.x, self.y, self.wt = t(np.repeat(ax, n)), t(np.tile(ax, n)), t(wt)
        self.umax = float("%.12g" % abs(p["vlim"]))
        self.geometry(*_vertices(b, p["warp"]))
        fill = b["fill"]
        self.macro = t(np.stack([fill["D"], fill["U"], fill["V"], 1.0 / fill["T"]], -1))
        self.f = torch.zeros((self.ni + 2 * self.G, self.nj + 2 * self.G, n * n, 2), dtype=torch.float64, device=dev)
        q = torch.zeros((self.ni, self.nj, 2), dtype=torch.float64, device=dev)
        self.inner = self.f[self.G:-self.G, self.G:-self.G]
        self.inner.copy_(_equilibrium(self.macro, q, self.x, self.y, self.wt))
        self.macro = _primary(_moments(self.inner, self.x, self.y))
        self.Q = _heat_flux(self.inner, self.macro, self.x, self.y)
        self.cover = torch.zeros((max(self.ni, self.nj), 4, 4), dtype=torch.float64, device=dev)

    def geometry(self, x, y):
        G, ni, nj = self.G, self.ni, self.nj
        xy = np.zeros((ni + 2 * G + 1, nj + 2 * G + 1, 2))
        xy[G:G + ni + 1, G:G + nj + 1, 0], xy[G:G + ni + 1, G:G + nj + 1, 1] = x, y
        for k in range(1, G + 1):  # ghost vertices continue the edge cells
            xy[G:-G, G + nj + k] = xy[G:-G, G + nj] + k * (xy[G:-G, G + nj] - xy[G:-G, G + nj - 1])
            xy[G + ni + k, G:-G] = xy[G + ni, G:-G] + k * (xy[G + ni, G:-G] - xy[G + ni - 1, G:-G])
            xy[G:-G, G - k] = xy[G:-G, G] + k * (xy[G:-G, G] - xy[G:-G, G + 1])
            xy[G - k, G:-G] = xy[G, G:-G] + k * (xy[G, G:-G] - xy[G + 1, G:-G])
        A, B, C, E = xy[1:, :-1], xy[1:, 1:], xy[:-1, 1:], xy[:-1, :-1]
        area = 0.5 * sum((P[..., 0] + O[..., 0]) * (P[..., 1] - O[..., 1]) for P, O in ((B, A), (C, B), (E, C), (A, E)))
        with np.errstate(all="ignore"):
            c = [1.0 / (6.0 * area) * s * sum((P[..., 1 - k] - O[..., 1 - k]) *
                                              (O[..., k] ** 2 + O[..., k] * P[..., k] + P[..., k] ** 2)
                                              for P, O in ((B, A), (C, B), (E, C), (A, E)))
                 for k, s in ((0, 1.0), (1, -1.0))]
            centre = np.stack(c, -1)
            normals, lens, mids = [], [], []
            for P, O in ((A, E), (E, C)):
                d = P - O
                lens.append(np.sqrt((d ** 2).sum(-1)))
                normals.append(np.stack([-d[..., 1], d[..., 0]], -1) / lens[-1][..., None])
                mids.append(0.5 * (P + O))
        self.t = t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)
        g = slice(G, -G)
        self.area = t(area[g, g])
        self.centre, self.normal = t(centre), [t(a) for a in normals]
        self.len, self.mid = [t(a) for a in lens], [t(a) for a in mids]
        edges = [np.abs(P - O) for P, O in ((A, B), (C, B), (C, E), (A, E), (C, A), (B, E))]
        ext = np.max(np.stack(edges), axis=0)[g, g]
        self.dx, self.dy = t(ext[..., 0]), t(ext[..., 1])

    def frequency(self):
        m = self.macro
        sos = torch.sqrt(0.5 * _GAM / m[..., 3])
        sc = (math.erf(10 * (self.Kn - 1e-3)) + 1) / 2.0
        sp = []
        for k in (1, 2):
            a = m[..., k].abs() + sos
            lo, hi = a.clamp(max=self.umax), a.clamp(min=self.umax)
            sp.append(sc * (hi - lo) + lo)
        return float(((self.dx * sp[0] + self.dy * sp[1]) / self.area).max())

    def flux(self, d, dt):
        """Face fluxes (per velocity and summed) of direction d: 0 the faces
        south of each cell, 1 the faces west of it."""
        G, ni, nj = self.G, self.ni, self.nj
        nf = (ni, nj + 1) if d == 0 else (ni + 1, nj)

        def at(a, o):  # cells o steps from the face along its normal
            i0, j0 = G + (o if d else 0), G + (0 if d else o)
            return a[i0:i0 + nf[0], j0:j0 + nf[1]]

        n, mid, ln = at(self.normal[d], 0), at(self.mid[d], 0), at(self.len[d], 0)
        nx, ny = n[..., 0:1], n[..., 1:2]
        u, v = self.x * nx + self.y * ny, self.y * nx - self.x * ny
        L, M = (5, 2) if self.scheme == "WENO5" else (3, 1)
        norm = lambda a: torch.sqrt((a * a).sum(-1))
        val, slp = [], []
        for sign in (1, -1):
            cells = [(-(M + 1) + s) if sign > 0 else (M - s) for s in range(L)]
            c, c2 = at(self.centre, cells[M]), at(self.centre, cells[M - 1])
            ds, il = norm(mid - c)[..., None, None], 1.0 / norm(c - c2)[..., None, None]
            s = _slope(self.scheme, [at(self.f, o) for o in cells], il, ds)
            slp.append(s)
            val.append(at(self.f, cells[M]) + s * ds)
        up = (u > 0).unsqueeze(-1)
        f, s = torch.where(up, val[0], val[1]), torch.where(up, slp[0], slp[1])
        del val, slp
        W = _moments(f, u, v)
        p = _primary(W)
        r, U, V, lam = p.unbind(-1)
        # half-range moments, slopes on both sides and in time
        sl, g = torch.sqrt(lam), 0.5 * torch.exp(-lam * U * U) / torch.sqrt(_PI * lam)
        half = []
        for sg in (1.0, -1.0):
            m = [0.5 * torch.special.erfc(-sg * sl * U)]
            m.append(U * m[0] + sg * g)
            for i in range(2, 7):
                m.append(U * m[-1] + 0.5 * (i - 1) * m[-2] / lam)
            half.append(m)
        full = [a + b for a, b in zip(*half)]
        mv = [torch.ones_like(V), V]
        for i in range(2, 5):
            mv.append(V * mv[-1] + 0.5 * (i - 1) * mv[-2] / lam)
        mx = [torch.ones_like(V), 0.5 * _K / lam, (_K * _K + 2.0 * _K) / (4.0 * lam * lam)]
        side = []
        for k, sg in ((-1, 1.0), (0, -1.0)):
            w = _moments(at(self.f, k), u, v)
            side.append(_micro_slope(p, sg * (W - w) / norm(mid - at(self.centre, k))[..., None]))
        e = lambda a: a.unsqueeze(-1)
        aT = _micro_slope(p, -e(r) * (_moment_au(side[0], half[0], mv, mx, 1, 0) +
                                      _moment_au(side[1], half[1], mv, mx, 1, 0)))
        tau = _tau(p, self.Kn)
        ex = torch.exp(-dt / tau)
        t3 = tau * (1.0 - ex)
        t4 = -tau * dt * ex + tau * t3
        t0 = dt - t3
        t1 = -tau * t0 + t4
        t2 = dt * dt / 2.0 - tau * t0
        g0 = e(r) * (e(t0) * _moment_uv(full, mv, mx, 1, 0, 0) +
                     e(t1) * (_moment_au(side[0], half[0], mv, mx, 2, 0) +
                              _moment_au(side[1], half[1], mv, mx, 2, 0)) +
                     e(t2) * _moment_au(aT, full, mv, mx, 1, 0))
        q = _heat_flux(f, p, u, v)
        h, b = _maxwellian(p, u, v, self.wt)
        sh, sb = _shakhov(p, q, u, v, h, b)
        T0, T1, T2, T3, T4 = (e(a) for a in (t0, t1, t2, t3, t4))
        zh = u * (T0 * sh + T3 * f[..., 0] - T4 * u * s[..., 0])
        zb = u * (T0 * sb + T3 * f[..., 1] - T4 * u * s[..., 1])
        uu, kb, k2 = u * u + v * v, e(mx[1]), e(mx[2])
        ph = lambda a: e(a[0]) + e(a[1]) * u + e(a[2]) * v + 0.5 * e(a[3]) * (uu + kb)
        pb = lambda a: kb * (e(a[0]) + e(a[1]) * u + e(a[2]) * v + 0.5 * e(a[3]) * uu) + 0.5 * e(a[3]) * k2
        pos = u > 0
        ah, ab = torch.where(pos, ph(side[0]), ph(side[1])), torch.where(pos, pb(side[0]), pb(side[1]))
        fh = zh + u * h * (T0 + T1 * u * ah + T2 * ph(aT))
        fb = zb + u * h * (T0 * kb + T1 * u * ab + T2 * pb(aT))
        mac = g0 + torch.stack([zh.sum(-1), (u * zh).sum(-1), (v * zh).sum(-1), 0.5 * (uu * zh + zb).sum(-1)], -1)
        dist = torch.stack([fh, fb], -1) * ln[..., None, None]
        mac = mac * ln[..., None]
        for wall in ((0, 2) if d == 0 else (1, 3)):  # faces of the walls
            c = self.bc[wall]
            if c[0] not in ("diffuse", "adsorbing"):
                continue
            k = -1 if wall < 2 else 0
            pick = lambda a: a[:, k] if d == 0 else a[k]
            fw, um = self.wall(wall, c, pick(f), pick(u), pick(v), pick(n), dt)
            scale = dt * pick(ln)
            pick(dist).copy_(um.unsqueeze(-1) * fw * scale[:, None, None])
            m4 = _moments(um.unsqueeze(-1) * fw, um, pick(v))
            pick(mac).copy_(m4 * scale[:, None])
        nx, ny = n[..., 0], n[..., 1]
        mac = torch.stack([mac[..., 0], nx * mac[..., 1] - ny * mac[..., 2], ny * mac[..., 1] + nx * mac[..., 2],
                           mac[..., 3]], -1)
        return dist, mac

    def wall(self, wall, c, f, u, v, n, dt):
        """The distribution at the faces of a diffuse or adsorbing wall."""
        rot = -1.0 if wall < 2 else 1.0
        out = u * rot > 0
        dl = out.double()
        Uw = c[2] if c[0] == "diffuse" else 0.0
        p = torch.stack([torch.ones_like(n[:, 0]), Uw * n[:, 0], -Uw * n[:, 1],
                         torch.full_like(n[:, 0], 1.0 / float("%.12g" % c[1]))], -1)
        M = torch.stack(_maxwellian(p, u, v, self.wt), -1)
        if c[0] == "diffuse":
            ratio = (u * (1 - dl) * f[..., 0]).sum(-1) / -(u * dl * M[..., 0]).sum(-1)
            return torch.where(out.unsqueeze(-1), ratio[:, None, None] * M, f), u
        gamma_f, alpha_p, k_des = 0.5, 1.0, 0.01
        nw = f.shape[0]
        theta = self.cover[:nw, wall, 0].clone()
        total = -rot * u * (1 - dl) * f[..., 0]
        ads = total * gamma_f * (1.0 - theta)[:, None]
        s0, s1 = (total - ads).sum(-1), ads.sum(-1)
        gain = torch.minimum(dt * alpha_p * s1, 1 - theta)
        ads_final = torch.where(dt * alpha_p * s1 > 1 - theta, gain / dt * alpha_p, s1)
        des = k_des * theta / alpha_p
        gain = gain - dt * alpha_p * des
        des = torch.where(theta + gain < 0, theta / (dt * alpha_p), des)
        refl = s0 + s1 - ads_final
        self.cover[:nw, wall] = torch.stack([theta + gain, refl, ads_final, des], -1)
        ratio = refl / (rot * u * dl * M[..., 0]).sum(-1)
        wd = p.clone()
        wd[:, 0] = 2 * des * torch.sqrt(_PI * p[:, 3])
        again = torch.stack(_maxwellian(wd, u, v, self.wt), -1)
        return torch.where(out.unsqueeze(-1), ratio[:, None, None] * M + again, f), u

    def update(self, dt):
        S, mS = self.flux(0, dt)
        W, mW = self.flux(1, dt)
        old, A = self.macro, self.area.unsqueeze(-1)
        q = _heat_flux(self.inner, old, self.x, self.y)
        new = _primary(_conserved(old) + (mS[:, :-1] - mS[:, 1:] + mW[:-1] - mW[1:]) / A)
        self.Q, self.old, self.macro = q, old, new
        e = lambda a: a.unsqueeze(-1).unsqueeze(-1)
        to, tn = e(_tau(old, self.Kn)), e(_tau(new, self.Kn))
        eo, en = (_equilibrium(p, q, self.x, self.y, self.wt) for p in (old, new))
        net = (S[:, :-1] - S[:, 1:] + W[:-1] - W[1:]) / e(self.area)
        self.next = (self.inner + net + 0.5 * dt * (en / tn + (eo - self.inner) / to)) / (1.0 + 0.5 * dt / tn)

    def ghosts(self, blocks):
        G, f = self.G, self.f
        for face, c in enumerate(self.bc):
            a = f if face in (0, 2) else f.transpose(0, 1)  # along the face, across it
            a = a[G:-G]
            last = a.shape[1] - G - 1
            for k in range(1, G + 1):
                g, e1, e0 = (last + k, last, last - 1) if face < 2 else (G - k, G, G + 1)
                if c[0] in ("diffuse", "adsorbing"):
                    a[:, g] = a[:, e1] + float(k) * (a[:, e1] - a[:, e0])
                elif c[0] == "adjacent":
                    o = blocks[c[1]]
                    b = (o.f if face in (0, 2) else o.f.transpose(0, 1))[G:-G]
                    a[:, g] = b[:, G + k - 1] if face < 2 else b[:, b.shape[1] - G - k]
                else:
                    i = -1 if face == 1 else 0
                    p = self.macro[i].clone()
                    p[:, 0], p[:, 3] = c[1], 1.0
                    a[:, g] = _equilibrium(p, self.Q[i], self.x, self.y, self.wt)


def _solve(p, steps, dev):
    blocks = [_Block(b, p, dev) for b in p["blocks"]]
    for b in blocks:
        b.ghosts(blocks)
    dt = _CFL / max(b.frequency() for b in blocks)
    for _ in range(steps):
        for b in blocks:
            b.update(dt)
        for b in blocks:
            b.inner.copy_(b.next)
            b.next = None
        # the step length may grow to twice the last one, which it never does here
        dt = min(2.0 * dt, _CFL / max(b.frequency() for b in blocks))
        for b in blocks:
            b.ghosts(blocks)
    return blocks


def _deviation(f, p):
    """f as the mixed storage lays it out: deviations from a Maxwellian at
    rest, velocities paired along u."""
    cells = sum(b["ni"] * b["nj"] for b in p["blocks"])
    rho = sum(float(b["fill"]["D"].sum()) for b in p["blocks"]) / cells
    T = [c[1] for b in p["blocks"] for c in b["bc"] if c[0] in ("diffuse", "adsorbing")]
    lam = 1.0 / float(np.mean(T))
    n, ax, wt, _ = _velocities(p["m"], p["vlim"])
    x, y = np.repeat(ax, n), np.tile(ax, n)
    M = torch.from_numpy(wt * (rho * lam / _PI) * np.exp(-lam * (x * x + y * y))).to(f.device)
    lead = f.shape[:2]
    out = torch.zeros(lead + (n + 1, n, 2), dtype=torch.float64, device=f.device)
    out[:, :, :n] = (f - torch.stack([M, 0.5 * _K / lam * M], -1)).reshape(lead + (n, n, 2))
    return out.reshape(lead + ((n + 1) // 2, 2, n, 2)).permute(0, 1, 2, 4, 5, 3).reshape(lead + (-1, 4)).contiguous()


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    out = []
    for p in _problems(case, seed):
        for b in _solve(p, case["steps"], dev):
            f = b.f
            if case["precision"] == "mixed":
                # the cells that nothing fills keep the deviation 0
                f = _deviation(f, p)
                G = b.G
                for i in (slice(0, G), slice(-G, None)):
                    for j in (slice(0, G), slice(-G, None)):
                        f[i, j] = 0.0
            out.append(dict(f=f, macro=b.macro))
            if case["kind"] == "channel":
                out[-1]["cover"] = b.cover
    return dict(solves=out, steps=None, residual=None) if case["kind"] == "serve" else out

"""Workloads of the library's main path, for timing and for comparing results.

Every case goes through the Python interface a user's program calls
(grace_b200.host).  Families:
  step      one SSP-RK3 step on a brick of same-level blocks: substeps, ghost
            fills, primitives passes, Runge-Kutta combinations
  fmr_step  the same on a two-level hierarchy (gather-map fill, refluxing)
  substep   one Runge-Kutta combination and one substep, on a smooth flow
  c2p       batched conservative-to-primitive recovery
  fmr       restriction into coarse buffers, prolongation into ghost zones
  mlp       gradient of the bracket network's loss (forward and backward)
Sizes come from the benchmark configurations and the tests (blocks of 8^3 and
16^3, the 1024 x 16 x 16 shock tube, the blast wave's spacing) or are generic.
"""
import functools
import math

import numpy as np
import torch

from grace_b200 import abi, fmr, params
from grace_b200.host import Blocks, Fields, GRMHDEquationsSystem

G = 4  # ghost width
CFL = 0.25
MAX_ZONES = 1536 * 16 ** 3  # the largest listed brick


def listed():
    step = {"kind": "step", "eos": "ideal", "metric": "flat", "mode": "tuned", "ranges": "full", "emf": "gs",
            "recon": "wenoz", "riemann": "hll", "static": False, "graph": False, "dt": False}
    bench = dict(step, ranges="next", static=True, dt=True, nx=16, ny=16, nz=16)
    return [
        # a test-sized grid, launched call by call: launches and host work
        dict(step, name="step_8x8^3", nbx=2, nby=2, nbz=2, nx=8, ny=8, nz=8),
        # a small share of a run on one GPU, replayed as a CUDA graph
        dict(bench, name="step_64x16^3_graph", nbx=4, nby=4, nbz=4, graph=True),
        # the benchmark's blast wave at a size that fills the GPU
        dict(bench, name="step_1536x16^3", nbx=12, nby=16, nbz=8),
        # a handle as it is created (plain mode), which a host code that
        # replaces its own kernels one by one starts with
        dict(step, name="step_plain_48x16^3", mode="plain", nbx=4, nby=4, nbz=3, nx=16, ny=16, nz=16),
        # the shock tube: upwind CT, no FOFC, periodic in y and z
        dict(step, name="step_tube_64x16^3_uct", emf="uct", nbx=64, nby=1, nbz=1, nx=16, ny=16, nz=16),
        # a curved metric with shift and curvature, hybrid equation of state,
        # every cell written; blocks that are no power of two
        dict(step, name="step_curved_120x12^3", eos="hybrid", metric="curved", nbx=5, nby=4, nbz=6, nx=12, ny=12,
             nz=12),
        # two refinement levels: 56 coarse and 64 fine blocks
        {"name": "fmr_step_120x16^3", "kind": "fmr_step", "nb": 4, "n": 16},
        # one substep alone, the slope-limited scheme, ragged blocks
        dict(step, name="substep_210x14x10x18_mc2", kind="substep", metric="curved", recon="mc2", riemann="llf",
             nbx=6, nby=7, nbz=5, nx=14, ny=10, nz=18),
        # a handful of states, an odd number: one launch's latency
        {"name": "c2p_1001", "kind": "c2p", "n": 1001, "metric": "flat", "cons_out": False},
        # states of a run: curved metric, consistent conservatives wanted
        {"name": "c2p_2e6_curved", "kind": "c2p", "n": (1 << 21) + 5, "metric": "curved", "cons_out": True},
        # the ghost-zone transfer between levels, all three element kinds
        {"name": "fmr_512x16^3", "kind": "fmr", "nq": 512, "n": 16},
        # one training batch of the bracket network
        {"name": "mlp_grad_16384", "kind": "mlp", "n": 16384},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "substep", "c2p", "c2p", "fmr", "fmr_step", "mlp"])
    if kind == "c2p":
        return {"kind": kind, "n": _log_int(rng, 500, 1 << 21), "metric": rng.choice(["flat", "curved"]),
                "cons_out": rng.random() < 0.5}
    if kind == "mlp":
        return {"kind": kind, "n": _log_int(rng, 64, 32768)}
    if kind == "fmr":
        return {"kind": kind, "nq": _log_int(rng, 8, 512), "n": rng.choice([8, 10, 12, 14, 16])}
    if kind == "fmr_step":
        return {"kind": kind, "nb": rng.choice([4, 5]), "n": rng.choice([8, 10, 12, 14, 16])}
    case = {"kind": kind, "mode": rng.choice(["tuned", "tuned", "tuned", "plain"]), "graph": False}
    case.update(rng.choice([{"eos": "ideal", "metric": "flat"}, {"eos": "hybrid", "metric": "curved"}]))
    # most runs take the same extent along each axis; odd extents do occur on
    # grids without refinement
    if rng.random() < 0.6:
        nx = ny = nz = rng.choice([8, 12, 16, 16, 20, 24])
    else:
        nx, ny, nz = (rng.randint(8, 24) for _ in range(3))
    zones = math.exp(rng.uniform(math.log(8 * 8 ** 3), math.log(MAX_ZONES / 4)))
    side = max(1.0, zones / (nx * ny * nz)) ** (1 / 3)
    nb = [max(1, round(side * rng.uniform(0.8, 1.25))) for _ in range(3)]
    case.update(nbx=nb[0], nby=nb[1], nbz=nb[2], nx=nx, ny=ny, nz=nz)
    if kind == "substep":
        # the smooth flow's case: schemes by their own independent evaluation
        case.update(emf="gs", recon=rng.choice(["wenoz", "mc2", "minmod"]), riemann=rng.choice(["hll", "llf"]),
                    metric="curved", eos="ideal", ranges="full", static=False, dt=False)
        return case
    emf = rng.choice(["gs", "gs", "gs", "uct"])
    case.update(emf=emf, recon=rng.choice(["wenoz", "wenoz", "wenoz", "mc2"]),
                riemann=rng.choice(["hll", "hll", "hll", "llf"]), ranges=rng.choice(["full", "next"]),
                static=rng.random() < 0.5, dt=rng.random() < 0.5)
    if rng.random() < 0.25 and case["mode"] == "tuned":
        case["graph"] = True
    return case


# ---- parameters ---------------------------------------------------------------
_RECON = {"wenoz": abi.RECON_WENOZ, "mc2": abi.RECON_MC2, "minmod": abi.RECON_MINMOD}


def _params(case):
    gs = case["emf"] == "gs"
    kw = dict(emf=abi.EMF_GS if gs else abi.EMF_UCT, fofc_enable=int(gs), recon=_RECON[case["recon"]],
              riemann=abi.RIEMANN_LLF if case["riemann"] == "llf" else abi.RIEMANN_HLL,
              ranges=abi.RANGES_NEXT_STAGE if case["ranges"] == "next" else abi.RANGES_FULL, max_sigma=1.0e4)
    if case["eos"] == "hybrid":
        return params.hybrid_pwpoly(100.0, [2.0], [], gamma_th=1.8, **kw)
    return params.ideal_gas(4.0 / 3.0, **kw)


# ---- 3+1 algebra (symmetric components xx, xy, xz, yy, yz, zz) ------------------
_SYM = ((0, 1, 2), (1, 3, 4), (2, 4, 5))


def _low(g, v):
    return [sum(g[_SYM[i][j]] * v[j] for j in range(3)) for i in range(3)]


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _det_inv(g):
    c = [g[3] * g[5] - g[4] ** 2, g[2] * g[4] - g[1] * g[5], g[1] * g[4] - g[2] * g[3], g[0] * g[5] - g[2] ** 2,
         g[1] * g[2] - g[0] * g[4], g[0] * g[3] - g[1] ** 2]
    det = g[0] * c[0] + g[1] * c[1] + g[2] * c[2]
    return det, [x / det for x in c]


def _comoving(g, beta, alp, z, B):
    """W, b^0, b^i, b^2 of ideal MHD, z^i = W v^i, B^i in the Eulerian frame."""
    W = torch.sqrt(1.0 + _dot(z, _low(g, z)))
    Bz = _dot(B, _low(g, z))
    b0 = Bz / alp
    bu = [(B[i] + Bz * (z[i] - W * beta[i] / alp)) / W for i in range(3)]
    return W, b0, bu, (_dot(B, _low(g, B)) + Bz * Bz) / W ** 2


def _conserved(g, beta, alp, rho, press, eps, z, B, s):
    """Undensitized D, S_i, tau, D s (the electron fraction's is 0)."""
    W, b0, bu, b2 = _comoving(g, beta, alp, z, B)
    bl, betal, zl = _low(g, bu), _low(g, beta), _low(g, z)
    h = rho * (1.0 + eps) + press + b2
    D = rho * W
    S = [h * W * zl[i] - alp * b0 * (bl[i] + betal[i] * b0) for i in range(3)]
    tau = h * W * W - press - 0.5 * b2 - (alp * b0) ** 2 - D
    return [D, *S, tau, torch.zeros_like(D), s * D]


def _kerr_schild(x, y, z):
    """Schwarzschild in Cartesian Kerr-Schild coordinates (M = 1): g, beta, alpha."""
    r = torch.sqrt(x * x + y * y + z * z)
    h2 = 2.0 / r
    l = [x / r, y / r, z / r]
    g = [(1.0 if i == j else 0.0) + h2 * l[i] * l[j] for i in range(3) for j in range(i, 3)]
    return g, [h2 * l[i] / (1 + h2) for i in range(3)], 1.0 / torch.sqrt(1 + h2)


def _curvature(x, y, z, h=1e-5):
    """K_ij = (d_i beta_j + d_j beta_i) / (2 alpha) by central differences."""
    def low(d, s):
        p = [x, y, z]
        p[d] = p[d] + s * h
        g, b, _ = _kerr_schild(*p)
        return _low(g, b)

    db = [[(a - b) / (2 * h) for a, b in zip(low(d, 1), low(d, -1))] for d in range(3)]
    alp = _kerr_schild(x, y, z)[2]
    return [(db[i][j] + db[j][i]) / (2 * alp) for i in range(3) for j in range(i, 3)]


def _thermo(eos, rho, press=None, eth=None):
    """(press, eps, T, s): the ideal gas (Gamma = 4/3) from press, the hybrid
    equation of state (K = 100, Gamma = 2, Gamma_th = 1.8) from eth."""
    if eos == "ideal":
        eps = 3.0 * press / rho
        return press, eps, eps / 3.0, 3.0 * torch.log(eps) - torch.log(rho)
    return (100.0 * rho ** 2 + 0.8 * rho * eth, 100.0 * rho + eth, 0.8 * eth,
            torch.log(eth * rho ** -0.8) / 0.8)


# ---- initial data ---------------------------------------------------------------
def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _write(f, aux, g6, beta, alp, K, rho, th, z):
    """Metric, primitives and conservatives of every cell; B from the faces."""
    st = f.state
    for a in range(6):
        st[:, abi.GXX + a] = g6[a]
        if K is not None:
            st[:, abi.KXX + a] = K[a]
    st[:, abi.ALP] = alp
    for a in range(3):
        st[:, abi.BETAX + a] = beta[a]
    sq = torch.sqrt(_det_inv(g6)[0])
    B = [0.5 * (f.bx[..., 1:] + f.bx[..., :-1]) / sq, 0.5 * (f.by[:, :, 1:] + f.by[:, :, :-1]) / sq,
         0.5 * (f.bz[:, 1:] + f.bz[:, :-1]) / sq]
    press, eps, T, s = th
    for v, c in enumerate(_conserved(g6, beta, alp, rho, press, eps, z, B, s)):
        st[:, v] = sq * c
    for v, x in ((abi.RHO, rho), (abi.PRESS, press), (abi.EPS, eps), (abi.TEMP, T), (abi.ENTROPY, s)):
        aux[:, v] = x
    for a in range(3):
        aux[:, abi.ZVECX + a] = z[a]
        aux[:, abi.BX + a] = B[a]


def _centres(origin, dx, n):
    """Cell centres x, y, z, ghosts included, of blocks at the given origins."""
    out = []
    for a in range(3):
        i = torch.arange(n[a] + 2 * G, device="cuda", dtype=torch.float64) - G + 0.5
        shape = [1, 1, 1, 1]
        shape[3 - a] = -1
        out.append(origin[:, a].view(-1, 1, 1, 1) + i.view(shape) * dx[:, a].view(-1, 1, 1, 1))
    full = torch.broadcast_shapes(*(t.shape for t in out))
    return [t.expand(full) for t in out]


def _blast(f, aux, x, y, z, seed, centre):
    """The blast wave: rho 1e-4 / p 5e-4 outside, rho 1e-2 / p 1 inside r < 0.8,
    uniform B^x, pressure noise of 1e-3."""
    r2 = (x - centre[0]) ** 2 + (y - centre[1]) ** 2 + (z - centre[2]) ** 2
    inside = r2 < 0.64
    rho = torch.where(inside, 1e-2, 1e-4).to(torch.float64)
    noise = 2.0 * torch.rand(rho.shape, generator=_rng(seed), device="cuda", dtype=torch.float64) - 1.0
    press = torch.where(inside, 1.0, 5e-4) * (1.0 + 1e-3 * noise)
    f.bx.fill_(0.1)
    zero, one = torch.zeros_like(rho), torch.ones_like(rho)
    _write(f, aux, [one, zero, zero, one, zero, one], [zero] * 3, one, None, rho, _thermo("ideal", rho, press),
           [zero] * 3)


def _tube(f, aux, x, seed):
    """A magnetised shock tube (the 1024 x 16 x 16 problem's states) with 1e-3
    of pressure noise."""
    left = x < 0.0
    rho = torch.where(left, 1.0, 0.125).to(torch.float64)
    noise = 2.0 * torch.rand(rho.shape[:1] + rho.shape[3:], generator=_rng(seed), device="cuda", dtype=torch.float64) - 1.0
    press = torch.where(left, 1.0, 0.1) * (1.0 + 1e-3 * noise[:, None, None, :])
    f.bx.fill_(0.5)
    f.by.copy_(torch.where(left[:, :, :1], 1.0, -1.0).to(torch.float64).expand(f.by.shape))
    zero, one = torch.zeros_like(rho), torch.ones_like(rho)
    _write(f, aux, [one, zero, zero, one, zero, one], [zero] * 3, one, None, rho, _thermo("ideal", rho, press),
           [zero] * 3)


def _curved(f, aux, x, y, z, dx, seed, eos, smooth):
    """A rotating magnetised blob on the Kerr-Schild metric; smooth: gentle
    gradients that no limiter of the scheme's fallback acts on."""
    r = _rng(seed)
    c = 0.2 * (torch.rand(4, generator=r, device="cuda", dtype=torch.float64) - 0.5)
    q2 = ((x - 4.0 - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2) / 0.25
    if smooth:
        rho = 1e-3 * (1.0 + 0.3 * torch.exp(-q2) + 0.05 * torch.sin(3.0 * x + 2.0 * y - z + 5.0 * c[3]))
        zv = [0.1 * torch.sin(2.0 * y + c[0]), 0.1 * torch.cos(1.5 * z + c[1]), 0.05 * torch.sin(1.2 * x + c[2])]
    else:
        rho = 1e-3 * torch.exp(-q2) + 1e-7
        e = 0.1 * torch.exp(-0.5 * q2)
        zv = [-y * e, (x - 4.0 - c[0]) * e, 0.3 * e]
    th = _thermo("ideal", rho, 0.05 * rho * (1.0 + 0.1 * torch.cos(2.0 * x - y))) if eos == "ideal" else \
        _thermo("hybrid", rho, eth=torch.full_like(rho, 1.25e-4))
    # the field: the discrete curl of A_z on the z edges, divergence free
    i = lambda t: torch.cat([t[..., :1] - dx[0], t], -1) + 0.5 * dx[0]
    j = lambda t: torch.cat([t[:, :, :1] - dx[1], t], 2) + 0.5 * dx[1]
    xe, ye, ze = i(x[:, :, :1, :]), j(y[..., :1]), z[:, :, :1, :1]
    Az = 2e-3 * torch.exp(-((xe - 4.0 - c[0]) ** 2 + (ye - c[1]) ** 2 + (ze - c[2]) ** 2) / (1.0 if smooth else 0.25))
    if not smooth:
        Az = 0.1 * Az
    f.bx.copy_((Az[:, :, 1:, :] - Az[:, :, :-1, :]) / dx[1])
    f.by.copy_(-(Az[..., 1:] - Az[..., :-1]) / dx[0])
    g6, beta, alp = _kerr_schild(x, y, z)
    _write(f, aux, g6, beta, alp, _curvature(x, y, z), rho, th, zv)


def _brick(case, seed):
    """(blocks, state, aux, nb, periodic, dx) of a brick case."""
    nb, n = [case["nb" + a] for a in "xyz"], [case["n" + a] for a in "xyz"]
    N = [a * b for a, b in zip(nb, n)]
    tube = nb[1] == nb[2] == 1 and nb[0] > 8
    if case["metric"] == "curved":
        lo, dx = (3.0, -1.0, -1.0), [2.0 / max(8, m) for m in N]
    elif tube:
        lo, dx = (-0.5, 0.0, 0.0), [1.0 / N[0]] * 3
    else:
        d = max(12.0 / 256, 3.0 / max(N))
        lo, dx = [-0.5 * d * m for m in N], [d] * 3
    nq = nb[0] * nb[1] * nb[2]
    q = torch.arange(nq, device="cuda")
    ijk = torch.stack([q % nb[0], (q // nb[0]) % nb[1], q // (nb[0] * nb[1])], 1).double()
    size = torch.tensor([dx[a] * n[a] for a in range(3)], device="cuda", dtype=torch.float64)
    origin = torch.tensor(lo, device="cuda", dtype=torch.float64) + ijk * size
    d = torch.tensor(dx, device="cuda", dtype=torch.float64).expand(nq, 3)
    blocks = Blocks(*n, G, nq, 1.0 / d)
    f, aux = blocks.new_fields(), blocks.new_aux()
    x, y, z = _centres(origin, d, n)
    if case["metric"] == "curved":
        _curved(f, aux, x, y, z, dx, seed, case["eos"], case["kind"] == "substep")
    elif tube:
        _tube(f, aux, x, seed)
    else:
        c = 0.3 * (torch.rand(3, generator=_rng(seed + 1), device="cuda", dtype=torch.float64) - 0.5)
        _blast(f, aux, x, y, z, seed, c)
    return blocks, f, aux, nb, (False, tube, tube), dx


# ---- states ---------------------------------------------------------------------
class _State:
    """What a user's program keeps for one case."""


def _system(case, P, blocks):
    g = GRMHDEquationsSystem(P)
    if case.get("mode", "tuned") == "tuned":
        g.set_mode(abi.MODE_TUNED)
    g.reserve(blocks)
    return g


def _autotune(s, new):
    # its trial runs use the handle's scratch, the cell-centred E among it,
    # which the primitives pass leaves for the next substep
    s.g.autotune(new, s.f, s.aux)
    s.g.compute_auxiliary_quantities(s.f, s.aux)


def _prepare_step(case, seed):
    s = _State()
    if case["kind"] == "fmr_step":
        H, maps, lists = _hierarchy(case["nb"], case["n"])
        n = [case["n"]] * 3
        d = torch.tensor(np.array([H.dx(l) for l, _ in H.leaves]), device="cuda")
        origin = torch.tensor(np.array([H.lo + np.asarray(b) * H.n * H.dx(l) for l, b in H.leaves]), device="cuda")
        s.blocks = Blocks(*n, G, H.nq, 1.0 / d)
        s.f, s.aux = s.blocks.new_fields(), s.blocks.new_aux()
        c = 0.3 * (torch.rand(3, generator=_rng(seed + 1), device="cuda", dtype=torch.float64) - 0.5)
        _blast(s.f, s.aux, *_centres(origin, d, n), seed, c)
        P = params.blast()
        P.ranges = abi.RANGES_NEXT_STAGE
        s.g = _system({}, P, s.blocks)
        s.g.set_reflux(lists)
        g = s.g
        s.bc = lambda f: g.fill_ghosts_gather(f, maps)
        s.dt, static, dt = CFL * float(d.min()), True, True
    else:
        s.blocks, s.f, s.aux, nb, per, dx = _brick(case, seed)
        d = torch.tensor(dx, device="cuda", dtype=torch.float64).repeat(s.blocks.nq, 1)
        s.g = _system(case, _params(case), s.blocks)
        g = s.g
        s.bc = lambda f: g.fill_ghosts_brick(f, nb, per)
        s.dt, static, dt = CFL * min(dx), case["static"], case["dt"]
    s.bc(s.f)
    if static:
        s.g.set_static_metric(s.f)
    s.g.compute_auxiliary_quantities(s.f, s.aux)
    s.fp, s.fpp = s.f.clone(), s.f.clone()
    s.dt_out = torch.zeros(1, device="cuda", dtype=torch.float64) if dt else None
    s.next_dt = (d, CFL, s.dt_out) if dt else None
    if case.get("mode", "tuned") == "tuned":
        _autotune(s, s.fp)
    s.graph = None
    if case.get("graph"):
        keep = [t.clone() for t in (s.f.state, s.f.bx, s.f.by, s.f.bz, s.aux)]
        s.g.rk3_step(s.dt, s.f, s.fp, s.fpp, s.aux, s.bc, next_dt=s.next_dt)
        for t, k in zip((s.f.state, s.f.bx, s.f.by, s.f.bz, s.aux), keep):
            t.copy_(k)
        s.g.compute_auxiliary_quantities(s.f, s.aux)
        s.fp.copy_(s.f)
        s.fpp.copy_(s.f)
        torch.cuda.synchronize()
        s.graph, _ = s.g.capture_rk3_step(s.dt, s.f, s.fp, s.fpp, s.aux, s.bc, next_dt=s.next_dt)
    return s


@functools.lru_cache(maxsize=None)
def _hierarchy(nb, n):
    """A cube of nb^3 blocks, its central blocks refined once: the hierarchy and
    the fill maps and refluxing lists that a run builds at each regrid."""
    mid = {nb // 2 - 1, nb // 2} if nb % 2 == 0 else {nb // 2}
    H = fmr.Hierarchy((nb,) * 3, n, (-3.0,) * 3, (3.0,) * 3, lambda l, b: l == 0 and all(x in mid for x in b), 1,
                      periodic=(False,) * 3)
    return H, H.gather_maps(), H.reflux_lists()


def _prepare_substep(case, seed):
    s = _State()
    s.blocks, s.f, s.aux, nb, per, dx = _brick(case, seed)
    s.g = _system(case, _params(case), s.blocks)
    s.dt = CFL * min(dx)
    s.g.compute_auxiliary_quantities(s.f, s.aux)
    s.new = s.f.clone()
    if case["mode"] == "tuned":
        _autotune(s, s.new)
    return s


def _c2p_inputs(case, seed):
    """cons (10, n), metric (10, n) or None, prims (13, n): rho, thermal energy,
    Lorentz factor and magnetisation spread as in the c2p benchmark."""
    n, r = case["n"], _rng(seed)
    u = lambda lo, hi: lo + (hi - lo) * torch.rand(n, generator=r, device="cuda", dtype=torch.float64)

    def unit(g):
        v = list(torch.randn(3, n, generator=r, device="cuda", dtype=torch.float64))
        k = 1.0 / torch.sqrt(_dot(v, _low(g, v)))
        return [a * k for a in v]

    if case["metric"] == "curved":
        rr, v = u(2.5, 20.0), list(torch.randn(3, n, generator=r, device="cuda", dtype=torch.float64))
        k = rr / torch.sqrt(_dot(v, v))
        g6, beta, alp = _kerr_schild(*[a * k for a in v])
    else:
        one, zero = torch.ones(n, device="cuda", dtype=torch.float64), torch.zeros(n, device="cuda", dtype=torch.float64)
        g6, beta, alp = [one, zero, zero, one, zero, one], [zero] * 3, one
    rho, eth, W, sig = 10 ** u(-12, -3), 10 ** u(-6, 1), u(1.0, 50.0), 10 ** u(-4, 3)
    press, eps, T, ent = _thermo("hybrid", rho, eth=eth)
    wv = torch.sqrt(W * W - 1.0)
    z = [wv * a for a in unit(g6)]
    d = unit(g6)
    b = torch.sqrt(sig * rho / ((1.0 + _dot(d, _low(g6, z)) ** 2) / W ** 2))
    B = [b * a for a in d]
    sq = torch.sqrt(_det_inv(g6)[0])
    cons = torch.stack([sq * c for c in _conserved(g6, beta, alp, rho, press, eps, z, B, ent) + B])
    zero = torch.zeros_like(rho)
    prims = torch.stack([rho, press, *z, zero, T, eps, ent, *B, zero])
    metric = torch.stack([*g6, *beta, alp]) if case["metric"] == "curved" else None
    return cons, metric, prims


def _prepare_c2p(case, seed):
    s = _State()
    s.cons, s.metric, _ = _c2p_inputs(case, seed)
    s.g = GRMHDEquationsSystem(params.c2p_bench())
    s.g.set_mode(abi.MODE_TUNED)
    s.cons_out = torch.empty_like(s.cons) if case["cons_out"] else None
    s.err = torch.zeros(case["n"], device="cuda", dtype=torch.int32)
    return s


def _fmr_inputs(case, seed):
    """Fields of nq fine blocks, zeroed coarse buffers, the transfer's lists."""
    nq, n, r = case["nq"], case["n"], _rng(seed)
    blocks = Blocks(n, n, n, G, nq, np.ones((nq, 3)))
    fine, cbuf = blocks.new_fields(), blocks.new_fields()
    for t in (fine.state, fine.bx, fine.by, fine.bz, cbuf.state, cbuf.bx, cbuf.by, cbuf.bz):
        t.copy_(1.0 + 0.1 * torch.randn(t.shape, generator=r, device="cuda", dtype=torch.float64))
    q = torch.arange(nq, device="cuda")
    child = (q % 8).to(torch.uint8)
    elems = []
    for kind, ids in ((0, 6), (1, 12), (2, 8)):
        # one element of each kind per block, the sides of a face by its block
        hf = torch.zeros(nq, 3, 2, device="cuda", dtype=torch.int8)
        elems.append((kind, q, q, ((q * 7 + kind) % ids).to(torch.uint8), hf))
    return blocks, fine, cbuf, q, child, elems


def _prepare_fmr(case, seed):
    s = _State()
    s.blocks, s.fine, s.cbuf, s.q, s.child, s.elems = _fmr_inputs(case, seed)
    s.g = _system({}, params.blast(), s.blocks)
    return s


_FMR_LO, _FMR_HO = tuple(range(abi.N_HRSC)), tuple(range(abi.N_HRSC, abi.N_EVOL_VARS))


def _mlp_inputs(case, seed):
    """A parameter block, raw features and targets of n states."""
    r = _rng(seed)
    P = torch.zeros(abi.MLP_NUM_PARAMS, device="cuda")
    o = 0
    for rows, cols, scale in ((64, 16, 1.0), (64, 1, 0.05), (64, 64, 0.3), (64, 1, 0.05), (64, 64, 0.3), (64, 1, 0.05),
                              (64, 1, 0.2), (1, 1, 0.05)):
        P[o:o + rows * cols] = scale * (2.0 * torch.rand(rows * cols, generator=r, device="cuda") - 1.0)
        o += rows * cols
    P[o:o + 6] = torch.tensor([-7.0, -1.0, 0.5, -0.5, 0.5, -0.5], device="cuda")
    P[o + 6:o + 12] = torch.tensor([2.5, 1.0, 0.8, 1.5, 0.3, 0.5], device="cuda")
    P[o + 12:o + 15] = torch.tensor([3.0, 2.0, 0.1], device="cuda")
    feat = P[o:o + 6, None] + P[o + 6:o + 12, None] * torch.randn(6, case["n"], generator=r, device="cuda")
    tgt = 3.0 + 2.0 * torch.tanh((feat[1] + 1.0) * 0.7 - 0.4 * (feat[3] + 0.5)) + \
        0.1 * torch.randn(case["n"], generator=r, device="cuda")
    return P, feat.contiguous(), tgt


def _prepare_mlp(case, seed):
    s = _State()
    s.P, s.feat, s.tgt = _mlp_inputs(case, seed)
    s.g = GRMHDEquationsSystem(params.c2p_bench())
    return s


def prepare(case, seed):
    s = {"step": _prepare_step, "fmr_step": _prepare_step, "substep": _prepare_substep, "c2p": _prepare_c2p,
         "fmr": _prepare_fmr, "mlp": _prepare_mlp}[case["kind"]](case, seed)
    s.kind = case["kind"]
    return s


# ---- one pass -------------------------------------------------------------------
def run(s):
    if s.kind in ("step", "fmr_step"):
        if s.graph is not None:
            s.graph.replay()
        else:
            s.g.rk3_step(s.dt, s.f, s.fp, s.fpp, s.aux, s.bc, next_dt=s.next_dt)
        out = {"cons": s.f.state[:, :abi.N_HRSC], "bx": s.f.bx, "by": s.f.by, "bz": s.f.bz,
               "prims": s.aux[:, :abi.BDIV], "div": s.aux[:, abi.BDIV:abi.C2P_ERR], "err": s.aux[:, abi.C2P_ERR]}
        if s.dt_out is not None:
            out["dt"] = s.dt_out
        return out
    if s.kind == "substep":
        s.g.linop_apply(s.new, s.f, None, 1.0)
        s.g.advance_substep(0.0, s.dt, 1.0, s.new, s.f, s.aux)
        return {"cons": s.new.state[:, :abi.N_HRSC], "bx": s.new.bx, "by": s.new.by, "bz": s.new.bz}
    if s.kind == "c2p":
        out = {"prims": s.g.conservs_to_prims(s.cons, s.metric, cons_out=s.cons_out, err=s.err), "err": s.err}
        if s.cons_out is not None:
            out["cons"] = s.cons_out
        return out
    if s.kind == "fmr":
        s.g.restrict_to_coarse(s.fine, s.cbuf, s.q, s.q, s.child, _FMR_LO, _FMR_HO)
        for kind, fq, cq, el, hf in s.elems:
            s.g.prolong_to_ghosts(s.fine, s.cbuf, kind, fq, cq, el, hf, _FMR_LO, _FMR_HO)
        return {"coarse": s.cbuf.state, "cbx": s.cbuf.bx, "cby": s.cbuf.by, "cbz": s.cbuf.bz, "fine": s.fine.state,
                "bx": s.fine.bx, "by": s.fine.by, "bz": s.fine.bz}
    grad, loss = s.g.mlp_grad(s.P, s.feat, s.tgt)
    return {"grad": grad, "loss": loss}


# ---- what a pass cannot do without ------------------------------------------------
# FP64 operations of one face: ten reconstructions of both states, the face
# metric, two states' speeds and fluxes, the HLL combination
_FACE_FLOPS = {"wenoz": 10 * 120 + 900, "mc2": 10 * 20 + 900, "minmod": 10 * 16 + 900}
_C2P_FLOPS = 700  # five evaluations of the master function, bracket, scalars


def work(case):
    k = case["kind"]
    if k == "c2p":
        b = 10 + 13 + (10 if case["metric"] == "curved" else 0) + (10 if case["cons_out"] else 0)
        return {"bytes": case["n"] * (8 * b + 4), "flops": 2 * _C2P_FLOPS * case["n"]}
    if k == "mlp":
        w = 64 * 16 + 2 * 64 * 64 + 64
        return {"bytes": 28 * case["n"] + 4 * 2 * abi.MLP_NUM_PARAMS, "flops": 6 * w * case["n"]}
    if k == "fmr":
        n, nq = case["n"], case["nq"]
        # restriction: 26 arrays, fine interior read, coarse image written;
        # prolongation: one face, edge and corner element per block, each read
        # from its coarse cells and written
        ghosts = G * n * n + G * G * n + G ** 3
        return {"bytes": 8 * 26 * nq * (n ** 3 * 9 // 8 + ghosts * 9 // 8),
                "flops": nq * (23 * (n // 2) ** 3 * 100 + 26 * ghosts * 30)}
    zones = case["nb"] ** 3 * case["n"] ** 3 if k == "fmr_step" else \
        case["nbx"] * case["nby"] * case["nbz"] * case["nx"] * case["ny"] * case["nz"]
    if k == "fmr_step":
        zones += 7 * (8 if case["nb"] % 2 == 0 else 1) * case["n"] ** 3
    per = 3 * _FACE_FLOPS[case.get("recon", "wenoz")] + 600
    if k == "substep":
        # the old state, metric, curvature and primitives read, the new state
        # and face fields written
        return {"bytes": 8 * zones * (7 + 3 + 16 + 10 + 10), "flops": zones * per}
    # a step's three stages: 66, 76 and 76 doubles of state, metric, curvature,
    # primitives and face fields per zone read or written once; the flow's
    # fluxes and sources and the recovery (twice with FOFC)
    c2p = _C2P_FLOPS * (2 if case.get("emf", "gs") == "gs" else 1)
    return {"bytes": 8 * zones * (66 + 76 + 76), "flops": 3 * zones * (per + c2p)}


def tolerance(case):
    k = case["kind"]
    if k == "fmr":
        # the transfer rounds every product and sum on its own
        return "exact"
    if k == "mlp":
        # bf16 activations, 32-bit sums (3e-6 / 7e-5 from 64 bits)
        return {"rel": 2e-5, "max": 5e-4}
    if k == "c2p":
        # the root's window of 1e-15 in mu, amplified by W^2 (W up to 50):
        # 5e-10 / 6e-7 between contracted and separate multiply-adds
        return {"rel": 3e-9, "max": 5e-6, "differ": 1e-4}
    if k == "substep":
        # 64-bit sums in another order (5e-14 / 9e-13, in the smallest field)
        return {"rel": 1e-12, "max": 1e-11}
    # the same over three stages with the recovery between them; the field's
    # divergence, a residue, differs most (2e-9 / 2e-8)
    return {"rel": 1e-8, "max": 1e-6}


# ---- independent evaluation ---------------------------------------------------------
def exact(case, seed):
    k = case["kind"]
    if k == "c2p":
        # the states' primitives are known: the conservatives were made of them
        cons, _, prims = _c2p_inputs(case, seed)
        out = {"prims": prims, "err": None}
        if case["cons_out"]:
            # the field's rows come back without the metric's determinant
            out["cons"] = torch.cat([cons[:abi.C_BSX], prims[abi.P_BX:abi.P_CS2]])
        return out
    if k == "mlp":
        return _exact_mlp(case, seed)
    if k == "fmr":
        return _exact_fmr(case, seed)
    if k == "substep":
        return _exact_substep(case, seed)
    # a whole step's fallback and recovery branch on the flow; the path has no
    # second evaluation here (its parts are the other families)
    return None


def _exact_mlp(case, seed):
    P, feat, tgt = (t.double() for t in _mlp_inputs(case, seed))
    bf = lambda t: t.float().bfloat16().double()
    o, W, b = 0, [], []
    for rows, cols in ((64, 16), (64, 64), (64, 64), (1, 64)):
        w = P[o:o + rows * cols].view(rows, cols).clone().requires_grad_()
        o += rows * cols
        c = P[o:o + rows].clone().requires_grad_()
        o += rows
        W.append(w)
        b.append(c)
    mu, sd, tmu, tsd = P[o:o + 6, None], P[o + 6:o + 12, None], P[o + 12], P[o + 13]
    v = (feat - mu) / sd
    hi = bf(v)
    # the model's own rounding: hidden weights and activations in bf16, passed
    # straight through by the gradient
    st = lambda t: t + (bf(t) - t).detach()
    h = torch.cat([hi, bf(v - hi), torch.zeros(4, v.shape[1], device=v.device, dtype=v.dtype)])
    for layer in range(3):
        h = st(torch.relu(st(W[layer]) @ h + b[layer][:, None]))
    y = (W[3] @ h + b[3][:, None])[0]
    loss = ((y - (tgt - tmu) / tsd) ** 2).mean()
    grads = torch.autograd.grad(loss, [t for pair in zip(W, b) for t in pair])
    return {"grad": torch.cat([g.reshape(-1) for g in grads]), "loss": loss.item()}


def _lagrange(offsets, at):
    """Weights of the Lagrange polynomial through `offsets`, evaluated at `at`."""
    return [math.prod((at - q) / (p - q) for q in offsets if q != p) for p in offsets]


def _exact_fmr(case, seed):
    n = case["n"]
    blocks, fine, cbuf, q, child, elems = _fmr_inputs(case, seed)
    N, h = n + 2 * G, n // 2
    u, c = fine.state, cbuf.state
    ins = slice(G, G + n)
    mid = slice(G, G + h)
    # restriction: averages of 8 cells and of 4 faces; the 5-point polynomial,
    # its stencil kept inside the interior and biased by the half of the parent
    lo = u[:, :7, ins, ins, ins].reshape(-1, 7, h, 2, h, 2, h, 2).mean((3, 5, 7))
    R = torch.zeros(2, h, N, device="cuda", dtype=torch.float64)
    for half in range(2):
        for i in range(h):
            p = 2 * i + G
            off = 0 if n + G - p - 1 == 1 else 3 if p == G else 1 if n + G - p - 1 == 2 else (1 if half else 2)
            cells = [off - 3 + t for t in range(5)]
            R[half, i, [p + t for t in cells]] = torch.tensor(_lagrange(cells, 0.5), device="cuda", dtype=torch.float64)
    bit = [(child.long() >> a) & 1 for a in range(3)]
    ho = torch.einsum("qcz,qvzyx->qvcyx", R[bit[2]], u[:, 7:])
    ho = torch.einsum("qcy,qvzyx->qvzcx", R[bit[1]], ho)
    ho = torch.einsum("qcx,qvzyx->qvzyc", R[bit[0]], ho)
    c[:, :7, mid, mid, mid], c[:, 7:, mid, mid, mid] = lo, ho
    face = slice(G, G + n + 1, 2)
    fm = slice(G, G + h + 1)
    cbuf.bx[:, mid, mid, fm] = fine.bx[:, ins, ins, face].reshape(-1, h, 2, h, 2, h + 1).mean((2, 4))
    cbuf.by[:, mid, fm, mid] = fine.by[:, ins, face, ins].reshape(-1, h, 2, h + 1, h, 2).mean((2, 5))
    cbuf.bz[:, fm, mid, mid] = fine.bz[:, face, ins, ins].reshape(-1, h + 1, h, 2, h, 2).mean((3, 5))
    # prolongation: along each axis a region below, above or across the interior
    length = (G, G, n)
    first_f, first_c = (0, n + G, G), (G // 2, G + h, G)
    Pm = []
    for w in range(3):
        m = torch.zeros(length[w], N, device="cuda", dtype=torch.float64)
        for f in range(length[w]):
            k = first_c[w] + f // 2
            m[f, k - 2:k + 3] = torch.tensor(_lagrange(range(-2, 3), 0.25 if f % 2 else -0.25), device="cuda",
                                             dtype=torch.float64)
        Pm.append(m)
    minmod = lambda a, b: torch.where(a * b > 0, torch.sign(a) * torch.minimum(a.abs(), b.abs()), 0.0 * a)
    for kind, fq, cq, el, _ in elems:
        for e in range((6, 12, 8)[kind]):
            sel = (el == e).nonzero()[:, 0]
            if not len(sel):
                continue
            if kind == 0:
                w = [(e & 1) if a == e >> 1 else 2 for a in range(3)]
            elif kind == 1:
                others = [a for a in range(3) if a != e >> 2]
                w = [2 if a == e >> 2 else (e >> others.index(a)) & 1 for a in range(3)]
            else:
                w = [(e >> a) & 1 for a in range(3)]
            dst = tuple(slice(first_f[t], first_f[t] + length[t]) for t in reversed(w))
            v = torch.einsum("fx,qvzyx->qvzyf", Pm[w[0]], c[sel, 7:])
            v = torch.einsum("fy,qvzyx->qvzfx", Pm[w[1]], v)
            u[(sel, slice(7, None)) + dst] = torch.einsum("fz,qvzyx->qvfyx", Pm[w[2]], v)
            src = [slice(first_c[t], first_c[t] + length[t] // 2) for t in reversed(w)]
            mid_v = c[sel, :7][(Ellipsis, *src)]
            val = mid_v
            for a in range(3):
                ax = 2 - a
                shift = lambda d: c[sel, :7][(Ellipsis, *[slice(s.start + d * (t == ax), s.stop + d * (t == ax))
                                                          for t, s in enumerate(src)])]
                slope = 0.25 * minmod(mid_v - shift(-1), shift(1) - mid_v)
                if a == 0:
                    val = mid_v.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)
                slope = slope.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)
                sign = torch.tensor([-1.0, 1.0], device="cuda", dtype=torch.float64).repeat(val.shape[2 + ax] // 2)
                shape = [1] * 5
                shape[2 + ax] = -1
                val = val + sign.view(shape) * slope
            u[(sel, slice(0, 7)) + dst] = val
    # the divergence-preserving fill of the fine faces has none here
    return {"coarse": c, "cbx": cbuf.bx, "cby": cbuf.by, "cbz": cbuf.bz, "fine": u, "bx": None, "by": None, "bz": None}


def _edges(kind, u):
    """Left and right states at face i (between cells i-1 and i) from the six
    cells i-3 .. i+2."""
    a, b, c, d, e, f = u

    def weno(m2, m1, u0, p1, p2):  # the value at the face above u0
        b0 = 13 / 12 * (m2 - 2 * m1 + u0) ** 2 + 0.25 * (m2 - 4 * m1 + 3 * u0) ** 2
        b1 = 13 / 12 * (m1 - 2 * u0 + p1) ** 2 + 0.25 * (m1 - p1) ** 2
        b2 = 13 / 12 * (u0 - 2 * p1 + p2) ** 2 + 0.25 * (3 * u0 - 4 * p1 + p2) ** 2
        t = (b0 - b2).abs()
        w = [k * (1 + (t / (x + 1e-42)) ** 2) for k, x in ((0.1, b0), (0.6, b1), (0.3, b2))]
        q = [(2 * m2 - 7 * m1 + 11 * u0) / 6, (-m1 + 5 * u0 + 2 * p1) / 6, (2 * u0 + 5 * p1 - p2) / 6]
        return (w[0] * q[0] + w[1] * q[1] + w[2] * q[2]) / (w[0] + w[1] + w[2])

    if kind == "wenoz":
        return weno(a, b, c, d, e), weno(f, e, d, c, b)

    def slope(l, r):
        m = torch.minimum(l.abs(), r.abs())
        if kind == "mc2":
            m = torch.minimum(2 * m, 0.5 * (l + r).abs())
        return torch.where(l * r > 0, torch.sign(l) * m, 0 * m)

    return c + 0.5 * slope(c - b, d - c), d - 0.5 * slope(d - c, e - d)


def _exact_substep(case, seed):
    """u + dt (flux differences and sources) of the smooth flow (ideal gas,
    Gamma = 4/3), which the first-order fallback leaves alone."""
    blocks, f, aux, nb, per, dx = _brick(case, seed)
    n = [case["n" + a] for a in "xyz"]
    st, dt = f.state, CFL * min(dx)
    fb = [f.bx, f.by, f.bz]

    def part(t, lo, hi):  # t[z, y, x] on index ranges given per axis x, y, z
        return t[(Ellipsis, slice(lo[2], hi[2]), slice(lo[1], hi[1]), slice(lo[0], hi[0]))]

    def cells(t, d, o, wide):
        """t at cell (face index + o) along d, for the faces g .. g + n along d
        and the cells g - wide .. g + n + wide across."""
        lo = [G - wide if a != d else G + o for a in range(3)]
        return part(t, lo, [G + n[a] + wide if a != d else G + n[a] + 1 + o for a in range(3)])

    flux, eface = [], []
    for d in range(3):
        face4 = lambda t: 0.5625 * (cells(t, d, -1, 1) + cells(t, d, 0, 1)) - 0.0625 * (cells(t, d, -2, 1) + cells(t, d, 1, 1))
        met = [face4(st[:, abi.GXX + a]) for a in range(10)]
        g, alp, beta = met[:6], met[6], met[7:]
        det, gi = _det_inv(g)
        sq = torch.sqrt(det)
        rec = {v: _edges(case["recon"], [cells(aux[:, v], d, o, 1) for o in range(-3, 3)])
               for v in (abi.RHO, abi.ZVECX, abi.ZVECY, abi.ZVECZ, abi.TEMP, abi.ENTROPY, abi.BX, abi.BY, abi.BZ)}
        bn = cells(fb[d], d, 0, 1) / sq
        U, F, E, speeds = [], [], [], []
        for s in range(2):
            rho, T, ent = rec[abi.RHO][s], rec[abi.TEMP][s], rec[abi.ENTROPY][s]
            z = [rec[abi.ZVECX + a][s] for a in range(3)]
            B = [bn if a == d else rec[abi.BX + a][s] for a in range(3)]
            eps = 3.0 * T
            press = rho * T
            cs2 = 4.0 / 9.0 * eps / (1 + 4.0 / 3.0 * eps)
            W, b0, bu, b2 = _comoving(g, beta, alp, z, B)
            vt = [alp * z[a] / W - beta[a] for a in range(3)]
            h = rho * (1 + eps) + press + b2
            pt = press + 0.5 * b2
            bl = [x + y * b0 for x, y in zip(_low(g, bu), _low(g, beta))]
            u = _conserved(g, beta, alp, rho, press, eps, z, B, ent)
            vl = [x + y for x, y in zip(_low(g, beta), _low(g, vt))]
            fl = [u[0] * vt[d]]
            fl += [h * W ** 2 * vt[d] / alp * vl[a] + alp * ((pt if a == d else 0.0) - bu[d] * bl[a]) for a in range(3)]
            fl += [h * W ** 2 * vt[d] + pt * beta[d] - alp ** 2 * b0 * bu[d] - fl[0], 0 * rho, ent * fl[0]]
            # fast speed from the quadratic in the coordinate frame
            va = b2 / h
            c2 = va + cs2 * (1 - va)
            u0, ud = W / alp, W * vt[d] / alp
            A = (1 - c2) * u0 ** 2 + c2 / alp ** 2
            Bq = -2 * (1 - c2) * u0 * ud + 2 * c2 * beta[d] / alp ** 2
            C = (1 - c2) * ud ** 2 - c2 * (gi[_SYM[d][d]] - beta[d] ** 2 / alp ** 2)
            disc = torch.sqrt(torch.clamp(Bq ** 2 - 4 * A * C, min=0))
            speeds.append(((-Bq - disc) / (2 * A), (-Bq + disc) / (2 * A)))
            # E = -v x B and the field, for the two transverse components
            e1, e2 = [a for a in range(3) if a != d]
            E.append([(vt[d] * B[e2] - vt[e2] * B[d], B[e2]), (vt[d] * B[e1] - vt[e1] * B[d], B[e1])])
            U.append(u)
            F.append(fl)
        cm = torch.clamp(-torch.minimum(speeds[0][0], speeds[1][0]), min=0)
        cp = torch.clamp(torch.maximum(speeds[0][1], speeds[1][1]), min=0)
        if case["riemann"] == "llf":
            cp = torch.stack([x.abs() for p in speeds for x in p]).amax(0)
            cm = cp
        hll = lambda fl, fr, ul, ur: (cp * fl + cm * fr - cp * cm * (ur - ul)) / (cp + cm)
        flux.append([sq * hll(F[0][v], F[1][v], U[0][v], U[1][v]) for v in range(7)])
        # transport of B^e along d gives +-E of the third axis
        eface.append([sq * hll(E[0][k][0], E[1][k][0], E[0][k][1], E[1][k][1]) for k in range(2)])

    # cell-centred E = -v x B, densitized
    g, alp, beta = [st[:, abi.GXX + a] for a in range(6)], st[:, abi.ALP], [st[:, abi.BETAX + a] for a in range(3)]
    det, gi = _det_inv(g)
    sq = torch.sqrt(det)
    z = [aux[:, abi.ZVECX + a] for a in range(3)]
    B = [aux[:, abi.BX + a] for a in range(3)]
    W, b0, bu, b2 = _comoving(g, beta, alp, z, B)
    vt = [alp * z[a] / W - beta[a] for a in range(3)]
    Ec = [sq * (B[(a + 1) % 3] * vt[(a + 2) % 3] - B[(a + 2) % 3] * vt[(a + 1) % 3]) for a in range(3)]

    def on_edges(t, a, d, o):
        """Face data of direction d at the edges along axis a, shifted by o (0 or
        -1) along the third axis."""
        r = 3 - a - d
        lo, hi = [0, 0, 0], [0, 0, 0]
        lo[a], hi[a] = 1, 1 + n[a]                # the cells along the edge
        lo[d], hi[d] = 0, n[d] + 1                # faces start at g
        lo[r], hi[r] = 1 + o, n[r] + 2 + o        # cells across start at g - 1
        return part(t, lo, hi)

    def centre(t, a, d, o, r, p):
        lo, hi = [0, 0, 0], [0, 0, 0]
        lo[a], hi[a] = G, G + n[a]
        lo[d], hi[d] = G + o, G + n[d] + 1 + o
        lo[r], hi[r] = G + p, G + n[r] + 1 + p
        return part(t, lo, hi)

    emf = []
    for a in range(3):
        # axes p < q around the edge; E_a on the faces normal to p and to q
        p, q = [x for x in range(3) if x != a]
        sgn = {(0, 2): 1.0, (0, 1): -1.0}

        def e_on(d, o):
            # transport of B^e along d: e the remaining axis, E_a = +-(v_d B_e - v_e B_d)
            e = 3 - a - d
            k = [x for x in range(3) if x != d][::-1].index(e)
            even = (a, d, e) in ((0, 1, 2), (1, 2, 0), (2, 0, 1))
            return (-1.0 if even else 1.0) * on_edges(eface[d][k], a, d, o)

        ep, epm, eq, eqm = e_on(p, 0), e_on(p, -1), e_on(q, 0), e_on(q, -1)
        NE, SW = centre(Ec[a], a, p, 0, q, 0), centre(Ec[a], a, p, -1, q, -1)
        NW, SE = centre(Ec[a], a, p, -1, q, 0), centre(Ec[a], a, p, 0, q, -1)  # one step down along p; along q
        up = lambda d, o: torch.copysign(torch.ones((), device="cuda", dtype=torch.float64), on_edges(flux[d][0], a, d, o))
        s, sm, w, wm = up(p, 0), up(p, -1), up(q, 0), up(q, -1)
        dN = (1 - s) * (NE - eq) + (1 + s) * (NW - eqm)
        dS = (1 - sm) * (eq - SE) + (1 + sm) * (eqm - SW)
        dE = (1 - w) * (NE - ep) + (1 + w) * (SE - epm)
        dW = (1 - wm) * (ep - NW) + (1 + wm) * (epm - SW)
        emf.append(0.25 * (ep + epm + eq + eqm) + 0.125 * (dS - dN) + 0.125 * (dW - dE))

    # geometric sources on interior cells, sixth-order metric derivatives
    inner = lambda t, o=(0, 0, 0): part(t, [G + x for x in o], [G + n[i] + o[i] for i in range(3)])

    def der(t, d):
        s = lambda k: inner(t, [k if a == d else 0 for a in range(3)])
        return (45 * (s(1) - s(-1)) - 9 * (s(2) - s(-2)) + s(3) - s(-3)) / (60 * dx[0])

    gI, aI, bI, giI = [inner(t) for t in g], inner(alp), [inner(t) for t in beta], [inner(t) for t in gi]
    zI, BI = [inner(t) for t in z], [inner(t) for t in B]
    rho, press, eps = (inner(aux[:, v]) for v in (abi.RHO, abi.PRESS, abi.EPS))
    W, b0, bu, b2 = _comoving(gI, bI, aI, zI, BI)
    h, pt = rho * (1 + eps) + press + b2, press + 0.5 * b2
    uu = [W / aI] + [zI[a] - W * bI[a] / aI for a in range(3)]
    bb = [b0] + bu
    gup = [[None] * 4 for _ in range(4)]
    gup[0][0] = -1 / aI ** 2
    for i in range(3):
        gup[0][i + 1] = gup[i + 1][0] = bI[i] / aI ** 2
        for j in range(3):
            gup[i + 1][j + 1] = giI[_SYM[i][j]] - bI[i] * bI[j] / aI ** 2
    T = [[h * uu[m] * uu[k] + pt * gup[m][k] - bb[m] * bb[k] for k in range(4)] for m in range(4)]
    K = [inner(st[:, abi.KXX + a]) for a in range(6)]
    tau = -sum((T[0][0] * bI[i] + T[0][i + 1]) * der(alp, i) for i in range(3))
    for i in range(3):
        for j in range(3):
            tau = tau + (T[0][0] * bI[i] * bI[j] + 2 * T[0][i + 1] * bI[j] + T[i + 1][j + 1]) * K[_SYM[i][j]]
    src = [0.0, None, None, None, aI * tau, 0.0, 0.0]
    for d in range(3):
        dg, db, da = [der(t, d) for t in g], [der(t, d) for t in beta], der(alp, d)
        # g_00 = -alpha^2 + g_ij beta^i beta^j, g_0i = g_ij beta^j
        dl = [x + y for x, y in zip(_low(dg, bI), _low(gI, db))]
        d00 = -2 * aI * da + _dot(bI, _low(dg, bI)) + 2 * _dot(_low(gI, bI), db)
        acc = 0.5 * T[0][0] * d00 + sum(T[0][i + 1] * dl[i] for i in range(3))
        for i in range(3):
            for j in range(3):
                acc = acc + 0.5 * T[i + 1][j + 1] * dg[_SYM[i][j]]
        src[1 + d] = aI * acc
    cons = st[:, :7].clone()
    sqI = inner(sq)
    for v in range(7):
        new = inner(st[:, v]) + dt * sqI * src[v]
        for d in range(3):
            lo, hi = [1, 1, 1], [1 + n[a] for a in range(3)]
            lo[d], hi[d] = 0, n[d]
            low = part(flux[d][v], lo, hi)
            lo[d], hi[d] = 1, n[d] + 1
            new = new + dt * (low - part(flux[d][v], lo, hi)) / dx[d]
        inner(cons[:, v]).copy_(new)
    out = []
    for d in range(3):
        # dB^d/dt = -(curl E)^d on the faces g .. g + n along d
        p, q = (d + 1) % 3, (d + 2) % 3
        nw = fb[d].clone()
        lo = [G, G, G]
        hi = [G + n[a] + (1 if a == d else 0) for a in range(3)]

        def diff(t, ax):
            a, b = [slice(None)] * 3, [slice(None)] * 3
            a[2 - ax], b[2 - ax] = slice(1, None), slice(None, -1)
            return t[(Ellipsis, *a)] - t[(Ellipsis, *b)]

        part(nw, lo, hi).add_(-dt * (diff(emf[q], p) / dx[p] - diff(emf[p], q) / dx[q]))
        out.append(nw)
    return {"cons": cons, "bx": out[0], "by": out[1], "bz": out[2]}

"""The recovery of the tuned stage passes on states with known primitives:
conservatives of sampled flows (thermal energies to 1e4, magnetisations to
1e3, Lorentz factors to 26), the same perturbed by 0.1 to 10 %, and with
momenta beyond the limiter, in the cells of a block; ideal gases and the hybrid
equation of state, flat and curved metric, entropy backup on and off.  The
tuned aux pass is compared with the generating primitives and with the plain
pass, the tuned FOFC flag with the plain one."""
import ctypes

import numpy as np
import pytest
import torch

import _oracle
from curved import ks_fields
from grace_b200 import abi, params
from grace_b200.host import Blocks, Fields, GRMHDEquationsSystem

pytestmark = pytest.mark.gpu

N, G, NQ = 12, 4, 6
M = N + 2 * G
KAPPA = 100.0
GM = {"4/3": 1.0 / 3.0, "5/3": 2.0 / 3.0, "2": 1.0, "hybrid": 0.8}
ATMO = 1 << 20  # the error bit of a reset to the atmosphere


def make_params(eos, backup, **kw):
    if eos == "hybrid":
        return params.hybrid_pwpoly(KAPPA, [2.0], [], gamma_th=1.8, max_sigma=1e4, use_ent_backup=backup, **kw)
    return params.ideal_gas(GM[eos] + 1.0, max_sigma=1e4, use_ent_backup=backup, **kw)


def unit(rng, shape):
    v = rng.standard_normal((3,) + shape)
    return v / np.linalg.norm(v, axis=0)


def sampled(eos, metric, seed):
    """(prims (13, cells), state, bx, by, bz, metric (10, cells)); cells in the
    order (q, k, j, i)."""
    rng = np.random.default_rng(seed)
    shape = (NQ, M, M, M)
    if metric == "curved":
        x = rng.uniform(2.5, 6.0, shape)
        y, z = rng.uniform(-3.0, 3.0, (2,) + shape)
        g, beta, alp = ks_fields(x, y, z)
    else:
        g, beta, alp = np.zeros((6,) + shape), np.zeros((3,) + shape), np.ones(shape)
        g[0] = g[3] = g[5] = 1.0
    mat = np.moveaxis(g[[0, 1, 2, 1, 3, 4, 2, 4, 5]].reshape((3, 3) + shape), (0, 1), (-2, -1))
    sq = np.sqrt(np.linalg.det(mat))
    # each face field constant along its own axis: a cell's mean of two faces
    # is that value, and cells differ in all three components
    top = -2.0 if eos == "hybrid" else 0.0
    amp = lambda s: rng.choice([-1.0, 1.0], s) * 10 ** rng.uniform(top - 4.0, top, s)
    fb = [amp((NQ, M, M, 1)), amp((NQ, M, 1, M)), amp((NQ, 1, M, M))]
    B = np.stack([np.broadcast_to(b, shape) for b in fb]) / sq
    z = unit(rng, shape)
    W = rng.uniform(1.0, 26.0, shape)
    dot = lambda u, v: np.einsum("...ab,a...,b...->...", mat, u, v)
    z *= np.sqrt((W * W - 1.0) / dot(z, z))
    b2 = (dot(B, B) + dot(B, z) ** 2) / (W * W)
    rho = np.clip(b2 / 10 ** rng.uniform(-4, 3, shape), 1e-11, 1e-3 if eos == "hybrid" else 1.0)
    gm = GM[eos]
    if eos == "hybrid":
        eth = 10 ** rng.uniform(-6, 1, shape)
        eps, press = KAPPA * rho + eth, KAPPA * rho * rho + gm * rho * eth
        ent = np.log(eth * rho ** -gm) / gm
    else:
        eps = eth = 10 ** rng.uniform(-3, 4, shape)
        press = gm * rho * eps
        ent = np.log(eps) / gm - np.log(rho)
    pr = np.zeros((13,) + shape)
    pr[abi.P_RHO], pr[abi.P_PRESS], pr[abi.P_EPS] = rho, press, eps
    pr[abi.P_TEMP], pr[abi.P_ENT] = gm * eth, ent
    pr[abi.P_ZX:abi.P_ZZ + 1], pr[abi.P_BX:abi.P_BZ + 1] = z, B
    pr = np.ascontiguousarray(pr.reshape(13, -1))
    met = np.ascontiguousarray(np.concatenate([g, beta, alp[None]]).reshape(10, -1))
    cons = np.zeros((10, pr.shape[1]))
    _oracle.lib("orc").orc_prims_to_conservs(ctypes.byref(params.defaults()), pr.shape[1], _oracle.p(pr),
                                             _oracle.p(met), _oracle.p(cons))
    state = np.zeros((NQ, abi.N_EVOL_VARS, M, M, M))
    state[:, :7] = np.moveaxis(cons[:7].reshape((7,) + shape), 0, 1)
    state[:, abi.GXX:abi.GXX + 6] = np.moveaxis(g, 0, 1)
    state[:, abi.BETAX:abi.BETAX + 3] = np.moveaxis(beta, 0, 1)
    state[:, abi.ALP] = alp
    faces = [np.ascontiguousarray(np.repeat(f, M + 1, axis=3 - a)) for a, f in enumerate(fb)]
    return pr, state, faces, mat, sq


def changed(kind, state, mat, sq, seed):
    """exact: the sampled states; perturbed: each conserved variable off by a
    normal deviate of 0.1 to 10 %; limited: those with |S| / D up to three
    times the q + 1 it is limited to."""
    if kind == "exact":
        return state
    rng = np.random.default_rng(seed)
    state = state.copy()
    a = 10 ** rng.uniform(-3, -1, state[:, 0].shape)
    for v in range(7):
        state[:, v] *= 1.0 + a * rng.standard_normal(a.shape)
    if kind == "limited":
        S = np.moveaxis(state[:, abi.SX:abi.SX + 3], 1, 0)
        s2 = np.einsum("...ab,a...,b...->...", np.linalg.inv(mat), S, S)
        S *= rng.uniform(1.0, 3.0, a.shape) * (state[:, abi.TAU] + state[:, abi.DENS]) / np.sqrt(s2)
    return state


def setup(P, mode, tuning, state, faces):
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to("cuda:0")
    g = GRMHDEquationsSystem(P)
    g.reserve(Blocks(N, N, N, G, NQ, np.ones((NQ, 3)), device="cuda:0"))
    g.set_mode(mode)
    if tuning is not None:
        g.set_tuning(*tuning)
    f = Fields(dev(state), *[dev(b) for b in faces])
    aux = torch.zeros((NQ, abi.N_AUX_VARS, M, M, M), dtype=torch.float64, device="cuda:0")
    g.compute_auxiliary_quantities(f, aux)
    return g, f, aux


def aux_pass(P, mode, tuning, state, faces):
    _, f, aux = setup(P, mode, tuning, state, faces)
    a = np.moveaxis(aux.cpu().numpy(), 1, 0).reshape(abi.N_AUX_VARS, -1)
    return a, np.moveaxis(f.state[:, :7].cpu().numpy(), 1, 0).reshape(7, -1)


def tolerance(rho, eps, press, W, B2):
    """Relative difference in rho = D / W of two converged solves.  Brent ends
    within 1e-15 + 2^-51 mu of a sign change, mu = 1 / (h W), and W passes a
    relative shift of mu on W^2-fold; q - b^2/2 of the solve carries the
    rounding of the field's energy, B^2 / rho of the rest mass."""
    h = 1.0 + eps + press / rho
    return W * W * (1e-15 * h * W + 2.0 ** -52 * (1.0 + B2 / rho))


@pytest.mark.parametrize("metric", ["flat", "curved"])
@pytest.mark.parametrize("eos", list(GM))
def test_tuned_aux_pass_recovers_known_primitives(eos, metric):
    for backup in (1, 0):
        P = make_params(eos, backup)
        pr, state, faces, mat, sq = sampled(eos, metric, 7)
        for kind in ("exact", "perturbed", "limited"):
            st = changed(kind, state, mat, sq, 8)
            a, sa = aux_pass(P, abi.MODE_PLAIN, None, st, faces)
            # the forms of the tuned pass: one thread a cell, work queue, deferred backups
            for form in ((0, 3, 6) if kind == "exact" else (0,)):
                b, sb = aux_pass(P, abi.MODE_TUNED, (0, 0, 0, form), st, faces)
                where = (eos, metric, backup, kind, form)
                same = a[abi.C2P_ERR] == b[abi.C2P_ERR]
                # (a decision may lie within rounding of its threshold)
                assert np.mean(~same) <= 1e-4, (where, np.mean(~same))
                ok = same & ((a[abi.C2P_ERR].astype(np.int64) & ATMO) == 0)
                assert np.mean(ok) > 0.8, (where, np.mean(ok))
                rho, eps, press = a[abi.RHO], a[abi.EPS], a[abi.PRESS]
                # W of the solve (the velocity limit then acts on z alone)
                W = st[:, abi.DENS].reshape(-1) / sq.reshape(-1) / rho
                B2 = np.einsum("...ab,a...,b...->...", mat, pr[abi.P_BX:abi.P_BZ + 1].reshape((3,) + sq.shape),
                               pr[abi.P_BX:abi.P_BZ + 1].reshape((3,) + sq.shape)).reshape(-1)
                tol = tolerance(rho, eps, press, W, B2)
                # each of the two solves within twice its tolerance of the root
                d = np.abs(b[abi.RHO] / rho - 1.0)
                assert np.all(d[ok] <= 4.0 * tol[ok]), (where, np.max((d / tol)[ok]))
                d = np.abs(sb[0] / sa[0] - 1.0)
                assert np.all(d[ok] <= 4.0 * tol[ok]), (where, np.max((d / tol)[ok]))
                for v in range(3):
                    z = b[abi.ZVECX + v] - a[abi.ZVECX + v]
                    assert np.all(np.abs(z)[ok] <= 4.0 * (W * np.maximum(tol, 1e-15))[ok]), where
                # pressure: of the scale of the energy density it is left over from
                d = np.abs(b[abi.PRESS] - press)
                scale = rho + rho * eps + press + B2
                assert np.all(d[ok] <= 4.0 * (tol * scale)[ok]), (where, np.max((d / (tol * scale))[ok]))
                if kind == "exact":
                    # the conservatives' own rounding, once more
                    d = np.abs(b[abi.RHO] / pr[abi.P_RHO] - 1.0)
                    assert np.all(d[ok] <= 8.0 * tol[ok]), (where, np.max((d / tol)[ok]))
                    assert np.mean(ok) == 1.0, where


def test_tuned_aux_pass_keeps_a_hot_fast_state():
    """Gamma = 2, eps about 1e5, W about 23: f at the bracket's top lies below
    its own rounding, and the root is a factor of 10^4 away in density."""
    P = params.ideal_gas(2.0, max_sigma=1e4)
    state = np.zeros((NQ, abi.N_EVOL_VARS, M, M, M))
    state[:, abi.GXX] = state[:, abi.GYY] = state[:, abi.GZZ] = state[:, abi.ALP] = 1.0
    state[:, abi.DENS], state[:, abi.TAU] = 0.011179975010051533, 3448.2786117315713
    for v, s in enumerate((2205.073125311711, 2490.511039582831, 908.6778857852215)):
        state[:, abi.SX + v] = s
    state[:, abi.ENTROPYSTAR] = 0.18380599770959746
    B = (0.05781621755338407, -0.018243328497907104, -0.015377565851736701)
    faces = [np.full([NQ] + [M + (a == 2 - k) for k in range(3)], B[a]) for a in range(3)]
    for mode in (abi.MODE_PLAIN, abi.MODE_TUNED):
        a, s = aux_pass(P, mode, None, state, faces)
        assert np.all(np.abs(a[abi.RHO] / 4.92525698e-4 - 1.0) < 1e-8), (mode, a[abi.RHO, 0])
        assert np.all(a[abi.C2P_ERR] == 8), (mode, a[abi.C2P_ERR, 0])  # the entropy re-synchronised, nothing reset
        assert np.all(s[0] == state[0, abi.DENS, 0, 0, 0])


@pytest.mark.parametrize("eos", list(GM))
def test_tuned_fofc_flag_decides_as_plain(eos):
    """A substep of no length: the flag's dry run sees the sampled states
    themselves.  None is floored; of the perturbed ones plain and tuned flag
    the same."""
    P = make_params(eos, 1, dmp_enable=0, recon=abi.RECON_MINMOD)
    pr, state, faces, mat, sq = sampled(eos, "flat", 11)
    for kind in ("exact", "perturbed"):
        st = changed(kind, state, mat, sq, 12)
        tags = []
        for mode, flags in ((abi.MODE_PLAIN, (0,)), (abi.MODE_TUNED, (0, 3))):
            for flag in flags:
                g, f, aux = setup(P, mode, (0, flag, 0, 0) if mode == abi.MODE_TUNED else None, st, faces)
                f.state.copy_(torch.from_numpy(st))
                g.advance_substep(0.0, 0.0, 1.0, f.clone(), f, aux)
                s = g.status()
                tags.append((s.fofc_faces, s.fofc_edges))
        assert tags[0] == tags[1] == tags[2], (kind, tags)
        if kind == "exact":
            assert tags[0] == (0, 0)

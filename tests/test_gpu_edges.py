"""GPU parity at the sizes where a kernel's split can go wrong, against the
CPU oracle: the TMA flux tiles (rows of one, of two and of more warps of
cells, the widest row a tile holds and the first it does not, both sides of
the one-launch limit), the shared-memory FMR operators up to the largest
block they take and past it, in-place and deferred c2p batches, linop on
unaligned arrays, the network's gradient at ragged batch sizes, and the tuned
c2p on NaN, infinite and huge conservatives."""
import numpy as np
import pytest
import torch

import _oracle
from grace_b200 import abi, params, workloads
from grace_b200.host import Blocks, Fields, GRMHDEquationsSystem
from parity import prim_tol, state_residual
from test_gpu_amr import G, NELEM
from test_gpu_paths import _check_state, _gpu, _oracle_run
from test_mlp_oracle import feats_targets, random_params

pytestmark = pytest.mark.gpu


def dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).to("cuda:0")


# x faces: rows of nx + 4 cells over warps of 31 (28: one warp; 58, 60: two,
# with a row end inside the second's overlap); 120 is the widest row of the
# 128-thread tile, 122 falls back to global loads; 540 and 600 tiles lie on
# the two sides of one wave; odd extents fall back as a whole
@pytest.mark.parametrize("nb,n,recon", [
    ((1, 1, 1), (28, 8, 10), abi.RECON_WENOZ),
    ((1, 1, 1), (58, 8, 8), abi.RECON_WENOZ),
    ((1, 1, 1), (60, 8, 8), abi.RECON_MC2),
    ((1, 1, 1), (120, 8, 8), abi.RECON_WENOZ),
    ((1, 1, 1), (122, 8, 8), abi.RECON_WENOZ),
    ((1, 2, 1), (9, 11, 8), abi.RECON_WENOZ),
    ((3, 3, 2), (8, 8, 8), abi.RECON_MINMOD),
    ((5, 2, 2), (8, 8, 8), abi.RECON_WENOZ),
])
@pytest.mark.parametrize("flux", [1, 2])
def test_flux_tiles_match_oracle(flux, nb, n, recon):
    P = params.blast()
    P.recon = recon
    hi = [0.09375 * 0.5 * b * c for b, c in zip(nb, n)]  # cubic cells, the sphere in the middle
    su, f = workloads.blast(nb=nb, n=n, lo=[-x for x in hi], hi=hi)
    dt = 0.25 / su.idx().max()
    gs, _, g = _gpu(P, su, f, dt, 1, abi.MODE_TUNED, tuning=(flux, 1, 1, 1), static_metric=True)
    os_, _, counts = _oracle_run(P, su, f, dt, 1)
    _check_state(gs, os_, su.ngz)
    assert (g.status().fofc_faces, g.status().fofc_edges) == counts
    assert g.status().device_flags == 0


# one launch up to a wave of tiles, else one a direction; every timed scope is a launch
@pytest.mark.parametrize("nb,launches", [((3, 3, 2), 1), ((5, 2, 2), 3)])
@pytest.mark.parametrize("flux", [0, 1, 2])
def test_flux_launches_are_counted_once(flux, nb, launches):
    su, (st, bx, by, bz, aux) = workloads.blast(nb=nb, n=(8, 8, 8))
    g = GRMHDEquationsSystem(params.blast())
    g.reserve(Blocks(*su.n, su.ngz, su.nq, su.idx(), device="cuda:0"))
    g.set_mode(abi.MODE_TUNED)
    g.set_tuning(flux=flux)
    old, a = Fields(dev(st), dev(bx), dev(by), dev(bz)), dev(aux)
    new = old.clone()
    g.compute_auxiliary_quantities(old, a)
    g.set_kernel_timing(True)
    before = g.status().launches
    g.advance_substep(0.0, 1e-3, 1.0, new, old, a)
    count = {k: c for k, (_, c) in g.kernel_times().items()}
    assert count["flux"] == (launches if flux else 3)
    # flux, EMF, flag, the three FOFC passes (one scope), update, CT
    assert g.status().launches - before == count["flux"] + 7
    assert sum(count.values()) == count["flux"] + 5


# 24 is the largest interior whose contractions fit shared memory
@pytest.mark.parametrize("n", [6, 10, 22, 24, 26])
def test_fmr_restriction_sizes_match_oracle_bitwise(n):
    rng = np.random.default_rng(70 + n)
    nq, M = 8, n + 2 * G
    st = rng.standard_normal((nq, abi.N_EVOL_VARS, M, M, M))
    q, child = np.arange(nq, dtype=np.int64), np.arange(nq).astype(np.uint8)
    g = GRMHDEquationsSystem(params.blast())
    g.reserve(Blocks(n, n, n, G, nq, np.ones((nq, 3)), device="cuda:0"))
    fine = Fields(dev(st), None, None, None)
    cb = Fields(torch.zeros_like(fine.state), None, None, None)
    g.restrict_to_coarse(fine, cb, dev(q), dev(q), dev(child), [0], [1, 7, 22], faces=False)
    want = np.zeros_like(st)
    _oracle.restrict_cells("orc", n, G, abi.N_EVOL_VARS, st, want, q, q, child, [0], [1, 7, 22])
    np.testing.assert_array_equal(cb.state.cpu().numpy(), want)


@pytest.mark.parametrize("n", [6, 10, 24, 26])
@pytest.mark.parametrize("kind", [0, 1, 2])
def test_fmr_prolongation_sizes_match_oracle_bitwise(kind, n):
    rng = np.random.default_rng(80 + 3 * n + kind)
    nq, M = 2, n + 2 * G
    vho = [1, 2, 3, 4, 9, 13, 14, 21, 22]  # one more than the corners' group of 8
    st = rng.standard_normal((nq, abi.N_EVOL_VARS, M, M, M))
    cst = rng.standard_normal((nq, abi.N_EVOL_VARS, M, M, M))
    fq = np.repeat(np.arange(nq), NELEM[kind]).astype(np.int64)
    el = np.tile(np.arange(NELEM[kind]), nq).astype(np.uint8)
    g = GRMHDEquationsSystem(params.blast())
    g.reserve(Blocks(n, n, n, G, nq, np.ones((nq, 3)), device="cuda:0"))
    fine, cb = Fields(dev(st), None, None, None), Fields(dev(cst), None, None, None)
    g.prolong_to_ghosts(fine, cb, kind, dev(fq), dev(nq - 1 - fq), dev(el), None, [], vho, faces=False)
    want = st.copy()
    _oracle.prolong_cells("orc", kind, n, G, abi.N_EVOL_VARS, want, cst, fq, nq - 1 - fq, el, [], vho)
    np.testing.assert_array_equal(fine.state.cpu().numpy(), want)


# 37888 = two CTAs of 128 per SM: the largest in-place batch
@pytest.mark.parametrize("n", [1, 127, 129, 37888, 37889])
def test_c2p_batch_sizes_match_oracle(n):
    P = params.c2p_bench()
    cons, _ = workloads.c2p_states(37889, seed=17)
    cons = np.ascontiguousarray(cons[:, :n])
    g = GRMHDEquationsSystem(P)
    g.set_mode(abi.MODE_TUNED)
    c_d, err = dev(cons), torch.zeros(n, dtype=torch.int32, device="cuda:0")
    out = torch.zeros_like(c_d)
    pr = g.conservs_to_prims(c_d, cons_out=out, err=err).cpu().numpy()
    pr_o, co_o, err_o, _, _, _ = _oracle.c2p_batch(P, cons)
    same = err.cpu().numpy().view(np.uint32) == err_o
    assert same.mean() > 0.999
    tol = prim_tol(pr_o)
    assert np.all(state_residual(pr[:, same], pr_o[:, same]) < tol[same])
    # D = rho W changes by less than the primitives' tolerance
    assert np.all(np.abs(out.cpu().numpy()[0] / co_o[0] - 1)[same] < tol[same])


def test_c2p_odd_conservatives_match_oracle():
    """NaN, infinite, huge, zero and negative entries in one conserved variable
    of a sampled state, in the tuned batch (in place and deferred) and in the
    tuned aux pass (cells of a block): the same error bits and finite
    primitives as the oracle.  Left out: densities beyond the equation of state (1e100),
    where the result hangs on whether exp(log(eps_max)) rounds below
    eps_max, and NaN fields, whose cells no solve reaches."""
    P = params.c2p_bench()
    vals = [np.nan, np.inf, -np.inf, 0.0, -0.0, 1e300, -1e300, 1e-300, -1.0]
    pick = [(v, x) for v in (1, 2, 3, 4, 5, 6) for x in vals]
    cons, _ = workloads.c2p_states(8 * len(pick), seed=19)
    for i, (v, x) in enumerate(pick * 8):
        cons[v, i] = x
    cons[0, 0], cons[0, 1], cons[0, 2] = np.nan, 0.0, -np.inf
    pr_o, _, err_o, _, _, _ = _oracle.c2p_batch(P, cons)
    for pad in (1, 100):  # 432 states in place, 43 200 deferred
        c = np.ascontiguousarray(np.tile(cons, (1, pad)))
        g = GRMHDEquationsSystem(P)
        g.set_mode(abi.MODE_TUNED)
        err = torch.zeros(c.shape[1], dtype=torch.int32, device="cuda:0")
        pr = g.conservs_to_prims(dev(c), err=err).cpu().numpy()
        np.testing.assert_array_equal(err.cpu().numpy().view(np.uint32), np.tile(err_o, pad))
        np.testing.assert_array_equal(np.isfinite(pr[:9]), np.tile(np.isfinite(pr_o[:9]), (1, pad)))
    # the aux pass: the same entries in cells of a uniform block
    su, f = workloads.blast(nb=(1, 1, 1), n=(12, 12, 12))
    st, bx, by, bz, aux = [x.copy() for x in f]
    cells = [(k, j, i) for k in range(4, 16, 3) for j in range(4, 16, 3) for i in range(4, 16, 3)]
    for (v, x), c in zip(pick, cells):
        st[(0, v) + c] = x
    PB = params.blast()
    h = GRMHDEquationsSystem(PB)
    h.reserve(Blocks(*su.n, su.ngz, su.nq, su.idx(), device="cuda:0"))
    h.set_mode(abi.MODE_TUNED)
    S, A = Fields(dev(st), dev(bx), dev(by), dev(bz)), dev(aux)
    h.compute_auxiliary_quantities(S, A)
    want = [x.copy() for x in (st, bx, by, bz)]
    aux_o = aux.copy()
    _oracle.Stage(PB, *su.n, su.ngz, su.nq).compute_aux(su.idx().copy(), want, aux_o)
    got = A.cpu().numpy()
    sel = tuple(np.array(cells[:len(pick)]).T)
    np.testing.assert_array_equal(got[0, abi.C2P_ERR][sel], aux_o[0, abi.C2P_ERR][sel])
    for v in (abi.RHO, abi.EPS):
        np.testing.assert_array_equal(np.isfinite(got[0, v]), np.isfinite(aux_o[0, v]))


def test_handles_of_several_threads():
    """Four host threads, each with a handle and a stream of its own, whose
    tiles want different amounts of shared memory: a substep in both tile
    sizes and an FMR restriction and prolongation, ten times over, bit for bit
    what one thread gets."""
    from concurrent.futures import ThreadPoolExecutor
    sizes = [(28, 8, 10), (58, 8, 8), (120, 8, 8), (8, 8, 8)]
    rng = np.random.default_rng(91)

    def case(k):
        su, f = workloads.blast(nb=(1, 1, 1), n=sizes[k])
        n = (6, 10, 22, 24)[k]
        return su, f, n, rng.standard_normal((8, abi.N_EVOL_VARS) + (n + 2 * G,) * 3)

    cases = [case(k) for k in range(4)]

    def work(k):
        torch.cuda.set_device(0)
        su, (st, bx, by, bz, aux), n, fine = cases[k]
        out = []
        with torch.cuda.stream(torch.cuda.Stream()):
            for flux in (1, 2):
                g = GRMHDEquationsSystem(params.blast())
                g.reserve(Blocks(*su.n, su.ngz, su.nq, su.idx(), device="cuda:0"))
                g.set_mode(abi.MODE_TUNED)
                g.set_tuning(flux=flux)
                old, a = Fields(dev(st), dev(bx), dev(by), dev(bz)), dev(aux)
                new = old.clone()
                g.compute_auxiliary_quantities(old, a)
                g.advance_substep(0.0, 1e-3, 1.0, new, old, a)
                out += [new.state, new.bx]
            q = np.arange(8, dtype=np.int64)
            g = GRMHDEquationsSystem(params.blast())
            g.reserve(Blocks(n, n, n, G, 8, np.ones((8, 3)), device="cuda:0"))
            F = Fields(dev(fine), None, None, None)
            C = Fields(torch.zeros_like(F.state), None, None, None)
            g.restrict_to_coarse(F, C, dev(q), dev(q), dev(q.astype(np.uint8)), [], [1, 7, 22], faces=False)
            g.prolong_to_ghosts(F, C, 0, dev(q[:6]), dev(q[:6]), dev(q[:6].astype(np.uint8)), None, [], [1, 7],
                                faces=False)
            out += [C.state, F.state]
            torch.cuda.current_stream().synchronize()
        return [x.cpu().numpy() for x in out]

    with ThreadPoolExecutor(4) as pool:  # before the one-thread run: the limits are still to be raised
        runs = [list(pool.map(work, range(4))) for _ in range(10)]
    want = [work(k) for k in range(4)]
    for run in runs:
        for got, ref in zip(run, want):
            for x, y in zip(got, ref):
                np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n", [(5, 6, 7), (16, 4, 5)])
def test_linop_unaligned_arrays(n, shift):
    """linop_apply on arrays that start on an 8-byte boundary, and of odd
    lengths: b x + c y on every entry, to its two roundings."""
    su, f = workloads.blast(nb=(1, 1, 2), n=n)
    rng = np.random.default_rng(5)
    host = [[rng.standard_normal(a.shape) for a in f[:4]] for _ in range(2)]

    def put(a):
        t = torch.empty(a.size + shift, dtype=torch.float64, device="cuda:0")[shift:]
        t.copy_(dev(a).reshape(-1))
        return t.view(a.shape)

    X, Y = (Fields(*[put(a) for a in h]) for h in host)
    O = Fields(*[put(np.zeros_like(a)) for a in host[0]])
    g = GRMHDEquationsSystem(params.blast())
    g.reserve(Blocks(*n, su.ngz, su.nq, su.idx(), device="cuda:0"))
    b, c = 0.3, -1.7
    for C, cc in ((Y, c), (None, 0.0)):
        g.linop_apply(O, X, C, b, cc)
        for o, x, y in zip((O.state, O.bx, O.by, O.bz), *host):
            want = b * x + cc * y
            assert np.all(np.abs(o.cpu().numpy() - want) <= 2.0 ** -52 * (np.abs(b * x) + np.abs(cc * y)))


# 64-sample tiles: one sample, a tile less one, one more; 65600: more partial
# gradients than the handle keeps
@pytest.mark.parametrize("n", [1, 63, 65, 65600])
def test_mlp_gradient_sizes_match_oracle(n):
    P = random_params(9)
    _, f, t = feats_targets(n, 47)
    s = GRMHDEquationsSystem(params.c2p_bench())
    got, loss = s.mlp_grad(dev(P), dev(f), dev(t))
    loss_o, want = _oracle.mlp_loss_grad(P, f, t, emulate=True)
    # an activation within FP32 rounding of a BF16 boundary may land on its
    # other side, 2^-8 away: at most that on each of the three hidden layers
    tol = 3 * 2.0 ** -8
    assert abs(loss - loss_o) <= tol * loss_o
    assert np.linalg.norm(got.cpu().numpy() - want) <= tol * np.linalg.norm(want)


# 2, 10, 16 and 1025 tiles (the last: an own buffer); the sums take every eighth row
@pytest.mark.parametrize("n,tiles", [(65, (0, 1)), (581, (0, 7, 8, 9)), (1024, (0, 7, 8, 15)),
                                     (65600, (0, 7, 8, 511, 1023, 1024))])
def test_mlp_gradient_counts_every_tile_once(n, tiles):
    """Targets on the network's own outputs except in one tile of 64 samples,
    which then is the whole gradient and loss: left out or taken twice, either
    is off by its full size."""
    P = random_params(9)
    _, f, _ = feats_targets(n, 48)
    s = GRMHDEquationsSystem(params.c2p_bench())
    fit = s.mlp_eval(dev(f), dev(P)).cpu().numpy()
    for k in tiles:
        t, at = fit.copy(), slice(64 * k, min(64 * (k + 1), n))
        t[at] *= 1.5
        got, loss = s.mlp_grad(dev(P), dev(f), dev(t))
        loss_o, want = _oracle.mlp_loss_grad(P, np.ascontiguousarray(f[:, at]), t[at], emulate=True)
        share = (at.stop - at.start) / n
        tol = 3 * 2.0 ** -8  # as above
        assert abs(loss / share - loss_o) <= tol * loss_o, k
        assert np.linalg.norm(got.cpu().numpy() / share - want) <= tol * np.linalg.norm(want), k

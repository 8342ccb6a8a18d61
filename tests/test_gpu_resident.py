"""The on-chip CG (the default of the mixed and the FP64 solver wherever the state
fits in registers and shared memory) against the oracle, at the sizes where its split into
warp tiles, blocks and clusters changes: lattices smaller than a tile, partial
tiles in both directions, one block, one cluster, a grid of blocks up to the
largest that fits.

Solutions: the stop rule leaves a relative residual of 1e-12 on both sides and the
masses are those of the other mixed-solver tests, so the same 5e-12 holds; the
recurrences and reliable updates are those of the solver's other forms, so iteration
counts agree with theirs within 2 plus 1% (not with the FP64 oracle's: on the smallest
lattices an FP64 CG ends exactly after as many steps as there are unknowns)."""
import numpy as np
import pytest

from helpers import bound, cgauss, hot_links, rel, to_dev, to_host
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

SIZES = [(2, 2), (3, 5), (31, 2), (33, 7), (32, 32), (64, 64), (65, 31), (100, 37), (128, 128), (40, 250), (257, 66),
         (256, 256), (330, 97), (350, 370), (512, 512), (544, 400)]


F64_SITES = 148 * 15 * 64   # what FP64 holds; beyond, the solver's other forms run


@pytest.fixture(params=["mixed", "f64"])
def q(request):
    import qed2d
    qed2d.set_precision(request.param)
    qed2d.prec = request.param
    yield qed2d
    qed2d.set_precision("f64")


def solve(q, prm, U, b, am0, mu=0.0, maxiter=20000, eps=1e-24, x=None):
    x = q.cfield(*prm.iL) if x is None else x
    q.set_schedule(prm, -1, q.prec)
    if mu:
        it = q.CG(x, U, b, am0, mu, maxiter, eps, q.gamm5Dw_sqr_musq, prm, None, so_as_guess=bool(x.any()))
    else:
        it = q.CG(x, U, b, am0, maxiter, eps, q.gamm5Dw_sqr_msq, prm, None)
    return it, x


@pytest.mark.parametrize("L1,L2", SIZES)
def test_solution_vs_oracle(q, L1, L2):
    if q.prec == "f64" and L1 * L2 > F64_SITES:
        pytest.skip("not on chip in FP64")
    prm = q.LattParm((L1, L2), 4.0)
    U, b = hot_links(L1, L2, 61), cgauss(L1, L2, 62, 2)
    am0 = 0.25
    st, xo, _, _ = Oracle(L1, L2, 4.0).cg(U, b, am0, 20000, 1e-24)
    assert st == 0
    Ud, bd = to_dev(U), to_dev(b)
    q.set_schedule(prm, 1, q.prec)
    ito = q.CG(q.cfield(L1, L2), Ud, bd, am0, 20000, 1e-24, q.gamm5Dw_sqr_msq, prm, None)
    it, x = solve(q, prm, Ud, bd, am0)
    assert q.get_schedule(prm, q.prec) in ((5, 6) if q.prec == "mixed" else (1, 2))
    bound("on-chip CG vs oracle", rel(to_host(x), xo), 5e-12)
    assert abs(it - ito) <= 2 + ito // 100, (it, ito)
    _, x2 = solve(q, prm, Ud, bd, am0)   # deterministic
    assert np.array_equal(to_host(x2), to_host(x))


@pytest.mark.parametrize("L1,L2", [(33, 7), (64, 48), (256, 192)])
def test_shift_guess_cap_and_zero(q, L1, L2):
    """Method 2 with a shift and with a warm start; a capped solve returns the same
    iterate as the solver's first form (FP32 rounding of a few iterations: 1e-6, as
    for the other forms) and reports non-convergence; a zero source gives zero."""
    prm = q.LattParm((L1, L2), 4.0)
    U, b = hot_links(L1, L2, 71), cgauss(L1, L2, 72, 2)
    am0, mu = 0.2, 0.3
    o = Oracle(L1, L2, 4.0)
    st, xo, _, _ = o.cg(U, b, am0, 20000, 1e-24, mu=mu)
    assert st == 0
    Ud, bd = to_dev(U), to_dev(b)
    it, x = solve(q, prm, Ud, bd, am0, mu)
    bound("on-chip CG (shift) vs oracle", rel(to_host(x), xo), 5e-12)
    guess = x + 1e-3 * to_dev(cgauss(L1, L2, 73, 2))
    it2, xg = solve(q, prm, Ud, bd, am0, mu, x=guess)
    assert 0 < it2 <= it
    # (a warm start stops elsewhere within the stop rule's ball than the oracle's cold start)
    q.set_schedule(prm, 1, q.prec)
    x1 = x + 1e-3 * to_dev(cgauss(L1, L2, 73, 2))
    q.CG(x1, Ud, bd, am0, mu, 20000, 1e-24, q.gamm5Dw_sqr_musq, prm, None, so_as_guess=True)
    bound("on-chip CG (warm start) vs first form", rel(to_host(xg), to_host(x1)), 5e-12)
    it3, xs = solve(q, prm, Ud, bd, am0, mu, x=xg.clone())   # already solved
    assert it3 == 0 and np.array_equal(to_host(xs), to_host(xg))
    for cap in (1, 7, 8):
        out = []
        for sched in (-1, 1):
            q.set_schedule(prm, sched, q.prec)
            xc = q.cfield(L1, L2)
            with pytest.raises(q.Qed2dError):
                q.CG(xc, Ud, bd, am0, cap, 1e-24, q.gamm5Dw_sqr_msq, prm, None)
            assert q.last_solve(prm)[0] == cap
            out.append(to_host(xc))
        bound("on-chip capped solve vs first form", rel(out[0], out[1]), 1e-6)
    with pytest.raises(q.Qed2dError):   # no iteration allowed
        solve(q, prm, Ud, bd, am0, maxiter=0)
    it, x = solve(q, prm, Ud, to_dev(np.zeros_like(b)), am0)
    assert it == 0 and not to_host(x).any()


def test_non_unitary_links_and_nan_source(q):
    """Links of any modulus are taken as they are; a NaN source ends unconverged."""
    L1, L2 = 48, 36
    prm = q.LattParm((L1, L2), 4.0)
    U = hot_links(L1, L2, 81) * (1.0 + 0.05 * np.random.default_rng(3).standard_normal((2, L2, L1)))
    b = cgauss(L1, L2, 82, 2)
    st, xo, _, _ = Oracle(L1, L2, 4.0).cg(U, b, 0.4, 20000, 1e-24)
    assert st == 0
    _, x = solve(q, prm, to_dev(U), to_dev(b), 0.4)
    bound("on-chip CG (non-unitary links) vs oracle", rel(to_host(x), xo), 5e-12)
    b[0, 3, 5] = np.nan
    with pytest.raises(q.Qed2dError):
        solve(q, prm, to_dev(U), to_dev(b), 0.4, maxiter=30)
    b[0, 3, 5] = 1.0
    solve(q, prm, to_dev(U), to_dev(b), 0.4)   # the context stays usable


def batch_solve(b, U, src, am0, sched):
    b.schedule = sched
    x = b.field()
    its, upd = b.cg(x, U, src, am0, 20000, 1e-24)
    return list(its), list(upd), to_host(x)


@pytest.mark.parametrize("L,am0", [(40, -0.14), (40, -0.10)])
def test_near_critical_mass(q, L, am0):
    """Where FP32 rounding and the jumps of reliable updates show: the recurrences stay
    as sound as those of the solver's first form (a quarter more iterations at most; single
    runs differ by a few per cent)."""
    rng = np.random.default_rng(12)
    U = np.exp(1j * 0.45 * rng.standard_normal((2, L, L)))
    b = (rng.standard_normal((2, L, L)) + 1j * rng.standard_normal((2, L, L))) / np.sqrt(2)
    prm = q.LattParm((L, L), 4.0)
    Ud, bd = to_dev(U), to_dev(b)
    its = {}
    for schedule in (1, -1):
        q.set_schedule(prm, schedule, q.prec)
        x = q.cfield(*prm.iL)
        cap = its[1] + its[1] // 4 if its else 20000
        its[schedule] = q.CG(x, Ud, bd, am0, cap, 1e-20, q.gamm5Dw_sqr, prm, None)
        r = q.cfield(*prm.iL)
        q.gamm5Dw_sqr(r, Ud, x, am0, prm)
        assert rel(to_host(r), b) < 2e-10   # the stop rule's 1e-10, and rounding


@pytest.mark.parametrize("nrep,L1,L2", [(2, 33, 7), (37, 64, 64), (20, 96, 128), (5, 256, 256), (3, 500, 300)])
def test_equal_batch_vs_lean_schedule(nrep, L1, L2):
    """Equal-size batches on chip: one cluster per replica, more clusters than fit at a
    time, teams of the whole GPU that take the replicas in turn.  Against schedule 5,
    the same recurrences in the other solver: as schedules 8 and 9 are (1e-11)."""
    import qed2d
    b = qed2d.Batch(nrep, L1, L2, 4.0)
    U, src = b.field(), b.field()
    for r in range(nrep):
        U[r] = to_dev(hot_links(L1, L2, 500 + r))
        src[r] = to_dev(cgauss(L1, L2, 600 + r, 2))
    src[nrep - 1].zero_()   # one replica with a zero source
    am0 = [0.2 + 0.1 * (r % 3) for r in range(nrep)]
    it, upd, x = batch_solve(b, U, src, am0, -1)
    assert b.schedule == 9 and b.tile_rows in (4, 8, 16)
    it2, _, x2 = batch_solve(b, U, src, am0, -1)
    assert it2 == it and np.array_equal(x, x2)   # deterministic
    it5, _, x5 = batch_solve(b, U, src, am0, 5)
    assert it[nrep - 1] == 0 and not x[nrep - 1].any()
    bound("on-chip equal batch vs schedule 5", rel(x, x5), 1e-11)
    assert all(abs(p - q) <= 2 + q // 100 for p, q in zip(it, it5)), (it, it5)


@pytest.mark.parametrize("big", [False, True])
def test_uneven_batch_vs_grid_solver(big):
    """Uneven batches on chip: more size classes than side streams, odd sizes, several
    replicas of a size; with and without sizes whose teams exceed a cluster."""
    import qed2d
    sizes = [(32, 32), (48, 48), (64, 64), (33, 20), (100, 37), (17, 90), (128, 128), (2, 3), (64, 48), (31, 31), (96, 96)]
    sizes = sizes * 2 + ([(256, 256), (300, 200), (256, 256)] if big else [])
    b = qed2d.Batch.ragged(sizes, [4.0] * len(sizes))
    U, src = b.field(), b.field()
    for r, (l1, l2) in enumerate(sizes):
        b.replica(U, r).copy_(to_dev(hot_links(l1, l2, 700 + r)))
        b.replica(src, r).copy_(to_dev(cgauss(l1, l2, 800 + r, 2)))
    am0 = [0.2 + 0.05 * (r % 5) for r in range(len(sizes))]
    it, upd, x = batch_solve(b, U, src, am0, -1)
    assert b.schedule == 6
    assert np.array_equal(batch_solve(b, U, src, am0, -1)[2], x)
    it2, _, x2 = batch_solve(b, U, src, am0, 2)
    bound("on-chip uneven batch vs grid solver", rel(x, x2), 1e-11)
    tiny = [l1 * l2 < 100 for l1, l2 in sizes]   # fewer unknowns than steps: the count is rounding
    assert all(t or abs(p - q) <= 2 + q // 100 for p, q, t in zip(it, it2, tiny)), (it, it2)
    with pytest.raises(qed2d.Qed2dError):   # capped
        b.schedule = -1
        b.cg(b.field(), U, src, am0, 5, 1e-24)
    assert np.array_equal(batch_solve(b, U, src, am0, -1)[2], x)


@pytest.mark.parametrize("L1,L2,n", [(12, 12, 2), (33, 7, 5), (64, 64, 12), (100, 37, 7), (128, 128, 12), (40, 90, 32),
                                     (180, 200, 12)])
def test_multishift_vs_grid_solver(L1, L2, n):
    """The on-chip multishift solve (the default where its vectors fit) against the grid
    kernel's schedule 1, the same recurrences: the layouts and schedules of that kernel
    are held to 1e-13 of one another, iteration counts to 1.  The smallest shift is not
    the first."""
    import qed2d
    prm = qed2d.LattParm((L1, L2), 4.0)
    U, src = to_dev(hot_links(L1, L2, 91)), to_dev(cgauss(L1, L2, 92, 2))
    mus = [0.05 * 1.3 ** i for i in range(n)]
    mus = mus[1:] + mus[:1] if n > 2 else mus
    out = []
    try:
        for sched in (-1, -1, 1):
            qed2d.set_schedule(prm, sched, "multishift")
            xs = [qed2d.cfield(L1, L2) for _ in mus]
            it = qed2d.multishift_CG(xs, U, src, 0.2, mus, 20000, 1e-24, prm)
            out.append((it, np.stack([to_host(x) for x in xs])))
        assert np.array_equal(out[0][1], out[1][1])   # deterministic
        assert abs(out[0][0] - out[2][0]) <= 1
        for i in range(n):
            bound("on-chip multishift vs grid kernel", rel(out[0][1][i], out[2][1][i]), 1e-13)
        qed2d.set_schedule(prm, -1, "multishift")
        xs = [to_dev(cgauss(L1, L2, 93 + i, 2)) for i in range(n)]   # capped: not converged; zero source: zero
        with pytest.raises(qed2d.Qed2dError):
            qed2d.multishift_CG(xs, U, src, 0.2, mus, 3, 1e-24, prm)
        assert qed2d.multishift_CG(xs, U, torch_zeros_like(src), 0.2, mus, 20000, 1e-24, prm) == 0
        assert not any(bool(x.any()) for x in xs)
    finally:
        qed2d.set_schedule(prm, -1, "multishift")


def torch_zeros_like(t):
    import torch
    return torch.zeros_like(t)


@pytest.mark.parametrize("L1,L2", [(2, 2), (3, 5), (33, 7), (32, 32), (64, 64), (100, 37), (128, 128), (350, 370), (512, 512),
                                   (544, 400)])
def test_gauge_md_vs_separate_kernels(L1, L2):
    """Pure-gauge OMF4 integration on chip (the default where links and momenta fit)
    against the same kicks and link updates made one by one with the library's
    kernels: the same operations, contracted differently by the compiler, so links and
    momenta agree to rounding over the 22 updates (1e-13)."""
    import torch
    import qed2d
    beta, eps, ns = 5.0, 0.2, 2
    prm = qed2d.LattParm((L1, L2), beta)
    U = to_dev(hot_links(L1, L2, 31))
    mom = torch.from_numpy(np.random.default_rng(5).standard_normal((2, L2, L1))).cuda()
    U1, m1 = U.clone(), mom.clone()
    qed2d.OMF4_(m1, U1, eps, ns, prm, None)
    r1, r2, r3, r4 = 0.08398315262876693, 0.2539785108410595, 0.6822365335719091, -0.03230286765269967
    r5, r6 = 0.5 - r1 - r3, 1.0 - 2.0 * (r2 + r4)
    f1, f2 = torch.empty_like(mom), torch.empty_like(mom)
    for _ in range(ns):
        for k, c in enumerate((r1, r3, r5, r5, r3, r1)):
            qed2d.krnl_force_(f1, f2, U, prm)
            mom += c * eps * (f1 + f2)
            if k < 5:
                qed2d.updt_fld_(U, mom, eps * (r2, r4, r6, r4, r2)[k])
    bound("on-chip gauge MD links vs separate kernels", rel(to_host(U1), to_host(U)), 1e-13)
    bound("on-chip gauge MD momenta vs separate kernels", rel(to_host(m1), to_host(mom)), 1e-13)
    U2 = to_dev(hot_links(L1, L2, 31))   # deterministic
    m2 = torch.from_numpy(np.random.default_rng(5).standard_normal((2, L2, L1))).cuda()
    qed2d.OMF4_(m2, U2, eps, ns, prm, None)
    assert torch.equal(U1, U2) and torch.equal(m1, m2)


@pytest.mark.parametrize("L1,L2", [(32, 8888), (64, 4448), (576, 576), (1024, 1000)])
def test_large_gauge_md_vs_separate_kernels(L1, L2):
    """The same beyond what fits on chip: one pass per link update and kick, tiles of 8 and of
    16 rows, one tile across (it is its own neighbour), passes in both directions."""
    test_gauge_md_vs_separate_kernels(L1, L2)

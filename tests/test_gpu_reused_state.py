"""Calls that reuse what an earlier call left behind -- recorded graphs,
buffers, rows -- give the answers that first calls give.

Bars: solutions to 1e-9 where both sides are solved to 1e-11 or below (the
operators' condition is below 1e2 here)."""
import ctypes

import numpy as np
import pytest

from helpers import rel_l2

pytestmark = pytest.mark.gpu


def system(vdr, oracle, dims, seed, aM=10.0):
    """A theta step on a ragged mesh: problem, element matrices, right-hand
    side, diagonal, start and the oracle's solution.  (aM 200: some 50
    iterations on the large meshes.  BiCG by atomics comes near a breakdown
    once in a hundred times where it takes 250.)"""
    prob = vdr.problems.rotation_shear(*dims, seed=seed)
    m = prob.mesh
    told = np.cos(0.37 * np.arange(m.nnode))
    bb, b, diag = oracle.assemble(prob.variant, m.xx, m.yy, m.zz, m.iss, prob.vel, prob.lam,
                                  prob.pdec, prob.q, kod=m.kod, robin_alpha=0.0, aH=2.0, aM=aM,
                                  cf=3.0, rM=aM, t_old=told, nthreads=8)
    b[prob.bc == 1] = 0.0
    diag[prob.bc == 1] = 1.0
    x0 = np.where(prob.bc == 1, 0.0, told)
    ref, _, _, st = oracle.bicgstab(b, x0, bb, m.iss, diag, prob.bc, tol=1e-12, itmax=5000)
    assert st == 0
    return prob, bb, b, diag, x0, ref


def dropin(vdr, sys_, x0=None, tol=1e-11, scale=1.0):
    prob, bb, b, diag, start, _ = sys_
    m = prob.mesh
    d = np.where(prob.bc == 1, 1.0, diag * scale)
    return vdr.kernel_dbcg_simple(m.nnode, b * scale, start if x0 is None else x0, tol, 5000,
                                  bb * scale, m.iss, d, m.nax, m.nay, m.naz, prob.bc)


def test_recorded_graphs_belong_to_their_arrays(vdr, gpu_lib):
    """Two pairs of arrays whose addresses differ by 2 d and by d, d a power
    of two (as blocks of an allocator do), one after the other: each solve's
    true residual below twice its tolerance."""
    torch = pytest.importorskip("torch")
    prob = vdr.problems.rotation_shear(19, 13, 11, seed=31)
    free = torch.tensor(prob.bc == 0, device="cuda")
    d = 1 << 20
    pool = torch.zeros(3 << 20, dtype=torch.float64, device="cuda")
    at = (-pool.data_ptr()) % (8 * d) // 8

    def arrays(off_b, off_x, n):
        return (pool[at + off_b // 8:at + off_b // 8 + n],
                pool[at + off_x // 8:at + off_x // 8 + n])

    def each(solve, n):
        want = []
        for pair in ((0, 4 * d), (2 * d, 5 * d)):
            b, x = arrays(*pair, n)
            assert (b.data_ptr() ^ 2 * x.data_ptr()) == \
                (pool.data_ptr() + 8 * at) ^ 2 * (pool.data_ptr() + 8 * at + 4 * d)
            b.copy_(torch.randn(n, dtype=torch.float64, device="cuda") * free)
            x.zero_()
            want.append((b, x, solve(b, x)))
        return want

    with vdr.Solver(prob, vdr.Options(scatter="atomic"), aH=2.0, aM=10.0) as s:
        for solve in (lambda b, x: s.solve_device(b, x, tol=1e-11, itmax=2000)[2],
                      lambda b, x: s.solve_gcr_device(b, x, tol=1e-11, itmax=2000)[2]):
            for b, x, st in each(solve, s.N):
                assert st == 0 and s.true_residual_device(b, x) < 2e-11
        s.set_segments(np.array([0, s.N]))
        for b, x, st in each(lambda b, x: s.solve_segmented_device(b, x, tol=1e-11,
                                                                   itmax=2000)[3], s.N):
            assert st == 0 and s.true_residual_device(b, x) < 2e-11


@pytest.mark.parametrize("solver", ["gcr", "bicgstab"])
@pytest.mark.parametrize("change", ["smoothing", "conv", "network"])
def test_recorded_graphs_follow_the_network(vdr, gpu_lib, solver, change):
    """A preconditioned solve after the network's settings changed, or with
    another network: its residual after a few iterations is the one that a
    handle with those settings from the start gives.  BF16 roundings that
    flip with the features' order of summation move it by 1e-3; the bar is 2
    per cent, and the solve before the change is further off."""
    torch = pytest.importorskip("torch")
    prob = vdr.problems.rotation_shear(19, 13, 11, seed=35)
    first = {"seed": 3, "steps": 1, "conv": "tcgen05"}
    then = dict(first, **{"smoothing": {"steps": 4}, "conv": {"conv": "mma"},
                          "network": {"seed": 4, "steps": 0}}[change])
    free = torch.tensor(prob.bc == 0, device="cuda")
    b = torch.tensor(np.cos(0.37 * np.arange(prob.mesh.nnode)), device="cuda") * free
    x = torch.empty_like(b)

    def solve(s, net):
        x.zero_()
        if solver == "gcr":
            _, err, _, _ = s.solve_gcr_device(b, x, net=net, tol=0.0, itmax=3)
        else:
            _, err, _, _ = s.solve_learned_device(net, b, x, tol=0.0, itmax=3)
        return err, s.stats()["kernel_launches"]

    def configured(s, c):
        net = vdr.LearnedNet(s, seed=c["seed"])
        p = net.get_params()
        p[:] = np.random.default_rng(c["seed"]).standard_normal(p.size) * 0.05
        net.set_params(p)
        net.update_features()
        net.set_smoothing(c["steps"])
        net.set_conv(c["conv"])
        return net

    with vdr.Solver(prob, aH=2.0, aM=10.0) as s:
        net = configured(s, then)
        want, launches = solve(s, net)
        net.close()
    with vdr.Solver(prob, aH=2.0, aM=10.0) as s:
        net = configured(s, first)
        before, _ = solve(s, net)
        if change == "network":
            net.close()
            net = configured(s, then)
        net.set_smoothing(then["steps"])
        net.set_conv(then["conv"])
        got, n = solve(s, net)
        net.close()
    assert abs(got - want) <= 0.02 * want, (before, got, want)
    assert n == launches
    if change != "conv":
        assert abs(before - want) > 0.02 * want


def test_dropin_after_a_nonfinite_call(vdr, oracle, gpu_lib):
    """A start that holds a NaN spoils its own call only: the next, on the
    same planes but fewer of them, solves."""
    tall = system(vdr, oracle, (9, 8, 19), 32)
    low = system(vdr, oracle, (9, 8, 9), 33)
    m = tall[0].mesh
    plane = np.arange(m.nnode) // (m.nax * m.nay)
    bad = tall[4].copy()
    bad[np.flatnonzero((tall[0].bc == 0) & (plane == 10))] = np.nan
    for _ in range(2):
        _, _, err = dropin(vdr, tall, x0=bad)
        assert not err <= 1e-11
        x, _, err = dropin(vdr, low)
        assert err <= 1e-11 and rel_l2(x, low[5]) < 1e-9
        x, _, err = dropin(vdr, tall)
        assert err <= 1e-11 and rel_l2(x, tall[5]) < 1e-9


def test_dropin_sizes_up_and_down(vdr, oracle, gpu_lib):
    """Tall, low, tall meshes on the same planes and others of the same node
    count, below and above the one-launch limit: rows, pair vectors and pads
    at other offsets in the same buffers."""
    for dims in ((12, 9, 30), (12, 9, 5), (12, 9, 30), (9, 12, 30), (30, 9, 12), (75, 63, 32),
                 (75, 63, 31), (75, 63, 4), (63, 75, 32), (12, 9, 5)):
        sys_ = system(vdr, oracle, dims, 36, aM=200.0)
        x, _, err = dropin(vdr, sys_)
        assert err <= 1e-11 and rel_l2(x, sys_[5]) < 1e-9, dims


# entries just below the store's 2^120, in the middle, just above its 2^-100
@pytest.mark.parametrize("power", [119, 60, -60, -95])
@pytest.mark.parametrize("dims", [(12, 9, 8), (75, 63, 32)])
def test_systems_across_the_stores_range(vdr, oracle, gpu_lib, dims, power):
    """The system times a power of two has the same solution, whether it runs
    as one launch or as kernels: by BiCGStab, in mixed precision, as a
    segment; on the small mesh also by the drop-in (BiCG) and as columns."""
    torch = pytest.importorskip("torch")
    sys_ = system(vdr, oracle, dims, 34)
    prob, bb, b = sys_[:3]
    big = np.abs(bb).max()
    small = np.abs(bb[bb != 0]).min()
    e = power - int(np.ceil(np.log2(big))) if power > 0 else power - int(np.floor(np.log2(small)))
    if power > 0 and np.log2(small) + e < -99:
        pytest.skip("the entries' own range")
    scale = 2.0 ** e
    if dims == (12, 9, 8):
        x, _, err = dropin(vdr, sys_, scale=scale)
        assert err <= 1e-11 and rel_l2(x, sys_[5]) < 1e-9
    bd, aM = torch.tensor(b, device="cuda"), 10.0
    for precision in ("fp64", "mixed"):
        with vdr.Solver(prob, vdr.Options(precision=precision), aH=2.0, aM=aM) as s:
            for f in (1.0, scale):
                s.set_operator(2.0 * f, aM * f)
                xd = torch.tensor(sys_[4], device="cuda")
                it, err, st = s.solve_device(bd * f, xd, tol=1e-11, itmax=2000)
                assert st == 0 and err <= 1e-11, (precision, f, it, err, st)
                assert rel_l2(xd.cpu().numpy(), sys_[5]) < 1e-9
                if precision == "mixed":
                    continue
                if dims == (12, 9, 8):
                    X = torch.zeros(s.N, 16, dtype=torch.float64, device="cuda")
                    _, _, errs, st = s.solve_block_device((bd * f)[:, None].repeat(1, 16), X,
                                                          tol=1e-11)
                    assert st == 0 and rel_l2(X[:, 3].cpu().numpy(), sys_[5]) < 1e-9
            s.set_segments(np.array([0, s.N]))
            xd.zero_()
            _, _, _, st = s.solve_segmented_device(bd * scale, xd, tol=1e-11, itmax=2000)
            assert st == 0 and rel_l2(xd.cpu().numpy(), sys_[5]) < 1e-9


def test_meeting_times_out_and_recovers(vdr, oracle, gpu_lib):
    """The meetings of the whole-solve launches are bounded: with one block of
    three absent the others give up after ~1 ms, the call's outcome is the
    timeout although one of them stores a success after it, and solves on the
    same handle, cluster and grid forms of FP64 and mixed, run as before."""
    import importlib
    torch = pytest.importorskip("torch")
    L = importlib.import_module(vdr.__name__ + "._lib")
    for dims in ((12, 9, 8), (32, 24, 12)):
        sys_ = system(vdr, oracle, dims, 37)
        prob, _, b, _, x0, ref = sys_
        for precision in ("fp64", "mixed"):
            with vdr.Solver(prob, vdr.Options(precision=precision), aH=2.0, aM=10.0) as s:
                for _ in range(2):
                    assert s.lib.vdr_diag_meeting_timeout(s.h) == L.TIMEOUT
                    x = torch.tensor(x0, device="cuda")
                    _, err, st = s.solve_device(torch.tensor(b, device="cuda"), x, tol=1e-11,
                                                itmax=2000)
                    assert st == 0 and err <= 1e-11 and rel_l2(x.cpu().numpy(), ref) < 1e-9


CLUSTER, WHOLE_SOLVE, ROWS, OTHER_ROOM = 1, 2, 4, 8


def test_segmented_solve_after_rows_were_refused(vdr, oracle, gpu_lib):
    """Rows formed by a segmented solve, then a plain solve for whose pair
    vectors there is no room (all rows go), then the segmented solve again."""
    torch = pytest.importorskip("torch")
    sys_ = system(vdr, oracle, (12, 9, 8), 38)
    prob, _, b, _, x0, ref = sys_
    bd = torch.tensor(b, device="cuda")
    with vdr.Solver(prob, aH=2.0, aM=10.0) as s:
        s.set_segments(np.array([0, s.N]))

        def segmented():
            x = torch.tensor(x0, device="cuda")
            _, _, _, st = s.solve_segmented_device(bd, x, tol=1e-11, itmax=2000)
            assert st == 0 and rel_l2(x.cpu().numpy(), ref) < 1e-9

        segmented()
        assert s.lib.vdr_diag_without(s.h, ROWS) == 0
        x = torch.tensor(x0, device="cuda")
        _, _, st = s.solve_device(bd, x, tol=1e-11, itmax=2000)
        assert st == 0 and rel_l2(x.cpu().numpy(), ref) < 1e-9
        for without in (ROWS, 0):
            assert s.lib.vdr_diag_without(s.h, without) == 0
            segmented()
            s.set_operator(2.0, 10.0)


@pytest.mark.parametrize("without", [CLUSTER, WHOLE_SOLVE, CLUSTER | WHOLE_SOLVE, ROWS,
                                     CLUSTER | WHOLE_SOLVE | ROWS])
@pytest.mark.parametrize("dims", [(12, 9, 8), (32, 24, 12)])
def test_solves_without(vdr, oracle, gpu_lib, dims, without):
    """What the solves fall back to where the device refuses clusters, whole
    solves in one launch, or memory for rows: the same solutions."""
    torch = pytest.importorskip("torch")
    sys_ = system(vdr, oracle, dims, 39)
    prob, _, b, _, x0, ref = sys_
    bd = torch.tensor(b, device="cuda")
    for opts in ({}, {"solver": "bicg"}, {"precision": "mixed"}):
        with vdr.Solver(prob, vdr.Options(**opts), aH=2.0, aM=10.0) as s:
            assert s.lib.vdr_diag_without(s.h, without) == 0
            s.set_segments(np.array([0, s.N]))
            calls = [lambda x: s.solve_device(bd, x, tol=1e-11, itmax=2000)[2]]
            if not opts:
                calls += [lambda x: s.solve_segmented_device(bd, x, tol=1e-11, itmax=2000)[3],
                          lambda x: s.solve_gcr_device(bd, x, tol=1e-11, itmax=2000)[2]]
            for call in calls:
                for start in (np.zeros_like(x0), x0):
                    x = torch.tensor(start, device="cuda")
                    assert call(x) == 0
                    assert rel_l2(x.cpu().numpy(), ref) < 1e-9
            if not opts:
                X = torch.tensor(x0, device="cuda")[:, None].repeat(1, 16)
                _, _, errs, st = s.solve_block_device(bd[:, None].repeat(1, 16), X, tol=1e-11)
                assert st == 0 and rel_l2(X[:, 7].cpu().numpy(), ref) < 1e-9


def test_applies_leave_no_rows_behind(vdr, oracle, gpu_lib):
    """A caller's applies take one kernel and no memory each, however many
    they are, and their products do not change when a solve has formed rows:
    each against the oracle's element matrices to 1e-13 (FP64 sums of pair
    products, 2^-47 each)."""
    torch = pytest.importorskip("torch")
    prob, bb, b = system(vdr, oracle, (33, 17, 21), 40)[:3]
    m = prob.mesh
    x = np.random.default_rng(8).standard_normal(m.nnode)
    xd, bd = torch.tensor(x, device="cuda"), torch.tensor(b, device="cuda")
    y = torch.empty_like(xd)
    ref = [oracle.matvec0(m.iss, bb, prob.bc, x, transpose=t)[0] for t in (False, True)]
    with vdr.Solver(prob, aH=2.0, aM=10.0) as s:
        s.apply_device(xd, y)  # builds the operator
        s.solve_gcr_device(bd, torch.zeros_like(bd), tol=1e-8, itmax=5)
        s.set_operator(2.0, 10.0)
        for solved in (False, True):
            s.apply_device(xd, y)
            if solved:
                s.solve_device(bd, torch.zeros_like(bd), tol=1e-8, itmax=500)
            torch.cuda.synchronize()
            free, launches = torch.cuda.mem_get_info()[0], vdr.kernel_launch_count()
            for k in range(4):
                s.apply_device(xd, y, transpose=k % 2 == 1)
                torch.cuda.synchronize()
                assert rel_l2(y.cpu().numpy(), ref[k % 2]) < 1e-13, (solved, k)
                s.apply_accumulate_device(xd, y, transpose=k % 2 == 1)
            assert vdr.kernel_launch_count() - launches == 8
            assert torch.cuda.mem_get_info()[0] == free


def test_products_on_rows_in_training(vdr, gpu_lib):
    """The residual loss's gradient, A and A^T in it, before and after a solve
    formed the operator's rows: apart by the gradient's own atomics (2e-7) and
    what 1e-14 in the products turns over in FP32 and BF16 roundings."""
    torch = pytest.importorskip("torch")
    prob = vdr.problems.rotation_shear(64, 32, 32, seed=41)  # large enough for rows
    free = torch.tensor(prob.bc == 0, device="cuda")
    b = torch.tensor(np.cos(0.37 * np.arange(prob.mesh.nnode)), device="cuda") * free
    with vdr.Solver(prob, aH=2.0, aM=10.0) as s, vdr.LearnedNet(s, seed=5) as net:
        net.update_features()
        rhat = (torch.randn(s.N, dtype=torch.float64, device="cuda") * free).float()
        got = []
        for solved in (False, True):
            if solved:
                s.solve_device(b, torch.zeros_like(b), tol=1e-10, itmax=500)
            loss = net.residual_loss_grad(rhat)
            got.append((loss, net.get_grads().astype(np.float64)))
        assert abs(got[0][0] - got[1][0]) <= 1e-6 * abs(got[0][0])
        assert rel_l2(got[1][1], got[0][1]) < 1e-4


@pytest.mark.parametrize("dims,rows", [((75, 63, 31), True), ((75, 63, 32), False)])
def test_bicg_holds_rows_for_whole_solves_only(vdr, gpu_lib, dims, rows):
    """One plane above the largest whole solve BiCG applies by elements: its
    first solve takes its vectors' memory (64 bytes a node), not the rows'
    (236)."""
    torch = pytest.importorskip("torch")
    prob = vdr.problems.rotation_shear(*dims, seed=42)
    b = torch.tensor(np.cos(0.37 * np.arange(prob.mesh.nnode)) * (prob.bc == 0), device="cuda")
    x = torch.zeros_like(b)
    with vdr.Solver(prob, vdr.Options(solver="bicg"), aH=2.0, aM=200.0) as s:
        s.apply_device(b, x)
        x.zero_()
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        _, err, st = s.solve_device(b, x, tol=1e-10, itmax=2000)
        assert st == 0 and err <= 1e-10
        held = free - torch.cuda.mem_get_info()[0]
    assert (held > 150 * prob.mesh.nnode) == rows, held


@pytest.mark.parametrize("dims", [(1, 1, 1), (6, 19, 19), (13, 5, 7), (40, 39, 38)])
@pytest.mark.parametrize("order", ["own", "permuted"])
def test_noalloc_solve_is_the_same_every_time(vdr, oracle, gpu_lib, dims, order):
    """vdr_bicg_noalloc_device on the reference's own numbering: the same bits
    from call to call (its sums have one order), and the oracle's solution; with
    the elements listed in another order (atomics) the solution."""
    torch = pytest.importorskip("torch")
    prob, bb, b, diag, x0, ref = system(vdr, oracle, dims, 43, aM=200.0)
    m, E, iss = prob.mesh, prob.mesh.nelem, prob.mesh.iss
    if order == "permuted":
        perm = np.random.default_rng(9).permutation(E)
        bb = np.ascontiguousarray(bb.reshape(E, 64)[perm]).ravel()
        iss = np.ascontiguousarray(iss.reshape(8, E)[:, perm]).ravel()
    dev = [torch.tensor(v, device="cuda") for v in (b, bb, diag)]
    ints = [torch.tensor(np.asarray(v, dtype=np.int32), device="cuda") for v in (iss, prob.bc)]
    got = []
    for _ in range(6):
        x = torch.tensor(x0, device="cuda")
        torch.cuda.synchronize()
        it, err = ctypes.c_int(-1), ctypes.c_double(-1.0)
        ptr = [ctypes.c_void_p(t.data_ptr()) for t in (*dev, *ints, x)]
        st = gpu_lib.vdr_bicg_noalloc_device(m.nnode, m.nax, m.nay, m.naz, ptr[0], ptr[5], 1e-12,
                                             5000, ptr[1], ptr[3], ptr[2], ptr[4], None,
                                             ctypes.byref(it), ctypes.byref(err))
        assert st == 0 and err.value <= 1e-12
        got.append((it.value, x.cpu().numpy()))
        assert rel_l2(got[-1][1], ref) < 1e-9
    if order == "own":
        assert all(n == got[0][0] and np.array_equal(x, got[0][1]) for n, x in got)


@pytest.mark.parametrize("dims,robin", [((1, 1, 1), 0.0), ((2, 1, 3), 0.3), ((6, 19, 19), 0.4),
                                        ((33, 17, 21), 0.0), ((75, 63, 31), 0.0)])
def test_time_loop_is_the_same_every_time(vdr, oracle, gpu_lib, dims, robin):
    """Up to the largest whole solve a step's sums have one order, from both
    builds (by geometric factors, and with a Robin term by coordinates): the
    right-hand side and the diagonal are the oracle's, to 1e-12, and repeat bit
    for bit, as do the time loop's counts, masses and field."""
    torch = pytest.importorskip("torch")
    prob = vdr.problems.rotation_shear(*dims, seed=44)
    prob.pdec[:] = 0.2
    prob.robin_alpha = robin
    if np.all(prob.bc == 1):
        prob.bc[:] = 0
    m, aM = prob.mesh, max(10.0, 0.3 * max(dims))
    told = np.cos(0.37 * np.arange(m.nnode))
    _, b, diag = oracle.assemble(prob.variant, m.xx, m.yy, m.zz, m.iss, prob.vel, prob.lam,
                                 prob.pdec, prob.q, kod=m.kod, robin_alpha=robin, aH=2.0, aM=aM,
                                 cf=3.0, rM=aM, t_old=told, nthreads=8)
    b[prob.bc == 1] = 0.0
    diag[prob.bc == 1] = 1.0
    seen = set()
    for solver in ("bicg", "bicgstab") * 3:
        with vdr.Solver(prob, vdr.Options(solver=solver), aH=2.0, aM=aM) as s:
            rhs, d = s.assemble_rhs(3.0, aM, told), s.diag()
            assert rel_l2(rhs, b) < 1e-12 and rel_l2(d, diag) < 1e-12
            t = torch.tensor(told * (prob.bc == 0), device="cuda")
            torch.cuda.synchronize()
            masses, its, errs, st, done = s.time_steps_device(t, 3, 3.0, aM, tol=1e-10, itmax=5000)
            assert st == 0 and done == 3
            seen.add((solver, tuple(its), masses.tobytes(), t.cpu().numpy().tobytes(),
                      rhs.tobytes(), d.tobytes()))
    assert len(seen) == 2


def test_block_solve_after_copy_waits_ran_out(vdr, oracle, gpu_lib):
    """The ring of copies of the products on rows gives up on a copy that is
    never issued, drains and reports it; block solves on the same handle
    before and after give the oracle's solution."""
    import importlib
    torch = pytest.importorskip("torch")
    L = importlib.import_module(vdr.__name__ + "._lib")
    sys_ = system(vdr, oracle, (12, 9, 8), 45)
    prob, _, b, _, _, ref = sys_
    B = torch.tensor(b, device="cuda")[:, None].repeat(1, 32)
    with vdr.Solver(prob, aH=2.0, aM=10.0) as s:
        for _ in range(3):
            X = torch.zeros_like(B)
            _, _, errs, st = s.solve_block_device(B, X, tol=1e-11)
            assert st == 0 and np.all(errs <= 1e-11)
            assert rel_l2(X[:, 30].cpu().numpy(), ref) < 1e-9
            assert s.lib.vdr_diag_wait_timeout(s.h) == L.TIMEOUT


@pytest.mark.parametrize("call", ["block", "gcr", "loop", "mixed", "half", "network"])
def test_rows_make_room(vdr, oracle, gpu_lib, call):
    """Calls that need memory beside the rows of an earlier solve and find
    none: the rows are given back for it, the call's result is the oracle's,
    and later solves run by elements, in mixed precision too."""
    torch = pytest.importorskip("torch")
    sys_ = system(vdr, oracle, (12, 9, 8), 46)
    prob, bb, b, diag, x0, ref = sys_
    m = prob.mesh
    bd = torch.tensor(b, device="cuda")

    def solved(x):
        return rel_l2(x.cpu().numpy(), ref) < 1e-9

    with vdr.Solver(prob, aH=2.0, aM=10.0) as s:
        x = torch.tensor(x0, device="cuda")
        assert s.solve_device(bd, x, tol=1e-11, itmax=2000)[2] == 0 and solved(x)
        assert s.stats()["kernel_launches"] == 1
        assert s.lib.vdr_diag_without(s.h, OTHER_ROOM) == 0
        x = torch.tensor(x0, device="cuda")
        if call == "block":
            X = torch.zeros(s.N, 16, dtype=torch.float64, device="cuda")
            _, _, errs, st = s.solve_block_device(bd[:, None].repeat(1, 16), X, tol=1e-11)
            assert st == 0 and solved(X[:, 9])
        elif call == "gcr":
            assert s.solve_gcr_device(bd, x, tol=1e-11, itmax=2000)[2] == 0 and solved(x)
        elif call == "loop":
            told = np.cos(0.37 * np.arange(m.nnode))
            t = torch.tensor(told, device="cuda")
            torch.cuda.synchronize()
            _, its, _, st, done = s.time_steps_device(t, 1, 3.0, 10.0, tol=1e-11, itmax=2000)
            assert st == 0 and done == 1 and solved(t)
        elif call == "mixed":
            s.set_mixed_operator("half")
            assert s.solve_mixed_device(bd, x, tol=1e-11, inner_tol=1e-3)[3] == 0 and solved(x)
        elif call == "half":
            y = torch.empty(s.N, dtype=torch.float32, device="cuda")
            s.apply_half_device((bd / bd.abs().max()).float(), y)
            torch.cuda.synchronize()
            want, _ = oracle.matvec0(m.iss, bb, prob.bc, b / np.abs(b).max() / diag)
            assert rel_l2(y.double().cpu().numpy(), want) < 2e-3
        else:
            with vdr.LearnedNet(s, seed=2) as net:
                net.update_features()
                assert s.solve_learned_device(net, bd, x, tol=1e-9, itmax=2000)[2] == 0
                assert rel_l2(x.cpu().numpy(), ref) < 1e-7
        for without in (OTHER_ROOM, 0):
            assert s.lib.vdr_diag_without(s.h, without) == 0
            x = torch.tensor(x0, device="cuda")
            assert s.solve_device(bd, x, tol=1e-11, itmax=2000)[2] == 0 and solved(x)
            assert s.stats()["kernel_launches"] > 1
            x = torch.tensor(x0, device="cuda")
            assert s.solve_mixed_device(bd, x, tol=1e-11, inner_tol=1e-4)[3] == 0 and solved(x)


@pytest.mark.parametrize("call", ["gcr", "learned"])
def test_few_products_form_no_rows(vdr, gpu_lib, call):
    """GCR and preconditioned solves take the rows that another solve has
    formed, but form none (236 bytes a node): the same residual after three
    iterations without them and with them, to BF16 roundings in the network."""
    torch = pytest.importorskip("torch")
    prob = vdr.problems.rotation_shear(75, 63, 31, seed=47)
    free_nodes = torch.tensor(prob.bc == 0, device="cuda")
    b = torch.tensor(np.cos(0.37 * np.arange(prob.mesh.nnode)), device="cuda") * free_nodes
    x = torch.zeros_like(b)
    with vdr.Solver(prob, aH=2.0, aM=200.0) as s, vdr.LearnedNet(s, seed=6) as net:
        net.update_features()

        def solve():
            x.zero_()
            if call == "gcr":
                return s.solve_gcr_device(b, x, tol=0.0, itmax=3)[1]
            return s.solve_learned_device(net, b, x, tol=0.0, itmax=3)[1]

        s.apply_device(b, x)
        s.true_residual_device(b, x)  # the solver's vectors
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        first = solve()
        vectors = 41 * 8 if call == "gcr" else 0  # GCR(20)'s own, bytes a node
        assert free - torch.cuda.mem_get_info()[0] < (vectors + 100) * s.N
        s.solve_device(b, torch.zeros_like(b), tol=1e-8, itmax=500)
        assert abs(solve() - first) <= (1e-9 if call == "gcr" else 0.02) * first

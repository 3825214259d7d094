"""The assembled 27-point operator of the structured numbering: A x and
A^T x against the oracle and against the element-wise apply (scatter
"atomic"), and the solve on it.

Bars: 1e-12 relative L2 (FP64), as for every stored apply; each row is a sum
of at most 64 pair products whose pairs carry 2^-47, 64 * 2^-47 = 4.5e-13.
"""
import numpy as np
import pytest

from helpers import kat_problem, rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-12
# one element, single rows, a row longer than a block, ragged, several blocks
DIMS = [(1, 1, 1), (1, 2, 1), (2, 1, 3), (31, 1, 2), (9, 7, 5), (300, 2, 3), (33, 17, 21)]


def oracle_bb(oracle, prob, aH, aM):
    m = prob.mesh
    bb, _, _ = oracle.assemble(prob.variant, m.xx, m.yy, m.zz, m.iss, prob.vel, prob.lam,
                               prob.pdec, prob.q, kod=m.kod, robin_alpha=prob.robin_alpha,
                               aH=aH, aM=aM, want_b=False, want_diag=False)
    return bb


@pytest.mark.parametrize("dims", DIMS)
def test_apply_matches_oracle(vdr, oracle, gpu_lib, dims):
    prob = vdr.problems.rotation_shear(*dims, seed=81)
    prob.pdec[:] = 0.2
    aH, aM = 2.0, 7.0
    bb = oracle_bb(oracle, prob, aH, aM)
    x = np.random.default_rng(3).standard_normal(prob.mesh.nnode)
    with vdr.Solver(prob, aH=aH, aM=aM) as s:
        s.apply(x)  # the rows are assembled from the second apply on
        for tr in (False, True):
            ref, _ = oracle.matvec0(prob.mesh.iss, bb, prob.bc, x, transpose=tr)
            y = s.apply(x, transpose=tr)
            assert rel_l2(y, ref) < TOL, (dims, tr)
            assert np.all(y[prob.bc == 1] == 0.0)


def test_dirichlet_values_scale_and_nonfinite(vdr, oracle, gpu_lib):
    """Whatever lies on Dirichlet nodes is ignored; inputs of any magnitude
    keep their relative accuracy; a non-finite entry reaches exactly the
    rows that the element-wise apply gives it to."""
    prob = vdr.problems.rotation_shear(13, 6, 5, seed=82)
    m = prob.mesh
    free = np.flatnonzero(prob.bc == 0)
    bb = oracle_bb(oracle, prob, 2.0, 7.0)
    rng = np.random.default_rng(4)
    with vdr.Solver(prob, aH=2.0, aM=7.0) as s, \
            vdr.Solver(prob, vdr.Options(scatter="atomic"), aH=2.0, aM=7.0) as e:
        x = rng.standard_normal(m.nnode)
        s.apply(x)
        ref, _ = oracle.matvec0(m.iss, bb, prob.bc, x)
        for fill in (np.nan, np.inf, 1e300):
            xd = np.where(prob.bc == 1, fill, x)
            assert rel_l2(s.apply(xd), ref) < TOL
        for scale in (1e-250, 1e-30, 1e30, 1e250):
            assert rel_l2(s.apply(x * scale) / scale, ref) < TOL
        for bad in (np.nan, np.inf):
            xb = x.copy()
            xb[free[len(free) // 2]] = bad
            for tr in (False, True):
                a, b = s.apply(xb, transpose=tr), e.apply(xb, transpose=tr)
                ok = np.isfinite(b)
                assert np.array_equal(ok, np.isfinite(a))
                assert rel_l2(a[ok], b[ok]) < TOL


@pytest.mark.parametrize("solver", ["bicgstab", "bicg"])
@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 1, 3), (19, 13, 11), (70, 40, 30)])
def test_solve_matches_element_wise(vdr, gpu_lib, dims, solver):
    """Both to 1e-12: their distance is bounded by the residuals times the
    condition of the theta-step operator (below 1e3 here)."""
    prob = vdr.problems.rotation_shear(*dims, seed=83)
    if np.all(prob.bc == 1):
        prob.bc[:] = 0
    xs = []
    for scatter in ("auto", "atomic"):
        with vdr.Solver(prob, vdr.Options(scatter=scatter, solver=solver), aH=2.0,
                        aM=0.3 * max(dims)) as s:
            b = s.assemble_rhs(3.0, 0.3 * max(dims), np.linspace(0, 1, prob.mesh.nnode))
            x, it, err, st = s.solve(b, tol=1e-12, itmax=2000)
            assert st == 0 and err <= 1e-12
            xs.append(x)
    assert rel_l2(xs[0], xs[1]) < 1e-9


def test_operator_follows_fields_and_mask(vdr, oracle, gpu_lib):
    prob = vdr.problems.rotation_shear(9, 8, 6, seed=84)
    m = prob.mesh
    x = np.random.default_rng(5).standard_normal(m.nnode)
    with vdr.Solver(prob, aH=2.0, aM=7.0) as s:
        s.apply(x)
        s.apply(x)
        prob.vel *= -0.5
        prob.lam *= 3.0
        prob.bc[:] = vdr.problems.inflow_mask(m, prob.vel)
        s.set_fields(prob.vel, prob.lam, prob.pdec, prob.q)
        s.set_dirichlet(prob.bc)
        ref, _ = oracle.matvec0(m.iss, oracle_bb(oracle, prob, 2.0, 7.0), prob.bc, x)
        for _ in range(2):  # element-wise, then from the new rows
            assert rel_l2(s.apply(x), ref) < TOL


def test_recorded_case(vdr, oracle, gpu_lib):
    prob = kat_problem(vdr)
    bb = oracle_bb(oracle, prob, 2.0, 0.03)
    x = np.random.default_rng(6).standard_normal(prob.mesh.nnode)
    with vdr.Solver(prob, aH=2.0, aM=0.03) as s:
        s.apply(x)
        for tr in (False, True):
            ref, _ = oracle.matvec0(prob.mesh.iss, bb, prob.bc, x, transpose=tr)
            assert rel_l2(s.apply(x, transpose=tr), ref) < TOL


# node counts at the edges of the whole-solve kernel's launch shapes: one
# cluster of 64, 128 and 192 threads a CTA (1024, 2048, 3072 nodes and one
# plane more), grids of 128, 256, 512, 768 and 1024 threads a CTA on 152 SMs,
# and the first size that runs as separate kernels
SHAPES = [(15, 15, 3), (15, 15, 4), (15, 7, 15), (15, 15, 8), (15, 15, 11), (15, 15, 12),
          (75, 31, 7), (75, 31, 8), (75, 31, 15), (75, 63, 15), (75, 63, 16), (75, 63, 23),
          (75, 63, 31), (75, 63, 32)]


@pytest.mark.parametrize("dims", SHAPES)
def test_whole_solve_launch_shapes(vdr, gpu_lib, dims):
    """From a warm and from a zero start, to 1e-11 against the element-wise
    solve (distance bounded as above), and the reported residual against the
    true one."""
    torch = pytest.importorskip("torch")
    prob = vdr.problems.rotation_shear(*dims, seed=85)
    N, aM = prob.mesh.nnode, 0.3 * max(dims)
    told = torch.tensor(np.cos(0.37 * np.arange(N)), device="cuda")
    xs = {}
    for scatter in ("auto", "atomic"):
        with vdr.Solver(prob, vdr.Options(scatter=scatter), aH=2.0, aM=aM) as s:
            b = torch.empty(N, dtype=torch.float64, device="cuda")
            s.assemble_rhs_device(b, 3.0, aM, told)
            for x0 in ("zero", "warm"):
                x = torch.zeros_like(b) if x0 == "zero" else told.clone()
                it, err, st = s.solve_device(b, x, tol=1e-11, itmax=2000)
                assert st == 0 and err <= 1e-11, (dims, scatter, x0)
                assert s.true_residual_device(b * torch.tensor(prob.bc == 0, device="cuda"),
                                              x) < 2e-11
                xs[scatter, x0] = x.cpu().numpy()
    for x0 in ("zero", "warm"):
        assert rel_l2(xs["auto", x0], xs["atomic", x0]) < 1e-8


# the mixed solve's inner kernel: odd node counts, then 128 to 1024 threads of
# one pair of nodes and 768 / 1024 threads of two (152 SMs), the last with its
# neighbours across the edge, and the separate kernels beyond
MIXED_SHAPES = [(2, 2, 2), (4, 2, 6), (15, 15, 3), (75, 31, 15), (75, 31, 16), (75, 63, 15),
                (75, 63, 16), (75, 63, 31), (75, 63, 32), (75, 63, 63), (76, 62, 64),
                (75, 63, 95), (75, 127, 63), (75, 127, 64)]


@pytest.mark.parametrize("dims", MIXED_SHAPES)
def test_mixed_launch_shapes(vdr, gpu_lib, dims):
    """The refinement on the binary16 rows reaches the FP64 tolerance (its
    true residual recomputed in FP64) and the FP64 solve's solution: both to
    1e-10, apart by at most the residuals times the condition (below 1e3)."""
    torch = pytest.importorskip("torch")
    prob = vdr.problems.rotation_shear(*dims, seed=86)
    N, aM = prob.mesh.nnode, 0.3 * max(dims)
    if np.all(prob.bc == 1):
        prob.bc[:] = 0
    told = torch.tensor(np.cos(0.37 * np.arange(N)), device="cuda")
    xs = []
    for precision in ("mixed", "fp64"):
        with vdr.Solver(prob, vdr.Options(precision=precision), aH=2.0, aM=aM) as s:
            b = torch.empty(N, dtype=torch.float64, device="cuda")
            s.assemble_rhs_device(b, 3.0, aM, told)
            x = torch.zeros_like(b)
            it, err, st = s.solve_device(b, x, tol=1e-10, itmax=2000)
            assert st == 0 and err <= 1e-10, (dims, precision, st, err)
            free = torch.tensor(prob.bc == 0, device="cuda")
            assert s.true_residual_device(b * free, x) < 1.1e-10
            xs.append(x.cpu().numpy())
    assert rel_l2(xs[0], xs[1]) < 1e-7


BICG_SHAPES = [(1, 1, 1), (2, 1, 3), (15, 15, 3), (75, 31, 7), (75, 31, 8), (75, 31, 16),
               (75, 63, 15), (75, 63, 16), (75, 63, 31), (75, 63, 32)]


@pytest.mark.parametrize("dims", BICG_SHAPES)
def test_dropin_launch_shapes(vdr, oracle, gpu_lib, dims):
    """kernel_dbcg_simple_ at the launch shapes of the whole-solve BiCG (128 to
    1024 threads a CTA, then separate kernels), sizes going up and down so that
    its buffers are reused: solution to 1e-9 of the oracle's BiCG at 1e-12, and
    to the tolerance where elements are listed in another order (the
    element-wise path)."""
    prob = vdr.problems.rotation_shear(*dims, seed=87)
    m, aM = prob.mesh, 0.3 * max(dims)
    if np.all(prob.bc == 1):
        prob.bc[:] = 0
    told = np.cos(0.37 * np.arange(m.nnode))
    bb, b, diag = oracle.assemble(prob.variant, m.xx, m.yy, m.zz, m.iss, prob.vel, prob.lam,
                                  prob.pdec, prob.q, kod=m.kod, robin_alpha=0.0, aH=2.0,
                                  aM=aM, cf=3.0, rM=aM, t_old=told, nthreads=8)
    b[prob.bc == 1] = 0.0
    diag[prob.bc == 1] = 1.0
    x0 = np.where(prob.bc == 1, 0.0, told)
    ref, _, _, st = oracle.bicgstab(b, x0, bb, m.iss, diag, prob.bc, tol=1e-12, itmax=5000)
    assert st == 0
    args = (m.nax, m.nay, m.naz, prob.bc)
    x, it, err = vdr.kernel_dbcg_simple(m.nnode, b, x0, 1e-11, 5000, bb, m.iss, diag, *args)
    assert err <= 1e-11 and rel_l2(x, ref) < 1e-9
    E = m.nelem
    perm = np.random.default_rng(7).permutation(E)
    x2, it2, err2 = vdr.kernel_dbcg_simple(
        m.nnode, b, x0, 1e-11, 5000, np.ascontiguousarray(bb.reshape(E, 64)[perm]).ravel(),
        np.ascontiguousarray(m.iss.reshape(8, E)[:, perm]).ravel(), diag, *args)
    assert err2 <= 1e-11 and rel_l2(x2, ref) < 1e-9


def test_many_meshes_on_assembled_rows(vdr, oracle, gpu_lib):
    """Uneven meshes in one handle, a mesh of one element and one of a single
    row among them: every mesh's solution against the element-wise segmented
    solve (scatter "atomic") and its true residual by the oracle; a non-finite
    source stays in its own mesh; a second solve at another tolerance."""
    torch = pytest.importorskip("torch")
    P = vdr.problems
    probs = [P.rotation_cube(7, 91), P.rotation_shear(1, 1, 1, seed=92),
             P.rotation_cube(12, 93), P.rotation_shear(19, 1, 2, seed=94),
             P.rotation_shear(40, 31, 9, seed=95)]
    union = P.concat(probs)
    off, aM = union.mesh.node_off, 10.0
    bad_mesh = 2
    out = {}
    for scatter in ("auto", "atomic"):
        with vdr.Solver(union, vdr.Options(scatter=scatter), aH=2.0, aM=aM) as s:
            s.set_segments(off)
            told = torch.tensor(np.cos(0.37 * np.arange(union.mesh.nnode)), device="cuda")
            b = torch.empty_like(told)
            s.assemble_rhs_device(b, 3.0, aM, told)
            b *= torch.tensor(union.bc == 0, device="cuda")
            for tol in (1e-6, 1e-12):
                x = torch.zeros_like(b)
                its, errs, sts, st = s.solve_segmented_device(b, x, tol=tol, itmax=2000)
                assert st == 0 and np.all(sts == 0) and np.all(errs <= tol)
            out[scatter] = (x.cpu().numpy(), b.cpu().numpy())
            bad = b.clone()
            bad[int(off[bad_mesh]) + 900] = float("inf")
            y = torch.zeros_like(b)
            _, _, sts, _ = s.solve_segmented_device(bad, y, tol=1e-12, itmax=2000)
            assert np.all(np.delete(sts, bad_mesh) == 0)
            keep = np.r_[0:off[bad_mesh], off[bad_mesh + 1]:off[-1]]
            assert rel_l2(y.cpu().numpy()[keep], out[scatter][0][keep]) < 1e-9
    x, b = out["auto"]
    for m, p in enumerate(probs):
        sl = slice(off[m], off[m + 1])
        assert rel_l2(x[sl], out["atomic"][0][sl]) < 1e-9, m
        ax, _ = oracle.matvec0(p.mesh.iss, oracle_bb(oracle, p, 2.0, aM), p.bc, x[sl])
        nb = np.linalg.norm(b[sl])
        assert np.linalg.norm(b[sl] - ax) <= 2e-12 * nb or nb == 0.0, m


@pytest.mark.parametrize("K", [16, 32, 64])
@pytest.mark.parametrize("dims", [(1, 1, 1), (6, 2, 1), (7, 3, 30), (8, 7, 5), (15, 16, 9),
                                  (33, 17, 12)])
def test_block_solve_launch_shapes(vdr, oracle, gpu_lib, dims, K):
    """The block solve on assembled rows where its tiles (8 or 16 nodes along
    x, 4 or 8 along y), its blocks' shares of the planes and the last plane
    end: every column's true residual by the oracle, and against the
    element-wise solve (scatter "atomic"); columns of very different size, a
    zero one, a start from a nonzero X."""
    torch = pytest.importorskip("torch")
    prob = vdr.problems.rotation_shear(*dims, seed=96)
    m, aM, tol = prob.mesh, 10.0, 1e-11
    rng = np.random.default_rng(sum(dims) + K)
    B = rng.standard_normal((m.nnode, K)) * 10.0 ** rng.integers(-200, 200, K)
    B[prob.bc == 1] = 0.0
    B[:, 3] = 0.0
    X0 = np.zeros_like(B)
    X0[:, 5] = B[:, 5]
    got = {}
    for scatter in ("auto", "atomic"):
        with vdr.Solver(prob, vdr.Options(scatter=scatter), aH=2.0, aM=aM) as s:
            X = torch.tensor(X0, device="cuda")
            _, _, errs, st = s.solve_block_device(torch.tensor(B, device="cuda"), X, tol=tol,
                                                  inner_tol=1e-4)
            torch.cuda.synchronize()
            assert st == 0 and np.all(errs <= tol)
            got[scatter] = X.cpu().numpy()
    bb = oracle_bb(oracle, prob, 2.0, aM)
    assert np.all(got["auto"][prob.bc == 1] == 0.0) and np.all(got["auto"][:, 3] == 0.0)
    for k in range(K):
        x, b = got["auto"][:, k], B[:, k]
        if not b.any():
            continue
        scale = np.abs(b).max()
        ax, _ = oracle.matvec0(m.iss, bb, prob.bc, x / scale)
        assert np.linalg.norm(b / scale - ax) <= 1.01 * tol * np.linalg.norm(b / scale), k
        assert rel_l2(x / scale, got["atomic"][:, k] / scale) < 1e-8, k


def test_recorded_apply_follows_the_operator(vdr, oracle, gpu_lib):
    """An apply recorded by its caller, after applies that already run on
    assembled rows, and replayed after the operator was built anew gives the
    new operator's product."""
    torch = pytest.importorskip("torch")
    prob = vdr.problems.rotation_shear(13, 6, 5, seed=97)
    m = prob.mesh
    x = np.random.default_rng(5).standard_normal(m.nnode)
    with vdr.Solver(prob, aH=2.0, aM=7.0) as s:
        for _ in range(3):
            s.apply(x)
        xd = torch.tensor(x, device="cuda")
        yd = torch.empty_like(xd)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(s.stream()),
                              capture_error_mode="thread_local"):
            assert s.lib.vdr_apply_device(s.h, xd.data_ptr(), yd.data_ptr(), 0) == 0
        for aM in (7.0, 19.0):
            s.set_operator(2.0, aM)
            s.apply(x)  # builds it
            graph.replay()
            torch.cuda.synchronize()
            ref, _ = oracle.matvec0(m.iss, oracle_bb(oracle, prob, 2.0, aM), prob.bc, x)
            assert rel_l2(yd.cpu().numpy(), ref) < TOL, aM


def test_block_solve_of_unaligned_arrays(vdr, gpu_lib):
    """B or X starting off a 16-byte boundary is solved as aligned ones are."""
    torch = pytest.importorskip("torch")
    prob = vdr.problems.rotation_shear(7, 6, 5, seed=98)
    N, K = prob.mesh.nnode, 16
    B = np.random.default_rng(6).standard_normal((N, K))
    B[prob.bc == 1] = 0.0
    with vdr.Solver(prob, aH=2.0, aM=10.0) as s:
        got = []
        for ob, ox in ((0, 0), (1, 0), (0, 1)):
            Bd = torch.zeros(N * K + 1, dtype=torch.float64, device="cuda")[ob:ob + N * K]
            Xd = torch.zeros(N * K + 1, dtype=torch.float64, device="cuda")[ox:ox + N * K]
            Bd, Xd = Bd.view(N, K), Xd.view(N, K)
            Bd.copy_(torch.tensor(B, device="cuda"))
            torch.cuda.synchronize()
            _, _, errs, st = s.solve_block_device(Bd, Xd, tol=1e-11, inner_tol=1e-4)
            torch.cuda.synchronize()
            assert st == 0 and np.all(errs <= 1e-11)
            got.append(Xd.cpu().numpy().copy())
    assert rel_l2(got[1], got[0]) < 1e-9 and rel_l2(got[2], got[0]) < 1e-9

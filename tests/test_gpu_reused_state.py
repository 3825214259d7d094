"""Calls that reuse what an earlier call left behind -- recorded graphs,
buffers, rows -- give the answers that first calls give."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


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

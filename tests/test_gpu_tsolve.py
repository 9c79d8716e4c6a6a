"""T = R11^{-1} R12 of given skeletons whose columns differ in size or nearly depend on one another."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def skeleton_matrix(kind, k, n):
    """n columns, the first k of them (in this order) the skeleton."""
    rng = np.random.Generator(np.random.Philox(key=k))
    A = rng.standard_normal((k + 40, n))
    j = np.arange(k)
    if kind == "ascending":          # 2^0 in the first block of 64 columns up to 2^60 in the last
        A[:, :k] *= 2.0 ** (60 * (j // 64) // ((k - 1) // 64))
    elif kind == "descending":
        A[:, :k] *= 2.0 ** -(60 * (j // 64) // ((k - 1) // 64))
    elif kind == "mixed":            # sizes without any order
        A[:, :k] *= 2.0 ** rng.integers(-30, 31, k)
    elif kind == "pairs":            # every second column its neighbour's within 1e-6
        A[:, 1:k:2] = A[:, 0:k - k % 2:2] + 1e-6 * A[:, 1:k:2]
    elif kind == "blocks":           # a block of 64 columns follows the one before within 1e-6
        A[:, 64:k] = A[:, :k - 64] + 1e-6 * A[:, 64:k]
    return A


def substitution(R, B):
    R, X = R.astype(np.longdouble), B.astype(np.longdouble)
    for i in range(len(R) - 1, -1, -1):
        X[i] /= R[i, i]
        X[:i] -= np.outer(R[:i, i], X[i])
    return X


@pytest.mark.parametrize("kind", ["ascending", "descending", "mixed", "pairs", "blocks"])
@pytest.mark.parametrize("k,nc", [(128, 33), (130, 33), (257, 33), (700, 33),    # substitution, one block, 3 of 128, 3 of 256
                                  (100, 9100), (128, 5600)])
def test_T_of_skeletons_in_any_order_and_scale(kind, k, nc):
    from robust_blockwise_random_pivoting_gb300.rbrp import Handle
    from robust_blockwise_random_pivoting_gb300.sketch_ids import fixed_skeleton
    n = k + nc
    A = torch.from_numpy(skeleton_matrix(kind, k, n)).cuda().t().contiguous().t()
    with Handle(0) as h:
        perm, T = fixed_skeleton(h, A, torch.arange(k, dtype=torch.int32), b=64)
        R = h.L().cpu().numpy()[perm.cpu().numpy()].T
    T, k = T.cpu().numpy(), T.shape[0]      # (columns whose residual norm is lost in rounding are not taken)
    R11 = R[:, :k]
    want = substitution(R11, R[:, k:])
    # in the scaling 2^-f of R11's columns: a residual of (4 k + 256) eps of the row's largest entry
    # times the largest of T's column - the slices' cuts and the sums over k, and the block inverses
    # that are not refined (largest entry 128) - carried through |R11^-1|
    f = np.abs(R11).max(0)
    Rs, Y = R11 / f, np.abs(T) * f[:, None]
    inv = np.abs(substitution(Rs, np.eye(k))).astype(np.float64)
    bound = (4 * k + 256) * EPS * (inv @ np.abs(Rs).max(1))[:, None] * Y.max(0) / f[:, None]
    assert np.all(np.abs(T - want) <= bound), float((np.abs(T - want) / bound).max())


def test_T_without_room_for_its_operands():
    """The T solve on a device that has no room for the slices' operands takes the FP64 pipe."""
    from robust_blockwise_random_pivoting_gb300.rbrp import Handle
    A = torch.from_numpy(skeleton_matrix("pairs", 300, 340)).cuda().t().contiguous().t()
    with Handle(0) as h:
        h.set_tsolve_fp64(True)
        want = h.column_id(A, b=50, tol=None, kmax=300, seed=2)
    with Handle(0) as h:
        h.column_id(A, b=50, tol=None, kmax=300, seed=2, compute_T=False)
        h.set_memory_limit(300 * 40 * 8)       # room for T alone
        got = h.column_id(A, b=50, tol=None, kmax=300, seed=2)
    assert torch.equal(got.perm, want.perm) and torch.equal(got.T, want.T)


@pytest.mark.parametrize("k", [128, 200])      # (the first by its rank, the second after the slices)
def test_T_of_a_factor_that_slices_do_not_solve(k):
    """A_S = R11 with 1 on the diagonal and -1 above, R12 = R11 X, all of it exact: the inverse's
    entries grow as 2^k and their products cancel past any refinement; the substitution on the
    FP64 pipe, which has to solve, gives X itself."""
    from robust_blockwise_random_pivoting_gb300.rbrp import Handle
    from robust_blockwise_random_pivoting_gb300.sketch_ids import fixed_skeleton
    n = k + 32
    R = np.eye(k) - np.triu(np.ones((k, k)), 1)
    X = np.random.Generator(np.random.Philox(key=1)).integers(-1000, 1001, (k, n - k)).astype(np.float64)
    A = np.zeros((k + 72, n))
    A[:k] = np.hstack([R, R @ X])
    A = torch.from_numpy(A).cuda().t().contiguous().t()
    with Handle(0) as h:
        perm, T = fixed_skeleton(h, A, torch.arange(k, dtype=torch.int32), b=1)
        assert "T_fp64" in h.form()
    assert np.array_equal(perm.cpu().numpy(), np.arange(n)) and np.array_equal(T.cpu().numpy(), X)


@pytest.mark.parametrize("k", [128, 300, 600])
def test_T_of_smooth_kernel_skeletons(k):
    """Skeletons in no order of a smooth kernel: blocks whose inverses cancel and are refined."""
    from robust_blockwise_random_pivoting_gb300.rbrp import Handle
    from robust_blockwise_random_pivoting_gb300.sketch_ids import fixed_skeleton
    rng = np.random.Generator(np.random.Philox(key=k))
    x, y = rng.random((k + 60, 3)), rng.random((k + 40, 3))
    A = np.exp(-2.0 * ((x[:, None] - y[None]) ** 2).sum(-1)) + 1e-10 * rng.standard_normal((k + 60, k + 40))
    A = torch.from_numpy(A).cuda().t().contiguous().t()
    with Handle(0) as h:
        perm, T = fixed_skeleton(h, A, torch.arange(k, dtype=torch.int32), b=64)
        R = h.L().cpu().numpy()[perm.cpu().numpy()].T.astype(np.longdouble)
    T = T.cpu().numpy()
    k = len(T)
    # per column, against the largest entry of |R11| |T|: the sums over k of the substitution (eps
    # each) and what a cancellation of 2^6 may leave of a block that is not refined
    res = np.abs(R[:, :k] @ T - R[:, k:]).max(0)
    assert np.all(res <= (k + 64) * EPS * (np.abs(R[:, :k]) @ np.abs(T)).max(0))


@pytest.mark.parametrize("k", [1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 128])
@pytest.mark.parametrize("nc", [1, 7, 8, 9, 300])
def test_T_of_small_ranks(k, nc):
    """Up to rank 128 the substitution on the FP64 pipe, a warp per column: entry by entry within the
    rounding of k + 3 operations on rows that were divided by their diagonal first, twice over for the
    reciprocal."""
    from robust_blockwise_random_pivoting_gb300.rbrp import Handle
    from robust_blockwise_random_pivoting_gb300.sketch_ids import fixed_skeleton
    A = torch.from_numpy(skeleton_matrix("mixed", k, k + nc)).cuda().t().contiguous().t()
    with Handle(0) as h:
        perm, T = fixed_skeleton(h, A, torch.arange(k, dtype=torch.int32), b=min(k, 16))
        assert "T_fp64" in h.form() and T.shape == (k, nc)
        R = h.L().cpu().numpy()[perm.cpu().numpy()].T
    R11, T = R[:, :k], T.cpu().numpy()
    want = substitution(R11, R[:, k:])
    inv = np.abs(substitution(R11, np.eye(k))).astype(np.float64)
    bound = (2 * k + 8) * EPS * (inv @ (np.abs(R11) @ np.abs(T)))
    assert np.all(np.abs(T - want) <= bound), float((np.abs(T - want) / bound).max())

"""The FP64 form's tensor-core products (exact BF16 slices) against the FP64 pipe."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def colmajor(A):
    return torch.from_numpy(np.asfortranarray(A)).cuda().t().contiguous().t()


def first_block(A, b, variant):
    """perm, L = A^T Q of a run of one block (both variants form the same Q on the FP64 pipe)."""
    from robust_blockwise_random_pivoting_gb300.rbrp import Handle
    with Handle(0) as h:
        h.set_variant(variant)
        r = h.column_id(colmajor(A), b=b, tol=None, kmax=min(4 * b if b <= 8 else b, *A.shape), seed=3, compute_T=False)
        assert len(r.ranks) >= 1
        k1 = int(r.ranks[0])
        return r.perm.cpu().numpy(), h.L().cpu().numpy()[:, :k1], k1


def matrix(kind, m, n):
    rng = np.random.Generator(np.random.Philox(key=m * 4099 + n))
    A = rng.standard_normal((m, n))
    if kind == "scaled":        # column scales over the whole exponent range, entries over 60 binades, zero columns
        A *= 2.0 ** rng.integers(-60, 1, (m, n))
        A *= 2.0 ** rng.integers(-400, 400, n)
        A[:, 5] = 0.0
    elif kind == "digits":      # every digit of every entry near its largest magnitude, one sign: the largest class sums
        A = np.full((m, n), float(0x1F7F7F7F7F7F7F) * 2.0 ** -53) * (1.0 + 1e-3 * rng.standard_normal((1, n)))
        A[rng.integers(0, m, n), np.arange(n)] += 1.0
    elif kind == "ones":        # the largest sums of the top limbs
        A = np.ones((m, n)) * (2.0 - 2.0 ** -52) + 1e-9 * A
    return A


@pytest.mark.parametrize("kind", ["normal", "scaled", "digits", "ones"])
@pytest.mark.parametrize("m,n,b", [(1, 30, 1), (255, 100, 1), (257, 333, 2), (1000, 129, 4), (8193, 65, 8), (20000, 40, 1),
                                   (32768, 50, 7), (40, 129, 9), (63, 300, 16), (64, 140, 32), (65, 200, 33), (192, 128, 31),
                                   (193, 257, 64), (500, 1000, 48), (1100, 333, 64), (4000, 700, 40)])
def test_projection_matches_the_fp64_pipe(kind, m, n, b):
    A = matrix(kind, m, n)
    perm0, L0, k0 = first_block(A, b, 0)
    perm1, L1, k1 = first_block(A, b, 1)
    assert k0 == k1 and np.array_equal(perm0[:k0], perm1[:k1])
    # |fl(q^T a) - q^T a| <= gamma_m |q|^T |a| <= m eps ||a|| for the FMA chain and ||q|| = 1; the slices
    # add the representation (2^-54 of each row's largest entry per value) and the dropped classes
    norm = np.array([np.linalg.norm(c / s) * s if s > 0 else 0.0 for c, s in zip(A.T, np.abs(A).max(0))])
    bound = (m + 1) * EPS * norm[:, None] + m * 2.0 ** -53 * np.abs(A).max(0)[:, None]
    if b == 1:      # one column's panel is normalised twice by reciprocals: a few eps of it
        bound = bound + 8 * EPS * norm[:, None]
    assert np.isfinite(L0).all() and np.isfinite(L1).all()
    rest = perm0[k0:]
    assert np.all(np.abs(L0 - L1)[rest] <= bound[rest])


# (the last three take the Gram-Schmidt products as slices: m i b >= 2e7, one and two column halves,
# ragged row tiles and blocks of the basis)
@pytest.mark.parametrize("m,n,b,kmax", [(300, 900, 20, 150), (700, 650, 64, 300), (5000, 400, 40, 250),
                                        (9000, 500, 30, 330), (6401, 700, 64, 600)])
def test_blocks_after_the_first_follow_the_same_skeleton(m, n, b, kmax):
    from robust_blockwise_random_pivoting_gb300.rbrp import Handle
    A = colmajor(matrix("normal", m, n))
    got = []
    for variant in (0, 1):
        with Handle(0) as h:
            h.set_variant(variant)
            r = h.column_id(A, b=b, tol=None, kmax=kmax, seed=1)
            got.append((r.perm.cpu().numpy(), r.ranks, r.T.cpu().numpy()))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    # a Gaussian matrix of these shapes: kappa(A_S) < 30, one Gram-Schmidt pass, m eps kappa^2
    d = np.linalg.norm(got[0][2] - got[1][2]) / np.linalg.norm(got[1][2])
    assert d <= m * EPS * 900, d


@pytest.mark.parametrize("k,n", [(1, 40), (63, 95), (64, 129), (65, 128), (255, 400), (256, 257), (257, 700),
                                 (520, 66200), (900, 1000)])
def test_T_solve_matches_the_fp64_pipe(k, n):
    """T = R11^{-1} R12 as slice products against the substitution on the FP64 pipe, at the
    edges of its blocks of 256 rows, tiles of 128 x 64 and passes of 65536 columns."""
    from robust_blockwise_random_pivoting_gb300.rbrp import Handle
    rng = torch.Generator(device="cuda").manual_seed(k)
    m = k + 40
    A = torch.randn(n, m, generator=rng, device="cuda", dtype=torch.float64).t()
    A = (A * 2.0 ** -(torch.arange(n, device="cuda") % 50)).t().contiguous().t()     # graded columns
    Ts = []
    for fp64 in (True, False):
        with Handle(0) as h:
            h.set_tsolve_fp64(fp64)
            r = h.column_id(A, b=min(64, k), tol=None, kmax=k, sampler="greedy")
            assert r.k == k
            Ts.append(r.T)
    # substitution: |dT| <= c k eps |R^-1| |R| |T|, row by row; greedy pivots keep |R^-1| |R| of these
    # Gaussian factors below 20 sqrt(k)
    scale = Ts[0].abs().amax(0).clamp_min(1e-300)
    d = ((Ts[1] - Ts[0]).abs().amax(0) / scale).max().item()
    assert d <= 4 * k * EPS * 20 * k ** 0.5, d


def test_slice_gemm_timeout_is_clean():
    """The projection's bounded waits run out under a budget of one clock: status 7, and the
    same handle reproduces an untouched one's results afterwards."""
    from robust_blockwise_random_pivoting_gb300._lib import RBRPError
    from robust_blockwise_random_pivoting_gb300.rbrp import Handle
    A = colmajor(matrix("normal", 900, 700))
    with Handle(0) as fresh:
        want = fresh.column_id(A, b=64, tol=None, kmax=200, seed=0)
    with Handle(0) as h:
        h.set_wait_budget(1)
        with pytest.raises(RBRPError) as e:
            h.column_id(A, b=64, tol=None, kmax=200, seed=0)
        assert e.value.status == 7
        h.set_wait_budget(0)
        got = h.column_id(A, b=64, tol=None, kmax=200, seed=0)
    assert torch.equal(got.perm, want.perm) and torch.equal(got.T, want.T)


@pytest.mark.parametrize("b", [1, 8, 48])
def test_a_basis_that_is_not_finite_is_an_error(b):
    """Given skeletons of exactly dependent columns: where the second Cholesky factorisation of a
    panel breaks down the run says so (status 5), as with the FP64 pipe's products, and otherwise
    |q^T a| <= ||a|| for its basis vectors of norm 1."""
    from robust_blockwise_random_pivoting_gb300._lib import RBRPError
    from robust_blockwise_random_pivoting_gb300.rbrp import Handle
    from robust_blockwise_random_pivoting_gb300.sketch_ids import fixed_skeleton
    S = torch.arange(48, dtype=torch.int32)
    with Handle(0) as h:
        for seed in range(400):
            rng = np.random.default_rng(seed)
            r, m = int(rng.integers(1, 20)), int(rng.integers(64, 300))
            if seed % 2:
                A = rng.standard_normal((m, r)) @ rng.standard_normal((r, 80))
            else:
                A = rng.integers(-3, 4, (m, r)).astype(float) @ rng.integers(-3, 4, (r, 80))
            A[:, 48:] += rng.standard_normal((m, 32))
            try:
                fixed_skeleton(h, colmajor(A), S, b=b)
            except RBRPError as e:
                assert e.status == 5, seed
                continue
            L = h.L().cpu().numpy()
            assert np.isfinite(L).all(), seed
            assert np.all(np.abs(L) <= 1.01 * np.linalg.norm(A, axis=0)[:, None]), seed


def test_the_form_of_a_run_is_told():
    """Which arithmetic a run took, with and without room for its scratch (256 x 400 slices: 2 MB)."""
    from robust_blockwise_random_pivoting_gb300.rbrp import Handle
    A = colmajor(matrix("normal", 256, 400))

    def form(h, **kw):
        h.column_id(A, kmax=100, **kw)
        return h.form()
    for limit in (0, 1 << 20):
        room = limit == 0
        with Handle(0) as h:
            form(h, b=20, tol=1e-10)               # the workspace that every run has to have
            h.set_memory_limit(limit)
            f = form(h, b=20, tol=1e-4)
            assert ("slices" in f) == room and "fixed_point" not in f and "fixed_order" not in f
            f = form(h, b=4, tol=None, sampler="greedy")
            assert ("fixed_point" in f) == (room or 256 * 400 * 8 <= limit // 2) and "slices" not in f
            f = form(h, b=20, tol=1e-10)
            assert "fixed_order" in f and "slices" not in f
    with Handle(0) as h:
        h.column_id(A.float(), b=20, tol=1e-10, kmax=100)
        assert h.form() <= {"T_fp64"}


@pytest.mark.parametrize("sampler", ["np", "es", "greedy"])
@pytest.mark.parametrize("b,kmax", [(8, None), (8, 220), (24, None), (40, 215)])
def test_draws_past_the_depth_follow_the_fixed_order(sampler, b, kmax):
    """Draws from weights below 1e-8 of the start (the spectrum exp(-i / 12) has its numerical rank
    near 230) follow the order of the sums: a run without a tolerance that gets there takes the
    columns, bit for bit, that one to a tolerance below any residual takes."""
    from robust_blockwise_random_pivoting_gb300.rbrp import Handle
    from robust_blockwise_random_pivoting_gb300.workloads import gaussian_exp
    A = colmajor(gaussian_exp(400, 400, decay=12.0, seed=0))
    with Handle(0) as h:
        for seed in range(3):
            got = h.column_id(A, b=b, tol=None, kmax=kmax, seed=seed, sampler=sampler)
            assert "fixed_order" in h.form()
            want = h.column_id(A, b=b, tol=1e-30, kmax=kmax, seed=seed, sampler=sampler)
            assert "fixed_order" in h.form()
            assert torch.equal(got.perm, want.perm) and np.array_equal(got.ranks, want.ranks)
            assert np.array_equal(got.residuals, want.residuals) and got.draws == want.draws
            assert torch.equal(got.T, want.T)
            if kmax:     # above the depth the order is free
                h.column_id(A, b=b, tol=None, kmax=40, seed=seed, sampler=sampler)
                assert "fixed_order" not in h.form()


@pytest.mark.parametrize("m,n,b", [(64, 120, 16), (193, 150, 33), (300, 400, 40), (1100, 333, 64), (777, 100, 48),
                                   (500, 200, 8), (600, 150, 3), (900, 100, 1)])
def test_projection_error_is_that_of_the_operands_digits(m, n, b):
    """The first block's products against exact ones.  Unit columns e_j beside the data give its basis,
    Q(j, :) = Q^T e_j.  What may be off: entries of q and a cut 55 bits below 2^e > |.|max, uniformly, their
    products' dropped classes, Q(j, :) read back in 53 bits and one rounding of the result: four times the
    root mean square of that (without its lowest class of 2^-60 products the error is ten times)."""
    rng = np.random.Generator(np.random.Philox(key=m))
    B = rng.standard_normal((m, n))
    A = np.hstack([B, np.eye(m)])
    err = []
    for variant in (0, 1):
        perm, L, k1 = first_block(A, b, variant)
        assert (perm[:k1] < n).all()               # the data's norms are far above the unit columns'
        rest = np.setdiff1d(np.arange(n), perm[:k1])
        Q = L[n:].astype(np.longdouble)
        exact = B[:, rest].T.astype(np.longdouble) @ Q
        err.append((L[rest] - exact).astype(np.float64))
    Q, X = Q.astype(np.float64), B[:, rest]
    eq, ea = 2.0 ** np.frexp(np.abs(Q).max(0))[1], 2.0 ** np.frexp(np.abs(X).max(0))[1]
    u = 1.0 / np.sqrt(12.0)                        # of a unit, uniform
    var = (u * 2.0 ** -54 * ea[:, None] * np.linalg.norm(Q, axis=0)) ** 2 \
        + (u * 2.0 ** -54 * eq * np.linalg.norm(X, axis=0)[:, None]) ** 2 \
        + (u * 2.0 ** -52) ** 2 * ((X ** 2).T @ Q ** 2) \
        + (u * 2.0 ** -52 * np.abs(X.T @ Q)) ** 2 \
        + (2.0 ** -60 * ea[:, None] * eq * np.sqrt(5.0 * m) * 128 ** 2 / 3 / 256 ** 2) ** 2
    rms = lambda e: float(np.sqrt(np.mean(e ** 2)))
    assert rms(err[0]) <= 4 * np.sqrt(var.mean())
    assert rms(err[0]) <= rms(err[1])              # and no more than the FP64 pipe's


@pytest.mark.parametrize("gen,m,n,b,tol,kmax,sampler", [
    ("exp", 700, 900, 40, 1e-4, None, "np"), ("exp", 1300, 600, 64, 1e-7, None, "np"), ("exp", 600, 800, 33, 1e-6, None, "es"),
    ("normal", 900, 500, 64, None, 300, "np"), ("normal", 640, 1200, 8, None, 100, "np"),
    ("normal", 500, 700, 1, None, 60, "greedy"), ("normal", 5000, 400, 48, None, 200, "np")])
def test_free_order_runs_take_the_oracles_columns(gen, m, n, b, tol, kmax, sampler):
    """The forms with free sums (slices, fixed point, L D L^T panels, sliced Gram-Schmidt in the last case)
    against the CPU oracle: the same columns in the same order, ranks and residuals."""
    from oracle import rbrp_column_id
    from robust_blockwise_random_pivoting_gb300.rbrp import Handle
    from robust_blockwise_random_pivoting_gb300.workloads import gaussian_exp
    A = matrix("normal", m, n) if gen == "normal" else gaussian_exp(m, n, decay=30.0, seed=2)
    want = rbrp_column_id(A, b, tol=tol, seed=0, sampler="np" if sampler == "greedy" else sampler,
                          mode="gp" if sampler == "greedy" else "rp", kmax=kmax)
    with Handle(0) as h:
        got = h.column_id(colmajor(A), b=b, tol=tol, kmax=kmax, sampler=sampler)
        assert ("fixed_point" if b <= 8 else "slices") in h.form() and "fixed_order" not in h.form()
    assert got.k == want["k"] and np.array_equal(got.ranks, want["ranks"])
    assert np.array_equal(got.perm.cpu().numpy(), want["perm"])
    np.testing.assert_allclose(got.residuals, want["residuals"], rtol=1e-6, atol=1e-14)

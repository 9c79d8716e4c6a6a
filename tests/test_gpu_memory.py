"""Device memory that a handle keeps between calls, seen on a device that is (said to be) nearly full."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
MB = 1 << 20
M, N = 512, 1100


def matrix(dtype=torch.float64):
    g = torch.Generator(device="cuda").manual_seed(5)
    return torch.randn(N, M, generator=g, device="cuda", dtype=torch.float64).to(dtype).t()


def later_batch(h, A):
    from robust_blockwise_random_pivoting_gb300.rbrp import Batch
    Batch(h, [matrix(torch.float32)[:64, :64].t().contiguous().t()], b=16).run()


def later_adjoint(h, A):
    from robust_blockwise_random_pivoting_gb300.adjoint import fixed_skeleton_id_loss
    B = A[:200, :300].float().t().contiguous().t().requires_grad_()
    fixed_skeleton_id_loss(B, torch.arange(100, dtype=torch.int32), torch.ones(300, device="cuda"), 50, h).backward()


def later_sketch(h, A):
    from robust_blockwise_random_pivoting_gb300.sketch_ids import gaussian_sketch
    gaussian_sketch(A.float(), 64, handle=h)


def later_lupp(h, A):
    from robust_blockwise_random_pivoting_gb300.sketch_ids import lupp_pivots
    lupp_pivots(A[:50], handle=h)


LATER = {
    "host run": lambda h, A: h.column_id_host(A.cpu(), b=32, tol=None, kmax=100, sampler="greedy"),
    "T_matdivide": lambda h, A: h.T_matdivide(),
    "refine_T": lambda h, A: h.refine_T(A),
    "batch": later_batch,
    "adjoint": later_adjoint,
    "sketch": later_sketch,
    "lupp": later_lupp,
}


@pytest.mark.parametrize("name", list(LATER))
def test_every_allocation_gets_the_slices_memory(name):
    """After an FP64 run its slices (9 MB here) fill what the device has: the next call on the handle
    takes their memory instead of failing."""
    from robust_blockwise_random_pivoting_gb300.rbrp import Handle
    A = matrix()
    with Handle(0) as h:
        r = h.column_id(A, b=32, tol=None, kmax=100)
        assert r.k == 100 and "slices" in h.form()
        held = h.scratch_bytes()
        assert held > 8 * MB
        h.set_memory_limit(held)
        LATER[name](h, A)
        assert h.scratch_bytes() != held
        torch.cuda.synchronize()


def test_a_handle_keeps_scratch_of_up_to_a_sixteenth_of_the_device():
    from robust_blockwise_random_pivoting_gb300.rbrp import Handle
    total = torch.cuda.get_device_properties(0).total_memory
    m = 32000
    n = total // 16 // (14 * m) + 64           # 14 bytes of slices an entry
    for n, keep in ((1000, True), (n, False)):
        A = torch.randn(n, m, device="cuda", dtype=torch.float64).t()
        free = torch.cuda.mem_get_info()[0]
        with Handle(0) as h:
            for _ in range(2):
                h.column_id(A, b=16, tol=None, kmax=32, compute_T=False)
                assert "slices" in h.form() and (h.scratch_bytes() > 0) == keep
            if not keep:
                assert free - torch.cuda.mem_get_info()[0] < 1 << 30
        del A
        torch.cuda.empty_cache()


@pytest.mark.parametrize("mb,sliced_cgs", [(0, True), (72, True), (61, False)])
def test_the_basis_gets_what_the_slices_of_A_leave(mb, sliced_cgs):
    """2000 x 800 to rank 700: 32 MB for the slices of A and what goes with them, 20 MB for those of the
    whole basis.  Half of 72 MB holds 200 basis vectors' too, half of 61 MB none: the products
    with A stay on the tensor cores, those with the basis go there as far as there is room."""
    from robust_blockwise_random_pivoting_gb300.rbrp import Handle
    g = torch.Generator(device="cuda").manual_seed(7)
    A = torch.randn(800, 2000, generator=g, device="cuda", dtype=torch.float64).t()
    with Handle(0) as h:
        h.set_variant(1)
        want = h.column_id(A, b=64, tol=None, kmax=700)
    with Handle(0) as h:
        h.set_memory_limit(mb * MB)
        got = h.column_id(A, b=64, tol=None, kmax=700)
        assert h.form() - {"T_fp64"} == ({"slices", "sliced_cgs"} if sliced_cgs else {"slices"})
    assert torch.equal(got.perm, want.perm) and np.array_equal(got.ranks, want.ranks)
    # a Gaussian matrix: kappa(A_S) < 10, one Gram-Schmidt pass, m eps kappa^2
    assert (got.T - want.T).norm() <= 2000 * 2.0 ** -53 * 100 * want.T.norm()

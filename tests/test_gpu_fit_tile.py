"""GEMMs whose tile the plan picks itself, on one GPU: each of the tiles, with ragged rows and columns."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,swiglu", [
    (200, 3328, 1584, False), (320, 7000, 3000, False), (384, 648, 776, False),        # 128 or 256 wide, single CTAs
    (1984, 8200, 1000, False), (1090, 4104, 3832, False),      # CTA pairs, a short K: stores staged (59 k-blocks)
    (1090, 4104, 3848, False), (2100, 2056, 6000, False),      # one k-block more, and long: not staged
    (1024, 4096, 16384, False), (2300, 8192, 12288, False),    # 512-row tiles, or pairs cut along K
    (700, 1416, 1000, True), (1928, 3000, 2048, True), (400, 7392, 4096, True),
])
def test_tiles(M, N, K, swiglu):
    from tridist_b200.ops._gemm_common import gemm_nt
    for dt in (torch.float16, torch.bfloat16):
        g = torch.Generator(device="cuda").manual_seed(M)
        a = (torch.randn((M, K), generator=g, device="cuda") * 0.1).to(dt)
        b = (torch.randn((2 * N if swiglu else N, K), generator=g, device="cuda") * 0.1).to(dt)
        for ldc in (N, N + 8, N + 136):        # rows of the output on their own, beside others
            plane = torch.full((M + 1, ldc), 5.0, dtype=dt, device="cuda")
            out = plane[:M, :N]
            gemm_nt(a, b, out=out, swiglu=swiglu)
            torch.cuda.synchronize()
            exact = a.double() @ b.double().t()
            half_ulp = 2.0 ** -11 if dt == torch.float16 else 2.0 ** -8
            e = K * 2.0 ** -23 * (a.abs().double() @ b.abs().double().t())       # an fp32 sum of K products in any order
            if swiglu:
                gate, up = exact[:, :N], exact[:, N:]
                exact = F.silu(gate) * up
                e = exact.abs() * 2.0 ** -18 + 1.1 * e[:, :N] * up.abs() + F.silu(gate).abs() * e[:, N:]
            assert bool(((out.double() - exact).abs() <= exact.abs() * half_ulp * 1.01 + e + 2.0 ** -24).all())
            assert bool((plane[M] == 5.0).all()) and bool((plane[:, N:] == 5.0).all())


@pytest.mark.parametrize("M,N,K", [
    (384, 3328, 1584), (320, 28672, 8192),                     # 128 and 256 wide, single CTAs
    (1984, 8192, 1024), (1728, 12288, 12288), (512, 8192, 4096),     # CTA pairs, staged or not, tiles cut along K
    (1024, 8192, 28672),                                       # 512-row tiles
])
def test_tiles_that_give_up_leave_the_context_usable(M, N, K):
    """With the abort word raised every role leaves the first wait that looks at it, whatever the others still have on
    their way: the call reports it or is complete, and the calls after it are right."""
    from tridist_b200.ops import create_gemm_ar_intra_node_context, finalize_gemm_ar_context, gemm_ar_intra_node_op
    from tridist_b200.parallel.runtime import ProcessWorld, native
    C, w, dt = native(), ProcessWorld(0, 1), torch.bfloat16
    ctx = create_gemm_ar_intra_node_context(M, N, dt, dt, 0, 1, M_PER_CHUNK=64, world=w)
    g = torch.Generator(device="cuda").manual_seed(N)
    a, b = [(torch.randn((n, K), generator=g, device="cuda") * 0.1).to(dt) for n in (M, N)]
    c = torch.empty((M, N), dtype=dt, device="cuda")
    gemm_ar_intra_node_op(a, b, c, ctx)
    torch.cuda.synchronize()
    w.check()
    ref = c.clone()
    exact = a.double() @ b.double().t()
    assert (ref.double() - exact).norm() <= 2.0 ** -8 * exact.norm()
    for _ in range(5):
        c.zero_()
        C.fill_u32(w.abort_word, 1, 5)
        gemm_ar_intra_node_op(a, b, c, ctx)
        torch.cuda.synchronize()
        assert w.status()[0] == 5 or torch.equal(c, ref)
        w.clear_status()
        for _ in range(2):
            gemm_ar_intra_node_op(a, b, c, ctx)
        torch.cuda.synchronize()
        w.check()
        assert torch.equal(c, ref)
    finalize_gemm_ar_context(ctx)

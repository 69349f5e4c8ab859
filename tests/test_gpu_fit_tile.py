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

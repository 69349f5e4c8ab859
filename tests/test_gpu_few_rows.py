"""The GEMM for few rows (csrc/gemm/skinny_gemm.cuh) on one GPU, at the edges of its layout."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _rand(shape, seed, dt):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * 0.1).to(dt)


def _bound(a, b, exact, dt):
    """One rounding to 16 bits after an fp32 sum of K products in any order."""
    half_ulp = 2.0 ** -11 if dt == torch.float16 else 2.0 ** -8
    return exact.abs() * half_ulp * 1.01 + a.shape[1] * 2.0 ** -23 * (a.abs().double() @ b.abs().double().t()) + 2.0 ** -24


@pytest.mark.parametrize("M,N,K,swiglu,cluster", [
    (1, 8, 8, False, 1), (16, 264, 136, False, 1), (33, 1000, 64, False, 1),
    (64, 4096, 1376, False, 1),                # a share of 24 or 32 rows of B, last k-block short
    (65, 1000, 1024, False, 1), (128, 8192, 3584, False, 1), (128, 1408, 4096, False, 2),
    (100, 48, 8200, False, 4),                 # three shares, four ranges of K
    (64, 2048, 16384, False, 4), (128, 4096, 12288, False, 4),
    (128, 40000, 512, False, 1),               # several shares a CTA
    (96, 30000, 4096, False, 1), (128, 3584, 2048, True, 1), (100, 1416, 4104, True, 2), (40, 20000, 320, True, 1),
    (128, 128, 8192, True, 4),
])
def test_few_rows(M, N, K, swiglu, cluster):
    from tridist_b200.ops._gemm_common import gemm_nt
    from tridist_b200.parallel.runtime import native
    assert native().skinny_layout(M, N, K, swiglu, 148)["cluster"] == cluster
    for dt in (torch.float16, torch.bfloat16):
        wide_a, wide_b = _rand((M, K + 24), 1, dt), _rand((2 * N if swiglu else N, K + 8), 2, dt)
        a, b = wide_a[:, 8:K + 8], wide_b[:, :K]                # row strides of their own, a on a 16-byte boundary
        plane = torch.full((M + 2, N + 16), 7.0, dtype=dt, device="cuda")
        out = plane[1:M + 1, 8:N + 8]
        gemm_nt(a, b, out=out, swiglu=swiglu)
        first = out.clone()
        gemm_nt(a, b, out=out, swiglu=swiglu)
        torch.cuda.synchronize()
        assert torch.equal(first, out)
        edge = plane.clone()
        edge[1:M + 1, 8:N + 8] = 7.0
        assert bool((edge == 7.0).all())                        # nothing beside the output was written
        exact = a.double() @ b.double().t()
        if swiglu:
            gate, up = exact[:, :N], exact[:, N:]
            exact = F.silu(gate) * up
            # the fp32 sums' errors through silu (its slope is below 1.1), __expf and the fast divide: 2^-20
            e = K * 2.0 ** -23 * (a.abs().double() @ b.abs().double().t())
            bound = (exact.abs() * (2.0 ** -11 if dt == torch.float16 else 2.0 ** -8) * 1.01 + exact.abs() * 2.0 ** -18 +
                     1.1 * e[:, :N] * up.abs() + F.silu(gate).abs() * e[:, N:] + 2.0 ** -24)
        else:
            bound = _bound(a, b, exact, dt)
        assert bool(((out.double() - exact).abs() <= bound).all())


@pytest.mark.parametrize("M,N,K", [(8, 4096, 512), (64, 2048, 8192), (128, 8192, 1024)])
def test_few_rows_keep_infinities_to_their_rows(M, N, K):
    from tridist_b200.ops._gemm_common import gemm_nt
    dt = torch.bfloat16
    a, b = _rand((M, K), 3, dt), _rand((N, K), 4, dt)
    a[M // 2, K - 1] = float("inf")
    b[N - 3, 5] = float("nan")
    out = gemm_nt(a, b)
    torch.cuda.synchronize()
    exact = a.double() @ b.double().t()
    bad = ~torch.isfinite(exact)
    assert int(bad.sum()) == M + N - 1 and torch.equal(torch.isfinite(out), ~bad)
    assert torch.equal(torch.isnan(out), torch.isnan(exact))


def test_few_rows_on_streams_and_in_graphs():
    """Replays over other inputs, on two streams beside eager calls: the bits of the eager call."""
    from tridist_b200.ops._gemm_common import gemm_nt
    dt = torch.bfloat16
    for M, N, K in [(64, 4096, 1376), (128, 8192, 8192)]:
        b = _rand((N, K), 5, dt)
        a = [torch.zeros((M, K), dtype=dt, device="cuda") for _ in range(2)]
        outs = [torch.empty((M, N), dtype=dt, device="cuda") for _ in range(2)]
        gemm_nt(a[0], b)
        torch.cuda.synchronize()
        graphs, streams = [torch.cuda.CUDAGraph() for _ in range(2)], [torch.cuda.Stream() for _ in range(2)]
        for g, s, x, o in zip(graphs, streams, a, outs):
            with torch.cuda.graph(g, stream=s):
                gemm_nt(x, b, out=o)
                gemm_nt(x, b, out=o)
        for it in range(10):
            new = [_rand((M, K), 10 + 2 * it + i, dt) for i in range(2)]
            ref = [gemm_nt(x, b) for x in new]
            for x, y, o in zip(a, new, outs):
                x.copy_(y)
                o.zero_()
            torch.cuda.synchronize()
            for g, s in zip(graphs, streams):
                with torch.cuda.stream(s):
                    g.replay()
            between = gemm_nt(new[0], b)
            torch.cuda.synchronize()
            assert torch.equal(between, ref[0]) and all(torch.equal(o, r) for o, r in zip(outs, ref))


def test_few_rows_of_a_context_follow_the_kernel_in_front():
    """Each call reads what the call before it wrote, back to back."""
    from tridist_b200.ops import create_gemm_ar_intra_node_context, finalize_gemm_ar_context, gemm_ar_intra_node_op
    from tridist_b200.parallel.runtime import ProcessWorld
    w = ProcessWorld(0, 1)
    dt, M, N = torch.bfloat16, 64, 2048
    ctx = create_gemm_ar_intra_node_context(M, N, dt, dt, 0, 1, M_PER_CHUNK=64, world=w)
    x = [_rand((M, N), 6, dt), torch.empty((M, N), dtype=dt, device="cuda")]
    b = (_rand((N, N), 7, dt).float() * (10.0 / N ** 0.5)).to(dt)
    refs = [x[0].clone()]
    for _ in range(6):
        refs.append((refs[-1].double() @ b.double().t()).to(dt))
    for i in range(6):
        gemm_ar_intra_node_op(x[i & 1], b, x[~i & 1], ctx)
    torch.cuda.synchronize()
    w.check()
    err = (x[0].double() - refs[6].double()).norm() / refs[6].double().norm()
    assert err < 6 * 2.0 ** -8
    finalize_gemm_ar_context(ctx)


@pytest.mark.parametrize("M,N,K,swiglu,cluster", [
    (129, 8, 64, False, 1), (160, 264, 136, False, 1), (256, 6144, 592, False, 1), (192, 40000, 512, False, 1),
    (150, 4096, 4104, False, 2), (256, 11008, 4096, False, 2), (224, 1416, 4104, True, 2), (256, 8192, 28672, False, 4),
    (200, 48, 8200, False, 4), (193, 1664, 12288, False, 4), (130, 20000, 320, True, 1),
])
def test_two_blocks_of_rows(M, N, K, swiglu, cluster, monkeypatch):
    """129 to 256 rows, also where the plan would rather take the general kernel."""
    from tridist_b200.ops._gemm_common import gemm_nt
    from tridist_b200.parallel.runtime import native
    C = native()
    lay = C.skinny_layout(M, N, K, swiglu, 148)
    assert (lay["cluster"], lay["mb"]) == (cluster, 2)
    create = C.gemm_plan_create
    monkeypatch.setattr(C, "gemm_plan_create", lambda d: create(dict(d, few_rows=2)))
    for dt in (torch.float16, torch.bfloat16):
        a, b = _rand((M, K), 8, dt), _rand((2 * N if swiglu else N, K), 9, dt)
        plane = torch.full((M + 1, N + 8), 7.0, dtype=dt, device="cuda")
        out = plane[:M, :N]
        for _ in range(3):
            out.zero_()
            gemm_nt(a, b, out=out, swiglu=swiglu)
        torch.cuda.synchronize()
        assert bool((plane[M] == 7.0).all()) and bool((plane[:, N:] == 7.0).all())
        exact = a.double() @ b.double().t()
        bound = _bound(a, b, exact, dt)
        if swiglu:
            gate, up = exact[:, :N], exact[:, N:]
            exact = F.silu(gate) * up
            e = K * 2.0 ** -23 * (a.abs().double() @ b.abs().double().t())
            bound = (exact.abs() * (2.0 ** -11 if dt == torch.float16 else 2.0 ** -8) * 1.01 + exact.abs() * 2.0 ** -18 +
                     1.1 * e[:, :N] * up.abs() + F.silu(gate).abs() * e[:, N:] + 2.0 ** -24)
        assert bool(((out.double() - exact).abs() <= bound).all())


@pytest.mark.parametrize("M,N,K", [(64, 4096, 1376), (128, 8192, 28672), (64, 2048, 16384), (256, 11008, 4096)])
def test_few_rows_that_give_up_leave_the_context_usable(M, N, K):
    """With the abort word raised every role leaves the first wait that looks at it, whatever the others still have on
    their way: the call reports it or is complete, and the calls after it are right."""
    from tridist_b200.ops import create_gemm_ar_intra_node_context, finalize_gemm_ar_context, gemm_ar_intra_node_op
    from tridist_b200.parallel.runtime import ProcessWorld, native
    C, w, dt = native(), ProcessWorld(0, 1), torch.bfloat16
    ctx = create_gemm_ar_intra_node_context(M, N, dt, dt, 0, 1, M_PER_CHUNK=64, world=w)
    a, b = _rand((M, K), 11, dt), _rand((N, K), 12, dt)
    c = torch.empty((M, N), dtype=dt, device="cuda")
    gemm_ar_intra_node_op(a, b, c, ctx)
    torch.cuda.synchronize()
    w.check()
    ref = c.clone()
    exact = a.double() @ b.double().t()
    assert bool(((ref.double() - exact).abs() <= _bound(a, b, exact, dt)).all())
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


@pytest.mark.parametrize("M,N,K,swiglu", [
    (33, 1000, 15016, False), (64, 4096, 1384, False), (100, 48, 8200, False), (128, 4704, 7192, True), (96, 3128, 48024, False),
    (136, 2240, 12616, False), (200, 1256, 10024, True), (256, 520, 8008, False),
])
@pytest.mark.parametrize("few", [0, 1, 2])       # the general kernel, the rule's choice, the few-rows kernel
def test_rows_on_odd_multiples_of_16_bytes(M, N, K, swiglu, few, monkeypatch):
    from tridist_b200.ops import _gemm_common as common
    from tridist_b200.ops._gemm_common import gemm_nt
    from tridist_b200.parallel.runtime import native
    C, dt = native(), torch.bfloat16
    create, made = C.gemm_plan_create, []

    def record(d):
        d = dict(d, few_rows=few)
        made.append(C.gemm_choice(d, 148)["few_rows"])
        return create(d)

    monkeypatch.setattr(C, "gemm_plan_create", record)
    monkeypatch.setattr(common, "_plain_cache", common.PlanCache())      # (its key knows nothing of `few`)
    a, b = _rand((M, K), 8, dt), _rand((2 * N if swiglu else N, K), 9, dt)
    plane = torch.full((M + 1, N + 8), 7.0, dtype=dt, device="cuda")
    out = plane[:M, :N]
    gemm_nt(a, b, out=out, swiglu=swiglu)
    gemm_nt(a, b, out=out, swiglu=swiglu)
    torch.cuda.synchronize()
    assert few == 1 or made == [few == 2]
    assert bool((plane[M] == 7.0).all()) and bool((plane[:, N:] == 7.0).all())
    exact = a.double() @ b.double().t()
    bound = _bound(a, b, exact, dt)
    if swiglu:
        gate, up = exact[:, :N], exact[:, N:]
        exact = F.silu(gate) * up
        e = K * 2.0 ** -23 * (a.abs().double() @ b.abs().double().t())
        bound = (exact.abs() * 2.0 ** -8 * 1.01 + exact.abs() * 2.0 ** -18 + 1.1 * e[:, :N] * up.abs() +
                 F.silu(gate).abs() * e[:, N:] + 2.0 ** -24)
    assert bool(((out.double() - exact).abs() <= bound).all())

"""Repeated calls of one rank, launched natively: the same results, refusals and bookkeeping as first calls."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _world():
    import test_gpu_ops
    return test_gpu_ops._world1()


def _rand(shape, seed, dt=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * 0.1).to(dt)


def _close(out, a, b):
    exact = a.double() @ b.double().t()
    assert (out.double() - exact).norm() <= 2.0 ** -8 * exact.norm()


def test_repeats_and_their_refusals(monkeypatch):
    from tridist_b200.ops import (ag_gemm_intra_node_op, create_ag_gemm_intra_node_context,
                                  create_gemm_ar_intra_node_context, create_gemm_rs_intra_node_context,
                                  finalize_ag_gemm_context, finalize_gemm_ar_context, finalize_gemm_rs_context,
                                  gemm_ar_intra_node_op, gemm_rs_intra_node_op)
    w, dt, M, N, K = _world(), torch.bfloat16, 128, 512, 256
    a, b = _rand((M, K), 1), _rand((N, K), 2)
    c = torch.empty((M, N), dtype=dt, device="cuda")
    ar = create_gemm_ar_intra_node_context(M, N, dt, dt, 0, 1, M_PER_CHUNK=64, world=w)
    rs = create_gemm_rs_intra_node_context(M, N, dt, 0, 1, world=w)
    ag = create_ag_gemm_intra_node_context(M, K, dt, dt, 0, 1, M_PER_CHUNK=128, world=w)
    calls = [(ar, lambda x, y, z: gemm_ar_intra_node_op(x, y, z, ar)),
             (rs, lambda x, y, z: gemm_rs_intra_node_op(x, y, dt, 0, 1, rs, out=z)),
             (ag, lambda x, y, z: ag_gemm_intra_node_op(x, y, z, ag))]
    for ctx, call in calls:
        for i in range(4):
            a.copy_(_rand((M, K), 10 + i))
            c.zero_()
            assert call(a, b, c) is c
            _close(c, a, b)
        assert (ctx.plans.hits, ctx.plans.misses, ctx.plans.recent.hits) == (3, 1, 3)
        with pytest.raises(AssertionError):
            call(a[:, :128], b, c)                        # other K than b's
        with pytest.raises(AssertionError):
            call(a.to(torch.float16), b, c)
        if ctx is not ag:
            with pytest.raises(AssertionError):
                call(a[:100], b, c[:100])                 # rows not whole blocks
        wide = torch.zeros((M, N + 64), dtype=dt, device="cuda")
        call(a, b, wide[:, :N])                           # the same sizes, another row stride and address
        _close(wide[:, :N], a, b)
        monkeypatch.setenv("TRIDIST_FORCE_BN", "256")     # part of the cache's key
        misses = ctx.plans.misses
        call(a, b, c)
        assert ctx.plans.misses == misses + 1
        monkeypatch.delenv("TRIDIST_FORCE_BN")
        before = ctx.plans.recent.hits
        call(a, b, c)
        assert ctx.plans.recent.hits == before + 1
        _close(c, a, b)
    assert ag.flag_round == 7 and rs.round == 7           # rounds go on with every call
    # gate and up of one tensor, with and without the fused activation, are two calls
    h = torch.empty((M, N // 2), dtype=dt, device="cuda")
    for _ in range(2):
        ag_gemm_intra_node_op(a, b, h, ag, fuse_swiglu=True)
        exact = a.double() @ b.double().t()
        exact = torch.nn.functional.silu(exact[:, :N // 2]) * exact[:, N // 2:]
        assert (h.double() - exact).norm() <= 2.0 ** -7 * exact.norm()
    for ctx, fin in ((ar, finalize_gemm_ar_context), (rs, finalize_gemm_rs_context), (ag, finalize_ag_gemm_context)):
        fin(ctx)
        assert not ctx.plans.recent.launch(a, b, c, 0, 1)


def test_recency_of_native_hits_counts():
    """The plan that leaves a full cache is the least recently launched one, however it was launched."""
    from tridist_b200.ops import create_gemm_ar_intra_node_context, finalize_gemm_ar_context, gemm_ar_intra_node_op
    w, dt, M, N, K = _world(), torch.bfloat16, 64, 128, 128
    ctx = create_gemm_ar_intra_node_context(M, N, dt, dt, 0, 1, M_PER_CHUNK=64, world=w)
    ctx.plans.capacity = 2
    a, b = _rand((M, K), 1), _rand((N, K), 2)
    cs = [torch.empty((M, N), dtype=dt, device="cuda") for _ in range(3)]
    for i in (0, 1, 0, 0, 2, 0):             # 2 takes the place of 1
        gemm_ar_intra_node_op(a, b, cs[i], ctx)
    assert (ctx.plans.misses, ctx.plans.evictions, ctx.plans.recent.hits) == (3, 1, 3)
    gemm_ar_intra_node_op(a, b, cs[1], ctx)  # made anew
    assert ctx.plans.misses == 4
    torch.cuda.synchronize()
    for c in cs:
        _close(c, a, b)
    finalize_gemm_ar_context(ctx)


def test_moe_refusals():
    from tridist_b200.ops import (create_moe_a2a_intra_node_context, finalize_moe_a2a_context,
                                  moe_combine_intra_node_op, moe_dispatch_intra_node_op)
    w, dt, T, E, H, topk = _world(), torch.bfloat16, 32, 8, 256, 2
    ctx = create_moe_a2a_intra_node_context(E, H, dt, T, topk, 0, 1, BLOCK_H=H, world=w)
    tokens = _rand((T, H), 1)
    idx = torch.randint(0, E, (T, topk), device="cuda", dtype=torch.int32)
    out, wts = torch.empty_like(tokens), torch.rand((T, topk), device="cuda")
    moe_dispatch_intra_node_op(tokens, idx, ctx)
    rounds = ctx.meta_round
    for bad in [(tokens.half(), idx), (tokens[:, :128], idx), (tokens, idx.long()), (tokens, idx[:, :1]), (tokens[:8], idx),
                (torch.cat([tokens, tokens]), torch.cat([idx, idx])), (tokens.t().contiguous().t(), idx),
                (tokens, idx.t().contiguous().t())]:
        with pytest.raises(AssertionError):
            moe_dispatch_intra_node_op(*bad, ctx)
    assert ctx.meta_round == rounds
    ctx.out[:] = ctx.recv
    for bad in [(idx, out[:8], wts), (idx, out[:, :128], wts), (idx, out, wts.double()), (idx, out, wts.t().contiguous().t()),
                (idx, out.t().contiguous().t(), wts)]:
        with pytest.raises(AssertionError):
            moe_combine_intra_node_op(ctx, *bad)
    moe_combine_intra_node_op(ctx, idx, out, wts)
    exact = tokens.double() * wts.double().sum(1, keepdim=True)
    assert (out.double() - exact).norm() <= 2.0 ** -8 * exact.norm()
    finalize_moe_a2a_context(ctx)


def test_width_forced_where_the_free_choice_starts_from_it(monkeypatch):
    """A forced width of 256 and a free choice that has 256 in its key are two plans, natively remembered or not."""
    from tridist_b200.ops import ag_gemm_intra_node_op, create_ag_gemm_intra_node_context, finalize_ag_gemm_context
    w, dt, M, N, K = _world(), torch.bfloat16, 128, 4096, 512
    ag = create_ag_gemm_intra_node_context(M, K, dt, dt, 0, 1, M_PER_CHUNK=128, world=w)
    a, b = _rand((M, K), 1), _rand((N, K), 2)
    h = torch.empty((M, N // 2), dtype=dt, device="cuda")
    exact = a.double() @ b.double().t()
    exact = torch.nn.functional.silu(exact[:, :N // 2]) * exact[:, N // 2:]
    for i in range(3):
        for forced in (False, True):
            if forced:
                monkeypatch.setenv("TRIDIST_FORCE_BN", "256")
            else:
                monkeypatch.delenv("TRIDIST_FORCE_BN", raising=False)
            h.zero_()
            ag_gemm_intra_node_op(a, b, h, ag, fuse_swiglu=True)
            assert (h.double() - exact).norm() <= 2.0 ** -7 * exact.norm()
    assert (ag.plans.misses, ag.plans.hits, ag.plans.recent.hits) == (2, 4, 2)
    finalize_ag_gemm_context(ag)


def test_moe_combine_refusals():
    """What the combine kernels would read past the end of, or write in another type; and forms that stay accepted."""
    from tridist_b200.ops import (create_moe_a2a_intra_node_context, finalize_moe_a2a_context,
                                  moe_combine_intra_node_op, moe_dispatch_intra_node_op)
    w, dt, T, E, H, topk = _world(), torch.bfloat16, 32, 8, 256, 2
    ctx = create_moe_a2a_intra_node_context(E, H, dt, T, topk, 0, 1, BLOCK_H=H, world=w)
    tokens = _rand((T, H), 1)
    idx = torch.randint(0, E, (T, topk), device="cuda", dtype=torch.int32)
    out, wts = torch.empty_like(tokens), torch.rand((T, topk), device="cuda")
    for bad in [(tokens.cpu(), idx), (tokens, idx.cpu())]:
        with pytest.raises(AssertionError):
            moe_dispatch_intra_node_op(*bad, ctx)
    moe_dispatch_intra_node_op(tokens, idx, ctx)
    ctx.out[:] = ctx.recv
    two = torch.cat([idx, idx])
    for bad in [(idx.long(), out, wts), (idx[:, :1].contiguous(), out, wts), (idx[:1, :1].expand(T, topk), out, wts),
                (idx.t().contiguous().t(), out, wts), (two, torch.cat([out, out]), None), (idx, out, wts[:, :1].contiguous()),
                (idx, out, wts[:8]), (idx, out.float(), wts), (idx, out.half(), wts), (idx.cpu(), out, wts),
                (idx, out.cpu(), wts), (idx, out, wts.cpu())]:
        with pytest.raises(AssertionError):
            moe_combine_intra_node_op(ctx, *bad)
    exact = tokens.double() * wts.double().sum(1, keepdim=True)
    for good in [(idx, out, wts), (idx, out, wts.flatten()), (idx.unsqueeze(-1), out, wts), (idx.cpu().pin_memory(), out, wts)]:
        out.zero_()
        moe_combine_intra_node_op(ctx, *good)
        assert (out.double() - exact).norm() <= 2.0 ** -8 * exact.norm()
    moe_dispatch_intra_node_op(tokens.cpu().pin_memory(), idx, ctx)
    torch.cuda.synchronize()
    w.check()
    assert torch.equal(ctx.recv[ctx.scatter_idx.flatten().long()], tokens.repeat_interleave(topk, 0))
    finalize_moe_a2a_context(ctx)

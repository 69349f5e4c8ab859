"""Metadata and dispatch of a small batch in one kernel, at the edges of the rule that picks it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,H,topk", [
    (1, 1024, 8, 32),                        # one piece a row, most experts and rows per token
    (147, 3, 4104, 1), (149, 300, 2056, 6),
    (128, 1024, 64, 32), (512, 64, 4096, 8), (2048, 16, 512, 2),       # 4096 pairs: the last in one kernel
    (513, 64, 512, 8), (2049, 16, 512, 1),   # one more: two kernels
])
def test_small_rounds(T, E, H, topk):
    import test_gpu_ops
    test_gpu_ops.test_moe_round_of_any_size(T, E, H, topk, torch.bfloat16)


@pytest.mark.parametrize("T", [24, 600])      # one kernel, two kernels
def test_repeated_experts_and_rows_past_the_end(T):
    """An expert that a token names twice gets two rows; rows past the receive buffer are dropped and reported."""
    import test_gpu_ops
    from tridist_b200.ops import (create_moe_a2a_intra_node_context, finalize_moe_a2a_context,
                                  moe_dispatch_intra_node_op)
    from tridist_b200.parallel.runtime import TriDistError
    w = test_gpu_ops._world1()
    E, H, topk, dt = 16, 256, 8, torch.float16
    g = torch.Generator(device="cuda").manual_seed(1)
    tokens = torch.randn((T, H), generator=g, device="cuda").to(dt)
    idx = torch.randint(0, E, (T, topk), generator=g, device="cuda", dtype=torch.int32)
    for rows in (T * topk, T * topk - 40):
        ctx = create_moe_a2a_intra_node_context(E, H, dt, T, topk, 0, 1, BLOCK_H=H, world=w, max_recv_rows=rows)
        total = moe_dispatch_intra_node_op(tokens, idx, ctx)
        torch.cuda.synchronize()
        sc = ctx.scatter_idx.flatten().long()
        assert int(total.item()) == T * topk and int((sc < 0).sum()) == T * topk - rows
        kept = sc >= 0
        assert torch.equal(sc[kept].sort().values, torch.arange(rows, device="cuda"))
        of = torch.arange(T, device="cuda").repeat_interleave(topk)
        assert torch.equal(ctx.recv[sc[kept]], tokens[of[kept]])
        first, e = ctx.recv_seg.flatten().long(), idx.flatten().long()
        assert bool((sc[kept] >= first[e[kept]]).all())
        assert torch.equal(ctx.splits.long(), torch.bincount(e, minlength=E))
        if rows < T * topk:
            with pytest.raises(TriDistError):
                w.check()
            w.clear_status()
        else:
            w.check()
        finalize_moe_a2a_context(ctx)


@pytest.mark.parametrize("T", [24, 64, 400])
def test_tokens_written_by_the_kernel_in_front(T):
    """A GEMM, or the combine of the round before, writes the tokens right in front of a small dispatch, over inputs
    that change from round to round in the same buffers."""
    import test_gpu_ops
    from tridist_b200.ops import (create_moe_a2a_intra_node_context, finalize_moe_a2a_context,
                                  moe_combine_intra_node_op, moe_dispatch_intra_node_op)
    from tridist_b200.ops._gemm_common import gemm_nt
    w = test_gpu_ops._world1()
    E, H, topk, K, dt = 16, 4096, 4, 512, torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(T)
    ctx = create_moe_a2a_intra_node_context(E, H, dt, T, topk, 0, 1, BLOCK_H=H, world=w)
    b = (torch.randn((H, K), generator=g, device="cuda") * 0.05).to(dt)
    tokens = torch.empty((T, H), dtype=dt, device="cuda")
    of = torch.arange(T, device="cuda").repeat_interleave(topk)
    for _ in range(8):
        x = torch.randn((T, K), generator=g, device="cuda").to(dt)
        idx = torch.randint(0, E, (T, topk), generator=g, device="cuda", dtype=torch.int32)
        gemm_nt(x, b, out=tokens)
        moe_dispatch_intra_node_op(tokens, idx, ctx)
        sc = ctx.scatter_idx.flatten().long()
        got = ctx.recv[sc]
        assert torch.equal(got, tokens[of])
        ctx.out[sc] = got + 1
        idx2 = torch.randint(0, E, (T, topk), generator=g, device="cuda", dtype=torch.int32)
        moe_combine_intra_node_op(ctx, idx, tokens)
        moe_dispatch_intra_node_op(tokens, idx2, ctx)
        assert torch.equal(ctx.recv[ctx.scatter_idx.flatten().long()], tokens[of])
    w.check()
    finalize_moe_a2a_context(ctx)


def test_combine_that_gives_up_leaves_the_context_usable():
    """With the abort word raised the ring's warps leave the first wait that looks at it, whatever copies are on their
    way: the call reports it or is complete, and the rounds after it are right."""
    from tridist_b200.ops import (create_moe_a2a_intra_node_context, finalize_moe_a2a_context,
                                  moe_combine_intra_node_op, moe_dispatch_intra_node_op)
    from tridist_b200.parallel.runtime import ProcessWorld, native
    C, w = native(), ProcessWorld(0, 1)
    T, E, H, topk, dt = 2048, 16, 4096, 8, torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(3)
    tokens = torch.randn((T, H), generator=g, device="cuda").to(dt)
    idx = torch.randint(0, E, (T, topk), generator=g, device="cuda", dtype=torch.int32)
    ctx = create_moe_a2a_intra_node_context(E, H, dt, T, topk, 0, 1, BLOCK_H=H, world=w)
    out = torch.empty_like(tokens)
    for _ in range(5):
        moe_dispatch_intra_node_op(tokens, idx, ctx)
        ctx.out.copy_(ctx.recv)
        out.zero_()
        C.fill_u32(w.abort_word, 1, 5)
        moe_combine_intra_node_op(ctx, idx, out)
        torch.cuda.synchronize()
        assert w.status()[0] == 5 or torch.equal(out, tokens * topk)
        w.clear_status()
        moe_combine_intra_node_op(ctx, idx, out)
        torch.cuda.synchronize()
        w.check()
        assert torch.equal(out, tokens * topk)       # eight times a 16-bit number is exact
    finalize_moe_a2a_context(ctx)

"""What the native MoE calls refuse before anything is launched: addresses that the kernels could not follow, and fewer
elements behind them than the kernels read."""
import pytest
import torch

T, E, H, TOPK = 8, 4, 16, 2


def _handle():
    from tridist_b200.parallel.runtime import native
    d = dict(rank=0, R=1, E=E, H=H, topk=TOPK, max_recv_rows=T * TOPK, bf16=True)
    return native().MoeHandle(d, d, T)


def _dispatch(tokens=None, idx=None):
    tokens = torch.zeros((T, H), dtype=torch.bfloat16) if tokens is None else tokens
    idx = torch.zeros((T, TOPK), dtype=torch.int32) if idx is None else idx
    return _handle().dispatch(1, 1, tokens, idx, True)


def _combine(idx=None, weights=None, out=None):
    idx = torch.zeros((T, TOPK), dtype=torch.int32) if idx is None else idx
    out = torch.zeros((T, H), dtype=torch.bfloat16) if out is None else out
    return _handle().combine(1, 1, idx, weights, out)


def test_host_memory_never_reaches_a_kernel():
    """(Without a device the launch behind a check that lets them pass raises.)"""
    assert not _dispatch()
    assert not _combine() and not _combine(weights=torch.ones((T, TOPK)))


@pytest.mark.parametrize("bad", [
    dict(idx=torch.zeros((T, TOPK), dtype=torch.int64)),
    dict(idx=torch.zeros((T, TOPK - 1), dtype=torch.int32)),                        # read past its end
    dict(idx=torch.zeros((1, 1), dtype=torch.int32).expand(T, TOPK)),               # one element behind T * topk
    dict(idx=torch.zeros((2 * T, TOPK), dtype=torch.int32), out=torch.zeros((2 * T, H), dtype=torch.bfloat16)),
    dict(weights=torch.ones((T, TOPK - 1))),
    dict(weights=torch.ones((T - 1, TOPK))),
    dict(out=torch.zeros((T, H), dtype=torch.float32)),
    dict(out=torch.zeros((T, H), dtype=torch.float16)),
])
def test_combine_refuses(bad):
    from types import SimpleNamespace
    from tridist_b200.ops import moe_a2a
    assert not _combine(**bad)
    full = dict(idx=torch.zeros((T, TOPK), dtype=torch.int32), weights=None, out=torch.zeros((T, H), dtype=torch.bfloat16))
    full.update(bad)
    ctx = SimpleNamespace(max_tokens=T, topk=TOPK, hidden=H, input_dtype=torch.bfloat16)
    with pytest.MonkeyPatch.context() as mp:
        mp.setattr(moe_a2a, "_on_device", lambda t: True)       # the other checks, on host tensors
        with pytest.raises(AssertionError):
            moe_a2a._check_combine(ctx, full["idx"], full["out"], full["weights"])
        good = torch.zeros((T, TOPK), dtype=torch.int32)
        moe_a2a._check_combine(ctx, good, torch.zeros((T, H), dtype=torch.bfloat16), torch.ones(T * TOPK))

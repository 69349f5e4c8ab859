"""Repair of the tiles that a verification flags, for few rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_repair_touches_the_flagged_tiles_only():
    import test_gpu_ops
    from tridist_b200.ops import create_i1_context, i1_ag_tr_op, i1_table_write
    from tridist_b200.ops.ag_tr_pred import _verify_and_repair
    w, dt, M, K, N = test_gpu_ops._world1(), torch.bfloat16, 128, 256, 4096
    g = torch.Generator(device="cuda").manual_seed(5)
    a, b = [(torch.randn((n, K), generator=g, device="cuda") * 0.1).to(dt) for n in (M, N)]
    c = torch.empty((M, N), dtype=dt, device="cuda")
    ictx = create_i1_context(M, K, dt, dt, 0, 1, world=w)
    i1_table_write(ictx, 1, 0, 1, 0, 1)
    i1_ag_tr_op(a, b, c, ictx)
    torch.cuda.synchronize()
    exact = a.double() @ b.double().t()
    assert (c.double() - exact).norm() <= 2.0 ** -8 * exact.norm()
    c[5, 100] += 2.0 ** -7 * c[5, 100].abs()              # a digit that no tolerance sees, in a healthy tile
    good = c.clone()
    c[:, 2048:2304] = 0
    assert 1 <= _verify_and_repair(a, b, c, ictx) <= 2
    torch.cuda.synchronize()
    w.check()
    assert torch.equal(c[:, :2048], good[:, :2048]) and torch.equal(c[:, 2304:], good[:, 2304:])
    assert (c.double() - exact).norm() <= 2.0 ** -8 * exact.norm()

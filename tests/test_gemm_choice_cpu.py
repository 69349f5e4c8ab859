"""Which kernel and tile a descriptor gets, worked out on the host."""
import pytest


def _choice(**kw):
    from tridist_b200.ops._gemm_common import OP_PLAIN, SCHED_NATURAL
    from tridist_b200.parallel.runtime import native
    d = dict(op=OP_PLAIN, sched=SCHED_NATURAL, bn=256, R=1, rank=0, by_rounds=1, fit_tile=1, few_rows=1)
    d.update(kw)
    return native().gemm_choice(d, 148)


@pytest.mark.parametrize("M", [1, 64, 128, 192, 256])
def test_tile_list_stays_with_the_kernel_that_knows_it(M):
    """The few-rows kernel stores every tile; a repair names those that it may touch."""
    from tridist_b200.ops._gemm_common import SCHED_LIST
    kw = dict(M=M, N=4096, K=1376)
    assert _choice(**kw)["few_rows"]
    assert not _choice(sched=SCHED_LIST, list_len=1, **kw)["few_rows"]

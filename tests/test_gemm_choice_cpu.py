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


@pytest.mark.parametrize("K", [64, 1376, 3584, 3840, 4096])
def test_panels_of_several_ranks_keep_their_ring(K):
    """Local tiles of a short K leave through the staging area; the panel GEMMs of an exchange (``local=False``), whose
    width and height are given, keep the stage of the ring that it takes."""
    kw = dict(M=2048, N=8192, K=K, allow_wide=0)
    panel = _choice(fit_tile=0, few_rows=0, by_rounds=0, early_start=0, **kw)
    assert (panel["bn"], panel["cta_m"], panel["row_blocks"], panel["staging"]) == (256, 2, 1, False)
    own = _choice(**kw)
    assert own["staging"] == (own["cta_m"] == 2 and K <= 59 * 64)


def test_ranks_that_ship_tiles_have_the_staging_area():
    from tridist_b200.ops._gemm_common import OP_AG, OP_AR1, OP_AR2, OP_PLAIN, OP_RS
    for op in (OP_AG, OP_RS, OP_AR1, OP_AR2, OP_PLAIN):
        assert _choice(op=op, R=2, M=2048, N=8192, K=4096, fit_tile=0, few_rows=0, by_rounds=0)["staging"] == (op != OP_PLAIN)


def test_given_width_of_a_local_launch():
    kw = dict(M=2048, N=8192, allow_wide=0, fit_tile=0, few_rows=0)
    assert _choice(K=3584, **kw)["staging"] and not _choice(K=4096, **kw)["staging"]

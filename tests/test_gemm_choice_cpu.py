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


@pytest.mark.parametrize("M,N,K,swiglu,few", [
    (64, 10008, 20008, 0, False), (128, 3400, 21752, 1, False), (96, 4704, 14392, 1, False), (128, 20160, 24784, 1, False),
    (16, 10008, 20008, 0, True), (64, 4096, 1376, 0, True), (96, 5352, 14576, 0, True), (128, 8192, 28672, 0, True),
    (64, 712, 8680, 1, True), (128, 512, 22576, 1, True), (128, 2656, 37568, 1, True),
    (256, 2736, 5720, 1, False), (192, 2240, 12616, 0, False),
])
def test_few_rows_by_the_alignment_of_the_rows(M, N, K, swiglu, few):
    """At shapes whose times were measured; the general kernel then keeps the tile that it is given."""
    from tridist_b200.ops._gemm_common import choose_bn
    bn = choose_bn(M, N, bool(swiglu), K=K, local=True)
    got = _choice(M=M, N=N, K=K, epi=swiglu, bn=bn)
    assert got["few_rows"] == few
    if not few:
        assert got["bn"] == bn and got["cta_m"] == (2 if M > 128 and bn == 256 else 1)


@pytest.mark.parametrize("part", ["a", "b", "lda", "ldb"])
def test_alignment_is_that_of_addresses_and_strides(part):
    kw = dict(M=64, N=10008, K=20032, a=1 << 20, b=1 << 30, lda=20032, ldb=20032)
    assert _choice(**kw)["few_rows"]
    kw[part] += 16 if part in "ab" else 8
    assert not _choice(**kw)["few_rows"]


def test_sizes_that_a_plan_refuses_are_not_laid_out():
    for kw in (dict(M=64, N=0, K=64), dict(M=0, N=64, K=64), dict(M=64, N=64, K=0), dict(M=64, N=4, K=64)):
        assert not _choice(**kw)["few_rows"]


def test_stall_accounting_does_not_change_the_kernel():
    """What is timed beside the accounting is the kernel of other runs."""
    for M in (16, 128, 192):
        kw = dict(M=M, N=4096, K=1376)
        assert _choice(prof=4096, **kw) == _choice(**kw) and _choice(**kw)["few_rows"]


def test_a_plane_that_no_kernel_wrote_gives_no_accounting(monkeypatch):
    import torch
    from tridist_b200.ops import _gemm_common as common
    plane = torch.zeros((256, common.PROF_WIDTH), dtype=torch.int64)
    monkeypatch.setattr(common, "_prof_buf", plane)
    assert common.read_prof() == {}
    plane[3, 9] = 5000
    assert common.read_prof()["kernel"]["max"] == 5.0

"""Layout of the few-rows GEMM (csrc/gemm/skinny_gemm.cuh), worked out on the host: every column once, and what the
kernel will read and write inside the memory that it is given."""
import random

import pytest


@pytest.mark.parametrize("seed", range(4))
def test_layout_holds_for_every_shape(seed):
    from tridist_b200.parallel.runtime import native
    rnd = random.Random(seed)
    shapes = [(1, 8, 8, 0), (128, 8, 64, 1), (64, 4096, 1376, 0), (65, 8192, 3584, 0), (128, 3584, 8192, 1), (128, 106496, 16384, 0)]
    shapes += [(129, 8, 64, 0), (256, 12288, 24576, 0), (200, 53248, 16384, 1), (192, 16384, 8192, 1)]
    shapes += [(rnd.randint(1, 256), 8 * rnd.randint(1, rnd.choice([4, 300, 2400, 14000])), 8 * rnd.randint(1, rnd.choice([20, 4000])),
                rnd.randint(0, 1)) for _ in range(150)]
    for M, N, K, swiglu in shapes:
        p = native().skinny_layout(M, N, K, bool(swiglu), 148)
        what = (M, N, K, swiglu, p)
        cl = p["cluster"]
        assert cl in (1, 2, 4) and (cl == 1 or p["workers"] == p["shares"]) and p["workers"] * cl <= 148 and p["workers"] <= p["shares"], what
        # columns: runs of groups that follow one another, none larger than the boxes that hold it
        assert p["share"][0][0] == 0 and p["share"][-1][1] * 8 == N, what
        assert all(a[1] == b[0] for a, b in zip(p["share"], p["share"][1:])), what
        assert all(0 < 8 * (hi - lo) <= p["wr"] and -(-(hi - lo) // cl) <= p["own"] for lo, hi in p["share"]), what
        # every CTA of a cluster has a range of K of one stage at least
        assert p["ranges"][0] == 0 and p["ranges"][cl] == p["k_blocks"], what
        ranges = [p["ranges"][r + 1] - p["ranges"][r] for r in range(cl)]
        assert min(ranges) >= 1, what
        # shared memory: whole swizzle groups, A's 128 rows of the last k-block inside the pad, TMA's limits
        assert p["wr"] % 8 == 0 and p["wr"] <= p["nb"] and p["nb"] % 16 == 0 and p["wr"] <= 256, what
        assert p["ar"] % 8 == 0 and M <= p["ar"] <= 256 and 32 * p["warps"] >= M and p["mb"] == -(-M // 128), what
        block = (p["ar"] + p["nb"] * p["boxes"]) * 128
        assert p["kw"] in (1, 2, 4, 8) and p["stage_bytes"] == p["kw"] * block and block % 1024 == 0, what
        ring = p["stages"] * p["stage_bytes"]
        assert 1 <= p["stages"] <= 16, what
        assert (p["kw"] - 1) * p["ar"] * 128 + p["mb"] * 128 * 128 <= p["stage_bytes"] + p["pad"], what
        xbuf = (cl - 1) * p["boxes"] * p["own"] * 2 * 32 * p["warps"] * 16
        assert (max(ring + p["pad"], xbuf) if p["in_ring"] else ring + p["pad"] + xbuf) <= p["smem_bytes"] <= 225 * 1024, what
        # tensor memory and the MMA's shape
        bufs = 2 if p["shares"] > p["workers"] else 1
        assert p["mma_n"] % 16 == 0 and 16 <= p["mma_n"] <= 256 and p["acc_cols"] >= p["mma_n"], what
        assert p["mb"] * bufs * p["accs"] * p["acc_cols"] <= p["tmem_cols"] <= 512 and p["tmem_cols"] & (p["tmem_cols"] - 1) == 0, what
        assert 1 <= p["accs"] <= max(1, min(ranges) // 16), what
        assert p["accs"] <= -(-min(ranges) // p["kw"]), what


@pytest.mark.parametrize("instead", [dict(shares=140), dict(k_blocks=200), dict(wr=8), dict(ar=64), dict(own=0), dict(stages=17),
                                     dict(pad=-20000), dict(smem_bytes=4096), dict(smem_bytes=226 * 1024), dict(tmem_cols=32)])
def test_checked_mode_names_what_a_layout_would_miss(instead):
    """TRIDIST_DEBUG=1 looks at the layout that runs, as well as at the schedule of the calls that it does not take."""
    from tridist_b200.parallel.runtime import native
    C, shape = native(), (128, 4096, 12288, False)
    assert C.skinny_check(*shape, {}) == []
    bad = C.skinny_check(*shape, instead)
    assert bad and all(s.startswith("few-rows layout: ") for s in bad), bad


def test_checked_mode_passes_what_plans_make():
    from tridist_b200.ops._gemm_common import OP_PLAIN, SCHED_NATURAL
    from tridist_b200.parallel.runtime import native
    rnd = random.Random(9)
    for _ in range(200):
        M, N, K = rnd.randint(1, 256), 8 * rnd.randint(1, rnd.choice([4, 300, 2400])), 8 * rnd.randint(1, rnd.choice([20, 4000]))
        d = dict(op=OP_PLAIN, sched=SCHED_NATURAL, bn=256, R=1, rank=0, M=M, N=N, K=K, ldc=N, epi=rnd.randint(0, 1), few_rows=2,
                 fit_tile=1, by_rounds=1)
        assert native().gemm_choice(d, 148)["few_rows"]
        assert native().plan_check(d, dict(c_bytes=M * N * 2), 148) == [], d
        assert native().plan_check(d, dict(c_bytes=M * N * 2 - 2), 148) != [], d

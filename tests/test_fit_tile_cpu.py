"""The tile that a local launch picks by the time expected of it (fit_tile), replayed on the host."""
import itertools
import random

import pytest


def _dump(**kw):
    from tridist_b200.ops._gemm_common import OP_PLAIN, SCHED_NATURAL
    from tridist_b200.parallel.runtime import native
    d = dict(op=OP_PLAIN, sched=SCHED_NATURAL, bn=256, R=1, rank=0, by_rounds=1, fit_tile=1)
    d.update(kw)
    return native().schedule_dump(d, 148), native().plan_check(dict(d, ldc=d["N"]), dict(c_bytes=d["M"] * d["N"] * 2), 148)


@pytest.mark.parametrize("M,N,K,width,blocks", [
    (384, 3328, 1584, 128, 1), (320, 28672, 8192, 256, 1), (2112, 22016, 4096, 256, 2), (1728, 12288, 12288, 256, 2),
    (8192, 6144, 12288, 256, 4), (1024, 8192, 28672, 256, 4),
])
def test_choice(M, N, K, width, blocks):
    """At the shapes whose times stand at the rule."""
    out, bad = _dump(M=M, N=N, K=K)
    assert bad == []
    tiles = [(t[0], t[1]) for cta in out for t in cta if t[0] * 128 < M]
    assert sorted(tiles) == list(itertools.product(range(-(-M // 128)), range(-(-N // width))))
    pair = [(a[0][0] + max(1, blocks // 2), a[0][1]) == (b[0][0], b[0][1]) for a, b in zip(out[0::2], out[1::2])]
    assert (blocks > 1) == all(pair)
    wide = [a[0] + 1 == b[0] and a[1] == b[1] for cta in out for a, b in zip(cta[0::2], cta[1::2])]
    assert (blocks == 4) == (bool(wide) and all(wide))


def test_every_tile_once():
    rnd = random.Random(11)
    for _ in range(200):
        M, N = rnd.randint(1, 70) * 64, 8 * rnd.randint(1, 2000)
        K = 8 * rnd.randint(1, 3000)
        kw = dict(M=M, N=N, K=K, epi=rnd.randint(0, 1), allow_pair=rnd.randint(0, 3) > 0, allow_wide=rnd.randint(0, 1),
                  allow_splitk=rnd.randint(0, 3) > 0)
        kw = {k: int(v) for k, v in kw.items()}
        out, bad = _dump(**kw)
        assert bad == [] and len(out) <= 148, (kw, bad)


@pytest.mark.parametrize("M,N,K,epi,bn,cta_m,row_blocks", [
    (3589, 26240, 64, 0, 256, 2, 1), (1000, 12736, 800, 0, 256, 2, 1), (520, 24256, 608, 0, 256, 2, 1),
    (1184, 17856, 80, 0, 256, 2, 1), (2312, 12304, 112, 1, 256, 1, 1), (1020, 3616, 336, 1, 256, 1, 1),
])
def test_choice_where_the_epilogue_is_longer_than_the_product(M, N, K, epi, bn, cta_m, row_blocks):
    from tridist_b200.ops._gemm_common import OP_PLAIN, SCHED_NATURAL
    from tridist_b200.parallel.runtime import native
    got = native().gemm_choice(dict(op=OP_PLAIN, sched=SCHED_NATURAL, bn=256, R=1, rank=0, by_rounds=1, fit_tile=1, M=M, N=N,
                                    K=K, epi=epi), 148)
    assert (got["bn"], got["cta_m"], got["row_blocks"]) == (bn, cta_m, row_blocks)

"""A cached plan is found only by a call that would make the same plan: the width that the environment forces is part
of every key, also where the unforced call has the same width but may pick its tile (or, for few rows, its kernel) itself."""
from types import SimpleNamespace

import pytest
import torch

OPS = ("ag", "ag_swiglu", "rs", "ar", "plain", "plain_swiglu")


class _Native:
    """Plans are numbered and their descriptors kept; nothing is launched."""

    def __init__(self):
        from tridist_b200.parallel.runtime import native
        self.descs = {}
        self.launched = []
        self.settings = native().settings

    def gemm_plan_create(self, d):
        self.descs[len(self.descs) + 1] = d
        return len(self.descs)

    def gemm_plan_launch(self, pid, *args):
        self.launched.append(pid)

    class RecentCalls:
        hits = 0

        def launch(self, *args):
            return False

        def remember(self, *args):
            pass

        def drain(self):
            return []


class _Operand:
    """What the host code asks of a row-major matrix on the device."""

    is_cuda, dtype, device = True, torch.bfloat16, "cuda"

    def __init__(self, address, rows, cols):
        self._address, self.shape = address, (rows, cols)

    def data_ptr(self):
        return self._address

    def stride(self, i):
        return (self.shape[1], 1)[i]

    def storage_offset(self):
        return 0

    def element_size(self):
        return 2

    def untyped_storage(self):
        return SimpleNamespace(nbytes=lambda: 2 * self.shape[0] * self.shape[1])


def _caller(op, M, N, K, fake, monkeypatch):
    from tridist_b200.ops import _gemm_common as common
    from tridist_b200.ops import all_gather_gemm as ag, gemm_allreduce as ar, gemm_reduce_scatter as rs
    for module in (common, ag, ar, rs):
        monkeypatch.setattr(module, "native", lambda: fake)
    world = SimpleNamespace(kind="process", num_ranks=1, status_dev=0, abort_word=0, timeout_ns=1)
    swiglu = op.endswith("swiglu")
    a, b, c = _Operand(1 << 20, M, K), _Operand(2 << 20, N, K), _Operand(3 << 20, M, N // 2 if swiglu else N)
    ctx = SimpleNamespace(num_ranks=1, rank=0, world=world, K=K, N=N, max_M=M, M_PER_CHUNK=64, input_dtype=a.dtype,
                          output_dtype=a.dtype, flag_round=0, round=0, plans=common.PlanCache(), order_override=None,
                          observe=False, transport="push", push_ctas=-1, mode=None, mc=None, reduce_ctas=0, reduce_tail=0)
    if op.startswith("plain"):
        monkeypatch.setattr(common, "plain_world", lambda: world)
        monkeypatch.setattr(common, "_plain_cache", common.PlanCache())
        return lambda: common.gemm_nt(a, b, out=c, swiglu=swiglu)
    if op.startswith("ag"):
        return lambda: ag.ag_gemm_intra_node_op(a, b, c, ctx, fuse_swiglu=swiglu)
    if op == "rs":
        return lambda: rs.gemm_rs_intra_node_op(a, b, a.dtype, 0, 1, ctx, out=c)
    return lambda: ar.gemm_ar_intra_node_op(a, b, c, ctx)


@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("M,N,K", [(128, 8192, 8192), (2048, 8192, 4096)])       # widths of 256 either way
@pytest.mark.parametrize("first", [None, "256"])
def test_forced_width_is_part_of_the_key(op, M, N, K, first, monkeypatch):
    for name in ("TRIDIST_MAX_CTAS", "TRIDIST_FORCE_BN"):
        monkeypatch.delenv(name, raising=False)
    fake = _Native()
    call = _caller(op, M, N, K, fake, monkeypatch)

    def force(width):
        if width is None:
            monkeypatch.delenv("TRIDIST_FORCE_BN", raising=False)
        else:
            monkeypatch.setenv("TRIDIST_FORCE_BN", width)

    other = "256" if first is None else None
    for width in (first, other, first, other):
        force(width)
        call()
        d = fake.descs[fake.launched[-1]]
        assert d["bn"] == 256
        assert (d["fit_tile"], d["few_rows"]) == ((1, int(M <= 256)) if width is None else (0, 0)), (width, fake.launched)
    assert fake.launched == [1, 2, 1, 2]


@pytest.mark.parametrize("op", OPS)
def test_one_look_at_the_environment_a_call(op, monkeypatch):
    """A first call on new operands pays for every look-up."""
    import os
    from tridist_b200.ops import _gemm_common as common
    fake = _Native()
    looks = []
    settings = fake.settings
    fake.settings = lambda: looks.append(1) or settings()
    call = _caller(op, 256, 4096, 1024, fake, monkeypatch)
    asked = []
    get = os.environ.get
    monkeypatch.setattr(common, "env_int", lambda n, d: asked.append(n) or int(get(n) or d))
    call()
    assert looks == [1] and asked == []


def test_settings_are_those_of_the_process(monkeypatch):
    from tridist_b200.ops import _gemm_common as common
    from tridist_b200.parallel.runtime import native
    for name in list(native().settings()):
        monkeypatch.delenv(name)
    assert native().settings() == {} and common.plan_env() == common._PLAN_ENV
    monkeypatch.setenv("TRIDIST_SPLITK", "0")
    monkeypatch.setenv("TRIDIST_FORCE_BN", "")           # empty: the default
    monkeypatch.setenv("TRIDIST_VERIFY_TOL", "2e-2")     # not a plan's
    assert native().settings() == {"TRIDIST_SPLITK": "0", "TRIDIST_FORCE_BN": "", "TRIDIST_VERIFY_TOL": "2e-2"}
    assert common.plan_env() == {**common._PLAN_ENV, "TRIDIST_SPLITK": 0}
    monkeypatch.setenv("TRIDIST_FORCE_BN", "wide")
    with pytest.raises(ValueError):
        common.plan_env()

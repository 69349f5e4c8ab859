"""Single-GPU tests of the sm_100a kernels.

Numerics are compared against a plain fp32 PyTorch reference of the same op.
The cross-rank protocols (tickets, peer slots, segment tables) are exercised on
one GPU by running R virtual ranks inside one cooperative launch
(``EmulatedWorld``); real multi-process runs live in test_gpu_multi.py.
"""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _world1():
    from tridist_b200.parallel.runtime import ProcessWorld
    global _W1
    try:
        return _W1
    except NameError:
        _W1 = ProcessWorld(0, 1)
        return _W1


def _loaded_native():
    from tridist_b200.parallel.runtime import native
    C = native()
    assert C.__file__.endswith("_C.so")
    return C


TOL = 1e-2


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape,bn", [((128, 256, 64), 256), ((256, 128, 192), 128), ((384, 640, 1000), None),
                                      ((1024, 2048, 512), None), ((192, 384, 520), 256)])
def test_plain_gemm(shape, bn, dtype):
    from tridist_b200.ops._gemm_common import gemm_nt
    _loaded_native()
    M, N, K = shape
    torch.manual_seed(1)
    a = (torch.randn(M, K, device="cuda") * 0.05).to(dtype)
    b = (torch.randn(N, K, device="cuda") * 0.05).to(dtype)
    before = _loaded_native().launch_count()
    out = gemm_nt(a, b, bn=bn)
    torch.cuda.synchronize()
    assert _loaded_native().launch_count() == before + 1
    ref = a.float() @ b.float().t()
    assert (out.float() - ref).abs().max().item() < TOL


def test_gemm_swiglu_epilogue_and_kernel():
    from tridist_b200.ops import swiglu
    from tridist_b200.ops._gemm_common import gemm_nt
    torch.manual_seed(2)
    M, I, K = 512, 640, 384
    a = (torch.randn(M, K, device="cuda") * 0.1).to(torch.bfloat16)
    w = (torch.randn(2 * I, K, device="cuda") * 0.1).to(torch.bfloat16)
    h = a.float() @ w.float().t()
    ref = F.silu(h[:, :I]) * h[:, I:]
    fused = gemm_nt(a, w, swiglu=True)
    two_step = swiglu(gemm_nt(a, w))
    torch.cuda.synchronize()
    assert (fused.float() - ref).abs().max().item() < TOL
    assert (two_step.float() - ref).abs().max().item() < 3e-2   # h rounded to bf16 first
    # stand-alone kernel against torch on the same 16-bit input
    hh = (torch.randn(300, 2 * 264, device="cuda")).to(torch.float16)
    got = swiglu(hh)
    exp = (F.silu(hh[:, :264].float()) * hh[:, 264:].float())
    assert (got.float() - exp).abs().max().item() < 1e-2


@pytest.mark.parametrize("M,I", [(64, 264), (2112, 1408)])
def test_swiglu_reads_what_the_gemm_in_front_of_it_wrote(M, I):
    """The activation starts under the tail of the GEMM that writes its input, over the same buffer with other
    contents each time and without a synchronisation: the bits of a call on the finished buffer."""
    from tridist_b200.ops import swiglu
    from tridist_b200.ops._gemm_common import gemm_nt
    K, dt = 512, torch.bfloat16
    w = _rand((2 * I, K), 4, dt)
    h = torch.empty((M, 2 * I), dtype=dt, device="cuda")
    xs = [_rand((M, K), 5 + i, dt) for i in range(8)]
    got = []
    for x in xs:
        gemm_nt(x, w, out=h)
        got.append(swiglu(h))
    torch.cuda.synchronize()
    for x, g in zip(xs, got):
        ref = gemm_nt(x, w)
        torch.cuda.synchronize()
        assert torch.equal(g, swiglu(ref))


def test_public_api_single_rank():
    """R = 1 degenerates: every op collapses to the local GEMM / permutation."""
    from tridist_b200.ops import (ag_gemm_intra_node, create_ag_gemm_intra_node_context,
                                  create_gemm_ar_intra_node_context, create_gemm_rs_intra_node_context,
                                  create_moe_a2a_intra_node_context, gemm_ar_intra_node, gemm_rs_intra_node,
                                  moe_combine_intra_node_op, moe_dispatch_intra_node_op)
    from tridist_b200.utils.testing import fake_expert, moe_inputs
    w = _world1()
    torch.manual_seed(3)
    dt = torch.float16
    M, N, K = 512, 768, 256
    a = (torch.randn(M, K, device="cuda") * 0.05).to(dt)
    b = (torch.randn(N, K, device="cuda") * 0.05).to(dt)
    ref = a.float() @ b.float().t()
    ctx = create_ag_gemm_intra_node_context(M, K, dt, dt, 0, 1, M_PER_CHUNK=256, world=w)
    assert (ag_gemm_intra_node(a, b, False, ctx).float() - ref).abs().max().item() < TOL
    rs = create_gemm_rs_intra_node_context(M, N, dt, 0, 1, world=w)
    assert (gemm_rs_intra_node(a, b, rs).float() - ref).abs().max().item() < TOL
    ar = create_gemm_ar_intra_node_context(M, N, dt, dt, 0, 1, world=w)
    assert (gemm_ar_intra_node(a, b, ar).float() - ref).abs().max().item() < TOL
    E, H, topk, T = 8, 256, 2, 96
    moe = create_moe_a2a_intra_node_context(E, H, dt, T, topk, 0, 1, world=w)
    tokens, idx, wts = [x.cuda() for x in moe_inputs(0, T, H, E, topk, 0, dt)]
    n = int(moe_dispatch_intra_node_op(tokens, idx, moe).item())
    assert n == T * topk
    sc = moe.scatter_idx[:T].long()
    assert sorted(sc.flatten().tolist()) == list(range(n))          # bijection onto rows
    assert torch.equal(moe.recv[sc[:, 0]], tokens)                  # content
    moe.out[:n] = fake_expert(moe.recv[:n])
    out = torch.empty_like(tokens)
    moe_combine_intra_node_op(moe, idx, out, wts)
    exp = (wts.unsqueeze(-1) * (tokens.float().unsqueeze(1) * 2 + (sc % 5).float().unsqueeze(-1))).sum(1)
    torch.cuda.synchronize()
    w.check()
    assert (out.float() - exp).abs().max().item() < 2e-2


def _emu(R):
    from tridist_b200.parallel.runtime import EmulatedWorld
    return EmulatedWorld(R)


@pytest.mark.parametrize("R", [2, 4])
def test_ag_gemm_emulated(R):
    from tridist_b200.ops.all_gather_gemm import ag_gemm_emulated, create_ag_gemm_intra_node_context
    from tridist_b200.utils.testing import ag_inputs
    w = _emu(R)
    dt = torch.bfloat16
    m_pr, K, n_pr = 256, 512, 384
    ctxs = [create_ag_gemm_intra_node_context(m_pr * R, K, dt, dt, r, R, M_PER_CHUNK=128, world=w) for r in range(R)]
    for it in range(3):                                   # fresh data every round, both parities
        ins = [ag_inputs(r, R, m_pr, K, n_pr, it, dt, 0.05) for r in range(R)]
        a_list = [ins[r][0][r].cuda() for r in range(R)]
        b_list = [ins[r][1].cuda() for r in range(R)]
        c_list = [torch.empty(m_pr * R, n_pr, dtype=dt, device="cuda") for _ in range(R)]
        ag_gemm_emulated(ctxs, a_list, b_list, c_list)
        torch.cuda.synchronize()
        w.check()
        full = torch.cat([x.float() for x in a_list], 0)
        for r in range(R):
            ref = full @ b_list[r].float().t()
            assert (c_list[r].float() - ref).abs().max().item() < TOL, f"round {it} rank {r}"
            ws = ctxs[r].workspace(ctxs[r].flag_round & 1, m_pr * R)
            for s in range(R):
                if s != r:                                # pushed shards landed bit-exactly
                    assert torch.equal(ws[s * m_pr:(s + 1) * m_pr], a_list[s])
    # GEMM-only decomposition on the last workspace gives the same result
    c2 = [torch.empty_like(c) for c in c_list]
    ag_gemm_emulated(ctxs, a_list, b_list, c2, skip_comm=True)
    torch.cuda.synchronize()
    for r in range(R):
        assert torch.equal(c2[r], c_list[r])


@pytest.mark.parametrize("R,M", [(2, 512), (4, 512), (4, 256)])
def test_gemm_rs_emulated(R, M):
    from tridist_b200.ops.gemm_reduce_scatter import create_gemm_rs_intra_node_context, gemm_rs_emulated
    from tridist_b200.utils.testing import ks_inputs
    w = _emu(R)
    dt = torch.float16
    N, kl = 384, 256
    ctxs = [create_gemm_rs_intra_node_context(M, N, dt, r, R, world=w) for r in range(R)]
    for it in range(3):
        a_all, b_all = ks_inputs(R, M, N, kl, it, dt, 0.05)
        a_all = [x.cuda() for x in a_all]
        b_all = [x.cuda() for x in b_all]
        outs = gemm_rs_emulated(ctxs, a_all, b_all)
        torch.cuda.synchronize()
        w.check()
        ref = sum(a_all[s].float() @ b_all[s].float().t() for s in range(R))
        m_pr = M // R
        for r in range(R):
            err = (outs[r].float() - ref[r * m_pr:(r + 1) * m_pr]).abs().max().item()
            assert err < TOL, f"round {it} rank {r}: {err}"


@pytest.mark.parametrize("mode", ["one_shot", "two_shot"])
@pytest.mark.parametrize("R,M", [(2, 256), (4, 192)])
def test_gemm_ar_emulated(R, M, mode):
    from tridist_b200.ops.gemm_allreduce import create_gemm_ar_intra_node_context, gemm_ar_emulated
    from tridist_b200.utils.testing import ks_inputs
    w = _emu(R)
    dt = torch.bfloat16
    N, kl = 640, 192
    ctxs = [create_gemm_ar_intra_node_context(256, N, dt, dt, r, R, M_PER_CHUNK=64, world=w) for r in range(R)]
    for it in range(3):
        a_all, b_all = ks_inputs(R, M, N, kl, it, dt, 0.05)
        a_all = [x.cuda() for x in a_all]
        b_all = [x.cuda() for x in b_all]
        use_symm = (mode == "two_shot" and it == 2)
        c_list = [ctxs[r].symm_output(M) if use_symm else torch.empty(M, N, dtype=dt, device="cuda")
                  for r in range(R)]
        gemm_ar_emulated(ctxs, a_all, b_all, c_list, mode=mode)
        torch.cuda.synchronize()
        w.check()
        ref = sum(a_all[s].float() @ b_all[s].float().t() for s in range(R))
        for r in range(R):
            err = (c_list[r].float() - ref).abs().max().item()
            assert err < 2e-2, f"round {it} rank {r}: {err}"
            assert torch.equal(c_list[r], c_list[0]), "all-reduce result must be bit-identical on all ranks"


@pytest.mark.parametrize("zipf", [0.0, 1.2])
def test_moe_emulated(zipf):
    from tridist_b200.ops.moe_a2a import (create_moe_a2a_intra_node_context, moe_combine_emulated,
                                          moe_dispatch_emulated)
    from tridist_b200.utils.testing import fake_expert, moe_inputs
    R, E, H, topk, T = 4, 16, 512, 4, 200
    w = _emu(R)
    dt = torch.float16
    ctxs = [create_moe_a2a_intra_node_context(E, H, dt, T, topk, r, R, world=w) for r in range(R)]
    epr = E // R
    for it in range(2):
        ins = [[x.cuda() for x in moe_inputs(r, T, H, E, topk, it, dt, zipf)] for r in range(R)]
        toks = [i[0] for i in ins]
        idxs = [i[1] for i in ins]
        wts = [i[2] for i in ins]
        totals = moe_dispatch_emulated(ctxs, toks, idxs)
        torch.cuda.synchronize()
        w.check()
        seen = [set() for _ in range(R)]
        for r in range(R):
            n = int(totals[r].item())
            exp_n = sum(int(((idxs[s] // epr) == r).sum()) for s in range(R))
            assert n == exp_n
            # segment layout: (source, local expert) in order, counts match the routing
            counts = ctxs[r].recv_counts.cpu()
            for s in range(R):
                for k in range(epr):
                    assert int(counts[s, k]) == int((idxs[s] == r * epr + k).sum())
        for s in range(R):
            sc = ctxs[s].scatter_idx[:T].cpu()
            ic = idxs[s].cpu()
            for t in range(0, T, 7):
                for j in range(topk):
                    d = int(ic[t, j]) // epr
                    row = int(sc[t, j])
                    assert torch.equal(ctxs[d].recv[row], toks[s][t])            # content
            for t in range(T):
                for j in range(topk):
                    key = (int(ic[t, j]) // epr, int(sc[t, j]))
                    assert key[1] not in seen[key[0]]                               # bijection
                    seen[key[0]].add(key[1])
            # rows of (s -> d, expert) fall inside their segment
        for r in range(R):
            n = int(totals[r].item())
            assert seen[r] == set(range(n))
            ctxs[r].out[:n] = fake_expert(ctxs[r].recv[:n])
        outs = [torch.empty_like(t) for t in toks]
        moe_combine_emulated(ctxs, idxs, outs, wts)
        torch.cuda.synchronize()
        w.check()
        for s in range(R):
            sc = ctxs[s].scatter_idx[:T].long()
            exp = (wts[s].unsqueeze(-1) * (toks[s].float().unsqueeze(1) * 2 + (sc % 5).float().unsqueeze(-1))).sum(1)
            assert (outs[s].float() - exp).abs().max().item() < 3e-2


def test_bounded_wait_reports_status():
    """A wait on a flag nothing sets runs out, records a status and leaves the context usable."""
    from tridist_b200.parallel.runtime import TriDistError
    w = _world1()
    C = _loaded_native()
    w.clear_status()
    flag = torch.zeros(4, dtype=torch.int32, device="cuda")
    C.wait_flag_test(flag.data_ptr(), 7, w.status_dev, w.abort_word, 50_000_000)   # 50 ms limit
    torch.cuda.synchronize()
    st = w.status()
    assert st[0] == 1 and st[2] == 32 and st[3] == 7 and st[4] == 0
    with pytest.raises(TriDistError):
        w.check()
    w.clear_status()
    w.check()
    # the context still works
    x = torch.ones(8, device="cuda")
    assert float(x.sum()) == 8.0


def test_spot_verify_flags_bad_tile():
    from tridist_b200.ops._gemm_common import gemm_nt
    C = _loaded_native()
    torch.manual_seed(5)
    M, N, K = 256, 512, 256
    a = (torch.randn(M, K, device="cuda") * 0.1).to(torch.float16)
    b = (torch.randn(N, K, device="cuda") * 0.1).to(torch.float16)
    c = gemm_nt(a, b, bn=256)
    bad = torch.zeros(4, dtype=torch.int32, device="cuda")
    C.spot_verify(a.data_ptr(), b.data_ptr(), c.data_ptr(), M, N, K, K, K, N, False, 4, 2e-2, bad.data_ptr(), 256)
    torch.cuda.synchronize()
    assert bad.sum().item() == 0
    c[128:, 256:] += 1.0                                  # damage tile (1, 1)
    C.spot_verify(a.data_ptr(), b.data_ptr(), c.data_ptr(), M, N, K, K, K, N, False, 4, 2e-2, bad.data_ptr(), 256)
    torch.cuda.synchronize()
    assert bad.tolist() == [0, 0, 0, 1]


def test_skew_layer_order_table_and_observer_emulated():
    """Table-driven source order (device int32 table) gives the same C as the default order, and the
    consumer's arrival stamps come back for every remote source."""
    from tridist_b200.ops.all_gather_gemm import ag_gemm_emulated, create_ag_gemm_intra_node_context
    from tridist_b200.parallel.predictor import infer_straggler
    from tridist_b200.utils.testing import ag_inputs
    R = 4
    w = _emu(R)
    dt = torch.float16
    m_pr, K, n_pr = 128, 256, 256
    ctxs = [create_ag_gemm_intra_node_context(m_pr * R, K, dt, dt, r, R, M_PER_CHUNK=128, world=w) for r in range(R)]
    ins = [ag_inputs(r, R, m_pr, K, n_pr, 0, dt, 0.05) for r in range(R)]
    a_list = [ins[r][0][r].cuda() for r in range(R)]
    b_list = [ins[r][1].cuda() for r in range(R)]
    c_ref = [torch.empty(m_pr * R, n_pr, dtype=dt, device="cuda") for _ in range(R)]
    ag_gemm_emulated(ctxs, a_list, b_list, c_ref)
    torch.cuda.synchronize()
    for r, ctx in enumerate(ctxs):                         # own first, "straggler" (r+1) last
        order = [r] + [x for x in range(R) if x not in (r, (r + 1) % R)] + [(r + 1) % R]
        ctx.emu_order_table = torch.tensor(order, dtype=torch.int32, device="cuda")
        ctx.observe = True
        ctx.arrival_ns.fill_(torch.iinfo(torch.int64).max)
    c_tab = [torch.empty_like(c) for c in c_ref]
    ag_gemm_emulated(ctxs, a_list, b_list, c_tab)
    torch.cuda.synchronize()
    w.check()
    for r in range(R):
        assert torch.equal(c_tab[r], c_ref[r])
        stamps = ctxs[r].arrival_ns.cpu().tolist()
        remote = [s for s in range(R) if s != r]
        assert all(0 < stamps[s] < torch.iinfo(torch.int64).max for s in remote)
        assert infer_straggler(stamps, r) in remote


def test_verify_and_repair_single_rank(monkeypatch):
    from tridist_b200.ops import create_i1_context, i1_ag_tr_op, i1_observer_read, i1_table_peek, i1_table_write
    from tridist_b200.ops.ag_tr_pred import _verify_and_repair
    w = _world1()
    dt = torch.bfloat16
    M, K, N = 512, 256, 512
    torch.manual_seed(11)
    a = (torch.randn(M, K, device="cuda") * 0.1).to(dt)
    b = (torch.randn(N, K, device="cuda") * 0.1).to(dt)
    c = torch.empty(M, N, dtype=dt, device="cuda")
    ictx = create_i1_context(M, K, dt, dt, 0, 1, world=w)
    i1_table_write(ictx, 7, 0, 1, 0, 1)
    assert i1_table_peek(ictx)[:4] == [7, 0, 1, 1]
    i1_ag_tr_op(a, b, c, ictx)
    torch.cuda.synchronize()
    good = c.clone()
    assert (good.float() - a.float() @ b.float().t()).abs().max().item() < TOL
    assert _verify_and_repair(a, b, c, ictx) == 0         # nothing to repair
    c[128:256, 256:] = 0                                  # damage one tile of the result
    fixed = _verify_and_repair(a, b, c, ictx)
    torch.cuda.synchronize()
    assert fixed >= 1 and torch.equal(c, good)
    assert i1_observer_read(ictx)[1] == 0


def test_order_driven_ar_carrier_and_gates_single_rank():
    from tridist_b200.ops import (create_gemm_ar_rd_context, gemm_ar_pred_op, make_gate_flag, task_events)
    w = _world1()
    dt = torch.float16
    M, N, K = 256, 256, 128
    torch.manual_seed(12)
    a = (torch.randn(M, K, device="cuda") * 0.1).to(dt)
    b = (torch.randn(N, K, device="cuda") * 0.1).to(dt)
    ctx = create_gemm_ar_rd_context(M, N, dt, dt, 0, 1, world=w)
    ctx.chunk_rows = 64
    gate = make_gate_flag()
    gate[0] = 5                                           # already released
    c = torch.zeros(M, N, dtype=dt, device="cuda")
    gemm_ar_pred_op(a, b, c, ctx, order=[3, 1, 0, 2], gates=[(1, gate.data_ptr(), 5)])
    torch.cuda.synchronize()
    w.check()
    assert (c.float() - a.float() @ b.float().t()).abs().max().item() < TOL
    ev = task_events(ctx)
    assert len(ev) == 4 and all(e is not None and e[0].elapsed_time(e[1]) >= 0 for e in ev)


def test_symm_host_one_sided_calls():
    from tridist_b200.parallel.symm_host import SymmHost
    w = _world1()
    h = SymmHost(w)
    assert h.my_pe() == 0 and h.n_pes() == 1
    buf = h.malloc(4096)
    src = torch.arange(256, dtype=torch.int32, device="cuda")
    h.putmem(buf, 1024, src, pe=0)
    dst = torch.zeros_like(src)
    h.getmem(dst, buf, 1024, pe=0)
    h.quiet()
    assert torch.equal(src, dst) and h.ptr(buf, 0, 16) == buf.local_ptr + 16
    h.set_signal(buf, 3, 9, pe=0)
    h.wait_signal(buf, 3, 9, timeout_ms=200)
    h.barrier_all()
    torch.cuda.synchronize()
    w.check()
    h.free(buf)


@pytest.mark.parametrize("mode", ["ag_rs", "gemm_ar"])
def test_tp_mlp_single_rank(mode):
    from tridist_b200.models.tp_mlp import TPMLP, TPMLPConfig, reference_forward
    w = _world1()
    dt = torch.bfloat16
    M, K, I = 256, 256, 384
    torch.manual_seed(13)
    x = torch.randn(M, K, device="cuda").to(dt)
    w_gu = (torch.randn(2 * I, K, device="cuda") * 0.05).to(dt)
    w_d = (torch.randn(K, I, device="cuda") * 0.05).to(dt)
    ref = reference_forward(x, [w_gu], [w_d])
    for fuse in ([True, False] if mode == "ag_rs" else [False]):
        layer = TPMLP(TPMLPConfig(hidden=K, intermediate=I, max_tokens=M, dtype=dt, mode=mode, fuse_swiglu=fuse),
                      0, 1, w_gu, w_d, world=w)
        y = layer(x)
        torch.cuda.synchronize()
        w.check()
        assert (y.float() - ref).abs().max().item() < 3e-2


# ---------------------------------------------------------------------------------------------
# The persistent loop, the tile shapes and the edges (every CTA gets many tiles: accumulator
# reuse, ring wrap across tiles, late-joining pushers; odd block counts; ragged M and N)
# ---------------------------------------------------------------------------------------------
def _rand(shape, seed, dtype, scale=0.05):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * scale).to(dtype)


def _check_rows(out, a, b, rows=96, tol=TOL):
    idx = torch.randperm(a.shape[0], device="cuda")[:rows]
    ref = a[idx].float() @ b.float().t()
    err = (out[idx].float() - ref).abs().max().item()
    assert err < tol, err


@pytest.mark.parametrize("variant", ["wide", "pair", "single"])
@pytest.mark.parametrize("K", [2048, 12288])
def test_plain_gemm_many_tiles_per_cta(variant, K, monkeypatch):
    """16 CTAs for 4096 x 4096: every CTA (pair) walks 16 to 64 tiles, so both accumulators are
    reused many times and the operand ring wraps across tile boundaries."""
    from tridist_b200.ops._gemm_common import gemm_nt
    monkeypatch.setenv("TRIDIST_WIDE", "1" if variant == "wide" else "0")
    monkeypatch.setenv("TRIDIST_CTA_PAIR", "0" if variant == "single" else "1")
    a, b = _rand((4096, K), 21, torch.bfloat16), _rand((4096, K), 22, torch.bfloat16)
    out = gemm_nt(a, b, max_ctas=16)
    torch.cuda.synchronize()
    _check_rows(out, a, b)


@pytest.mark.parametrize("splitk", [1, 0])
@pytest.mark.parametrize("M,N,K,max_ctas", [(128, 2048, 4096, 0), (128, 1024, 8200, 0), (1536, 1024, 2048, 10),
                                            (2048, 2304, 1024, 20), (640, 648, 1024, 0), (1000, 520, 776, 0),
                                            (384, 768, 512, 0), (4224, 512, 256, 12)])
def test_plain_gemm_edges_and_split_k(M, N, K, max_ctas, splitk, monkeypatch):
    """Ragged M / N / K, odd numbers of row blocks under CTA pairs and 512-row tiles, and the K
    split of the last scheduling round (2 to 8 slices; K blocks that do not divide evenly)."""
    from tridist_b200.ops._gemm_common import gemm_nt
    monkeypatch.setenv("TRIDIST_SPLITK", str(splitk))
    for dt in (torch.float16, torch.bfloat16):
        a, b = _rand((M, K), 31, dt), _rand((N, K), 32, dt)
        out = gemm_nt(a, b, max_ctas=max_ctas)
        torch.cuda.synchronize()
        ref = a.float() @ b.float().t()
        assert (out.float() - ref).abs().max().item() < TOL


def test_split_k_slices_are_used(monkeypatch):
    from tridist_b200.ops._gemm_common import BM, OP_PLAIN, SCHED_NATURAL
    C = _loaded_native()
    for M, N, K in [(128, 2048, 4096), (128, 8192, 3584), (8192, 6144, 12288)]:
        cuts = C.splitk_dump(dict(op=OP_PLAIN, sched=SCHED_NATURAL, bn=256 if M > 128 else 128, R=1, rank=0,
                                  M=M, N=N, K=K), 148)
        assert cuts and all(2 <= c[3] <= 8 for c in cuts)


def test_gemm_variants_keep_their_tile_loop_in_registers():
    """Local memory per thread (stack and spills) of every variant: 32 bytes are the producer's table of
    observed shards, the rest are spills, at most what they were before tiles cut along K were summed
    by all their workers (80, 112 and 176 bytes)."""
    for bn, bf16, pair, staging, mt, regs, local in _loaded_native().gemm_variants():
        limit = 32 if not staging else 208 if mt == 2 else 144 if bn == 256 else 112
        assert regs <= 168 and local <= limit, (bn, bf16, pair, staging, mt, local)


@pytest.mark.parametrize("tiles", ["single", "pair", "wide"])
def test_fused_ops_emulated_many_tiles_per_cta(tiles, monkeypatch):
    """Two virtual ranks, 8 CTAs each, 2048-row problems: AG (pushing CTAs join late), RS and both
    AR forms walk many tiles per CTA, on single CTAs, CTA pairs and 512-row pair tiles."""
    from tridist_b200.ops.all_gather_gemm import ag_gemm_emulated, create_ag_gemm_intra_node_context
    from tridist_b200.ops.gemm_allreduce import create_gemm_ar_intra_node_context, gemm_ar_emulated
    from tridist_b200.ops.gemm_reduce_scatter import create_gemm_rs_intra_node_context, gemm_rs_emulated
    monkeypatch.setenv("TRIDIST_MAX_CTAS", "8")
    monkeypatch.setenv("TRIDIST_EMU_PAIR", "0" if tiles == "single" else "1")
    monkeypatch.setenv("TRIDIST_WIDE", "1" if tiles == "wide" else "0")
    monkeypatch.setenv("TRIDIST_PUSH_CTAS", "4")
    monkeypatch.setenv("TRIDIST_PUSH_SKIP", "1")
    R, dt = 2, torch.bfloat16
    w = _emu(R)
    M, N, K = 2048, 1024, 768
    m_pr = M // R
    ag = [create_ag_gemm_intra_node_context(M, K, dt, dt, r, R, M_PER_CHUNK=512, world=w) for r in range(R)]
    rs = [create_gemm_rs_intra_node_context(M, N, dt, r, R, world=w) for r in range(R)]
    ar = [create_gemm_ar_intra_node_context(M, N, dt, dt, r, R, M_PER_CHUNK=64, world=w) for r in range(R)]
    for it in range(2):
        a_sh = [_rand((m_pr, K), 40 + 7 * it + r, dt) for r in range(R)]
        bw = [_rand((N, K), 50 + 7 * it + r, dt) for r in range(R)]
        c = [torch.empty(M, N, dtype=dt, device="cuda") for _ in range(R)]
        ag_gemm_emulated(ag, a_sh, bw, c)
        torch.cuda.synchronize()
        w.check()
        full = torch.cat(a_sh, 0)
        for r in range(R):
            _check_rows(c[r], full, bw[r])
        a_k = [_rand((M, K), 60 + 7 * it + r, dt) for r in range(R)]
        ref = sum(a_k[s].float() @ bw[s].float().t() for s in range(R))
        outs = gemm_rs_emulated(rs, a_k, bw)
        torch.cuda.synchronize()
        w.check()
        for r in range(R):
            assert (outs[r].float() - ref[r * m_pr:(r + 1) * m_pr]).abs().max().item() < 2e-2
        for mode in ("one_shot", "two_shot"):
            cc = [torch.empty(M, N, dtype=dt, device="cuda") for _ in range(R)]
            gemm_ar_emulated(ar, a_k, bw, cc, mode=mode)
            torch.cuda.synchronize()
            w.check()
            for r in range(R):
                assert (cc[r].float() - ref).abs().max().item() < 2e-2, mode
                assert torch.equal(cc[r], cc[0])


@pytest.mark.parametrize("R,M", [(4, 768), (2, 384), (4, 1280)])
def test_gemm_rs_emulated_rows_per_rank_not_a_block_multiple(R, M):
    """Rows per rank of 192 / 320: row blocks with two owners take the per-row bulk path, and two
    owners of one block publish before either waits."""
    from tridist_b200.ops.gemm_reduce_scatter import create_gemm_rs_intra_node_context, gemm_rs_emulated
    w = _emu(R)
    dt = torch.float16
    N, kl = 640, 320
    ctxs = [create_gemm_rs_intra_node_context(M, N, dt, r, R, world=w) for r in range(R)]
    for it in range(2):
        a_all = [_rand((M, kl), 70 + it * 9 + r, dt) for r in range(R)]
        b_all = [_rand((N, kl), 80 + it * 9 + r, dt) for r in range(R)]
        outs = gemm_rs_emulated(ctxs, a_all, b_all)
        torch.cuda.synchronize()
        w.check()
        ref = sum(a_all[s].float() @ b_all[s].float().t() for s in range(R))
        m_pr = M // R
        for r in range(R):
            assert (outs[r].float() - ref[r * m_pr:(r + 1) * m_pr]).abs().max().item() < TOL


def test_fused_kernel_gives_up_cleanly_when_a_shard_never_arrives(monkeypatch):
    """The allowed form of a failure test: virtual rank 1 does not push, rank 0's producer waits
    for its shard with a 20 ms limit, the wait runs out, every role of the kernel unwinds (loads
    drained, MMAs retired, TMEM freed), the status names the site, and the next launch on the same
    context works."""
    from tridist_b200.ops.all_gather_gemm import ag_gemm_emulated, create_ag_gemm_intra_node_context
    from tridist_b200.parallel.runtime import TriDistError
    monkeypatch.setenv("TRIDIST_WAIT_TIMEOUT_MS", "20")
    R, dt = 2, torch.float16
    w = _emu(R)
    m_pr, K, N = 256, 512, 512
    ctxs = [create_ag_gemm_intra_node_context(m_pr * R, K, dt, dt, r, R, M_PER_CHUNK=128, world=w) for r in range(R)]
    a = [_rand((m_pr, K), 90 + r, dt) for r in range(R)]
    b = [_rand((N, K), 95 + r, dt) for r in range(R)]
    c = [torch.empty(m_pr * R, N, dtype=dt, device="cuda") for _ in range(R)]
    ag_gemm_emulated(ctxs, a, b, c)                      # a good round first
    torch.cuda.synchronize()
    w.check()
    ag_gemm_emulated(ctxs, a, b, c, mute_ranks=[1])      # rank 1's shard never arrives at rank 0
    torch.cuda.synchronize()
    with pytest.raises(TriDistError, match="all-gather chunk ticket"):
        w.check()
    st = w.status()
    assert st[0] == 1 and st[1] == 0 and st[2] == 1      # flag wait timed out, on rank 0, at the chunk ticket
    w.clear_status()
    ag_gemm_emulated(ctxs, a, b, c)                      # the context is still usable
    torch.cuda.synchronize()
    w.check()
    full = torch.cat(a, 0).float()
    for r in range(R):
        assert (c[r].float() - full @ b[r].float().t()).abs().max().item() < TOL


def test_a_rank_that_gives_up_raises_every_ranks_abort_word():
    """The abort buffer is symmetric: the kernel that runs out of time stores its code into the abort
    word of every rank, and a kernel that leaves a wait because of a raised word records why."""
    w = _emu(3)
    C = _loaded_native()
    w.clear_status()
    words = w.peer_abort_words()
    assert len(set(words)) == 3
    flag = torch.zeros(4, dtype=torch.int32, device="cuda")
    C.wait_flag_test(flag.data_ptr(), 9, w.status_dev, words[0], 20_000_000, words)
    torch.cuda.synchronize()
    raised = [int(w.abort_buf.tensor(torch.int32, (1,), 0, rank=r).item()) for r in range(3)]
    assert raised == [1, 1, 1]
    assert w.status()[0] == 1
    # a second waiter whose word is already raised leaves at once and records "gave up because ..."
    from tridist_b200.parallel.runtime import TriDistError
    w.C.status_clear(w.status_host)
    C.wait_flag_test(flag.data_ptr(), 9, w.status_dev, words[1], 2_000_000_000, [])
    torch.cuda.synchronize()
    assert w.status()[0] == 5
    with pytest.raises(TriDistError, match="another rank"):
        w.check()
    w.clear_status()
    assert [int(w.abort_buf.tensor(torch.int32, (1,), 0, rank=r).item()) for r in range(3)] == [0, 0, 0]


@pytest.mark.parametrize("R", [2, 4])
def test_ag_gemm_pull_transport_emulated(R):
    """The tile-ready entry points: stage, arrive tickets, pull through the copy engine, ready tickets."""
    from tridist_b200.ops.all_gather_gemm import ag_gemm_emulated
    from tridist_b200.ops.gemm_ag_tr import create_gemm_ag_tr_context
    w = _emu(R)
    dt = torch.float16
    m_pr, K, n_pr = 256, 1024, 384
    ctxs = [create_gemm_ag_tr_context(m_pr * R, K, dt, dt, r, R, chunk_rows=128, world=w) for r in range(R)]
    assert all(c.transport == "pull" for c in ctxs)
    for it in range(3):
        a = [_rand((m_pr, K), 200 + it * 5 + r, dt) for r in range(R)]
        b = [_rand((n_pr, K), 210 + it * 5 + r, dt) for r in range(R)]
        c = [torch.empty(m_pr * R, n_pr, dtype=dt, device="cuda") for _ in range(R)]
        ag_gemm_emulated(ctxs, a, b, c)
        torch.cuda.synchronize()
        w.check()
        full = torch.cat(a, 0).float()
        for r in range(R):
            assert (c[r].float() - full @ b[r].float().t()).abs().max().item() < TOL, f"round {it} rank {r}"
            ws = ctxs[r].workspace(ctxs[r].flag_round & 1, m_pr * R)
            for s in range(R):                      # own shard staged, the others pulled, all bit-exact
                assert torch.equal(ws[s * m_pr:(s + 1) * m_pr], a[s])


def test_skew_table_modes_give_the_same_result_emulated():
    """The full table [seq, degraded, mode, k_eff, order[R], budget[R]] read by the kernel: band-major
    (mode 0, two row bands), source-major (mode 1), degraded (default rotation) and small spin budgets
    only change which CTA computes which tile when."""
    from tridist_b200.ops.all_gather_gemm import ag_gemm_emulated, create_ag_gemm_intra_node_context
    R = 4
    w = _emu(R)
    dt = torch.bfloat16
    m_pr, K, n_pr = 512, 512, 512
    ctxs = [create_ag_gemm_intra_node_context(m_pr * R, K, dt, dt, r, R, M_PER_CHUNK=256, world=w) for r in range(R)]
    a = [_rand((m_pr, K), 300 + r, dt) for r in range(R)]
    b = [_rand((n_pr, K), 310 + r, dt) for r in range(R)]
    ref = [torch.empty(m_pr * R, n_pr, dtype=dt, device="cuda") for _ in range(R)]
    ag_gemm_emulated(ctxs, a, b, ref)
    torch.cuda.synchronize()
    w.check()
    full = torch.cat(a, 0).float()
    assert (ref[0].float() - full @ b[0].float().t()).abs().max().item() < 2e-2
    for seq, (deg, mode, k_eff, budget) in enumerate([(0, 0, 2, 128), (0, 1, 2, 128), (1, 1, 2, 128), (0, 0, 2, 1)]):
        tables = []
        for r, ctx in enumerate(ctxs):
            order = [r] + [x for x in range(R) if x not in (r, (r + 1) % R)] + [(r + 1) % R]
            t = torch.tensor([seq, deg, mode, k_eff] + order + [budget] * R, dtype=torch.int32, device="cuda")
            tables.append(t)
            ctx.emu_order_table = t[4:4 + R]
            ctx.emu_table_header = True
            ctx.plans.clear()
        out = [torch.empty_like(x) for x in ref]
        ag_gemm_emulated(ctxs, a, b, out)
        torch.cuda.synchronize()
        w.check()
        for r in range(R):
            assert torch.equal(out[r], ref[r]), (deg, mode, k_eff, budget, r)


def test_band_major_schedule_walks_bands_first():
    C = _loaded_native()
    from tridist_b200.ops._gemm_common import OP_AG, SCHED_SEGMENT
    R, M, N = 4, 4096, 1024
    d = dict(op=OP_AG, sched=SCHED_SEGMENT, bn=256, R=R, rank=1, M=M, N=N, K=1024, m_per_rank=M // R,
             seg_order=[1, 0, 3, 2], chunk_rows=256, n_chunks=4, seg_bands=2, allow_wide=0)
    tiles = sorted((t[4], t[0]) for cta in C.schedule_dump(d, 148) for t in cta)
    rows_per_seg = (M // R) // 128
    walk = []
    for _, mt in tiles:
        key = (mt // rows_per_seg, (mt % rows_per_seg) // (rows_per_seg // 2))     # (segment, band)
        if not walk or walk[-1] != key:
            walk.append(key)
    assert walk == [(s, b) for b in range(2) for s in [1, 0, 3, 2]]


def test_device_side_index_check_reports_and_skips():
    """A row index outside the receive buffer (made here by damaging the scatter table between dispatch
    and combine) is recorded as 'index out of range' and the access is skipped: nothing faults."""
    from tridist_b200.ops import (create_moe_a2a_intra_node_context, moe_combine_intra_node_op,
                                  moe_dispatch_intra_node_op)
    from tridist_b200.parallel.runtime import TriDistError
    from tridist_b200.utils.testing import moe_inputs
    w = _world1()
    w.clear_status()
    dt = torch.float16
    E, H, topk, T = 8, 256, 2, 64
    ctx = create_moe_a2a_intra_node_context(E, H, dt, T, topk, 0, 1, world=w)
    tokens, idx, wts = [x.cuda() for x in moe_inputs(0, T, H, E, topk, 3, dt)]
    moe_dispatch_intra_node_op(tokens, idx, ctx)
    ctx.out[:T * topk] = ctx.recv[:T * topk]
    ctx.scatter_idx[5, 1] = ctx.recv.shape[0] + 17
    out = torch.empty_like(tokens)
    moe_combine_intra_node_op(ctx, idx, out, wts)
    torch.cuda.synchronize()
    st = w.status()
    assert st[0] == 3 and st[2] == 11 and st[4] == ctx.recv.shape[0] + 17
    with pytest.raises(TriDistError, match="index out of range"):
        w.check()
    w.clear_status()
    assert bool(torch.isfinite(out.float()).all())


@pytest.mark.parametrize("R", [2, 4, 8])
def test_gemm_ar_rd_emulated(R):
    """Recursive-doubling panel exchange on virtual ranks: three panels over two staging slots (the
    third panel reuses slot 0 under the ack ticket), several calls on one context, and an M that
    changes between calls (tickets advance by a fixed stride per call)."""
    from tridist_b200.ops.gemm_ar_rd import create_gemm_ar_rd_context, gemm_ar_rd_emulated
    from tridist_b200.utils.testing import ks_inputs
    w = _emu(R)
    dt = torch.bfloat16
    N, kl = 640, 192
    ctxs = [create_gemm_ar_rd_context(384, N, dt, dt, r, R, chunk_rows=128, stage_slots=2, world=w)
            for r in range(R)]
    assert ctxs[0].rd.num_chunks == 3 and ctxs[0].rd.phases == R.bit_length() - 1
    for it, M in enumerate((384, 256, 384, 128)):
        a_all, b_all = ks_inputs(R, M, N, kl, it, dt, 0.05)
        a_all = [x.cuda() for x in a_all]
        b_all = [x.cuda() for x in b_all]
        c_list = [torch.empty(M, N, dtype=dt, device="cuda") for _ in range(R)]
        gemm_ar_rd_emulated(ctxs, a_all, b_all, c_list)
        torch.cuda.synchronize()
        w.check()
        ref = sum(a_all[s].float() @ b_all[s].float().t() for s in range(R))
        for r in range(R):
            err = (c_list[r].float() - ref).abs().max().item()
            assert err < 3e-2, f"call {it} rank {r}: {err}"
            assert torch.equal(c_list[r], c_list[0]), "all ranks must hold bit-identical results"


def test_gemm_ar_rd_keeps_its_tiles(monkeypatch):
    """The panel GEMMs of several ranks take neither the tile rules of one rank nor its overlapped start."""
    from tridist_b200.ops.gemm_ar_rd import create_gemm_ar_rd_context, gemm_ar_rd_emulated
    C = _loaded_native()
    made = []
    create = C.gemm_plan_create
    monkeypatch.setattr(C, "gemm_plan_create", lambda d: (made.append(dict(d)), create(d))[1])
    R, M, N, K, dt = 2, 512, 8192, 8192, torch.bfloat16
    w = _emu(R)
    ctxs = [create_gemm_ar_rd_context(M, N, dt, dt, r, R, chunk_rows=256, stage_slots=2, world=w) for r in range(R)]
    a, b = [_rand((M, K), 31 + r, dt) for r in range(R)], [_rand((N, K), 33 + r, dt) for r in range(R)]
    c = [torch.empty((M, N), dtype=dt, device="cuda") for _ in range(R)]
    gemm_ar_rd_emulated(ctxs, a, b, c)
    torch.cuda.synchronize()
    w.check()
    assert len(made) == 4        # (256-row panels, which one rank alone would cut from 256-wide pair tiles)
    assert all(d["bn"] == 128 and not d["by_rounds"] and not d["early_start"] for d in made)
    ref = sum(a[s].float() @ b[s].float().t() for s in range(R))
    assert all((x.float() - ref).abs().max().item() < 2e-2 for x in c)


def test_gemm_ar_rd_ack_wait_runs_out():
    """A staging slot whose previous occupant is never acknowledged: the exchange kernel's wait
    runs out (20 ms limit), the kernel returns with a status record naming the ack ticket, the
    other virtual rank leaves through the abort word, and the context stays usable."""
    from tridist_b200.ops.gemm_ar_rd import create_gemm_ar_rd_context, gemm_ar_rd_emulated
    from tridist_b200.parallel.runtime import TriDistError
    from tridist_b200.utils.testing import ks_inputs
    R, M, N, kl = 2, 128, 256, 64
    w = _emu(R)
    w.timeout_ms = 20
    dt = torch.float16
    ctxs = [create_gemm_ar_rd_context(M, N, dt, dt, r, R, chunk_rows=128, stage_slots=1, world=w) for r in range(R)]
    a_all, b_all = [[x.cuda() for x in xs] for xs in ks_inputs(R, M, N, kl, 0, dt, 0.05)]
    c_list = [torch.empty(M, N, dtype=dt, device="cuda") for _ in range(R)]
    ctxs[1].rd.last_ticket_per_slot[0] = 1 << 19          # an occupant nobody will ever acknowledge
    gemm_ar_rd_emulated(ctxs, a_all, b_all, c_list)
    torch.cuda.synchronize()
    with pytest.raises(TriDistError, match="recursive-doubling ack ticket"):
        w.check()
    w.clear_status()
    for ctx in ctxs:                                       # forget the poisoned slot; tickets only grow
        ctx.rd.last_ticket_per_slot[0] = 0
    gemm_ar_rd_emulated(ctxs, a_all, b_all, c_list)
    torch.cuda.synchronize()
    w.check()
    ref = sum(a_all[s].float() @ b_all[s].float().t() for s in range(R))
    assert (c_list[0].float() - ref).abs().max().item() < 2e-2 and torch.equal(c_list[0], c_list[1])


def test_own_first_band_walk_emulated():
    """The walk the multicast all-gather uses (own rows, then row unit b of every other source before
    unit b + 1 of any) on virtual ranks with the bulk-copy push: only the order of the tiles changes,
    the result is bit-identical to the source-major walk."""
    from tridist_b200.ops.all_gather_gemm import ag_gemm_emulated, create_ag_gemm_intra_node_context
    R = 4
    w = _emu(R)
    dt = torch.bfloat16
    m_pr, K, n_pr = 1024, 256, 512
    ctxs = [create_ag_gemm_intra_node_context(m_pr * R, K, dt, dt, r, R, M_PER_CHUNK=256, world=w) for r in range(R)]
    a = [_rand((m_pr, K), 700 + r, dt) for r in range(R)]
    b = [_rand((n_pr, K), 710 + r, dt) for r in range(R)]
    ref = [torch.empty(m_pr * R, n_pr, dtype=dt, device="cuda") for _ in range(R)]
    ag_gemm_emulated(ctxs, a, b, ref)
    torch.cuda.synchronize()
    w.check()
    assert (ref[1].float() - torch.cat(a, 0).float() @ b[1].float().t()).abs().max().item() < 2e-2
    for ctx in ctxs:
        ctx.seg_bands, ctx.seg_own_first = -1, 1
        ctx.plans.clear()
    for it in range(2):                              # both workspace parities
        out = [torch.empty_like(x) for x in ref]
        ag_gemm_emulated(ctxs, a, b, out)
        torch.cuda.synchronize()
        w.check()
        for r in range(R):
            assert torch.equal(out[r], ref[r]), (it, r)


@pytest.mark.parametrize("T,E,H,topk,dt", [
    (1, 1, 8, 1, torch.float16),               # one pair, one 16-byte piece per row
    (64, 64, 4096, 8, torch.bfloat16),         # one piece per lane
    (257, 16, 264, 8, torch.float16),          # 2056 pairs: two metadata CTAs; 33 pieces per row
    (37, 16, 1032, 6, torch.bfloat16),         # topk not a multiple of 8, a run with one piece
    (300, 1024, 520, 32, torch.float16),       # most experts, most rows per token
    (16500, 64, 256, 8, torch.bfloat16),       # 132000 pairs: more than 64 metadata CTAs of 2048
])
def test_moe_round_of_any_size(T, E, H, topk, dt):
    """Two rounds on one context (fewer tokens in the second), some pairs routed nowhere: segments,
    rows and the weighted sum follow from the routing alone."""
    from tridist_b200.ops import (create_moe_a2a_intra_node_context, finalize_moe_a2a_context,
                                  moe_combine_intra_node_op, moe_dispatch_intra_node_op)
    w = _world1()
    ctx = create_moe_a2a_intra_node_context(E, H, dt, T, topk, 0, 1, BLOCK_H=H, world=w)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(T + H)
    for n in (T, max(1, T // 3)):
        tokens = torch.randn((n, H), generator=gen, dtype=dt, device="cuda")
        idx = torch.rand((n, E), generator=gen, device="cuda").topk(topk, dim=1).indices.to(torch.int32).contiguous()
        if n > 8:
            idx[3, topk - 1], idx[5, 0] = -1, E                # no such experts: these pairs are dropped
        wts = torch.rand((n, topk), generator=gen, device="cuda")
        total = moe_dispatch_intra_node_op(tokens, idx, ctx)
        kept = (idx >= 0) & (idx < E)
        counts = torch.bincount(idx[kept], minlength=E)
        assert int(total.item()) == int(kept.sum())
        assert torch.equal(ctx.recv_counts.flatten().long(), counts) and torch.equal(ctx.splits.long(), counts)
        first = torch.cumsum(counts, 0) - counts
        assert torch.equal(ctx.recv_seg.flatten().long(), first)
        sc = ctx.scatter_idx[:n].long()
        assert bool((sc[~kept] == -1).all())
        assert torch.equal(sc[kept].sort().values, torch.arange(int(kept.sum()), device="cuda"))   # a bijection
        e = idx[kept].long()
        assert bool(((sc[kept] >= first[e]) & (sc[kept] < first[e] + counts[e])).all())
        t_of = torch.arange(n, device="cuda").unsqueeze(1).expand_as(idx)[kept]
        assert torch.equal(ctx.recv[sc[kept]], tokens[t_of])
        ctx.out[:int(kept.sum())] = ctx.recv[:int(kept.sum())]
        out = torch.empty_like(tokens)
        moe_combine_intra_node_op(ctx, idx, out, wts)
        exact = tokens.double() * (wts.double() * kept).sum(1, keepdim=True)
        torch.cuda.synchronize()
        w.check()
        # one rounding to 16 bits (half an ulp: 2^-11 of fp16's 11-bit, 2^-8 of bf16's 8-bit significand, or
        # half the smallest subnormal of fp16) after topk fp32 sums
        half_ulp = 2.0 ** -11 if dt == torch.float16 else 2.0 ** -8
        bound = exact.abs() * (half_ulp + 2 * topk * 2.0 ** -24) + 2.0 ** -25
        assert bool(((out.double() - exact).abs() <= bound).all())
    finalize_moe_a2a_context(ctx)


@pytest.mark.parametrize("T,E,H,topk,dt", [
    (592, 16, 4096, 6, torch.bfloat16),        # ring: fewest tokens, stages of six rows
    (600, 32, 8192, 20, torch.float16),        # two runs of a row, a last group of four rows
    (700, 16, 4096, 5, torch.float16),         # by registers: a ring stage would be too empty
    (480, 16, 4104, 3, torch.bfloat16),        # four pieces per lane, the last run one piece wide
    (300, 64, 4096, 17, torch.float16),        # two pieces per lane, five groups of four rows
    (2500, 8, 512, 2, torch.bfloat16),
    (3000, 8, 1016, 1, torch.float16),
])
def test_moe_combine_by_ring_and_by_registers(T, E, H, topk, dt):
    test_moe_round_of_any_size(T, E, H, topk, dt)


def test_moe_context_scratch_is_one_allocation():
    """The six tensors that only the MoE kernels use share one allocation, each on a 16-byte boundary; with the
    five that callers read, a context makes six allocations (eight before the metadata had scratch of its own)."""
    from tridist_b200.ops import create_moe_a2a_intra_node_context, finalize_moe_a2a_context
    w = _world1()
    ctx = create_moe_a2a_intra_node_context(7, 64, torch.float16, 5, 3, 0, 1, BLOCK_H=64, world=w)
    own = [ctx.counters, ctx.dst_row_base, ctx.done_counter, ctx.meta_counter, ctx.slots, ctx.cta_base]
    assert len({t.untyped_storage().data_ptr() for t in own}) == 1
    spans = sorted((t.data_ptr(), t.data_ptr() + t.numel() * 4) for t in own)
    assert all(a[1] <= b[0] for a, b in zip(spans, spans[1:])) and all(lo % 16 == 0 for lo, _ in spans)
    read = [ctx.scatter_idx, ctx.splits, ctx.recv_seg, ctx.recv_counts, ctx.recv_total_t]
    assert len({t.untyped_storage().data_ptr() for t in own + read}) == 6
    finalize_moe_a2a_context(ctx)


@pytest.mark.parametrize("T,H,topk", [(9, 264, 3), (600, 4096, 6)])
def test_moe_combine_of_infinities_and_dropped_pairs(T, H, topk):
    """Both forms: an expert's infinity or NaN reaches the token, a pair without a row adds weight times zero
    (a NaN where that weight is infinite), and other tokens are untouched."""
    from tridist_b200.ops import (create_moe_a2a_intra_node_context, finalize_moe_a2a_context,
                                  moe_combine_intra_node_op, moe_dispatch_intra_node_op)
    E, dt = 16, torch.bfloat16
    w = _world1()
    ctx = create_moe_a2a_intra_node_context(E, H, dt, T, topk, 0, 1, BLOCK_H=H, world=w)
    tokens = _rand((T, H), 5, dt, scale=1.0)
    idx = torch.stack([torch.arange(topk, device="cuda") + t % (E - topk) for t in range(T)]).to(torch.int32)
    idx[4, 1] = -1
    idx[6, 2] = E
    wts = torch.rand((T, topk), device="cuda") + 0.5
    wts[6, 2] = float("inf")
    wts[7, 0] = 0.0
    moe_dispatch_intra_node_op(tokens, idx, ctx)
    sc = ctx.scatter_idx[:T].long()
    ctx.out[:T * topk] = ctx.recv[:T * topk]
    ctx.out[sc[2, 1], 7] = float("inf")
    ctx.out[sc[7, 0], 8] = float("inf")          # times a weight of zero
    ctx.out[sc[8, 2], H - 1] = float("nan")
    rows = torch.where((sc >= 0).unsqueeze(2), ctx.out[sc.clamp(min=0)].double(), 0.0)
    exact = (rows * wts.double().unsqueeze(2)).sum(1)
    out = torch.empty_like(tokens)
    moe_combine_intra_node_op(ctx, idx, out, wts)
    torch.cuda.synchronize()
    w.check()
    bad = ~torch.isfinite(exact)
    assert int(bad.sum()) == H + 3 and torch.equal(torch.isnan(out), torch.isnan(exact))
    assert torch.equal(out[torch.isinf(exact)].double(), exact[torch.isinf(exact)])
    # one rounding to bf16 (2^-8) after topk fp32 sums of values up to 2^3 or so
    diff = (out.double() - exact)[~bad].abs()
    assert bool((diff <= exact[~bad].abs() * 2.0 ** -8 + 2 * topk * 2.0 ** -24 * 16).all())
    finalize_moe_a2a_context(ctx)


def _gemm_bound(a, b, exact, dt):
    """Largest error of one rounding to 16 bits (half an ulp: 2^-11 of fp16's 11-bit, 2^-8 of bf16's 8-bit
    significand) after an fp32 sum of K products in any order."""
    half_ulp = 2.0 ** -11 if dt == torch.float16 else 2.0 ** -8
    return exact.abs() * half_ulp * 1.01 + a.shape[1] * 2.0 ** -23 * (a.abs().double() @ b.abs().double().t()) + 2.0 ** -24


@pytest.mark.parametrize("M,N,K,bn,swiglu", [
    (128, 256, 8192, 256, False),              # one tile, eight workers: one 32-column share each
    (64, 4096, 1376, 128, False),              # half a row block, last k-block short
    (128, 648, 4096, 128, False),              # last share of a row 8 columns wide
    (200, 2048, 4104, 256, False),             # CTA pairs, second row block ragged
    (600, 2304, 4096, 256, False),             # 512-row units, the second one mostly empty
    (1024, 2560, 2048, 256, False),
    (128, 640, 4096, 256, True),               # gate and up columns shared alike
    (456, 1000, 2048, 256, True),
])
def test_split_tiles_are_summed_by_their_workers(M, N, K, bn, swiglu):
    """A last round cut along K and summed by all the workers of a tile: within the rounding of one fp32
    sum of the 64-bit product, and the same bits on every call."""
    from tridist_b200.ops._gemm_common import gemm_nt
    for dt in (torch.float16, torch.bfloat16):
        a, b = _rand((M, K), 41, dt), _rand((2 * N if swiglu else N, K), 42, dt)
        out = gemm_nt(a, b, bn=bn, swiglu=swiglu)
        again = gemm_nt(a, b, bn=bn, swiglu=swiglu)
        torch.cuda.synchronize()
        exact = a.double() @ b.double().t()
        assert torch.equal(out, again)
        if swiglu:
            exact = F.silu(exact[:, :N]) * exact[:, N:]
            assert (out.double() - exact).abs().max().item() < TOL
        else:
            assert bool(((out.double() - exact).abs() <= _gemm_bound(a, b, exact, dt)).all())


@pytest.mark.parametrize("N,K", [(1024, 4096), (2304, 4096)])      # eight and four slices
def test_split_tiles_have_the_bits_of_a_sum_by_one_worker(N, K):
    """A tile summed by all its workers against the same tiles summed by slice 0: a one-shot all-reduce of two
    virtual ranks, the second with zeros, on as many CTAs per rank."""
    from tridist_b200.ops._gemm_common import gemm_nt
    from tridist_b200.ops.gemm_allreduce import create_gemm_ar_intra_node_context, gemm_ar_emulated
    R, M, dt = 2, 128, torch.bfloat16
    w = _emu(R)
    ctxs = [create_gemm_ar_intra_node_context(M, N, dt, dt, r, R, M_PER_CHUNK=64, world=w) for r in range(R)]
    a, b = _rand((M, K), 91, dt), _rand((N, K), 92, dt)
    c = [torch.empty((M, N), dtype=dt, device="cuda") for _ in range(R)]
    gemm_ar_emulated(ctxs, [a, torch.zeros_like(a)], [b, b], c, mode="one_shot")
    out = gemm_nt(a, b, bn=128, max_ctas=74)
    torch.cuda.synchronize()
    w.check()
    assert torch.equal(out, c[0])


def test_split_k_on_several_streams_and_under_capture():
    """Launches that overlap on different streams do not share scratch; a capture on a stream that has not been used before works (what its replays
    compute with new inputs: test_captured_split_k_sums_the_partials_of_its_own_replay)."""
    from tridist_b200.ops._gemm_common import gemm_nt
    M, N, K, dt = 128, 4096, 4096, torch.bfloat16
    b = _rand((N, K), 52, dt)
    a = [_rand((M, K), 60 + i, dt) for i in range(6)]
    exact = [x.double() @ b.double().t() for x in a]
    ref = [gemm_nt(x, b).clone() for x in a]
    outs = [torch.empty((M, N), dtype=dt, device="cuda") for _ in a]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in a]
    for _ in range(20):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                gemm_nt(a[i], b, out=outs[i])
    torch.cuda.synchronize()
    for i in range(len(a)):
        assert bool(((outs[i].double() - exact[i]).abs() <= _gemm_bound(a[i], b, exact[i], dt)).all()), i
    assert all(torch.equal(o, r) for o, r in zip(outs, ref))
    graph = torch.cuda.CUDAGraph()
    outs[0].zero_()
    with torch.cuda.graph(graph):
        gemm_nt(a[0], b, out=outs[0])
        gemm_nt(a[0], b, out=outs[1])
    graph.replay()
    graph.replay()
    torch.cuda.synchronize()
    for o in outs[:2]:
        assert bool(((o.double() - exact[0]).abs() <= _gemm_bound(a[0], b, exact[0], dt)).all())


def test_split_k_on_more_streams_than_keep_their_scratch():
    """40 streams in turn, a small shape and then one that needs more scratch, all pending at once: every
    stream computes the bits of the default stream."""
    from tridist_b200.ops._gemm_common import gemm_nt
    dt = torch.bfloat16
    streams = [torch.cuda.Stream(priority=-(i & 1)) for i in range(40)]
    for M, N, K, bn in ((64, 512, 4096, 128), (128, 4096, 4096, 128), (600, 2304, 4096, 256)):
        b = _rand((N, K), 53, dt)
        a = [_rand((M, K), 70 + i, dt) for i in range(3)]
        ref = [gemm_nt(x, b, bn=bn) for x in a]
        outs = [torch.empty((M, N), dtype=dt, device="cuda") for _ in streams]
        torch.cuda.synchronize()
        for _ in range(4):
            for i, s in enumerate(streams):
                with torch.cuda.stream(s):
                    gemm_nt(a[i % 3], b, out=outs[i], bn=bn)
        torch.cuda.synchronize()
        for i, o in enumerate(outs):
            assert torch.equal(o, ref[i % 3]), (M, i)


@pytest.mark.parametrize("M,N,K,bn", [(128, 4096, 4096, 128),      # every tile cut: 32 x 4 slices
                                      (600, 2304, 4096, 256)])     # CTA pairs
def test_captured_split_k_sums_the_partials_of_its_own_replay(M, N, K, bn):
    """A captured GEMM that is cut along K, and two in one graph whose launches share scratch, replayed
    over other inputs each time, an eager call between two replays, and two graphs of one capture
    stream replayed at the same time: the bits of the eager call, within the rounding of the 64-bit
    product."""
    from tridist_b200.ops._gemm_common import OP_PLAIN, SCHED_NATURAL, gemm_nt
    dt = torch.bfloat16
    assert _loaded_native().splitk_dump(dict(op=OP_PLAIN, sched=SCHED_NATURAL, bn=bn, R=1, rank=0, M=M, N=N, K=K,
                                             by_rounds=1), 148)
    b = _rand((N, K), 52, dt)
    a = [torch.zeros((M, K), dtype=dt, device="cuda") for _ in range(3)]
    outs = [torch.empty((M, N), dtype=dt, device="cuda") for _ in range(3)]
    gemm_nt(a[0], b, bn=bn)                             # (the first call of a process allocates its status block)
    torch.cuda.synchronize()
    capture = torch.cuda.Stream()
    one, two = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(one, stream=capture):
        gemm_nt(a[0], b, out=outs[0], bn=bn)
    with torch.cuda.graph(two, stream=capture):
        gemm_nt(a[1], b, out=outs[1], bn=bn)
        gemm_nt(a[2], b, out=outs[2], bn=bn)
    replay = [torch.cuda.Stream(), torch.cuda.Stream()]
    for it in range(25):
        new = [_rand((M, K), 100 + 3 * it + i, dt) for i in range(3)]
        ref = [gemm_nt(x, b, bn=bn) for x in new]
        for i in range(3):
            a[i].copy_(new[i])
            outs[i].zero_()
        torch.cuda.synchronize()
        for graph, s in zip((one, two), replay):
            with torch.cuda.stream(s):
                graph.replay()
        between = gemm_nt(new[0], b, bn=bn)
        torch.cuda.synchronize()
        assert torch.equal(between, ref[0])
        for i in range(3):
            exact = new[i].double() @ b.double().t()
            assert torch.equal(outs[i], ref[i]), (it, i)
            assert bool(((outs[i].double() - exact).abs() <= _gemm_bound(new[i], b, exact, dt)).all()), (it, i)
    del one, two                                 # their scratch serves the next capture
    again = torch.cuda.CUDAGraph()
    with torch.cuda.graph(again, stream=capture):
        gemm_nt(a[0], b, out=outs[0], bn=bn)
    outs[0].zero_()
    again.replay()
    torch.cuda.synchronize()
    assert torch.equal(outs[0], ref[0])


def test_split_tiles_meet_again_after_a_launch_that_gave_up(monkeypatch):
    """Virtual rank 1 does not push, so rank 0's workers leave their cut tiles without having met
    (20 ms limit); the next launches on the same scratch, over other inputs, sum what they should."""
    from tridist_b200.ops._gemm_common import gemm_nt
    from tridist_b200.ops.all_gather_gemm import ag_gemm_emulated, create_ag_gemm_intra_node_context
    from tridist_b200.parallel.runtime import TriDistError
    monkeypatch.setenv("TRIDIST_WAIT_TIMEOUT_MS", "20")
    R, dt = 2, torch.bfloat16
    w = _emu(R)
    m_pr, K, N = 256, 4096, 512
    ctxs = [create_ag_gemm_intra_node_context(m_pr * R, K, dt, dt, r, R, M_PER_CHUNK=128, world=w) for r in range(R)]
    b = [_rand((N, K), 195 + r, dt) for r in range(R)]
    c = [torch.empty(m_pr * R, N, dtype=dt, device="cuda") for _ in range(R)]
    for it in range(3):
        a = [_rand((m_pr, K), 190 + 2 * it + r, dt) for r in range(R)]
        if it == 1:
            ag_gemm_emulated(ctxs, a, b, c, mute_ranks=[1])
            torch.cuda.synchronize()
            with pytest.raises(TriDistError, match="all-gather chunk ticket"):
                w.check()
            w.clear_status()
        ag_gemm_emulated(ctxs, a, b, c)
        plain = gemm_nt(a[0], b[0])
        torch.cuda.synchronize()
        w.check()
        full = torch.cat(a, 0)
        for r in range(R):
            exact = full.double() @ b[r].double().t()
            assert bool(((c[r].double() - exact).abs() <= _gemm_bound(full, b[r], exact, dt)).all()), (it, r)
        exact = a[0].double() @ b[0].double().t()
        assert bool(((plain.double() - exact).abs() <= _gemm_bound(a[0], b[0], exact, dt)).all()), it


@pytest.mark.parametrize("M,N,K,swiglu", [(128, 512, 1024, False), (384, 2048, 4096, False), (640, 1024, 512, True),
                                          (1152, 2048, 4096, False), (1920, 4096, 512, True)])
def test_local_ag_gemm_with_an_odd_number_of_row_blocks(M, N, K, swiglu):
    """One rank, CTA pairs whose second CTA stands past the last row block: it waits for no shard."""
    from tridist_b200.ops import (ag_gemm_intra_node_op, create_ag_gemm_intra_node_context, finalize_ag_gemm_context)
    w = _world1()
    dt = torch.bfloat16
    ctx = create_ag_gemm_intra_node_context(M, K, dt, dt, 0, 1, M_PER_CHUNK=128, world=w)
    a, b = _rand((M, K), 71, dt), _rand((2 * N if swiglu else N, K), 72, dt)
    c = torch.empty((M, N), dtype=dt, device="cuda")
    ag_gemm_intra_node_op(a, b, c, ctx, fuse_swiglu=swiglu)
    torch.cuda.synchronize()
    w.check()
    exact = a.double() @ b.double().t()
    if swiglu:
        exact = F.silu(exact[:, :N]) * exact[:, N:]
        assert (c.double() - exact).abs().max().item() < TOL
    else:
        assert bool(((c.double() - exact).abs() <= _gemm_bound(a, b, exact, dt)).all())
    finalize_ag_gemm_context(ctx)

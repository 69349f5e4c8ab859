"""All-gather GEMM whose transfer gives up, emulated ranks on one GPU."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("transport", ["push", "pull"])
def test_transfer_that_gives_up(transport):
    """With every rank's abort word raised the pushing threads leave the first wait that looks at it, with pieces on
    their way into the ring: the call reports it or is complete, and contexts made after it are right."""
    from tridist_b200.ops.all_gather_gemm import ag_gemm_emulated, create_ag_gemm_intra_node_context
    from tridist_b200.parallel.runtime import EmulatedWorld, native
    C, R, dt = native(), 2, torch.bfloat16
    m_pr, K, N = 1024, 4096, 512
    g = torch.Generator(device="cuda").manual_seed(7)
    a, b = [[(torch.randn((n, K), generator=g, device="cuda") * 0.1).to(dt) for _ in range(R)] for n in (m_pr, N)]
    full = torch.cat(a, 0).double()
    for raised in (True, True, False):
        w = EmulatedWorld(R)
        ctxs = [create_ag_gemm_intra_node_context(m_pr * R, K, dt, dt, r, R, M_PER_CHUNK=128, world=w, transport=transport)
                for r in range(R)]
        c = [torch.zeros((m_pr * R, N), dtype=dt, device="cuda") for _ in range(R)]
        if raised:
            for r in range(R):
                C.fill_u32(w.abort_word_of(r), 1, 5)
        ag_gemm_emulated(ctxs, a, b, c)
        torch.cuda.synchronize()
        if raised and w.status()[0] != 0:
            assert w.status()[0] == 5
            w.clear_status()
            continue
        w.check()
        for r in range(R):
            exact = full @ b[r].double().t()
            assert (c[r].double() - exact).norm() <= 2.0 ** -8 * exact.norm()

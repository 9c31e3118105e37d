"""Launches of one rank that come up while the one before ends: nothing is read before it is written, nor written while it is read."""
import os

import pytest
import torch

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("tokens", [3, 700])  # one wave of CTAs, several
def test_chain_eager_and_captured(tokens):
    """Norm, cast, GEMM, MoE and copies in a row, each on the output of the one before and over what that one has read;
    in a graph and eagerly the same bits as with a wait after every step."""
    os.environ.setdefault("UCCL_BOOTSTRAP_IFNAME", "lo")
    from unified_ccl_b200 import Communicator
    from unified_ccl_b200.ops import gemm_bf16
    from unified_ccl_b200.parallel import MoeDispatcher, allreduce_residual_rmsnorm

    comm = Communicator(0, 1)
    H, K = 512, 4
    g = torch.Generator(device="cuda").manual_seed(tokens)
    new = lambda *s, dtype=torch.bfloat16: torch.empty(*s, device="cuda", dtype=dtype)  # noqa: E731
    x0, res0 = (torch.randn(tokens, H, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    gamma = torch.ones(H, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(H, H, device="cuda", generator=g) * 0.04).to(torch.bfloat16)
    w2 = (torch.randn(2 * H, H, device="cuda", generator=g) * 0.04).to(torch.bfloat16)
    idx = torch.randint(0, 8, (tokens, K), device="cuda", generator=g, dtype=torch.int32)
    weight = torch.rand(tokens, K, device="cuda", generator=g)
    disp = MoeDispatcher(comm, tokens, H, 8, K)
    x, res, n, y, f, z, h = new(tokens, H), new(tokens, H), new(tokens, H), new(tokens, H), new(tokens, H, dtype=torch.float32), new(tokens, H), new(tokens, H)
    got = new(disp.recv_scale.numel(), dtype=torch.float32)
    fp8, scales = new(tokens * H, dtype=torch.float8_e4m3fn), new(tokens * H // 128, dtype=torch.float32)

    def steps():
        yield lambda: allreduce_residual_rmsnorm(comm, x, res, gamma, out=n)       # res in place
        yield lambda: gemm_bf16(n, w2, out=h, swiglu=True)
        yield lambda: gemm_bf16(h, w, out=y)
        yield lambda: comm.reduce_scatter_cast(y.view(-1), f.view(-1), 0.5)
        yield lambda: comm.reduce_scatter_cast(f.view(-1), z.view(-1), 2.0)
        yield lambda: comm.allreduce_cast(z.view(-1), fp8, 1.0, scales=scales)
        yield lambda: comm.reduce_scatter(z.view(-1), y.view(-1))                  # y has just been read
        yield lambda: disp.dispatch(y, idx)
        yield lambda: comm.reduce_scatter_cast(disp.recv_scale.view(-1), got, 1.0)  # bulk stores of the launch before
        yield lambda: allreduce_residual_rmsnorm(comm, y, res, gamma, out=x, residual_out=y)
        yield lambda: disp.expert_out[0].copy_(disp.recv_x[0])                     # a row's answer is the row, wherever it lies
        yield lambda: disp.combine(weight, out=n)
        yield lambda: allreduce_residual_rmsnorm(comm, n, y, gamma, out=x)
        yield lambda: comm.allgather(x.view(-1), n.view(-1))

    def run(wait):
        x.copy_(x0), res.copy_(res0)
        for _ in range(6):
            for step in steps():
                step()
                if wait:
                    torch.cuda.synchronize()

    # rows lie in the order of their arrival, another one each time
    arrived = lambda: got.sort().values  # noqa: E731
    out = (x, res, n, y, f, z, h, fp8.view(torch.uint8), scales)
    run(True)
    want, scale_rows = [t.clone() for t in out], arrived()
    for _ in range(3):
        for t in out:
            t.zero_()
        run(False)
        torch.cuda.synchronize()
        assert all(torch.equal(p, q) for p, q in zip(out, want)) and torch.equal(arrived(), scale_rows)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(False)
    for _ in range(3):
        for t in out:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(p, q) for p, q in zip(out, want)) and torch.equal(arrived(), scale_rows)
    del graph
    disp.close()
    comm.destroy()

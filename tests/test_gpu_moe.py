"""MoE routing, dispatch (+permute) and combine (+weighted sum) against PyTorch references."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_moe_world_of_one():
    sys.path.insert(0, HERE)
    from moe_worker import run
    fails = run(0, 1, torch.device("cuda", 0))
    assert not fails, fails


@pytest.mark.parametrize("tokens,hidden,experts,topk", [(1, 16, 32, 1), (1, 7168, 32, 8), (3, 1040, 64, 3), (300, 528, 512, 8), (2371, 48, 256, 2)])
def test_exchange_pieces(tokens, hidden, experts, topk):
    # rows are cut into 1 KiB pieces over all warps: one piece in all, a remainder of a piece, fewer and more pieces than warps
    sys.path.insert(0, HERE)
    from moe_worker import run
    fails = run(0, 1, torch.device("cuda", 0), tokens=tokens, hidden=hidden, experts=experts, topk=topk, iters=2)
    assert not fails, fails


def test_layers_without_tokens_and_token_counts_that_do_not_match():
    # a layer with no tokens sends none of the layer before it, and x and y have to fit what was routed
    from purlin_b200.parallel.expert_parallel import ExpertParallelContext
    dev = torch.device("cuda", 0)
    tokens, hidden, experts, topk = 48, 64, 32, 2
    ep = ExpertParallelContext(None, dev, max_tokens=64, hidden=hidden, experts=experts, topk=topk)
    g = torch.Generator(device=dev).manual_seed(4)
    x = torch.randn(tokens, hidden, generator=g, device=dev).to(torch.bfloat16)
    logits = torch.randn(tokens, experts, generator=g, device=dev)
    for n in (tokens, 0, tokens, 0, 1):
        for empty_plan in (False, True):
            if empty_plan and n == 0:
                ep.plan(ep.topk_idx[:0], ep.topk_weight[:0])
            else:
                ep.route(logits[:n])
            ep.recv_rows().fill_(3.0)
            rows, counts = ep.dispatch(x[:n])
            assert int(counts[:-1].sum()) == int(counts[-1]) == n * topk
            assert (rows[n * topk:] == 3).all()
            ep.out_rows().copy_(rows)
            y = ep.combine(n)
            ep.check()
            assert y.shape == (n, hidden) and torch.allclose(y.float(), x[:n].float(), rtol=2 ** -7, atol=1e-6)    # the gate weights sum to one
    ep.route(logits)
    with pytest.raises(RuntimeError, match="fewer tokens than were routed"):
        ep.dispatch(x[:8])
    padded = torch.cat([x, x[:16]])
    rows, counts = ep.dispatch(padded)                       # rows past the routed ones are allowed and not sent
    assert int(counts[-1]) == tokens * topk
    with pytest.raises(RuntimeError, match="more tokens than the matching dispatch sent"):
        ep.combine(64)
    ep.out_rows().copy_(rows)
    assert torch.allclose(ep.combine(8).float(), x[:8].float(), rtol=2 ** -7, atol=1e-6)
    ep.check()
    ep.close()


@pytest.mark.parametrize("experts,topk", [(32, 2), (64, 8)])
def test_a_captured_exchange_follows_the_plan_of_its_replay(experts, topk):
    # a decode server captures dispatch -> experts -> combine for its largest batch and replays it after plans of fewer tokens
    from purlin_b200.parallel.expert_parallel import ExpertParallelContext
    dev = torch.device("cuda", 0)
    most, hidden = 64, 1040
    ep = ExpertParallelContext(None, dev, max_tokens=most, hidden=hidden, experts=experts, topk=topk)
    g = torch.Generator(device=dev).manual_seed(6)
    x = torch.randn(most, hidden, generator=g, device=dev).to(torch.bfloat16)
    y = torch.empty_like(x)

    def layer():
        rows, _ = ep.dispatch(x)
        ep.out_rows().copy_(rows)
        ep.combine(most, y)

    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ep.route(torch.randn(most, experts, generator=g, device=dev))
        layer()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            layer()
        for n, routed in ((most, True), (8, False), (most, False), (33, True), (1, True), (0, False), (17, False)):
            logits = torch.randn(n, experts, generator=g, device=dev)
            if routed and n:
                ep.route(logits)
            else:
                ep.plan(logits.topk(topk, dim=1).indices.to(torch.int32), torch.full((n, topk), 1.0 / topk, device=dev))
            ep.recv_rows().fill_(3.0)
            graph.replay()
            torch.cuda.synchronize()
            ep.check()
            assert int(ep.recv_counts[-1]) == n * topk
            assert (ep.recv_rows()[n * topk:] == 3).all()                                           # rows past the routed ones are not sent
            assert torch.allclose(y[:n].float(), x[:n].float(), rtol=2 ** -7, atol=1e-6)             # the gate weights sum to one
    del graph
    ep.close()


def test_check_sees_a_wait_that_ran_out_in_the_experts_gemm():
    # a grouped GEMM over a k so long that the wait for its accumulator outlasts a limit of 1 ns, reporting where the block's report
    from purlin_b200.models.moe_block import ExpertParallelMoE
    from purlin_b200.ops.gemm import grouped_gemm
    moe = ExpertParallelMoE(hidden=128, intermediate=64, experts=32, topk=2, max_tokens=16, device="cuda:0")
    x = torch.ones(16, 128, device="cuda", dtype=torch.bfloat16)
    y = moe(x)
    moe.ep.check()
    a, w = torch.zeros(8, 1 << 21, device="cuda", dtype=torch.bfloat16), torch.zeros(1, 64, 1 << 21, device="cuda", dtype=torch.bfloat16)
    out = torch.zeros(8, 64, device="cuda", dtype=torch.bfloat16)
    grouped_gemm(a, w, torch.tensor([8], dtype=torch.int32, device="cuda"), 8, out, status_ptr=moe.ep.status_ptr, timeout_ns=1)
    with pytest.raises(RuntimeError, match="inside a GEMM of the experts timed out"):
        moe.ep.check()
    assert torch.equal(moe(x), y)                            # the report is cleared, the next layer runs
    moe.ep.check()
    moe.ep.close()


@pytest.mark.multigpu
def test_moe_all_gpus():
    n = torch.cuda.device_count()
    n = 8 if n >= 8 else 4 if n >= 4 else 2
    env = dict(os.environ)
    env.setdefault("NCCL_NVLS_ENABLE", "0")
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", f"--nproc-per-node={n}",
           "--master-addr", "127.0.0.1", "--master-port", "29585", os.path.join(HERE, "moe_worker.py")]
    res = subprocess.run(cmd, env=env, capture_output=True, text=True, timeout=600)
    sys.stdout.write(res.stdout[-3000:])
    sys.stderr.write(res.stderr[-3000:])
    assert res.returncode == 0


def test_moe_block_world_of_one_matches_fp32_reference():
    from purlin_b200.models.moe_block import ExpertParallelMoE
    moe = ExpertParallelMoE(hidden=512, intermediate=256, experts=32, topk=4, max_tokens=256, device="cuda:0", capacity_factor=4.0)
    g = torch.Generator(device="cuda:0").manual_seed(5)
    x = torch.randn(256, 512, generator=g, device="cuda:0").to(torch.bfloat16)
    y = moe(x)
    moe.ep.check()
    ref = moe.reference(x)
    err = (y.float() - ref).abs().max().item()
    assert err <= 3e-2 * ref.abs().max().item() + 2e-3, err
    y2 = moe(x)            # a second layer call reuses the buffers
    moe.ep.check()
    assert torch.equal(y, y2)


@pytest.mark.parametrize("tokens", [1, 7, 48, 120])
def test_moe_block_decode_batches_match_the_fp32_reference(tokens):
    # up to a dozen rows per expert the few-rows kernel computes the experts, above it the one on CTA pairs (15 rows at 120 tokens)
    from purlin_b200.models.moe_block import ExpertParallelMoE
    moe = ExpertParallelMoE(hidden=1024, intermediate=512, experts=32, topk=4, max_tokens=120, device="cuda:0", capacity_factor=1.0)
    g = torch.Generator(device="cuda:0").manual_seed(tokens)
    x = torch.randn(tokens, 1024, generator=g, device="cuda:0").to(torch.bfloat16)
    y = moe(x)
    moe.ep.check()
    ref = moe.reference(x)
    assert (y.float() - ref).abs().max().item() <= 3e-2 * ref.abs().max().item() + 2e-3
    stacked = moe.w_gu, moe.w_down
    moe.w_gu, moe.w_down = list(moe.w_gu), list(moe.w_down)                       # expert by expert: the same products
    assert ((moe(x).float() - y.float()).abs() <= 2 ** -6 * y.float().abs() + 2 ** -7 * ref.abs().max()).all()
    moe.w_gu, moe.w_down = stacked
    moe.ep.close()


def test_route_kernel_is_total_and_matches_the_host_restatement():
    """Rows of NaN, +inf, -inf and rows with fewer than top-k usable logits: the kernel must return k distinct experts
    inside [0, experts) with finite weights, equal to the host restatement of the same arithmetic."""
    sys.path.insert(0, HERE)
    from test_moe_route_cpu import route_host
    from purlin_b200.parallel.expert_parallel import ExpertParallelContext
    dev = torch.device("cuda", 0)
    tokens, experts, topk = 64, 64, 8
    ep = ExpertParallelContext(None, dev, max_tokens=tokens, hidden=256, experts=experts, topk=topk)
    g = torch.Generator(device=dev).manual_seed(2)
    logits = torch.randn(tokens, experts, generator=g, device=dev)
    logits[0] = float("nan")
    logits[1] = float("inf")
    logits[2] = float("-inf")
    logits[3] = float("-inf"); logits[3, 5] = 1.0; logits[3, 9] = 2.0
    logits[4, 7] = float("nan")
    logits[5, 11] = float("inf")
    idx, w = ep.route(logits)
    torch.cuda.synchronize()
    hi, hw = route_host(logits.cpu().numpy(), topk)
    assert int(idx.min()) >= 0 and int(idx.max()) < experts
    assert torch.equal(idx.cpu(), torch.from_numpy(hi))
    assert torch.isfinite(w).all()
    assert torch.allclose(w.cpu(), torch.from_numpy(hw), rtol=1e-4, atol=1e-6)
    x = torch.randn(tokens, 256, generator=g, device=dev).to(torch.bfloat16)
    ep.dispatch(x)          # ids are in range, so nothing is stored out of bounds
    ep.check()
    ep.close()

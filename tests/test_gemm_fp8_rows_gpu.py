"""fp8 down projection in its form for many rows per expert: the blocks of 128 token rows and their
half-fetched ends, the column and K tails, the stores to peers.  The sizes are such that the rule
takes that form (its tiles fill whole waves and it has half as many of them)."""

import pytest
import torch

from pplx_kernels_b200.models.configs import MoEModelConfig
from pplx_kernels_b200.models.moe import MoELayerFP8, moe_reference_fp8
from pplx_kernels_b200.ops.grouped_gemm import (
    grouped_gemm_fp8,
    grouped_gemm_fp8_reference,
    quantize_weight_blocks,
)
from pplx_kernels_b200.ops.quant import per_token_block_quant
from pplx_kernels_b200.utils.testing import as_index_tensor, routing

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [
    [1, 63, 64, 65, 127, 128, 129, 192, 193, 257],
    [257, 256, 255, 0, 0, 191, 2, 130, 66, 0],
])
def test_plain(counts):
    E, rows, K, N = 10, 257, 4112, 2064
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(3)
    x = torch.randn(E * rows, K, generator=g, device=dev)
    # Scales that differ from row to row and from K block to K block: a wrong one shows as a factor.
    x *= torch.exp2(torch.randint(-3, 4, (E * rows, 33), generator=g, device=dev).float()
                    ).repeat_interleave(128, dim=1)[:, :K]
    xq, sa = per_token_block_quant(x)
    xq, sa = xq.view(E, rows, K), sa.view(E, rows, -1)
    wq, sw = quantize_weight_blocks(torch.randn(E, N, K, generator=g, device=dev) * K ** -0.5)
    cnt = torch.tensor(counts, dtype=torch.int32, device=dev)
    # Rows beyond an expert's count must neither be written nor reach another row's result.
    for e, m in enumerate(counts):
        sa[e, m:] = float("nan")
    out = torch.full((E, rows, N), float("nan"), dtype=torch.bfloat16, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    grouped_gemm_fp8(xq, sa, wq, sw, cnt, out=out, status=status, expected_rows=E * rows)
    want = grouped_gemm_fp8_reference(xq, sa, wq, sw, cnt)
    assert int(status.item()) == 0
    for e, m in enumerate(counts):
        # fp32 sums of exact products, one bf16 rounding (2^-9), and the order of up to K sums
        err = (out[e, :m].float() - want[e, :m]).abs()
        bound = 2 ** -8 * want[e, :m].abs() + 1e-5 * want[e, :m].abs().amax() if m else err
        assert (err <= bound).all(), (e, m, float(err.max()))
        assert torch.isnan(out[e, m:].float()).all()


@pytest.mark.parametrize("world,dp_size", [(1, 1), (2, 1), (2, 2)])
def test_stores_to_peers(world, dp_size):
    """The fused layer, all ranks on one GPU, each step launched for all ranks before the next."""
    import pplx_kernels_b200 as pk

    cfg, m = MoEModelConfig("rows", 8, 2, 4096, 512), 1200 // world
    dev = torch.device("cuda", 0)
    atas = pk.AllToAll.local_world(m, cfg.num_experts, cfg.experts_per_token, world, dp_size,
                                   cfg.hidden_dim, cfg.hidden_dim, 32 * 4)
    layers = [MoELayerFP8(cfg, m, rank=r, world_size=world, dp_size=dp_size, device=dev,
                          ata=atas[r], init_std=0.05) for r in range(world)]
    gen = torch.Generator().manual_seed(4)
    data = []
    for _ in range(world // dp_size):
        x = torch.randn(m, cfg.hidden_dim, generator=gen).to(torch.bfloat16).to(dev)
        idx = routing(m, cfg.num_experts, cfg.experts_per_token, gen)
        w = torch.softmax(torch.randn(m, cfg.experts_per_token, generator=gen), dim=-1).to(dev)
        data.append((x, idx, w))
    mine = [data[r // dp_size] for r in range(world)]
    idx_dev = [as_index_tensor(d[1], dev) for d in mine]
    outs = [torch.full((m, cfg.hidden_dim), float("nan"), dtype=torch.bfloat16, device=dev)
            for _ in range(world)]
    deq = [l.dequantized_weights() for l in layers]
    w13, w2 = torch.cat([d[0] for d in deq]), torch.cat([d[1] for d in deq])
    for _ in range(2):
        for o in outs:
            o.fill_(float("nan"))
        pk.fused_dispatch_group(atas, [d[0] for d in mine], idx_dev, [None] * world, quantize=True)
        for l in layers:
            l.ata.fused_up_fp8(l.w13_q, l.w13_s, l.h, l.h_scale, l.counts, l.gemm_status)
        for l in layers:
            l.ata.fused_down_fp8(l.h, l.h_scale, l.w2_q, l.w2_s, l.gemm_status)
        pk.combine_group(atas, outs, idx_dev, [d[2] for d in mine], [l.expert_y for l in layers],
                         [None] * world, do_send=False, do_recv=True)
        torch.cuda.synchronize()
        for r, l in enumerate(layers):
            l.check_status()
            x, idx, w = mine[r]
            want = moe_reference_fp8(x, idx.to(dev), w, w13, w2)
            err = (outs[r].float() - want).abs()
            assert (err <= 0.06 * want.abs() + 0.03 * want.abs().amax()).all(), err.max()
    for l in layers:
        l.destroy()

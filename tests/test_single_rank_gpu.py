"""Dispatch and combine in a world of one rank (no staging, rows found by token order)."""

import pytest
import torch

import pplx_kernels_b200 as pk
from pplx_kernels_b200.utils.testing import MoEConfig
from pplx_kernels_b200.utils.verify import (
    RankBuffers,
    run_local_world,
    verify_combine,
    verify_dispatch,
    world_inputs,
)

pytestmark = pytest.mark.gpu


# Chunks of 512 bytes: rows below, at and just above one; entries (tokens x top-k) around the 512
# that a block ranks at a time, above 32 per token, and above 512 per token.
@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("tokens,experts,topk,hidden,in_dtype,max_blocks", [
    (1, 8, 1, 16, torch.float8_e4m3fn, 0),
    (1, 256, 8, 7168, torch.float8_e4m3fn, 0),
    (3, 4, 4, 512, torch.float8_e4m3fn, 1),
    (37, 40, 33, 528, torch.float8_e4m3fn, 0),
    (129, 16, 4, 264, torch.bfloat16, 1),
    (200, 64, 6, 2048, torch.bfloat16, 3),
    (301, 8, 2, 1032, torch.bfloat16, 0),
    (5, 600, 520, 64, torch.bfloat16, 2),
    (1500, 64, 6, 640, torch.float8_e4m3fn, 0),
])
def test_sizes(tokens, experts, topk, hidden, in_dtype, max_blocks, split):
    cfg = MoEConfig(num_experts=experts, experts_per_token=topk, hidden_dim=hidden,
                    max_num_tokens=tokens + 2, in_dtype=in_dtype)
    run_local_world(cfg, world=1, dp_size=1, seed=tokens, num_tokens=tokens, max_blocks=max_blocks,
                    split=split, iterations=2)
    run_local_world(cfg, world=1, dp_size=1, seed=tokens + 1, num_tokens=tokens, split=split,
                    use_bound_m=False, y_dtype=torch.float32)


def test_no_tokens():
    cfg = MoEConfig(num_experts=8, experts_per_token=2, hidden_dim=64, max_num_tokens=4)
    for split in (False, True):
        run_local_world(cfg, world=1, dp_size=1, seed=3, num_tokens=0, split=split, iterations=2)


def test_whole_calls_and_halves_mix():
    """Each of dispatch and combine may be one call or two, whatever the other was."""
    cfg = MoEConfig(num_experts=16, experts_per_token=4, hidden_dim=1024, max_num_tokens=48,
                    in_dtype=torch.float8_e4m3fn)
    device = torch.device("cuda", 0)
    ata = pk.AllToAll.intranode(cfg.max_num_tokens, cfg.num_experts, cfg.experts_per_token, 0, 1, 1,
                                cfg.hidden_dim, cfg.hidden_dim_bytes, cfg.hidden_dim_scale_bytes)
    ata.set_timeout_ms(3000)
    for n, (d_split, c_split) in enumerate([(False, True), (True, False), (False, False),
                                            (True, True), (False, True)]):
        inputs = world_inputs(cfg, 1, 1, seed=100 + n)
        buf = RankBuffers(cfg, 1, 1, inputs[0], device)
        d_args = (buf.counts, buf.expert_x, buf.expert_scale, buf.x, buf.x_scale, buf.indices,
                  buf.bound_m)
        for kw in ({"do_recv": False}, {"do_send": False}) if d_split else ({},):
            ata.dispatch(*d_args, **kw)
        torch.cuda.synchronize()
        verify_dispatch(cfg, inputs, 1, 0, buf)
        buf.make_expert_y()
        c_args = (buf.out, buf.indices, buf.weights, buf.expert_y, buf.bound_m)
        for kw in ({"do_recv": False}, {"do_send": False}) if c_split else ({},):
            ata.combine(*c_args, **kw)
        torch.cuda.synchronize()
        ata.check_status()
        verify_combine(cfg, inputs, 0, buf)
    ata.destroy()


def test_a_token_without_an_expert_is_reported():
    cfg = MoEConfig(num_experts=8, experts_per_token=2, hidden_dim=64, max_num_tokens=4)
    device = torch.device("cuda", 0)
    ata = pk.AllToAll.intranode(cfg.max_num_tokens, cfg.num_experts, cfg.experts_per_token, 0, 1, 1,
                                cfg.hidden_dim, cfg.hidden_dim_bytes, cfg.hidden_dim_scale_bytes)
    buf = RankBuffers(cfg, 1, 1, world_inputs(cfg, 1, 1, seed=7, num_tokens=4)[0], device)
    bad = buf.indices.view(torch.int32).clone()
    bad[2, 1] = cfg.num_experts
    ata.dispatch(buf.counts, buf.expert_x, None, buf.x, None, bad.view(torch.uint32), buf.bound_m)
    ata.combine(buf.out, buf.indices, buf.weights, buf.make_expert_y(), buf.bound_m)
    torch.cuda.synchronize()
    st = ata.status()
    assert (st["code"], st["peer"]) == (2, 2)
    assert torch.isnan(buf.out[2].float()).all() and not torch.isnan(buf.out[3].float()).any()
    ata.destroy()

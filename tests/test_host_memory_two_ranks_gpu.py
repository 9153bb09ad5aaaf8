"""Pinned host tensors in a world of two ranks on one GPU.  (A world of one rank runs kernels of its
own; these are the staged fetch of the general send and the host stores of the general reduction.)
The send halves wait for nobody and are launched rank by rank, the receive halves after them."""

import pytest
import torch

import pplx_kernels_b200 as pk
from pplx_kernels_b200.utils.testing import MoEConfig
from pplx_kernels_b200.utils.verify import RankBuffers, verify_combine, verify_dispatch, world_inputs

pytestmark = pytest.mark.gpu


def _world(cfg: MoEConfig, seed: int, num_tokens=None, max_blocks: int = 0):
    ranks = pk.AllToAll.local_world(cfg.max_num_tokens, cfg.num_experts, cfg.experts_per_token, 2, 1,
                                    cfg.hidden_dim, cfg.hidden_dim_bytes, cfg.hidden_dim_scale_bytes)
    for r in ranks:
        r.set_debug_checks(True)
        r.set_timeout_ms(3000)
        if max_blocks:
            r.set_max_blocks(max_blocks)
    inputs = world_inputs(cfg, 2, 1, seed, num_tokens=num_tokens)
    return ranks, inputs, [RankBuffers(cfg, 2, 1, i, torch.device("cuda", 0)) for i in inputs]


def _pinned(t: torch.Tensor) -> torch.Tensor:
    return t.cpu().pin_memory()


def _check(ranks):
    torch.cuda.synchronize()
    for r in ranks:
        r.check_status()


# 300 tokens on three blocks: a block fetches its tokens in several rounds.  528 bytes and 5 scales: a
# staged row that is no multiple of 128 bytes.
@pytest.mark.parametrize("tokens,experts,topk,hidden,max_blocks", [
    (24, 16, 4, 1024, 0), (300, 8, 2, 4096, 3), (7, 6, 3, 528, 1)])
@pytest.mark.parametrize("host_indices", [False, True])
def test_send_from_pinned_memory(tokens, experts, topk, hidden, max_blocks, host_indices):
    cfg = MoEConfig(num_experts=experts, experts_per_token=topk, hidden_dim=hidden,
                    max_num_tokens=tokens + 1, in_dtype=torch.float8_e4m3fn)
    ranks, inputs, bufs = _world(cfg, 31, num_tokens=[tokens, tokens - 2], max_blocks=max_blocks)
    for _ in range(2):
        for r, b in zip(ranks, bufs, strict=True):
            b.counts.fill_(-1)
            b.expert_x.view(torch.uint8).zero_()
            r.dispatch(b.counts, b.expert_x, b.expert_scale, _pinned(b.x), _pinned(b.x_scale),
                       _pinned(b.indices) if host_indices else b.indices, b.bound_m, do_recv=False)
            torch.cuda.synchronize()  # (the pinned copies live no longer than this)
        pk.dispatch_group(ranks, [b.counts for b in bufs], [b.expert_x for b in bufs],
                          [b.expert_scale for b in bufs], [b.x for b in bufs],
                          [b.x_scale for b in bufs], [b.indices for b in bufs],
                          [b.bound_m for b in bufs], do_send=False)
        _check(ranks)
        for r in range(2):
            verify_dispatch(cfg, inputs, 1, r, bufs[r])
            bufs[r].make_expert_y()
        pk.combine_group(ranks, [b.out for b in bufs], [b.indices for b in bufs],
                         [b.weights for b in bufs], [b.expert_y for b in bufs],
                         [b.bound_m for b in bufs])
        _check(ranks)
        for r in range(2):
            verify_combine(cfg, inputs, r, bufs[r])
    for r in ranks:
        r.destroy()


@pytest.mark.parametrize("lines", ["0", "1"])
def test_reduction_into_pinned_memory(lines, monkeypatch):
    monkeypatch.setenv("PPLX_B200_LL", lines)
    cfg = MoEConfig(num_experts=16, experts_per_token=4, hidden_dim=1032, max_num_tokens=32)
    ranks, inputs, bufs = _world(cfg, 32)
    pk.dispatch_group(ranks, [b.counts for b in bufs], [b.expert_x for b in bufs], [None, None],
                      [b.x for b in bufs], [None, None], [b.indices for b in bufs],
                      [b.bound_m for b in bufs])
    _check(ranks)
    for b in bufs:
        b.make_expert_y()
        b.out = _pinned(b.out)
    pk.combine_group(ranks, [b.out for b in bufs], [b.indices for b in bufs],
                     [_pinned(b.weights) for b in bufs], [b.expert_y for b in bufs],
                     [b.bound_m for b in bufs])
    _check(ranks)
    for r in range(2):
        verify_combine(cfg, inputs, r, bufs[r])
        ranks[r].destroy()

"""World of one rank: what the calls report and keep to where the input goes past a limit."""

import pytest
import torch

import pplx_kernels_b200 as pk
from pplx_kernels_b200.ops import _ops
from pplx_kernels_b200.ops.quant import per_token_block_quant
from pplx_kernels_b200.utils.testing import MoEConfig
from pplx_kernels_b200.utils.verify import (
    EXPERT_GAIN,
    RankBuffers,
    run_local_world,
    verify_combine,
    verify_dispatch,
    world_inputs,
)

pytestmark = pytest.mark.gpu

HALVES = ({"do_recv": False}, {"do_send": False})


def _object(cfg: MoEConfig, seed: int, num_tokens: int):
    ata = pk.AllToAll.intranode(cfg.max_num_tokens, cfg.num_experts, cfg.experts_per_token, 0, 1, 1,
                                cfg.hidden_dim, cfg.hidden_dim_bytes, cfg.hidden_dim_scale_bytes)
    ata.set_timeout_ms(300)
    inputs = world_inputs(cfg, 1, 1, seed=seed, num_tokens=num_tokens)
    return ata, inputs, RankBuffers(cfg, 1, 1, inputs[0], torch.device("cuda", 0))


def _dispatch(ata, buf, split):
    for kw in HALVES if split else ({},):
        ata.dispatch(buf.counts, buf.expert_x, buf.expert_scale, buf.x, buf.x_scale, buf.indices,
                     buf.bound_m, **kw)


def _combine(ata, buf, split, bound_m=None):
    for kw in HALVES if split else ({},):
        ata.combine(buf.out, buf.indices, buf.weights, buf.expert_y,
                    buf.bound_m if bound_m is None else bound_m, **kw)


@pytest.mark.parametrize("lines", [0, 1])
@pytest.mark.parametrize("split", [False, True])
def test_combine_of_more_tokens_than_dispatched_is_reported(split, lines, monkeypatch):
    """The places of the extra tokens are those of an earlier pass: their sums are not results."""
    monkeypatch.setenv("PPLX_B200_LL", str(lines))
    cfg = MoEConfig(num_experts=8, experts_per_token=2, hidden_dim=64, max_num_tokens=12)
    ata, _, buf = _object(cfg, 3, 12)
    _dispatch(ata, buf, split)
    buf.make_expert_y()
    _combine(ata, buf, split)
    buf.bound_m.view(torch.int32).fill_(5)
    _dispatch(ata, buf, split)
    torch.cuda.synchronize()
    ata.check_status()
    buf.out.fill_(float("nan"))
    more = torch.full((1,), 12, dtype=torch.int32, device=buf.out.device).view(torch.uint32)
    _combine(ata, buf, split, bound_m=more)
    torch.cuda.synchronize()
    assert ata.status()["code"] != 0
    out = buf.out.float()
    assert torch.isnan(out[5:]).all()
    if not split:
        assert not torch.isnan(out[:5]).any()
    ata.destroy()


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("lines", [0, 1])
def test_combine_of_fewer_tokens_than_dispatched(split, lines, monkeypatch):
    """The rest of the tokens is left alone, and the next pass of all of them is whole."""
    monkeypatch.setenv("PPLX_B200_LL", str(lines))
    cfg = MoEConfig(num_experts=8, experts_per_token=2, hidden_dim=64, max_num_tokens=12)
    ata, inputs, buf = _object(cfg, 4, 12)
    fewer = torch.full((1,), 5, dtype=torch.int32, device=buf.out.device).view(torch.uint32)
    whole = None
    for bound_m in (None, fewer, None, fewer, None):
        _dispatch(ata, buf, split)
        buf.make_expert_y()
        buf.out.fill_(float("nan"))
        _combine(ata, buf, split, bound_m)
        torch.cuda.synchronize()
        ata.check_status()
        m = 12 if bound_m is None else 5
        if whole is None:
            whole = buf.out.clone()
        assert torch.equal(buf.out[:m], whole[:m])
        assert torch.isnan(buf.out[m:].float()).all()
    ata.destroy()


def _blocks(ata, array: int) -> int:
    stamps = _ops.all_to_all_read_trace(ata._ptr)
    return sum(v != 0 for v in stamps[32 + 256 * array: 32 + 256 * (array + 1)])


@pytest.mark.parametrize("cap", [0, 1, 7, 150, 400])
def test_max_blocks_limits_the_blocks_of_a_launch(cap):
    cfg = MoEConfig(num_experts=64, experts_per_token=8, hidden_dim=4096, max_num_tokens=256)
    ata, inputs, buf = _object(cfg, 6, 256)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ata.set_trace(True)
    ata.set_max_blocks(cap)
    _dispatch(ata, buf, False)
    torch.cuda.synchronize()
    verify_dispatch(cfg, inputs, 1, 0, buf)
    buf.make_expert_y()
    _combine(ata, buf, False)
    torch.cuda.synchronize()
    ata.check_status()
    # (The trace holds the stamps of the first 256 blocks.)
    most = min(256, 2 * sms, cap or 2 * sms)
    assert 0 < _blocks(ata, 0) <= most and 0 < _blocks(ata, 2) <= most
    ata.destroy()


@pytest.mark.parametrize("split", [False, True])
def test_an_expert_named_twice_by_its_tokens(split):
    """Counts are those of the routing table in both forms, also beyond the capacity; the rows
    beyond it are dropped and reported."""
    cfg = MoEConfig(num_experts=4, experts_per_token=3, hidden_dim=64, max_num_tokens=4)
    ata, _, buf = _object(cfg, 5, 4)
    buf.indices = torch.zeros(4, 3, dtype=torch.int32, device=buf.out.device).view(torch.uint32)
    _ops.sleep_on_stream(0.05)  # both halves are issued before the host can see the failure
    _dispatch(ata, buf, split)
    torch.cuda.synchronize()
    assert buf.counts.tolist() == [12, 0, 0, 0]
    assert ata.status()["code"] == 4
    ata.verify_canaries()
    ata.destroy()


@pytest.mark.parametrize("quantised_half", ["send", "recv"])
def test_halves_of_dispatch_and_dispatch_quant(quantised_half):
    """The receive half takes what the send half staged, whichever call staged it."""
    dev = torch.device("cuda", 0)
    cfg = MoEConfig(num_experts=16, experts_per_token=4, hidden_dim=1024, max_num_tokens=600,
                    in_dtype=torch.float8_e4m3fn)
    ata, _, buf = _object(cfg, 8, 600)
    x = torch.randn(600, cfg.hidden_dim, generator=torch.Generator().manual_seed(9)).to(torch.bfloat16)
    xq, xs = per_token_block_quant(x)
    quant = (buf.counts, buf.expert_x, buf.expert_scale, x.to(dev), buf.indices, buf.bound_m)
    plain = (buf.counts, buf.expert_x, buf.expert_scale, xq.to(dev), xs.to(dev), buf.indices,
             buf.bound_m)
    rows, scales = [], []
    for mixed in (False, True):
        buf.expert_x.view(torch.uint8).zero_()
        buf.expert_scale.zero_()
        if quantised_half == "send":
            ata.dispatch_quant(*quant, do_recv=False)
        else:
            ata.dispatch(*plain, do_recv=False)
        if (quantised_half == "recv") == mixed:
            ata.dispatch_quant(*quant, do_send=False)
        else:
            ata.dispatch(*plain, do_send=False)
        torch.cuda.synchronize()
        ata.check_status()
        rows.append(buf.expert_x.view(torch.uint8).clone())
        scales.append(buf.expert_scale.clone())
        ata.combine(buf.out, buf.indices, buf.weights, buf.make_expert_y(), buf.bound_m)
    assert torch.equal(rows[0], rows[1]) and torch.equal(scales[0], scales[1])
    assert buf.counts.sum().item() == 600 * cfg.experts_per_token
    ata.destroy()


def test_object_whose_tables_do_not_fit_one_block():
    """9000 experts and 7000 rows per token: the kernels of larger worlds take it."""
    cfg = MoEConfig(num_experts=9000, experts_per_token=7000, hidden_dim=16, max_num_tokens=3)
    run_local_world(cfg, world=1, dp_size=1, seed=10, num_tokens=3, iterations=2)
    run_local_world(cfg, world=1, dp_size=1, seed=11, num_tokens=2, split=True)


def test_dispatch_quant_in_halves_equals_the_whole_call():
    dev = torch.device("cuda", 0)
    cfg = MoEConfig(num_experts=16, experts_per_token=4, hidden_dim=1408, max_num_tokens=130,
                    in_dtype=torch.float8_e4m3fn)
    ata, _, buf = _object(cfg, 12, 129)
    x = torch.randn(130, cfg.hidden_dim, generator=torch.Generator().manual_seed(13)).to(torch.bfloat16)
    got = []
    for halves in (({},), HALVES):
        buf.expert_x.view(torch.uint8).zero_()
        buf.expert_scale.zero_()
        for kw in halves:
            ata.dispatch_quant(buf.counts, buf.expert_x, buf.expert_scale, x.to(dev), buf.indices,
                               buf.bound_m, **kw)
        torch.cuda.synchronize()
        ata.check_status()
        got.append((buf.expert_x.view(torch.uint8).clone(), buf.expert_scale.clone(), buf.counts.clone()))
        ata.combine(buf.out, buf.indices, buf.weights, buf.make_expert_y(), buf.bound_m)
    assert all(torch.equal(a, b) for a, b in zip(*got, strict=True))
    ata.destroy()


def test_halves_on_two_streams():
    """Send halves on one stream, receive halves on another, ordered by events; many passes, so that
    launches overlap on both streams."""
    cfg = MoEConfig(num_experts=16, experts_per_token=4, hidden_dim=2048, max_num_tokens=64,
                    in_dtype=torch.float8_e4m3fn)
    ata, inputs, buf = _object(cfg, 14, 63)
    ata.set_timeout_ms(3000)
    send, recv = torch.cuda.Stream(), torch.cuda.Stream()
    buf.make_expert_y()
    d_args = (buf.counts, buf.expert_x, buf.expert_scale, buf.x, buf.x_scale, buf.indices, buf.bound_m)
    c_args = (buf.out, buf.indices, buf.weights, buf.expert_y, buf.bound_m)
    torch.cuda.synchronize()
    for _ in range(50):
        with torch.cuda.stream(send):
            ata.dispatch(*d_args, do_recv=False)
        recv.wait_stream(send)
        with torch.cuda.stream(recv):
            ata.dispatch(*d_args, do_send=False)
            buf.expert_y.copy_((buf.expert_x.to(torch.float32) * EXPERT_GAIN).to(cfg.out_dtype))
        send.wait_stream(recv)
        with torch.cuda.stream(send):
            ata.combine(*c_args, do_recv=False)
        recv.wait_stream(send)
        with torch.cuda.stream(recv):
            ata.combine(*c_args, do_send=False)
        send.wait_stream(recv)
    torch.cuda.synchronize()
    ata.check_status()
    verify_dispatch(cfg, inputs, 1, 0, buf)
    verify_combine(cfg, inputs, 0, buf)
    ata.destroy()

"""World of one rank: one half of the fused path with the other half of the plain one."""

import pytest
import torch

from pplx_kernels_b200.models.configs import MoEModelConfig
from pplx_kernels_b200.models.moe import MoELayer, MoELayerFP8, moe_reference, moe_reference_fp8
from pplx_kernels_b200.ops.grouped_gemm import grouped_gemm, grouped_gemm_fp8
from pplx_kernels_b200.utils.testing import as_index_tensor, routing

pytestmark = pytest.mark.gpu

CFG = MoEModelConfig("mixed", 16, 4, 512, 256)
M = 40


def _layer(kind: str):
    layer = (MoELayer(CFG, M, init_std=0.05) if kind == "bf16"
             else MoELayerFP8(CFG, M, init_std=0.05, pow2_scales=kind == "fp8pow2"))
    layer.ata.set_timeout_ms(2000)
    return layer


def _calls(kind: str, layer, x, idx, bound_m):
    """(fused dispatch, fused up, own up, own down, fused down, plain dispatch) of one kind."""
    l, a = layer, layer.ata
    if kind == "bf16":
        return (lambda: a.fused_dispatch(x, idx, bound_m),
                lambda: a.fused_up(l.w13, l.h, l.counts, l.gemm_status),
                lambda: grouped_gemm(l.expert_x, l.w13, l.counts, out=l.h, swiglu=True,
                                     status=l.gemm_status),
                lambda: grouped_gemm(l.h, l.w2, l.counts, out=l.expert_y, status=l.gemm_status),
                lambda: a.fused_down(l.h, l.w2, l.gemm_status),
                lambda **kw: a.dispatch(l.counts, l.expert_x, None, x, None, idx, bound_m, **kw))
    pow2 = l.pow2_scales
    return (lambda: a.fused_dispatch(x, idx, bound_m, quantize=True),
            lambda: a.fused_up_fp8(l.w13_q, l.w13_s, l.h, l.h_scale, l.counts, l.gemm_status),
            lambda: grouped_gemm_fp8(l.expert_x, l.expert_scale, l.w13_q, l.w13_s, l.counts,
                                     swiglu_quant=True, out=l.h, out_scale=l.h_scale,
                                     status=l.gemm_status, pow2_scales=pow2),
            lambda: grouped_gemm_fp8(l.h, l.h_scale, l.w2_q, l.w2_s, l.counts, out=l.expert_y,
                                     status=l.gemm_status, pow2_scales=pow2),
            lambda: a.fused_down_fp8(l.h, l.h_scale, l.w2_q, l.w2_s, l.gemm_status),
            lambda **kw: a.dispatch_quant(l.counts, l.expert_x, l.expert_scale, x, idx, bound_m,
                                          **kw))


@pytest.mark.parametrize("kind", ["bf16", "fp8", "fp8pow2"])
@pytest.mark.parametrize("first", ["up", "down"])
def test_fused_halves_with_plain_halves(kind, first):
    """fused up + own down + combine, and dispatch + own up + fused down + combine(recv): on a
    fresh object, and after passes of other routings and sizes."""
    dev = torch.device("cuda", 0)
    layer = _layer(kind)
    ata = layer.ata
    gen = torch.Generator().manual_seed(5)
    bound_m = torch.zeros(1, dtype=torch.int32, device=dev)
    weights = ((layer.w13, layer.w2) if kind == "bf16" else layer.dequantized_weights())
    both = ["up", "down"] if first == "up" else ["down", "up"]
    for n, (which, split, m) in enumerate([(both[0], False, M), (both[1], False, 7),
                                           (both[0], True, 23), (both[1], True, M)]):
        x = torch.randn(M, CFG.hidden_dim, generator=gen).to(torch.bfloat16).to(dev)
        idx = routing(M, CFG.num_experts, CFG.experts_per_token, gen)
        w = torch.softmax(torch.randn(M, CFG.experts_per_token, generator=gen), dim=-1).to(dev)
        bound_m.fill_(m)
        idx_dev = as_index_tensor(idx, dev)
        f_dispatch, f_up, own_up, own_down, f_down, dispatch = _calls(kind, layer, x, idx_dev,
                                                                      bound_m)
        out = torch.full((M, CFG.hidden_dim), float("nan"), dtype=torch.bfloat16, device=dev)
        c_args = (out, idx_dev, w, layer.expert_y, bound_m)
        if which == "up":
            f_dispatch()
            f_up()
            own_down()
            for kw in ({"do_recv": False}, {"do_send": False}) if split else ({},):
                ata.combine(*c_args, **kw)
        else:
            for kw in ({"do_recv": False}, {"do_send": False}) if split else ({},):
                dispatch(**kw)
            own_up()
            f_down()
            ata.combine(*c_args, do_send=False)
        torch.cuda.synchronize()
        layer.check_status()
        if kind == "bf16":
            want = moe_reference(x[:m], idx[:m].to(dev), w[:m], *weights)
            torch.testing.assert_close(out[:m].float(), want, rtol=3e-2, atol=3e-3)
        else:
            want = moe_reference_fp8(x[:m], idx[:m].to(dev), w[:m], *weights, pow2=kind == "fp8pow2")
            err = (out[:m].float() - want).abs()
            assert (err <= 0.06 * want.abs() + 0.03 * want.abs().amax()).all(), (n, err.max())
        assert torch.isnan(out[m:].float()).all()
    layer.destroy()


@pytest.mark.parametrize("kind", ["fp8", "fp8pow2"])
def test_fused_layer_with_more_than_64_experts(kind):
    cfg, m = MoEModelConfig("many", 200, 4, 256, 128), 90
    dev = torch.device("cuda", 0)
    layer = MoELayerFP8(cfg, m, init_std=0.05, pow2_scales=kind == "fp8pow2")
    gen = torch.Generator().manual_seed(6)
    x = torch.randn(m, cfg.hidden_dim, generator=gen).to(torch.bfloat16).to(dev)
    idx = routing(m, cfg.num_experts, cfg.experts_per_token, gen)
    w = torch.softmax(torch.randn(m, cfg.experts_per_token, generator=gen), dim=-1).to(dev)
    want = moe_reference_fp8(x, idx.to(dev), w, *layer.dequantized_weights(), pow2=kind == "fp8pow2")
    for _ in range(2):
        out = layer(x, as_index_tensor(idx, dev), w, fused=True)
        torch.cuda.synchronize()
        layer.check_status()
        err = (out[:m].float() - want).abs()
        assert (err <= 0.06 * want.abs() + 0.03 * want.abs().amax()).all(), err.max()
    layer.destroy()

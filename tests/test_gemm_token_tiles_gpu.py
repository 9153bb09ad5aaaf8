"""Expert GEMMs whose token tile follows the rows an expert has: row counts around the tile steps."""

import pytest
import torch

from pplx_kernels_b200.ops.grouped_gemm import (
    grouped_gemm_fp8,
    grouped_gemm_fp8_reference,
    quantize_weight_blocks,
)
from pplx_kernels_b200.ops.quant import block_dequant, per_token_block_quant

pytestmark = pytest.mark.gpu

# Steps of 16 tokens, widest tiles of 64 and 128: one below, at and above each; several equal tiles.
COUNTS = [1, 15, 16, 17, 0, 63, 64, 65, 127, 128, 129, 193, 257]


def _fp8_operands(E, rows, K, w_rows, seed):
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(seed)
    kblocks = (K + 127) // 128
    x = torch.randn(E * rows, K, generator=g, device=dev)
    # Scales that differ from row to row and from K block to K block by powers of two: a wrong
    # one shows as a factor.
    x *= torch.exp2(torch.randint(-3, 4, (E * rows, kblocks), generator=g, device=dev).float()
                    ).repeat_interleave(128, dim=1)[:, :K]
    w = torch.randn(E, w_rows, K, generator=g, device=dev) * K ** -0.5
    xq, sa = per_token_block_quant(x)
    return (xq.view(E, rows, K), sa.view(E, rows, -1), *quantize_weight_blocks(w))


@pytest.mark.parametrize("K,N", [(16, 16), (144, 272), (1024, 640)])
def test_fp8_plain(K, N):
    E, rows = len(COUNTS), max(COUNTS) + 3
    xq, sa, wq, sw = _fp8_operands(E, rows, K, N, seed=K)
    cnt = torch.tensor(COUNTS, dtype=torch.int32, device=xq.device)
    out = torch.full((E, rows, N), float("nan"), dtype=torch.bfloat16, device=xq.device)
    status = torch.zeros(1, dtype=torch.int32, device=xq.device)
    grouped_gemm_fp8(xq, sa, wq, sw, cnt, out=out, status=status)
    want = grouped_gemm_fp8_reference(xq, sa, wq, sw, cnt)
    assert int(status.item()) == 0
    for e, m in enumerate(COUNTS):
        # fp32 sums of exact products, one bf16 rounding (2^-9), and the order of up to K sums
        err = (out[e, :m].float() - want[e, :m]).abs()
        bound = 2 ** -8 * want[e, :m].abs() + 1e-5 * want[e, :m].abs().amax() if m else err
        assert (err <= bound).all(), (e, m, float(err.max()))
        assert torch.isnan(out[e, m:].float()).all()


@pytest.mark.parametrize("K,I", [(16, 128), (400, 256), (2048, 384)])
def test_fp8_swiglu(K, I):
    E, rows = len(COUNTS), max(COUNTS) + 3
    xq, sa, wq, sw = _fp8_operands(E, rows, K, 2 * I, seed=K + 1)
    cnt = torch.tensor(COUNTS, dtype=torch.int32, device=xq.device)
    hq = torch.zeros(E, rows, I, dtype=torch.uint8, device=xq.device).view(torch.float8_e4m3fn)
    hs = torch.full((E, rows, I // 128), float("nan"), device=xq.device)
    status = torch.zeros(1, dtype=torch.int32, device=xq.device)
    grouped_gemm_fp8(xq, sa, wq, sw, cnt, swiglu_quant=True, out=hq, out_scale=hs, status=status)
    want = grouped_gemm_fp8_reference(xq, sa, wq, sw, cnt, swiglu=True)
    assert int(status.item()) == 0
    for e, m in enumerate(COUNTS):
        assert torch.isnan(hs[e, m:]).all() and not hq[e, m:].view(torch.uint8).any()
        if m == 0:
            continue
        amax = want[e, :m].view(m, -1, 128).abs().amax(dim=2).clamp(min=1e-4) / 448.0
        torch.testing.assert_close(hs[e, :m], amax, rtol=1e-3, atol=0)
        # half an e4m3 step: 2^-4 of the value, 2^-10 of 448 scales below the normal range
        got = block_dequant(hq[e, :m], hs[e, :m])
        step = 2 ** -4 * want[e, :m].abs() + 2 ** -10 * amax.repeat_interleave(128, dim=1)
        assert ((got - want[e, :m]).abs() <= 1.02 * step).all()

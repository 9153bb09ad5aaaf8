"""fp8 expert GEMM with power-of-two scales where its token tiles can go wrong: the steps of 16, the
scales of tokens beyond the first 128, the change from two accumulators to one, equal tiles."""

import pytest
import torch

from pplx_kernels_b200.ops.grouped_gemm import (
    grouped_gemm_fp8,
    grouped_gemm_fp8_reference,
    quantize_weight_blocks,
)
from pplx_kernels_b200.ops.quant import block_dequant, per_token_block_quant

pytestmark = pytest.mark.gpu

# Widest tile 112 rows (two accumulators; more tiles than one per CTA) and 224 (one).
COUNTS = [[1, 15, 16, 17, 0, 33, 97, 112], [113, 128, 129, 224, 225, 1, 0, 460]]


def _operands(E, rows, K, w_rows, seed):
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(seed)
    kblocks = (K + 127) // 128
    x = torch.randn(E * rows, K, generator=g, device=dev)
    # Scales that differ from row to row and from K block to K block: a wrong one shows as a factor.
    x *= torch.exp2(torch.randint(-3, 4, (E * rows, kblocks), generator=g, device=dev).float()
                    ).repeat_interleave(128, dim=1)[:, :K]
    w = torch.randn(E, w_rows, K, generator=g, device=dev) * K ** -0.5
    w *= torch.exp2(torch.randint(-2, 3, (E, (w_rows + 127) // 128, 1), generator=g, device=dev)
                    .float()).repeat_interleave(128, dim=1)[:, :w_rows]
    xq, sa = per_token_block_quant(x, pow2=True)
    return (xq.view(E, rows, K), sa.view(E, rows, -1), *quantize_weight_blocks(w, pow2=True))


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("K,N", [(16, 16), (144, 272), (1024, 4096)])
def test_plain(counts, K, N):
    E, rows = len(counts), max(counts) + 3
    xq, sa, wq, sw = _operands(E, rows, K, N, seed=K)
    cnt = torch.tensor(counts, dtype=torch.int32, device=xq.device)
    out = torch.full((E, rows, N), float("nan"), dtype=torch.bfloat16, device=xq.device)
    status = torch.zeros(1, dtype=torch.int32, device=xq.device)
    grouped_gemm_fp8(xq, sa, wq, sw, cnt, out=out, status=status, pow2_scales=True)
    want = grouped_gemm_fp8_reference(xq, sa, wq, sw, cnt)
    assert int(status.item()) == 0
    for e, m in enumerate(counts):
        # fp32 sums of exact products, one bf16 rounding (2^-9), and the order of up to K sums
        err = (out[e, :m].float() - want[e, :m]).abs()
        bound = 2 ** -8 * want[e, :m].abs() + 1e-5 * want[e, :m].abs().amax() if m else err
        assert (err <= bound).all(), (e, m, float(err.max()))
        assert torch.isnan(out[e, m:].float()).all()


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("K,I", [(16, 128), (400, 256), (1024, 2560)])
def test_swiglu(counts, K, I):
    E, rows = len(counts), max(counts) + 3
    xq, sa, wq, sw = _operands(E, rows, K, 2 * I, seed=K + 1)
    cnt = torch.tensor(counts, dtype=torch.int32, device=xq.device)
    hq = torch.zeros(E, rows, I, dtype=torch.uint8, device=xq.device).view(torch.float8_e4m3fn)
    hs = torch.full((E, rows, I // 128), float("nan"), device=xq.device)
    status = torch.zeros(1, dtype=torch.int32, device=xq.device)
    grouped_gemm_fp8(xq, sa, wq, sw, cnt, swiglu_quant=True, out=hq, out_scale=hs, status=status,
                     pow2_scales=True)
    want = grouped_gemm_fp8_reference(xq, sa, wq, sw, cnt, swiglu=True)
    assert int(status.item()) == 0
    for e, m in enumerate(counts):
        assert torch.isnan(hs[e, m:]).all() and not hq[e, m:].view(torch.uint8).any()
        if m == 0:
            continue
        amax = want[e, :m].view(m, -1, 128).abs().amax(dim=2).clamp(min=1e-4) / 448.0
        # The next power of two; the maximum itself is known to 1e-3.
        assert torch.equal(torch.exp2(torch.log2(hs[e, :m]).round()), hs[e, :m])
        assert (hs[e, :m] >= amax * (1 - 1e-3)).all() and (hs[e, :m] <= 2 * amax * (1 + 1e-3)).all()
        # half an e4m3 step: 2^-4 of the value, 2^-10 of 448 scales below the normal range
        got = block_dequant(hq[e, :m], hs[e, :m])
        step = 2 ** -4 * want[e, :m].abs() + 2 ** -10 * hs[e, :m].repeat_interleave(128, dim=1)
        assert ((got - want[e, :m]).abs() <= 1.02 * step).all()

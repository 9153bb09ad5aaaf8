"""bf16 expert GEMM where its cut of the token rows and of the weight rows can go wrong: around the
steps of 16 and 32 rows, the 256-row tile, unequal tiles of one expert, and column tails."""

import pytest
import torch

from pplx_kernels_b200.ops.grouped_gemm import grouped_gemm, grouped_gemm_reference

pytestmark = pytest.mark.gpu

# Products of K terms are summed in fp32 (error far below a bf16 unit) and rounded once: half a
# unit in the last place, 2^-9 of the value.  The reference's SwiGLU is in fp32 as well; __expf
# and the division add a few fp32 units.  2^-8 leaves a factor of two; the absolute part covers
# results near zero, K sums of products of at most 1/8 with fp32 rounding.
RTOL, ATOL = 2.0 ** -8, 2e-4


@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize("cta_pair", [0, 1])
@pytest.mark.parametrize("counts,K,N,half_n", [
    ([1, 15, 16, 17, 31, 32, 33, 0], 136, 72, 0),
    ([255, 256, 257, 1], 64, 264, 0),
    ([1030, 7, 513], 72, 136, 0),       # five unequal tiles beside a single narrow one
    ([512, 481, 289, 256], 200, 264, 0),  # two MMAs per tile, equal and unequal
    ([300, 65, 0, 1], 320, 8, 16),      # the narrowest limit: ten tiles of 32 rows
])
def test_token_cut(swiglu, cta_pair, counts, K, N, half_n):
    dev = torch.device("cuda", 0)
    gen = torch.Generator().manual_seed(11)
    E, rows = len(counts), max(counts)
    x = (torch.randn(E, rows, K, generator=gen) * 0.5).to(torch.bfloat16).to(dev)
    w = (torch.randn(E, 2 * N if swiglu else N, K, generator=gen) * K ** -0.5).to(torch.bfloat16).to(dev)
    cnt = torch.tensor(counts, dtype=torch.int32, device=dev)
    # Rows beyond an expert's count must neither be written nor reach another row's result.
    for e, m in enumerate(counts):
        x[e, m:] = float("nan")
    out = torch.full((E, rows, N), float("nan"), dtype=torch.bfloat16, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    grouped_gemm(x, w, cnt, out=out, swiglu=swiglu, status=status, half_n=half_n, cta_pair=cta_pair)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    want = grouped_gemm_reference(x, w, cnt, swiglu)
    for e, m in enumerate(counts):
        torch.testing.assert_close(out[e, :m].float(), want[e, :m], rtol=RTOL, atol=ATOL)
        assert torch.isnan(out[e, m:].float()).all()

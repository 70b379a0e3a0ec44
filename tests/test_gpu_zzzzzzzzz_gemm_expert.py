"""GPU: grouped products with one tile of rows per expert (gemm_expert_kernel): units of 16 weight rows dealt over the CTAs."""
import ctypes as C

import pytest
import torch
import torch.nn.functional as F

from .util import cptr

pytestmark = pytest.mark.gpu
CASES = [([1], 16, 64), ([1], 8, 64), ([2, 0, 1], 24, 72), ([3], 148 * 16, 64), ([3], 148 * 16 + 2, 128), ([128, 1, 127], 148 * 64, 72), ([128, 1, 127], 148 * 32, 72), ([1, 0, 128], 4096, 2048),
         ([1] * 16, 8192, 136), ([5, 2, 0, 9] * 10, 1038, 200)]


@pytest.mark.parametrize("act", [0, 2])
@pytest.mark.parametrize("counts,N,K", CASES)
def test_grouped_product_of_few_rows(counts, N, K, act):
    """(The plain product of 256 rows and 148 x 64 columns takes gemm_wide_kernel: its tiles fill three quarters of a wave.)  One unit for the whole chip, one
    per CTA and one more, rows that do not fill a unit, shares that span several experts, tiles of 1 to 8 units; each sum of K bf16 products in fp32, rounded to bf16 (2^-8 of the result; the
    gated unit's slope stays below 16)."""
    from moshi_b200 import _lib
    M, E = sum(counts), len(counts)
    g = torch.Generator().manual_seed(M + N + act)
    x = torch.randn(M, K, generator=g).bfloat16().cuda()
    w = (torch.randn(E, N, K, generator=g) / K ** 0.5).bfloat16().cuda()
    cols = N // 2 if act == 2 else N
    for ld in (cols + 8, cols + 3):
        y = torch.full((M, ld), 7.0, dtype=torch.bfloat16, device="cuda")
        _lib.check(_lib.lib().b200_op_grouped_wide(cptr(x), cptr(w), cptr(y), (C.c_int32 * E)(*counts), E, M, N, K, ld, act, 1.5, C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        starts = [sum(counts[:e]) for e in range(E)]
        z = torch.cat([x[s:s + c].double() @ w[e].double().t() for e, (s, c) in enumerate(zip(starts, counts))])
        size = torch.cat([x[s:s + c].double().abs() @ w[e].double().abs().t() for e, (s, c) in enumerate(zip(starts, counts))])
        bound = (K + 8) * 2.0 ** -24 * size
        if act == 2:
            gt, u = z[:, 0::2].clamp(max=1.5), z[:, 1::2].clamp(-1.5, 1.5)
            z, bound = gt * torch.sigmoid(1.702 * gt) * (u + 1), 16 * (bound[:, 0::2] + bound[:, 1::2]) + 1e-6
        assert bool(((y[:, :cols].double() - z).abs() <= bound + 2.0 ** -8 * z.abs()).all())
        assert (y[:, cols:] == 7.0).all()

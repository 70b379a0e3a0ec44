"""GPU: the sums of linears of a few rows (csrc/gemm_row.cu) are as exact as fp32 FMAs make them."""
import ctypes as C

import pytest
import torch

from .util import cptr

pytestmark = pytest.mark.gpu


# (outputs, inputs, error of a kernel that adds with fp32 FMAs, in chains of up to 352 per thread and 8 threads a row): measured over the same draws
@pytest.mark.parametrize("M", [1, 2, 8])
@pytest.mark.parametrize("N,K,fma", [(12288, 4096, 7.4e-8), (4096, 11264, 8.5e-8), (3072, 1024, 5.5e-8), (1024, 2816, 6.5e-8)])
def test_sums_that_cancel(M, N, K, fma):
    """Every term comes with its negative in a random place, so a result is the error of its sum and bf16 keeps its size.  The rms over 4 M N >= 4096 results
    is known to 2 %; a tenth is allowed."""
    from moshi_b200 import _lib
    lib, st = _lib.lib(), C.c_void_p(torch.cuda.current_stream().cuda_stream)
    total, n = 0.0, 0
    for seed in range(4):
        g = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.randn(M, K // 2, device="cuda", generator=g).bfloat16()
        w = (torch.randn(N, K // 2, device="cuda", generator=g) / K ** 0.5).bfloat16()
        perm = torch.randperm(K, device="cuda", generator=g)
        x, w = torch.cat([x, x], 1)[:, perm].contiguous(), torch.cat([w, -w], 1)[:, perm].contiguous()
        tiles = torch.empty(lib.b200_op_packed_bytes(N, K, 0, 0), dtype=torch.uint8, device="cuda")
        y = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
        _lib.check(lib.b200_op_pack_tiles(cptr(w), cptr(tiles), N, K, 0, 0, st))
        _lib.check(lib.b200_op_linear_sk(cptr(x), cptr(tiles), cptr(y), cptr(None), M, N, K, 0, 0, 0, 0, 0, st))
        scale = x.double().norm(dim=1)[:, None] * w.double().norm(dim=1)[None] / K ** 0.5
        total += float((y.double() / scale).square().sum())
        n += y.numel()
    assert (total / n) ** 0.5 <= 1.1 * fma

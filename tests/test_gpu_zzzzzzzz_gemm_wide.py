"""GPU: the GEMM for many rows and its grouped form (csrc/gemm_wide.cu) against fp32 products."""
import ctypes as C

import pytest
import torch
import torch.nn.functional as F

from .util import cptr

pytestmark = pytest.mark.gpu


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _close(y, want, k):
    # fp32 sums in another order: k * 2^-24 of the rms product sum at most; the result is rounded to bf16 once (2^-9 relative)
    assert not torch.isnan(y.float()).any()
    err = (y.float() - want).abs()
    assert (err <= 2.0 ** -8 * want.abs() + k * 2.0 ** -22).all(), float((err - 2.0 ** -8 * want.abs()).max())


@pytest.mark.parametrize("splits", [0, 1, 3])
@pytest.mark.parametrize("packed", [1, 0])
@pytest.mark.parametrize("M,N,K", [(257, 128, 8), (256, 256, 64), (300, 264, 72), (1, 128, 64), (129, 385, 200), (511, 2048, 2048), (2048, 14848, 2048),
                                   (1009, 520, 4104)])
def test_wide_linear(M, N, K, packed, splits):
    """Edges of row and column tiles, one k-block and remainders of k, odd result strides, more tiles than CTAs; k whole and in ranges (the last one
    shorter or, with few blocks, missing)."""
    from moshi_b200 import _lib
    lib = _lib.lib()
    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g).bfloat16().cuda()
    w = (torch.randn(N, K, generator=g) / K ** 0.5).bfloat16().cuda()
    wt = w
    if packed:
        wt = torch.empty(lib.b200_op_packed_bytes(N, K, 0, 0), dtype=torch.uint8, device="cuda")
        _lib.check(lib.b200_op_pack_tiles(cptr(w), cptr(wt), N, K, 0, 0, _stream()))
    for ld in (N, N + 3):
        y = torch.full((M, ld), 7.0, dtype=torch.bfloat16, device="cuda")
        _lib.check(lib.b200_op_linear_wide(cptr(x), cptr(wt), cptr(y), M, N, K, ld, packed, splits, _stream()))
        torch.cuda.synchronize()
        _close(y[:, :N], x.float() @ w.float().t(), K)
        assert (y[:, N:] == 7.0).all()


@pytest.mark.parametrize("act", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("counts,N,K", [([1], 256, 64), ([0, 3, 0, 130, 1], 264, 72), ([128, 129, 127, 5], 512, 2048), ([2] * 16, 1030, 328),
                                        ([700, 1, 0, 400], 768, 136)])
def test_grouped_product(counts, N, K, act):
    """Experts without rows, single rows, tiles of exactly 128 rows, neighbours that share a box; every epilogue."""
    from moshi_b200 import _lib
    lib = _lib.lib()
    M, E = sum(counts), len(counts)
    g = torch.Generator().manual_seed(M + N + act)
    x = torch.randn(M, K, generator=g).bfloat16().cuda()
    w = (torch.randn(E, N, K, generator=g) / K ** 0.5).bfloat16().cuda()
    cols = N // 2 if act in (2, 3) else N
    y = torch.full((M, cols + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    _lib.check(lib.b200_op_grouped_wide(cptr(x), cptr(w), cptr(y), (C.c_int32 * E)(*counts), E, M, N, K, cols + 8, act, 1.5, _stream()))
    z = torch.cat([x[sum(counts[:e]):sum(counts[:e + 1])].float() @ w[e].float().t() for e in range(E)])
    if act == 1:
        z = z.clamp(min=0) ** 2
    elif act == 2:
        gt, u = z[:, 0::2].clamp(max=1.5), z[:, 1::2].clamp(-1.5, 1.5)
        z = gt * torch.sigmoid(1.702 * gt) * (u + 1)
    elif act == 3:
        z = F.silu(z[:, 0::2]) * z[:, 1::2]
    elif act == 4:
        z = F.gelu(z)
    _close(y[:, :cols], z, 16 * K)            # the epilogues' slopes stay below 16 for sums of unit size
    assert (y[:, cols:] == 7.0).all()

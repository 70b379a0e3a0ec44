"""GPU: linears of 1..16 rows with whole output rows per CTA (csrc/gemm_row.cu) against fp32 products and exact integer sums."""
import ctypes as C

import pytest
import torch
import torch.nn.functional as F

from oracle import quant

from .util import cptr

pytestmark = pytest.mark.gpu
STORE, RESADD, GATE = 0, 1, 2


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("M", [1, 2, 8, 9, 12, 16])
@pytest.mark.parametrize("N,K,epi", [(12, 72, STORE), (130, 8, STORE), (1192, 1024, RESADD), (600, 4104, GATE), (4096, 11264, RESADD), (22528, 4096, GATE),
                                     (32000, 512, STORE)])
def test_row_linear(M, N, K, epi):
    """Fewer units than CTAs, one and several per CTA (odd counts, across tiles), rows beyond the last, one k-block and more than registers hold, sums in
    one pass and in two (32000 outputs of 16 rows); two launches give the same bits, and another kernel other bits here and there only.  (16 gated rows of 22528 x 4096
    would take two passes and go to the register kernel.)"""
    from moshi_b200 import _lib
    lib = _lib.lib()
    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g).bfloat16().cuda()
    w = (torch.randn(N, K, generator=g) / K ** 0.5).bfloat16().cuda()
    rows = N // 2 if epi == GATE else 0
    res = torch.randn(M, N, generator=g).bfloat16().cuda() if epi == RESADD else None
    wt = torch.empty(lib.b200_op_packed_bytes(N, K, epi, rows), dtype=torch.uint8, device="cuda")
    _lib.check(lib.b200_op_pack_tiles(cptr(w), cptr(wt), N, K, epi, rows, _stream()))
    ys = [torch.full((M, rows or N), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(3)]
    before = lib.b200_op_set_gemv_max_rows(16)
    try:
        for y in ys[:2]:
            _lib.check(lib.b200_op_linear_sk(cptr(x), cptr(wt), cptr(y), cptr(res), M, N, K, epi, rows, 0, 0, 0, _stream()))
        lib.b200_op_set_gemv_max_rows(0)
        _lib.check(lib.b200_op_linear_sk(cptr(x), cptr(wt), cptr(ys[2]), cptr(res), M, N, K, epi, rows, 0, 0, 0, _stream()))
        torch.cuda.synchronize()
    finally:
        lib.b200_op_set_gemv_max_rows(before)
    z = x.float() @ w.float().t()
    if epi == RESADD:
        z = res.float() + z.bfloat16().float()
    elif epi == GATE:
        z = z.bfloat16()
        z = (F.silu(z[:, :rows].float()).bfloat16() * z[:, rows:]).float()
    # a bf16 rounding of the sums, one of the gate's activation and one of the result: three half ulps (2^-9) of values up to ~5, plus fp32 order
    assert torch.equal(ys[0], ys[1])
    torch.testing.assert_close(ys[0].float(), z, rtol=2.0 ** -7, atol=3e-2)
    torch.testing.assert_close(ys[0].float(), ys[2].float(), rtol=2.0 ** -7, atol=3e-2)
    # sums in another order move a result across a rounding now and then: some 1e-6 of its size against roundings 2^-8 apart, twice or thrice on the way
    assert (ys[0] != ys[2]).float().mean() < 0.02


@pytest.mark.parametrize("M", [1, 8, 13, 16])
@pytest.mark.parametrize("N,K,epi", [(130, 144, STORE), (4096, 2816, RESADD), (600, 4096, GATE), (22528, 256, GATE)])
def test_row_linear_int8_is_exact(M, N, K, epi):
    from moshi_b200 import _lib
    lib = _lib.lib()
    g = torch.Generator().manual_seed(M + N)
    x = torch.randn(M, K, generator=g).bfloat16()
    w = (torch.randn(N, K, generator=g) / K ** 0.5).bfloat16()
    rows = N // 2 if epi == GATE else 0
    res = torch.randn(M, N, generator=g).bfloat16() if epi == RESADD else None
    tiles = torch.empty(lib.b200_op_packed_bytes_i8(N, K, epi, rows), dtype=torch.uint8, device="cuda")
    sw = torch.empty(N, device="cuda")
    xd, wd, rd = x.cuda(), w.cuda(), res.cuda() if res is not None else None
    _lib.check(lib.b200_op_quant_pack_tiles(cptr(wd), cptr(tiles), cptr(sw), N, K, epi, rows, _stream()))
    xq, sa = torch.empty(M, K, dtype=torch.int8, device="cuda"), torch.empty(M, device="cuda")
    _lib.check(lib.b200_op_quantize_rows(cptr(xd), cptr(xq), cptr(sa), M, K, _stream()))
    y = torch.full((M, rows or N), float("nan"), dtype=torch.bfloat16, device="cuda")
    _lib.check(lib.b200_op_linear_i8(cptr(xq), cptr(sa), cptr(tiles), cptr(sw), cptr(y), cptr(rd), M, N, K, epi, rows, _stream()))
    torch.cuda.synchronize()
    z = quant.qlinear(x, w)
    if epi == GATE:
        # silu through another exponential: a bf16 ulp now and then
        want = F.silu(z[:, :rows].float()).bfloat16() * z[:, rows:]
        assert ((y.cpu().float() - want.float()).abs() <= 2.0 ** -6 * want.float().abs() + 1e-6).all()
    else:
        want = (res.float() + z.float()).bfloat16() if epi == RESADD else z
        assert torch.equal(y.cpu(), want)

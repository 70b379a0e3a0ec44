"""GPU: linears of 1..32 rows with the weights through registers (csrc/gemm_reg.cu) against fp32 products and exact integer sums."""
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


@pytest.mark.parametrize("M", [1, 3, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("N,K,epi", [(130, 72, STORE), (128, 8, STORE), (4096, 200, RESADD), (600, 4104, GATE), (4096, 11264, RESADD), (22528, 4096, GATE),
                                     (32000, 512, STORE)])
def test_register_linear(M, N, K, epi):
    """Edges of row blocks and tiles, remainders of k, one k-block, k whole and cut; two launches give the same bits, and so does the general
    entry point wherever its rule takes this kernel.  Gated pairs beyond 16 rows are not this kernel's and are refused."""
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
    if epi == GATE and M > 16:
        with pytest.raises(AssertionError, match="unsupported"):
            _lib.check(lib.b200_op_linear_reg(cptr(x), cptr(wt), cptr(ys[0]), cptr(res), M, N, K, epi, rows, _stream()))
        return
    for y in ys[:2]:
        _lib.check(lib.b200_op_linear_reg(cptr(x), cptr(wt), cptr(y), cptr(res), M, N, K, epi, rows, _stream()))
        torch.cuda.synchronize()
    before = lib.b200_op_set_gemv_max_rows(0)
    try:
        _lib.check(lib.b200_op_linear_sk(cptr(x), cptr(wt), cptr(ys[2]), cptr(res), M, N, K, epi, rows, 0, 0, 0, _stream()))
        torch.cuda.synchronize()
    finally:
        lib.b200_op_set_gemv_max_rows(before)
    if M <= 8 or -(-(rows or N) // 128) <= torch.cuda.get_device_properties(0).multi_processor_count:
        assert torch.equal(ys[0], ys[2])
    z = x.float() @ w.float().t()
    if epi == RESADD:
        z = res.float() + z.bfloat16().float()
    elif epi == GATE:
        z = z.bfloat16()
        z = (F.silu(z[:, :rows].float()).bfloat16() * z[:, rows:]).float()
    # a bf16 rounding of the sums, one of the gate's activation and one of the result: three half ulps (2^-9) of values up to ~5, plus fp32 order
    assert torch.equal(ys[0], ys[1])
    torch.testing.assert_close(ys[0].float(), z, rtol=2.0 ** -7, atol=3e-2)


@pytest.mark.parametrize("M", [1, 5, 16, 31])
@pytest.mark.parametrize("N,K,epi", [(130, 144, STORE), (4096, 2816, RESADD), (600, 4096, GATE)])
def test_register_linear_int8_is_exact(M, N, K, epi):
    """Exact sums; the gated pair of 31 rows goes to the kernel of gemm_sk.cu, on the other side of the line."""
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

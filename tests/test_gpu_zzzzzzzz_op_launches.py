"""GPU: the kernel-level entry points, launched early behind one another, read nothing before the kernel in front is done."""
import ctypes as C

import pytest
import torch

from .util import cptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 6, 20, 24, 104])      # whole rows, registers, swap-AB and non-swapped kernels
def test_linears_behind_the_kernels_that_write_their_operands(M):
    """Weights packed, rows written by a linear, and both used by the next linear, with and without a wait in between: the same bits."""
    from moshi_b200 import _lib
    lib, N = _lib.lib(), 4096
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    g = torch.Generator().manual_seed(M)
    x0 = torch.randn(M, N, generator=g).bfloat16().cuda()
    ws = [(torch.randn(N, N, generator=g) / N ** 0.5).bfloat16().cuda() for _ in range(3)]
    out = []
    for wait in (True, False):
        tiles = torch.empty(lib.b200_op_packed_bytes(N, N, 0, 0), dtype=torch.uint8, device="cuda")
        q = torch.empty(lib.b200_op_packed_bytes_i8(N, N, 0, 0), dtype=torch.uint8, device="cuda")
        sw, xq, sa = torch.empty(N, device="cuda"), torch.empty(M, N, dtype=torch.int8, device="cuda"), torch.empty(M, device="cuda")
        x, y = x0.clone(), torch.empty_like(x0)
        torch.cuda.synchronize()
        for w in ws:                          # the same buffers over and over: tiles and rows are rewritten right in front of their reader
            calls = [lambda: lib.b200_op_pack_tiles(cptr(w), cptr(tiles), N, N, 0, 0, st),
                     lambda: lib.b200_op_linear_sk(cptr(x), cptr(tiles), cptr(y), cptr(None), M, N, N, 0, 0, 0, 0, 0, st),
                     lambda: lib.b200_op_quant_pack_tiles(cptr(w), cptr(q), cptr(sw), N, N, 0, 0, st),
                     lambda: lib.b200_op_quantize_rows(cptr(y), cptr(xq), cptr(sa), M, N, st),
                     lambda: lib.b200_op_linear_i8(cptr(xq), cptr(sa), cptr(q), cptr(sw), cptr(x), cptr(None), M, N, N, 0, 0, st)]
            for call in calls:
                _lib.check(call())
                if wait:
                    torch.cuda.synchronize()
        torch.cuda.synchronize()
        out.append(x)
    assert not torch.isnan(out[0].float()).any()
    assert torch.equal(out[0], out[1])

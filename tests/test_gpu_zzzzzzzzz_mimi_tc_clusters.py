"""GPU: mimi_tc_kernel where k is cut over a cluster, where few rows exist of a tile, and with widths that do not fill its runs of columns."""
import ctypes as C

import pytest
import torch
import torch.nn.functional as F

from .util import cptr

pytestmark = pytest.mark.gpu

# B, cin, cout, k, stride, T; transposed convolutions (k = 2 stride) with a minus in front of k
CASES = [(b, 256, 256, 3, 1, 2) for b in (1, 3, 7, 8, 9, 31, 40, 56, 57, 63, 64, 65, 104)]           # rows of a tile from 2 to 128, features as the tensor core's rows below 113
CASES += [(2, 32, 128, k, 1, 2) for k in (1, 2, 3, 4, 5, 7, 8, 9, 15, 17, 33)]                       # k-blocks: clusters of 1 to 8, remainders, chains of one k-block and of four
CASES += [(3, 64, c, 7, 1, 32) for c in (16, 32, 48, 64, 80, 96, 112)]                               # columns: runs of four that do not deal out evenly
CASES += [(40, 64, c, 3, 1, 1920) for c in (32, 48, 64, 128)]                                        # many tiles, one CTA each, without clusters
CASES += [(1, 512, 1024, 16, 8, 16), (33, 512, 128, 16, 8, 16), (2, 1024, 512, -16, 8, 2), (41, 64, 2, -16, 8, 4), (3, 96, 6, -16, 8, 5)]


@pytest.mark.parametrize("B,cin,cout,k,stride,T", CASES)
def test_conv_against_64_bits(B, cin, cout, k, stride, T):
    """Per product 2^-21 for the parts that are left out or rounded; 48 additions of a chain that may cut off a bit of 2^-23 each, as many in fp32 behind them."""
    from moshi_b200 import _lib
    g = torch.Generator().manual_seed(B + cout)
    transposed, k = k < 0, abs(k)
    x = torch.randn(B, cin, T, generator=g).cuda()
    w = (torch.randn(*((cin, cout, k) if transposed else (cout, cin, k)), generator=g) / (cin * (2 if transposed else k)) ** 0.5).cuda()
    bias = torch.randn(cout, generator=g).cuda()
    P = 1 if transposed else k - stride
    prev = torch.randn(B, cin, max(P, 1), generator=g).cuda()[:, :, :P].contiguous()
    mask = torch.ones(B, dtype=torch.bool, device="cuda")
    xin = torch.cat([prev, F.elu(x)], -1).double()               # the carried rows are activations already
    if transposed:
        conv = lambda a, b: F.conv_transpose1d(a, b, stride=stride)[..., stride:stride * (T + 1)]
    else:
        conv = lambda a, b: F.conv1d(a, b, stride=stride)
    want, size = conv(xin, w.double()) + bias.double()[:, None], conv(xin.abs(), w.double().abs())
    y = torch.full(want.shape, float("nan"), device="cuda")
    _lib.check(_lib.lib().b200_op_tc_conv1d(cptr(x), cptr(w), cptr(bias), cptr(prev) if P > 0 else None, cptr(mask), cptr(y), B, cin, cout, T, k, stride, 1, 1, int(transposed),
                                            C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    assert not torch.isnan(y).any()
    bound = (2.0 ** -21 + 96 * 2.0 ** -23) * size + 2.0 ** -22 * (want.abs() + bias.double().abs()[:, None])
    assert bool(((y.double() - want).abs() <= bound).all())

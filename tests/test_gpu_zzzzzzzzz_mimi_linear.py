"""GPU: the linears of Mimi's bottleneck transformers at every kernel and tile that few tokens take (mimi_lin.cuh, mimi_tile.cuh), against 64 bits."""
import ctypes as C

import pytest
import torch
import torch.nn.functional as F

from .util import cptr

pytestmark = pytest.mark.gpu
STORE, GELU, RESIDUAL = 0, 1, 2


@pytest.mark.parametrize("N,K,norm,epi", [(1536, 512, True, STORE), (2048, 512, True, GELU), (512, 512, False, RESIDUAL), (512, 2048, False, RESIDUAL), (48, 512, False, STORE),
                                          (64, 1024, False, GELU), (4096, 512, True, STORE)])
@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33, 48, 49, 64, 130])
def test_linear_against_64_bits(M, N, K, norm, epi):
    """Every sum within the bound of fp32 sums whose chains are no longer than K / 8 additions, the norm's own rounding (eight more) included."""
    from moshi_b200 import _lib
    g = torch.Generator().manual_seed(M * 7 + N)
    x = (torch.randn(M, K, generator=g) + 0.5).cuda()
    w = (torch.randn(N, K, generator=g) / K ** 0.5).cuda()
    gamma, beta = (1 + 0.1 * torch.randn(K, generator=g)).cuda(), (0.1 * torch.randn(K, generator=g)).cuda()
    res, scale = torch.randn(M, N, generator=g).cuda(), (0.3 * torch.randn(N, generator=g)).cuda()
    y = torch.full((M + 1, N), float("nan"), device="cuda")
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(_lib.lib().b200_op_mimi_linear(cptr(x), cptr(gamma) if norm else None, cptr(beta) if norm else None, cptr(w), cptr(res), cptr(scale), cptr(y), M, N, K, epi, stream))
    torch.cuda.synchronize()
    xn = x.double()
    if norm:
        xn = F.layer_norm(xn, (K,), gamma.double(), beta.double(), 1e-5)
    want, size = xn @ w.double().t(), xn.abs() @ w.double().abs().t()
    bound = (K / 8 + 8) * 2.0 ** -24 * size + (2.0 ** -20 * size if norm else 0)
    if epi == GELU:                        # its slope is at most 1.13; erff itself is good to 2 units in the last place
        want, bound = F.gelu(want), 1.13 * bound + 2.0 ** -21 * want.abs()
    elif epi == RESIDUAL:
        want, bound = res.double() + scale.double() * want, scale.double().abs() * bound + 2.0 ** -22 * (res.double().abs() + size * scale.double().abs())
    assert torch.isnan(y[M]).all() and not torch.isnan(y[:M]).any()
    assert bool(((y[:M].double() - want).abs() <= bound + 1e-30).all())

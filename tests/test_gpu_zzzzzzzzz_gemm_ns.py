"""GPU: linears of 33..256 rows (gemm_ns_kernel): results through shared memory in pieces of eight columns, every unit and split of its plan."""
import ctypes as C

import pytest
import torch

from .util import cptr

pytestmark = pytest.mark.gpu
STORE, RESIDUAL, GATED = 0, 1, 2


@pytest.mark.parametrize("M", [1, 33, 64, 127, 128, 129, 200, 255, 256])
@pytest.mark.parametrize("N,K,epi,cluster", [(148 * 128, 128, STORE, 0), (149 * 128 - 8, 72, STORE, 0), (75 * 128 - 120, 200, RESIDUAL, 0), (74 * 128, 512, RESIDUAL, 0), (2056, 520, RESIDUAL, 0),
                                             (1032, 640, RESIDUAL, 0), (264, 4104, STORE, 0), (2 * 392, 328, GATED, 0), (648, 576, RESIDUAL, 3), (392, 576, STORE, 8), (392, 1032, STORE, 107)])
def test_linear_ns(M, N, K, epi, cluster):
    """One tile per SM, one more, K whole and cut (a range without a k-block among them), last tiles that are not full; every sum within the bound of K products in fp32, the
    bf16 roundings of the epilogue behind it (gated: of gate, value, unit and product, the unit's slope being at most 1.1)."""
    from moshi_b200 import _lib
    lib = _lib.lib()
    g = torch.Generator().manual_seed(M + N + K)
    gate = N // 2 if epi == GATED else 0
    x = torch.randn(M, K, generator=g).bfloat16().cuda()
    w = (torch.randn(N, K, generator=g) / K ** 0.5).bfloat16().cuda()
    cols = gate or N
    res = torch.randn(M, N, generator=g).bfloat16().cuda() if epi == RESIDUAL else None
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    wt = torch.empty(lib.b200_op_packed_bytes(N, K, epi, gate), dtype=torch.uint8, device="cuda")
    _lib.check(lib.b200_op_pack_tiles(cptr(w), cptr(wt), N, K, epi, gate, stream))
    y = torch.full((M + 1, cols), 7.0, dtype=torch.bfloat16, device="cuda")
    _lib.check(lib.b200_op_linear_ns(cptr(x), cptr(wt), cptr(y), cptr(res), M, N, K, epi, gate, cluster, stream))
    z, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    err = (K + 8) * 2.0 ** -23 * size
    if epi == GATED:
        a, u = z.chunk(2, -1)
        ea, eu = (err + 2.0 ** -8 * z.abs()).chunk(2, -1)
        s = a * torch.sigmoid(a)
        want = s * u
        err = (1.1 * ea + 2.0 ** -8 * s.abs()) * (u.abs() + eu) + s.abs() * eu + 2.0 ** -8 * want.abs()
    elif epi == RESIDUAL:
        want = res.double() + z
        err = err + 2.0 ** -8 * z.abs() + 2.0 ** -8 * (want.abs() + err)
    else:
        want, err = z, err + 2.0 ** -8 * z.abs()
    assert bool(((y[:M].double() - want).abs() <= err + 1e-30).all())
    assert (y[M] == 7.0).all()


@pytest.mark.parametrize("M", [128, 129, 200, 256])
@pytest.mark.parametrize("N,K,epi,cluster", [(4096, 4096, RESIDUAL, 0), (4096, 1024, STORE, 0), (2056, 520, RESIDUAL, 0), (640, 1024, STORE, 8), (648, 576, RESIDUAL, 102), (640, 1024, STORE, 108)])
def test_blocks_of_sessions_one_after_the_other(M, N, K, epi, cluster):
    """Two blocks of 128 sessions pass their sums through the same shared memory of a cluster: the second may overwrite what its neighbours have read.  Small whole numbers, whose
    sums are exact in whatever order they are added: the bits of the plain computation, launch after launch."""
    from moshi_b200 import _lib
    lib = _lib.lib()
    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randint(-8, 9, (M, K), generator=g).bfloat16().cuda()
    w = torch.randint(-8, 9, (N, K), generator=g).bfloat16().cuda()
    res = torch.randn(M, N, generator=g).bfloat16().cuda() if epi == RESIDUAL else None
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    wt = torch.empty(lib.b200_op_packed_bytes(N, K, epi, 0), dtype=torch.uint8, device="cuda")
    _lib.check(lib.b200_op_pack_tiles(cptr(w), cptr(wt), N, K, epi, 0, stream))
    y = torch.full((12, M, N), 7.0, dtype=torch.bfloat16, device="cuda")
    for i in range(12):
        _lib.check(lib.b200_op_linear_ns(cptr(x), cptr(wt), cptr(y[i]), cptr(res), M, N, K, epi, 0, cluster, stream))
    want = (x.double() @ w.double().t()).bfloat16()          # below 2^24: what fp32 holds exactly, rounded once
    if res is not None:
        want = (res.float() + want.float()).bfloat16()
    assert all(torch.equal(y[i], want) for i in range(12))

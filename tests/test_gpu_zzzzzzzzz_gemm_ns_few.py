"""GPU: gemm_ns_kernel from 17 rows on: boxes of as many activation rows as there are (to whole eights), what the tensor cores read beyond them, accumulators taken in turn, int8;
output rows shared out in sixteens: units inside a tile, across two or three, a last one that is not full, one more wave.  By its own entry point at every shape, and by the general
ones, which send some of the shapes of up to 32 rows to gemm_reg.cu and gemm_sk.cu (`general` has the kernel of each; test_op_routes_cpu.py holds it to that)."""
import ctypes as C

import pytest
import torch
import torch.nn.functional as F

from .util import cptr

pytestmark = pytest.mark.gpu
STORE, RESIDUAL, GATED = 0, 1, 2
SHAPES = [(130, 144, STORE), (264, 4112, RESIDUAL), (75 * 128, 80, RESIDUAL), (149 * 128 - 8, 256, STORE), (2 * 392, 336, GATED), (4096, 1024, RESIDUAL),
          (2 * 2824, 592, GATED), (2 * (148 * 32 + 8), 128, GATED), (2 * 18952, 80, GATED), (37896, 144, STORE),
          (2 * 11264, 512, GATED), (2 * 25600, 1024, GATED), (2 * 392, 4112, GATED), (2 * 2824, 4112, GATED), (2 * 18952, 4112, GATED), (149 * 128 - 8, 4112, STORE), (4096, 4112, RESIDUAL)]
ROWS = [17, 24, 25, 32, 33, 127, 129, 136, 256]


def general(M, N, K, epi, i8):
    """The kernels, one of which the general entry points take for these shapes."""
    if i8 and M > 32:
        tiles, blocks, ranks = -(-N // 128), -(-K // 128), 1            # few tiles: k over a cluster, each of whose CTAs finishes up to 64 rows
        while ranks < 8 and tiles * ranks * 2 <= 148 and blocks >= 8 * ranks and (ranks < 4 or tiles <= 15):
            ranks *= 2
        pad = -(-M // (8 * ranks)) * 8 * ranks
        return ("gemm_ck", "gemm_sk") if epi != GATED and ranks > 1 and pad <= 256 and pad <= 64 * ranks else ("gemm_sk",) if N % 8 else ("gemm_ns",)
    if M > 32 or (K >= 4096 and (i8 or epi != GATED)):
        return ("gemm_ns",)
    return ("gemm_sk",) if epi == GATED or (not i8 and N > 148 * 128) else ("gemm_reg",)


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _case(M, N, K, epi, whole):
    g = torch.Generator().manual_seed(M + N + K)
    if whole:
        x, w = (torch.randint(-127, 128, s, generator=g, dtype=torch.int8).cuda() for s in ((M, K), (N, K)))
    else:
        x, w = torch.randn(M, K, generator=g).bfloat16().cuda(), (torch.randn(N, K, generator=g) / K ** 0.5).bfloat16().cuda()
    return x, w, torch.randn(M, N, generator=g).bfloat16().cuda() if epi == RESIDUAL else None, N // 2 if epi == GATED else 0


@pytest.mark.parametrize("M", ROWS)
@pytest.mark.parametrize("N,K,epi", SHAPES)
def test_int8(M, N, K, epi):
    """Whole numbers, scaled by the same three products and rounded once: the bits of the plain computation; gated: the unit's two roundings apart (a bf16 step each of unit and
    product, the exponential's error far below)."""
    from moshi_b200 import _lib
    lib = _lib.lib()
    x, q, res, gate = _case(M, N, K, epi, True)
    w = q.float().bfloat16()
    w[:, 0] = 127.0                                     # every row's largest value: what is quantised comes out as it went in
    q = w.to(torch.int8)
    tiles = torch.empty(lib.b200_op_packed_bytes_i8(N, K, epi, gate), dtype=torch.uint8, device="cuda")
    sw = torch.empty(N, device="cuda")
    _lib.check(lib.b200_op_quant_pack_tiles(cptr(w), cptr(tiles), cptr(sw), N, K, epi, gate, _stream()))
    sw.copy_(torch.rand(N, generator=torch.Generator().manual_seed(K)))
    sa = torch.rand(M, generator=torch.Generator().manual_seed(M)).cuda()
    y = torch.full((M + 1, gate or N), 7.0, dtype=torch.bfloat16, device="cuda")
    _lib.check(lib.b200_op_linear_i8(cptr(x), cptr(sa), cptr(tiles), cptr(sw), cptr(y), cptr(res), M, N, K, epi, gate, _stream()))
    sums = (x.double() @ q.double().t()).float()
    z = sums * (sa[:, None] * sw[None, :] * torch.tensor(1.0 / 16129.0, dtype=torch.float32, device="cuda"))
    z = z.bfloat16().float()
    if epi == GATED:
        want = F.silu(z[:, :gate]).bfloat16().float() * z[:, gate:]
        assert bool(((y[:M].float() - want).abs() <= 2.0 ** -7 * want.abs() + 1e-30).all())
    else:
        assert torch.equal(y[:M], (res.float() + z).bfloat16() if epi == RESIDUAL else z.bfloat16())
    assert (y[M] == 7.0).all()


@pytest.mark.parametrize("N,K,epi", SHAPES)
@pytest.mark.parametrize("M,entry,shift", [(M, "ns", 0) for M in ROWS] + [(M, "general", shift) for M in ROWS if M <= 32 for shift in (0, 1)])
def test_bf16(M, N, K, epi, entry, shift):
    """Every sum within the bound of K products in fp32, the epilogue's bf16 roundings behind it; up to 32 rows by the general entry point too, with results on a 16-byte border and
    (other kernels) not."""
    if entry == "ns" and N % 8:
        pytest.skip("results of the kernel lie on 16 bytes")
    from moshi_b200 import _lib
    lib = _lib.lib()
    x, w, res, gate = _case(M, N, K, epi, False)
    wt = torch.empty(lib.b200_op_packed_bytes(N, K, epi, gate), dtype=torch.uint8, device="cuda")
    _lib.check(lib.b200_op_pack_tiles(cptr(w), cptr(wt), N, K, epi, gate, _stream()))
    cols = gate or N
    flat = torch.full((M * cols + 8,), 7.0, dtype=torch.bfloat16, device="cuda")
    y = flat[shift:shift + M * cols].view(M, cols)
    if entry == "ns":
        _lib.check(lib.b200_op_linear_ns(cptr(x), cptr(wt), cptr(y), cptr(res), M, N, K, epi, gate, 0, _stream()))
    else:
        _lib.check(lib.b200_op_linear_sk(cptr(x), cptr(wt), cptr(y), cptr(res), M, N, K, epi, gate, 0, 0, 0, _stream()))
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
    assert bool(((y.double() - want).abs() <= err + 1e-30).all())
    assert (flat[:shift] == 7.0).all() and (flat[shift + M * cols:] == 7.0).all()

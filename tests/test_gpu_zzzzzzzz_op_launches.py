"""GPU: the kernel-level entry points, launched early behind one another, read nothing before the kernel in front is done."""
import ctypes as C

import pytest
import torch

from .util import cptr

pytestmark = pytest.mark.gpu
STORE, RESADD, GATE = 0, 1, 2

# kernel -> (rows, outputs, inputs, epilogue, int8) of a linear that takes it; test_op_routes_cpu.py shows that it does.  Weights and rows of each fit what any of the
# writers leaves.
LINEARS = {
    "gemm_row_kernel": [(1, 1024, 384, STORE, False), (6, 1024, 384, GATE, False), (16, 1024, 384, RESADD, False), (9, 768, 1024, STORE, True)],
    "gemm_reg_kernel": [(20, 1024, 384, RESADD, False), (24, 768, 1024, STORE, True)],
    "gemm_sk_kernel": [(20, 1024, 384, GATE, False), (24, 768, 1024, GATE, True)],
    "gemm_ns_kernel": [(104, 1024, 384, STORE, False), (200, 1024, 384, RESADD, False)],
    "gemm_ck_kernel": [(104, 768, 1024, STORE, True)],
}
# linears whose results, as bytes, are what the next kernel reads
WRITERS = {"gemm_row_kernel": (16, 32000, 2048, STORE, False), "gemm_reg_kernel": (24, 18944, 2048, STORE, False), "gemm_ns_kernel": (104, 4096, 4096, STORE, False)}


def linear(lib, shape, x, tiles, out, res=None, sa=None, sw=None, st=None):
    M, N, K, epi, i8 = shape
    gate = N // 2 if epi == GATE else 0
    if i8:
        return lib.b200_op_linear_i8(x, sa, tiles, sw, out, res, M, N, K, epi, gate, st)
    return lib.b200_op_linear_sk(x, tiles, out, res, M, N, K, epi, gate, 0, 0, 0, st)


class Writer:
    """A linear into ``buf`` from other rows at every call."""

    def __init__(self, lib, name, calls):
        self.lib, self.shape = lib, WRITERS[name]
        M, N, K, _, _ = self.shape
        g = torch.Generator(device="cuda").manual_seed(N)
        w = torch.randn(N, K, device="cuda", generator=g).mul_(K ** -0.5).bfloat16()
        self.x = [torch.randn(M, K, device="cuda", generator=g).bfloat16() for _ in range(calls)]
        self.tiles = torch.empty(lib.b200_op_packed_bytes(N, K, 0, 0), dtype=torch.uint8, device="cuda")
        assert lib.b200_op_pack_tiles(cptr(w), cptr(self.tiles), N, K, 0, 0, _stream()) == 0
        self.buf = torch.zeros(M * N, dtype=torch.bfloat16, device="cuda")

    def __call__(self, i):
        assert linear(self.lib, self.shape, cptr(self.x[i]), cptr(self.tiles), cptr(self.buf), st=_stream()) == 0


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _twice(write, read, calls=4):
    """Results of `calls` pairs of writer and reader, with a wait behind every launch and without any."""
    got = []
    for wait in (True, False):
        write.buf.zero_()
        torch.cuda.synchronize()
        outs = []
        for i in range(calls):
            write(i)
            if wait:
                torch.cuda.synchronize()
            outs.append(read())
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        got.append(outs)
    for a, b in zip(*got):
        assert all(torch.equal(s.view(torch.uint8), t.view(torch.uint8)) for s, t in zip(a, b))
    assert not torch.equal(got[0][0][0], got[0][1][0])        # each writer's results matter


@pytest.mark.parametrize("writer", sorted(WRITERS))
@pytest.mark.parametrize("kernel,shape,role", [(k, s, r) for k, shapes in LINEARS.items() for s in shapes for r in ["weights", "rows"] + ["residual"] * (s[3] == RESADD)])
def test_linears_behind_the_kernel_that_writes_their_operands(kernel, shape, role, writer):
    from moshi_b200 import _lib
    lib = _lib.lib()
    M, N, K, epi, i8 = shape
    write, cols, es = Writer(lib, writer, 4), N // 2 if epi == GATE else N, 1 if i8 else 2
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K, device="cuda", generator=g)
    x = x.mul_(40).clamp_(-127, 127).to(torch.int8) if i8 else x.bfloat16()
    tiles = torch.randn(-(-N // 128) * -(-K * es // 128) * 8192, device="cuda", generator=g).mul_(0.05).bfloat16()
    sa, sw = torch.rand(M, device="cuda", generator=g), torch.rand(N, device="cuda", generator=g)
    res = torch.randn(M, cols, device="cuda", generator=g).bfloat16() if epi == RESADD else None
    need = {"weights": tiles.numel() * 2, "rows": M * K * es, "residual": M * cols * 2}[role]
    assert need <= write.buf.numel() * 2
    if role == "weights":
        tiles = write.buf
    elif role == "rows":
        x = write.buf
    else:
        res = write.buf

    def read():
        y = torch.empty(M, cols, dtype=torch.bfloat16, device="cuda")
        assert linear(lib, shape, cptr(x), cptr(tiles), cptr(y), cptr(res), cptr(sa), cptr(sw), _stream()) == 0
        return (y,)

    _twice(write, read)


@pytest.mark.parametrize("writer", sorted(WRITERS))
def test_row_quantisation_behind_the_kernel_that_writes_its_rows(writer):
    from moshi_b200 import _lib
    lib, write = _lib.lib(), Writer(_lib.lib(), writer, 4)

    def read():
        xq, sa = torch.empty(96, 4096, dtype=torch.int8, device="cuda"), torch.empty(96, device="cuda")
        assert lib.b200_op_quantize_rows(cptr(write.buf), cptr(xq), cptr(sa), 96, 4096, _stream()) == 0
        return xq, sa

    _twice(write, read)


@pytest.mark.parametrize("role", ["ring", "qkv"])
@pytest.mark.parametrize("writer", sorted(WRITERS))
def test_attention_step_behind_the_kernel_that_writes_its_ring(writer, role):
    """One session of two heads and 700 keys, and its projections, from what a linear has just written; the step appends to the ring itself."""
    from moshi_b200 import _lib
    lib, write = _lib.lib(), Writer(_lib.lib(), writer, 4)
    H, cap, D = 2, 800, 128
    g = torch.Generator(device="cuda").manual_seed(1)
    qkv = torch.randn(3 * H * D, device="cuda", generator=g).bfloat16()
    ring = torch.randn(2, H * cap * D, device="cuda", generator=g).bfloat16()
    pos, mask = torch.tensor([700], device="cuda"), torch.ones(1, dtype=torch.uint8, device="cuda")
    if role == "ring":
        assert 2 * H * cap * D <= write.buf.numel()
        ring = write.buf[:2 * H * cap * D].view(2, -1)
    else:
        qkv = write.buf

    def read():
        out = torch.empty(H * D, dtype=torch.bfloat16, device="cuda")
        _lib.check(lib.b200_op_attn_step(cptr(qkv), cptr(ring[0]), cptr(ring[1]), cptr(out), cptr(pos), cptr(mask), 1, H, cap, 0, 1e4, _stream()))
        return (out,)

    _twice(write, read)


def test_entry_points_in_a_graph_with_a_fork():
    """Captured behind one another, with a branch on a stream of its own: replays give the eager bits."""
    from moshi_b200 import _lib
    lib, write = _lib.lib(), Writer(_lib.lib(), "gemm_ns_kernel", 1)
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(20, 384, device="cuda", generator=g).bfloat16()
    y = [torch.empty(M, 1024, dtype=torch.bfloat16, device="cuda") for M in (1, 6, 16)]
    xq, sa = torch.empty(96, 4096, dtype=torch.int8, device="cuda"), torch.empty(96, device="cuda")
    side = torch.cuda.Stream()

    def work():
        write(0)
        here = torch.cuda.current_stream()
        side.wait_stream(here)
        with torch.cuda.stream(side):
            assert lib.b200_op_quantize_rows(cptr(write.buf), cptr(xq), cptr(sa), 96, 4096, _stream()) == 0
        for o, M in zip(y, (1, 6, 16)):
            assert linear(lib, (M, 1024, 384, STORE, False), cptr(x), cptr(write.buf), cptr(o), st=_stream()) == 0
        here.wait_stream(side)

    work()
    torch.cuda.synchronize()
    want = [t.clone() for t in (*y, xq, sa)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        work()
    for _ in range(3):
        for t in (*y, xq, sa, write.buf):
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip((*y, xq, sa), want))

"""Host state that belongs to one device (kernels' limits of shared memory, workspaces), with a second device in the same process."""
import ctypes as C
import re

import pytest

from moshi_b200.build import CSRC

from . import fake_cuda

STORE, RESADD, GATE = 0, 1, 2


@pytest.fixture
def fake(tmp_path):
    return fake_cuda.load(tmp_path)


def _linear(fake, M, N=4096, K=4096, epi=STORE, i8=False):
    p = C.create_string_buffer(64)
    at = C.c_void_p((C.addressof(p) + 15) // 16 * 16)
    rows, res = N // 2 if epi == GATE else 0, at if epi == RESADD else None
    if i8:
        return fake.b200_op_linear_i8(at, at, at, at, at, res, M, N, K, epi, rows, None)
    return fake.b200_op_linear_sk(at, at, at, res, M, N, K, epi, rows, 0, 0, 0, None)


@pytest.mark.parametrize("i8", [False, True])
def test_linears_of_few_rows_on_a_second_device(fake, i8):
    for dev in (0, 1, 0):
        fake.cudaSetDevice(dev)
        for M, epi in ((1, STORE), (2, RESADD), (6, GATE), (12, STORE)):
            fake_cuda.check(fake, _linear(fake, M, epi=epi, i8=i8))
            ((at, name),) = fake_cuda.launches(fake)
            assert at == dev and "gemm_row_kernel" in name


def test_a_refused_limit_is_asked_for_again(fake):
    fake_cuda.check(fake, _linear(fake, 20))          # what all kernels share
    fake.fake_refuse_attributes(1)
    assert _linear(fake, 1) != 0
    fake_cuda.check(fake, _linear(fake, 1))


def _stores(fake, op):
    p = C.create_string_buffer(1 << 22)
    return op(C.c_void_p((C.addressof(p) + 255) // 256 * 256))


@pytest.mark.parametrize("name,call", [
    ("gemm_sk_kernel", lambda f: _linear(f, 24, 22528, 4096, GATE)), ("gemm_ns_kernel", lambda f: _linear(f, 104)),
    ("gemm_ck_kernel", lambda f: _linear(f, 104, i8=True)), ("gemm_wide_kernel", lambda f: _stores(f, lambda p: f.b200_op_linear_wide(p, p, p, 512, 512, 512, 512, 1, 1, None))),
    ("mimi_tc_kernel", lambda f: _stores(f, lambda p: f.b200_op_tc_linear_f32(p, p, p, 64, 256, 64, None))),
    ("flash_attention_kernel", lambda f: _stores(f, lambda p: f.b200_op_prefill_attention(p, p, p, None, p, 128, 1, 0, 128, 1.0, None)))])
def test_other_kernels_on_a_second_device(fake, name, call):
    for dev in (0, 1):
        fake.cudaSetDevice(dev)
        fake_cuda.check(fake, call(fake))
        got = fake_cuda.launches(fake)
        assert any(name in n for _, n in got) and all(at == dev for at, _ in got)


def test_limits_are_raised_per_device_everywhere():
    """The one place that raises a kernel's limit is the one that keeps book per device (dep_fused.cu: with every handle)."""
    at = [(f.name, f.read_text().count("cudaFuncSetAttribute")) for f in sorted(CSRC.glob("*.cu*"))]
    assert {n for n, c in at if c} <= {"common.cuh", "dep_fused.cu"}
    for f in CSRC.glob("*.cu*"):
        assert not re.search(r"static (bool|const cudaError_t) \w*(attr|once)", f.read_text()), f.name


def _attention(fake, sessions, q8):
    def op(p):
        if q8:
            return fake.b200_op_attn_step_q8(p, p, p, p, p, p, p, p, sessions, 32, 3000, 0, 1e4, 1, None)
        return fake.b200_op_attn_step(p, p, p, p, p, p, sessions, 32, 3000, 0, 1e4, None)
    return _stores(fake, op)


@pytest.mark.parametrize("call,larger", [(lambda f: _linear(f, 20), None), (lambda f: _linear(f, 20, i8=True), None),
                                         (lambda f: _attention(f, 1, False), lambda f: _attention(f, 48, False)), (lambda f: _attention(f, 1, True), lambda f: _attention(f, 48, True))])
def test_workspaces_lie_on_the_device_of_the_call(fake, call, larger):
    """Partial results of work that is cut: another device's kernels could not write them.  They are kept, and grow with the largest call."""
    for dev in (0, 1):
        fake.cudaSetDevice(dev)
        before = fake.fake_held(dev)
        fake_cuda.check(fake, call(fake))
        once = fake.fake_held(dev)
        assert once > before
        fake_cuda.check(fake, call(fake))
        assert fake.fake_held(dev) == once
        if larger:
            fake_cuda.check(fake, larger(fake))
            assert (most := fake.fake_held(dev)) > once
            fake_cuda.check(fake, call(fake))
            assert fake.fake_held(dev) == most


@pytest.mark.parametrize("sessions", [1, 104])
def test_the_attention_says_how_much_l1_it_wants(fake, sessions):
    """On every device: the ring's keys and values on their way need most of an SM's L1, whose division a kernel without a preference takes over from the linear in front of it."""
    for dev in (0, 1):
        fake.cudaSetDevice(dev)
        fake_cuda.check(fake, _attention(fake, sessions, False))
        assert "attn_step_kernel" in fake_cuda.launches(fake)[-1][1]
        assert 10 <= fake.fake_share() <= 50            # four CTAs' shared memory, and room for what they have under way

"""Host state that belongs to one device (kernels' limits of shared memory, workspaces), with a second device in the same process."""
import ctypes as C

import pytest

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

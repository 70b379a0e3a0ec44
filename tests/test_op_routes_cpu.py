"""Which kernel an entry point takes, on the fake CUDA runtime."""
import ctypes as C

import pytest

from . import fake_cuda


def _kernel(fake, M):
    p = C.create_string_buffer(64)
    at = C.c_void_p((C.addressof(p) + 15) // 16 * 16)
    fake_cuda.launches(fake)
    fake_cuda.check(fake, fake.b200_op_linear_sk(at, at, at, None, M, 4096, 4096, 0, 0, 0, 0, 0, None))
    ((_, name),) = fake_cuda.launches(fake)
    return name


@pytest.mark.parametrize("name", ["B200_ROW_MAX_M", "B200_GEMV_MAX_M"])
def test_rows_up_to_which_whole_rows_per_cta_are_considered(tmp_path, monkeypatch, name):
    """The older name of the setting counts too."""
    monkeypatch.setenv(name, "2")
    fake = fake_cuda.load(tmp_path)
    assert "gemm_row_kernel" in _kernel(fake, 2)
    assert "gemm_reg_kernel" in _kernel(fake, 3)
    assert fake.b200_op_set_gemv_max_rows(16) == 2
    assert "gemm_row_kernel" in _kernel(fake, 3)

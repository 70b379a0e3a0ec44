"""Which kernel an entry point takes, on the fake CUDA runtime."""
import ctypes as C

import pytest

from . import fake_cuda
from . import test_gpu_zzzzzzzzz_gemm_expert as gemm_expert
from . import test_gpu_zzzzzzzzz_gemm_ns_few as ns_few
from .test_gpu_zzzzzzzz_op_launches import GATE, LINEARS, RESADD, STORE, WRITERS, linear


def _kernel(fake, shape):
    p = C.create_string_buffer(64)
    at = C.c_void_p((C.addressof(p) + 15) // 16 * 16)
    fake_cuda.launches(fake)
    fake_cuda.check(fake, linear(fake, shape, at, at, at, at if shape[3] == RESADD else None, at, at))
    ((_, name),) = fake_cuda.launches(fake)
    return name


def test_linears_of_the_early_launch_tests_take_the_kernels_they_name(tmp_path):
    fake = fake_cuda.load(tmp_path)
    for kernel, shapes in [*LINEARS.items(), *((k, [s]) for k, s in WRITERS.items())]:
        for shape in shapes:
            assert kernel in _kernel(fake, shape), (kernel, shape)


@pytest.mark.parametrize("shape,kernel", [((24, 32000, 2048, STORE, False), "gemm_sk_kernelILi0ELb0E"), ((24, 19072, 2048, STORE, False), "gemm_sk_kernelILi0ELb1E"),
                                          ((200, 2048, 4096, RESADD, True), "gemm_sk_kernelILi1ELb1E"), *(((24, 256 * tiles, k, GATE, False), "gemm_sk_kernelILi2ELb" + str(int(warps)) + "E")
                                          for tiles, k, warps in [(22, 2048, True), (74, 1024, True), (75, 1024, False), (88, 4096, False), (130, 4096, True), (130, 8192, False), (148, 8192, True),
                                                                  (152, 1024, True), (200, 1024, False), (200, 4096, False), (200, 5120, True)])])
def test_who_walks_the_loops_of_the_swapped_kernel(tmp_path, shape, kernel):
    """Whole warps where tiles are whole, for gated pairs also in few tiles and in long ones of several rounds; one thread elsewhere."""
    assert kernel in _kernel(fake_cuda.load(tmp_path), shape)


@pytest.mark.parametrize("M,N,K,kernel", [(24, 512, 11264, "reg"), (24, 520, 11264, "ns"), (25, 256, 11264, "ns"), (24, 256, 11256, "reg"), (24, 256, 8192, "ns"), (24, 1024, 22016, "reg"), (24, 1032, 22016, "ns"),
                                          (32, 512, 22016, "reg"), (32, 640, 22016, "ns"), (17, 128, 19200, "reg"), (32, 128, 19136, "ns")])
def test_few_rows_and_tiles_of_long_k(tmp_path, M, N, K, kernel):
    """Few tiles of long k are cut into more ranges by the kernel with weights in registers than a cluster has."""
    assert f"gemm_{kernel}_kernel" in _kernel(fake_cuda.load(tmp_path), (M, N, K, STORE, False))


@pytest.mark.parametrize("name", ["B200_ROW_MAX_M", "B200_GEMV_MAX_M"])
def test_rows_up_to_which_whole_rows_per_cta_are_considered(tmp_path, monkeypatch, name):
    """The older name of the setting counts too."""
    monkeypatch.setenv(name, "2")
    fake = fake_cuda.load(tmp_path)
    assert "gemm_row_kernel" in _kernel(fake, (2, 4096, 4096, 0, False))
    assert "gemm_reg_kernel" in _kernel(fake, (3, 4096, 4096, 0, False))
    assert fake.b200_op_set_gemv_max_rows(16) == 2
    assert "gemm_row_kernel" in _kernel(fake, (3, 4096, 4096, 0, False))


@pytest.mark.parametrize("q8", [False, True])
def test_attention_steps_refuse_null_pointers(tmp_path, q8):
    """On a GPU the kernel would read address 0."""
    fake = fake_cuda.load(tmp_path)
    p = C.create_string_buffer(64)
    for gone in range(8 if q8 else 6):
        at = [None if i == gone else C.addressof(p) for i in range(8 if q8 else 6)]
        rc = fake.b200_op_attn_step_q8(*at, 1, 2, 8, 0, 1e4, 1, None) if q8 else fake.b200_op_attn_step(*at, 1, 2, 8, 0, 1e4, None)
        assert rc != 0 and not fake_cuda.launches(fake)


@pytest.mark.parametrize("counts,N,K,act,units", [([1] * 2 + [0] * 14, 2048, 4096, 0, True), ([8] * 16, 2048, 4096, 0, False), ([128] + [8] * 15, 2048, 4096, 0, False), ([1] * 10 + [0] * 6, 2048, 4096, 0, True),
                                                  ([4] * 16, 8192, 2048, 2, True), ([16] * 16, 4096, 4096, 0, False), ([2] * 64, 8192, 2048, 3, False), ([64] * 64, 8192, 2048, 3, True),
                                                  ([129] + [1] * 15, 8192, 2048, 2, False),
                                                  *((*case, act, not (act == 0 and case[1] == 148 * 64)) for case in gemm_expert.CASES for act in (0, 2))])
def test_products_of_few_rows_per_expert(tmp_path, counts, N, K, act, units):
    """Units of weight rows dealt over the SMs where tiles would leave a last wave idle or have a gated unit behind them, tiles elsewhere and above 128 rows."""
    fake, p = fake_cuda.load(tmp_path), C.create_string_buffer(256)
    at, E = C.c_void_p((C.addressof(p) + 15) // 16 * 16), len(counts)
    fake_cuda.check(fake, fake.b200_op_grouped_wide(at, at, at, (C.c_int32 * E)(*counts), E, sum(counts), N, K, N, act, 1.0, None))
    ((_, name),) = fake_cuda.launches(fake)
    assert ("gemm_expert_kernel" if units else "gemm_wide_kernel") in name


@pytest.mark.parametrize("i8", [False, True])
def test_linears_of_the_sixteens_take_the_kernels_they_name(tmp_path, i8):
    """What the tests of gemm_ns_kernel send through the general entry points."""
    fake = fake_cuda.load(tmp_path)
    got = {(M, *shape): _kernel(fake, (M, *shape, i8)) for shape in ns_few.SHAPES for M in ns_few.ROWS if i8 or M <= 32}
    wrong = {shape: name for shape, name in got.items() if not any(k + "_kernel" in name for k in ns_few.general(*shape, i8))}
    assert not wrong
    assert any("gemm_ns" in n for s, n in got.items() if s[0] <= 32 and s[3] == (GATE if i8 else STORE))

"""Which kernels the depformer of a stream takes, and that streams do not disturb one another's."""
import pytest

from moshi_b200.config import tiny_lm_config

from . import fake_cuda


@pytest.fixture
def fake(tmp_path):
    return fake_cuda.load(tmp_path)


def _dep(launches):
    return [n for _, n in launches if "dep_reg_kernel" in n or "dep_fused_kernel" in n]


def test_a_second_stream_leaves_the_first_its_shared_memory(fake):
    """The limit of shared memory is the kernel's, not the handle's: a stream of fewer sessions, or of another model, must not lower it."""
    big, small = fake_cuda.LM(fake, tiny_lm_config()), fake_cuda.LM(fake, tiny_lm_config(card=48))
    big.begin(16)
    assert len(_dep(big.step())) == 1
    small.begin(9)
    assert len(_dep(small.step())) == 1
    assert len(_dep(big.step())) == 1
    big.close(), small.close()

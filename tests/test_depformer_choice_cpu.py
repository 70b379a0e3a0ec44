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


@pytest.mark.parametrize("sessions", [1, 2, 3, 16])
@pytest.mark.parametrize("layers,dep_q", [(2, 8), (16, 16), (40, 16)])
def test_few_sessions_of_deep_depformers(fake, sessions, layers, dep_q):
    """As many weights as its shared memory holds the addresses of: the kernel of few sessions."""
    lm = fake_cuda.LM(fake, tiny_lm_config(depformer_num_layers=layers, dep_q=dep_q, n_q=2 * dep_q))
    lm.begin(sessions)
    (name,) = _dep(lm.step())
    assert "dep_reg_kernel" in name
    lm.close()


@pytest.mark.parametrize("sessions", [1, 2, 3, 9, 16])
def test_few_sessions_of_depformers_whose_addresses_lie_in_memory(fake, sessions):
    """More addresses than fit beside the kernel's other shared memory, but no more than it took before that had grown."""
    lm = fake_cuda.LM(fake, tiny_lm_config(depformer_dim=64, depformer_num_heads=1, depformer_dim_feedforward=96, dep_q=16, n_q=32, depformer_num_layers=150))
    lm.begin(sessions)
    (name,) = _dep(lm.step())
    assert "dep_reg_kernel" in name
    lm.close()


@pytest.mark.parametrize("sessions", [1, 2, 3])
@pytest.mark.parametrize("over", [dict(card=9480), dict(depformer_dim=64, depformer_num_heads=1, depformer_dim_feedforward=96, dep_q=16, n_q=32, depformer_num_layers=190)])
def test_few_sessions_of_shapes_that_only_the_shared_memory_kernel_takes(fake, sessions, over):
    """More rows of logits than eight 8-row pieces a CTA, more weights than addresses fit: one and two sessions take a chain of launches, more the
    shared-memory kernel."""
    lm = fake_cuda.LM(fake, tiny_lm_config(**over))
    lm.begin(sessions)
    names = _dep(lm.step())
    assert (not names) if sessions <= 2 else "dep_fused_kernel" in names[0]
    lm.close()

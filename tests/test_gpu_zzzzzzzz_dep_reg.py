"""GPU: the depformer of few sessions (csrc/dep_reg.cuh)."""
import pytest
import torch

from moshi_b200.config import LMConfig
from moshi_b200.synth import synth_lm_state_dict

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lm():
    from moshi_b200.models import LMModel
    cfg = LMConfig(dim=512, num_heads=4, num_layers=1, context=64, text_card=4000, card=2048, depformer_dim=512, depformer_num_heads=8,
                   depformer_dim_feedforward=2112, depformer_num_layers=2)
    return LMModel(cfg, synth_lm_state_dict(cfg, seed=5, device="cuda"), device="cuda")


def _codes(lm, B):
    return torch.randint(0, lm.cfg.card, (B, 8, 1), generator=torch.Generator().manual_seed(B)).cuda()


@pytest.mark.parametrize("B", [1, 12])
def test_a_barrier_that_runs_out_is_reported(lm, B, monkeypatch):
    """With a limit of a nanosecond the blocks give up on one another at their first barriers and the kernel ends at once: the step's flag has
    its name, the next step fails, and one stream later all is well."""
    from moshi_b200 import _lib
    from moshi_b200.models import LMGen
    codes = _codes(lm, B)
    with monkeypatch.context() as m:
        m.setenv("B200_DEP_WAIT_NS", "1")
        gen = LMGen(lm, use_sampling=False)
        with gen.streaming(B):
            gen.step(codes)
            torch.cuda.synchronize()
            with pytest.raises(RuntimeError, match="wait"):
                gen.step(codes)
            assert gen.error_flags() == 8
            out = torch.empty(B, 9, dtype=torch.int64)
            with pytest.raises(RuntimeError, match="wait"):
                gen.step_host(codes[:, :, 0].cpu().contiguous(), None, out)
    gen = LMGen(lm, use_sampling=False)
    with gen.streaming(B):
        for _ in range(3):
            gen.step(codes)
        assert gen.error_flags() == 0
        assert _lib.lib().b200_lm_check_waits(gen._h) == 0


@pytest.mark.parametrize("B", [1, 12])
def test_stamps_of_every_barrier(lm, B, monkeypatch):
    """B200_DEP_TRACE: a stamp at the start and behind each of the 8 x (2 + 5 x layers) barriers, in order, and none beyond."""
    from moshi_b200.models import LMGen
    monkeypatch.setenv("B200_DEP_TRACE", "1")
    gen = LMGen(lm, use_sampling=False)
    with gen.streaming(B):
        gen.step(_codes(lm, B))
        t = gen.read_buffer("dep_trace", torch.int64, (512,)).cpu()
        assert gen.error_flags() == 0
    n = lm.cfg.dep_q * (2 + 5 * lm.cfg.depformer_num_layers)
    assert (t[:n + 1] > 0).all() and (t[n + 1:] == 0).all()
    assert (t[1:n + 1] >= t[:n]).all()

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


SHAPES = {"7b": dict(depformer_dim=1024, depformer_num_heads=16, depformer_dim_feedforward=4224, depformer_num_layers=6, card=2048),
          "odd": dict(depformer_dim=512, depformer_num_heads=8, depformer_dim_feedforward=2088, depformer_num_layers=2, card=2041)}


@pytest.fixture(scope="module", params=sorted(SHAPES))
def pair(request):
    """The same weights behind the persistent kernel and behind the chain of launches."""
    from moshi_b200.models import LMModel
    cfg = LMConfig(dim=512, num_heads=4, num_layers=1, context=64, text_card=4000, **SHAPES[request.param])
    sd = synth_lm_state_dict(cfg, seed=7, device="cuda")
    models = {}
    with pytest.MonkeyPatch.context() as m:
        for name, value in (("kernel", "1"), ("chain", "0")):
            m.setenv("B200_DEP_FUSED", value)
            models[name] = LMModel(cfg, sd, device="cuda")
    return cfg, models


@torch.no_grad()
@pytest.mark.parametrize("B", [1, 2, 8, 9, 13, 16])
def test_depformer_of_few_sessions_agrees_with_the_chain(pair, B):
    """One block of eight sessions and two, full and part empty, at the sizes of the 7B and with rows of logits that end inside a cache line:
    every sub-step's logits as the chain of launches has them, while the tokens chosen before are the same."""
    from moshi_b200 import _lib
    from moshi_b200.models import LMGen
    cfg, models = pair
    got = {}
    for name, lm in models.items():
        gen = LMGen(lm, use_sampling=False)
        gen.use_graph = False
        with gen.streaming(B):
            before = _lib.lib().b200_launch_count()
            rec = []
            for i in range(3):
                g = torch.Generator().manual_seed(100 * B + i)
                gen.step(torch.randint(0, cfg.card, (B, 8, 1), generator=g).cuda())
                rec.append((gen.read_buffer("dep_logits", torch.bfloat16, (cfg.dep_q, B, cfg.card)).float(),
                            gen.read_buffer("audio_tokens", torch.int64, (cfg.dep_q, B))))
            launches = _lib.lib().b200_launch_count() - before
            assert gen.error_flags() == 0
        got[name] = rec, launches
    assert got["chain"][1] - got["kernel"][1] >= 3 * 8 * cfg.depformer_num_layers * 4      # each of the two took its own way
    same = torch.ones(B, dtype=torch.bool, device="cuda")
    compared = 0
    for (lg, tg), (lw, tw) in zip(got["kernel"][0], got["chain"][0]):
        for k in range(cfg.dep_q):
            # every layer rounds four products' results to bf16 (2^-9 each), in either path at other sums: about a percent over six layers
            err = (lg[k] - lw[k]).norm(dim=-1) / lw[k].norm(dim=-1)
            assert (err[same] < 3e-2).all(), (k, err)
            compared += int(same.sum())
            # greedy picks of the kernel's own logits: the first of the largest
            first = torch.where(lg[k] == lg[k].max(-1, keepdim=True).values, torch.arange(cfg.card, device="cuda"), cfg.card).amin(-1)
            assert torch.equal(tg[k], first)
            same &= tg[k] == tw[k]
    assert compared >= B

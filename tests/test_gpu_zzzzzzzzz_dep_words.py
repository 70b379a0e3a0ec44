"""GPU: what the blocks of the depformer's kernel for few sessions pass to one another, word by word up to 8 sessions and across a barrier above (csrc/dep_reg.cuh)."""
import dataclasses

import pytest
import torch

from moshi_b200.config import LMConfig
from moshi_b200.synth import synth_lm_state_dict

pytestmark = pytest.mark.gpu
BASE = LMConfig(dim=512, num_heads=4, num_layers=1, context=64, text_card=4000, card=1023, depformer_dim=448, depformer_num_heads=7, depformer_dim_feedforward=2112,
                depformer_num_layers=3)


def _frames(lm, B, graph, frames=6):
    """Greedy frames: each one's tokens, and what the depformer's heads gave."""
    from moshi_b200.models import LMGen
    cfg, out = lm.cfg, []
    gen = LMGen(lm, use_sampling=False)
    gen.use_graph = graph
    with gen.streaming(B):
        for i in range(frames):
            g = torch.Generator().manual_seed(100 * B + i)
            gen.step(torch.randint(0, cfg.card, (B, cfg.n_q - cfg.dep_q, 1), generator=g).cuda())
            out.append((gen.read_buffer("dep_logits", torch.bfloat16, (cfg.dep_q, B, cfg.card)).float(), gen.read_buffer("audio_tokens", torch.int64, (cfg.dep_q, B))))
        assert gen.error_flags() == 0
    return out


@torch.no_grad()
@pytest.mark.parametrize("dep_q", [3, 8, 9, 16])
def test_sub_steps_and_replays(dep_q, monkeypatch):
    """Fewer sub-steps than a frame of the 7B has, as many, and the kernel for more; a width whose rows leave CTAs without a share of some products and k-blocks for seven warps,
    an odd count of codes.  Frame after frame out of one buffer: replays of the graph give the launches' bits, and every head's logits are the launch chain's while the tokens
    before were the same (a percent: three layers of four products rounded to bf16 at other sums)."""
    from moshi_b200.models import LMModel
    cfg = dataclasses.replace(BASE, n_q=2 * dep_q, dep_q=dep_q, depformer_context=dep_q, delays=(0,) * (2 * dep_q + 1))
    sd = synth_lm_state_dict(cfg, seed=5, device="cuda")
    lms = {}
    for name, value in (("kernel", "1"), ("chain", "0")):
        monkeypatch.setenv("B200_DEP_FUSED", value)
        lms[name] = LMModel(cfg, sd, device="cuda")
    for B in (1, 7, 8, 9, 16):
        got, again, want = _frames(lms["kernel"], B, True), _frames(lms["kernel"], B, False), _frames(lms["chain"], B, False)
        same = torch.ones(B, dtype=torch.bool, device="cuda")
        for (lg, tg), (la, ta), (lw, tw) in zip(got, again, want):
            assert torch.equal(lg, la) and torch.equal(tg, ta)
            for k in range(dep_q):
                err = (lg[k] - lw[k]).norm(dim=-1) / lw[k].norm(dim=-1)
                assert (err[same] < 3e-2).all(), (B, k, err)
                same &= tg[k] == tw[k]


DEEP = dict(card=200, depformer_dim=64, depformer_num_heads=1, depformer_dim_feedforward=96, depformer_num_layers=140)


@torch.no_grad()
@pytest.mark.parametrize("over,sessions", [(dict(card=9401, depformer_num_layers=8), 16), (DEEP, 1), (DEEP, 16)])
def test_addresses_in_memory(over, sessions, monkeypatch):
    """More weights than their addresses fit into shared memory: many rows of logits, many layers.  Replays of the graph give the launches' bits; every head's logits are the launch
    chain's while the tokens before were the same.  Two residual additions a layer, each rounded to bf16 (2^-9) on both sides: independent errors grow with the root of their number,
    and as much again for the roundings of the products."""
    from moshi_b200.models import LMModel
    cfg = dataclasses.replace(BASE, n_q=32, dep_q=16, depformer_context=16, delays=(0,) * 33, **over)
    tol = 2 * (2 * cfg.depformer_num_layers) ** 0.5 * 2.0 ** -8
    sd = synth_lm_state_dict(cfg, seed=5, device="cuda")
    lms = {}
    for name, value in (("kernel", "1"), ("chain", "0")):
        monkeypatch.setenv("B200_DEP_FUSED", value)
        lms[name] = LMModel(cfg, sd, device="cuda")
    got, again, want = _frames(lms["kernel"], sessions, True, 3), _frames(lms["kernel"], sessions, False, 3), _frames(lms["chain"], sessions, False, 3)
    same, compared = torch.ones(sessions, dtype=torch.bool, device="cuda"), 0
    for (lg, tg), (la, ta), (lw, tw) in zip(got, again, want):
        assert torch.equal(lg, la) and torch.equal(tg, ta)
        for k in range(cfg.dep_q):
            err = (lg[k] - lw[k]).norm(dim=-1) / lw[k].norm(dim=-1)
            assert (err[same] < tol).all(), (k, err)
            compared += int(same.sum())
            same &= tg[k] == tw[k]
    assert compared >= sessions

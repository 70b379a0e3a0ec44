"""GPU: the depformer of few sessions (csrc/dep_reg.cuh) as a server runs it, with sampling, and at the ends of the shapes it takes."""
import pytest
import torch

from moshi_b200.config import LMConfig
from moshi_b200.synth import synth_lm_state_dict

from .util import cptr

pytestmark = pytest.mark.gpu
BASE = dict(dim=512, num_heads=4, num_layers=1, context=64, text_card=4000)
SERVER = dict(BASE, depformer_dim=1024, depformer_num_heads=16, depformer_dim_feedforward=4224, depformer_num_layers=2, card=2048)
SHAPES = {
    # 1125 units of 8 logits: eight pieces for the fullest CTA
    "many_logits": dict(BASE, depformer_dim=512, depformer_num_heads=8, depformer_dim_feedforward=2112, depformer_num_layers=2, card=9000),
    # 16 x (4 x 17 + 1) weights
    "deep": dict(BASE, depformer_dim=256, depformer_num_heads=4, depformer_dim_feedforward=1056, depformer_num_layers=17, card=512, n_q=32, dep_q=16, depformer_context=16,
                 delays=[0, 0] + [2] * 15 + [0] + [2] * 15),
}


def _model(cfg, sd, **env):
    from moshi_b200.models import LMModel
    with pytest.MonkeyPatch.context() as m:
        for name, value in env.items():
            m.setenv(name, value)
        return LMModel(cfg, sd, device="cuda")


def _steps(lm, B, steps, sampling, noise_seed=0):
    from moshi_b200 import _lib
    from moshi_b200.models import LMGen
    cfg, rec = lm.cfg, []
    gen = LMGen(lm, use_sampling=sampling, temp=0.8, temp_text=0.7, top_k=250, top_k_text=25)
    gen.use_graph = False
    with gen.streaming(B):
        per_row = _lib.lib().b200_lm_noise_per_row(gen._h)
        before = _lib.lib().b200_launch_count()
        for i in range(steps):
            g = torch.Generator().manual_seed(100 * B + i)
            noise = torch.empty(B, per_row).exponential_(generator=torch.Generator().manual_seed(noise_seed + i)).cuda()
            gen.step(torch.randint(0, cfg.card, (B, cfg.n_q - cfg.dep_q, 1), generator=g).cuda(), noise=noise if sampling else None)
            rec.append((gen.read_buffer("dep_logits", torch.bfloat16, (cfg.dep_q, B, cfg.card)), gen.read_buffer("audio_tokens", torch.int64, (cfg.dep_q, B)), noise))
        launches = _lib.lib().b200_launch_count() - before
        assert gen.error_flags() == 0
    return rec, launches


@pytest.fixture(scope="module")
def server():
    cfg = LMConfig(**SERVER)
    return _model(cfg, synth_lm_state_dict(cfg, seed=3, device="cuda"))


@torch.no_grad()
@pytest.mark.parametrize("B", [1, 8, 13])
def test_sampled_tokens_are_those_of_the_sampler(server, B):
    """2048 logits, the 250 likeliest, noise that the test gives: the tokens that the sampler's own kernel draws from the same logits and noise (softmax sums in
    another order would move a token only between probabilities over noise that agree to 1e-6)."""
    from moshi_b200 import _lib
    lib, cfg, k = _lib.lib(), server.cfg, 250
    rec, _ = _steps(server, B, 3, True)
    seen = set()
    for logits, tokens, noise in rec:
        audio = noise[:, noise.shape[1] - k * cfg.dep_q:]
        for q in range(cfg.dep_q):
            want = torch.empty(B, dtype=torch.int64, device="cuda")
            rows, draws = logits[q].contiguous(), audio[:, q * k:(q + 1) * k].contiguous()
            _lib.check(lib.b200_op_sample(cptr(rows), cptr(draws), cptr(want), B, cfg.card, 1, 0.8, k, None))
            torch.cuda.synchronize()
            assert torch.equal(tokens[q], want), q
            seen.update(want.tolist())
            # and by the definition: the largest probability over noise among the 250 likeliest, in their order
            top, idx = torch.sort(rows.float(), dim=-1, descending=True, stable=True)
            p = torch.softmax(rows.double() / 0.8, -1).gather(1, idx[:, :k])
            score = p / draws.double()
            picked = idx[torch.arange(B, device="cuda"), score.argmax(-1)]
            assert torch.equal(tokens[q], picked), q
    assert len(seen) > B                                    # tokens are drawn, not the likeliest each time


@pytest.fixture(scope="module", params=sorted(SHAPES))
def pair(request):
    cfg = LMConfig(**SHAPES[request.param])
    sd = synth_lm_state_dict(cfg, seed=9, device="cuda")
    return cfg, _model(cfg, sd, B200_DEP_FUSED="1"), _model(cfg, sd, B200_DEP_FUSED="0")


@torch.no_grad()
@pytest.mark.parametrize("B", [1, 2, 9, 16])
def test_ends_of_the_shapes_agree_with_the_chain(pair, B):
    cfg, kernel, chain = pair
    (got, few), (want, many) = _steps(kernel, B, 2, False), _steps(chain, B, 2, False)
    assert many - few >= 2 * cfg.dep_q * cfg.depformer_num_layers * 4          # one kernel, and a chain of launches
    same, compared = torch.ones(B, dtype=torch.bool, device="cuda"), 0
    for (lg, tg, _), (lw, tw, _) in zip(got, want):
        for q in range(cfg.dep_q):
            a, b = lg[q].float(), lw[q].float()
            # every layer rounds four products' results to bf16 (2^-9 each), at other sums either way: a random walk of 68 such steps is 1.6e-2 at most layers
            err = (a - b).norm(dim=-1) / b.norm(dim=-1)
            assert (err[same] < 4e-2).all(), (q, err)
            compared += int(same.sum())
            first = torch.where(a == a.max(-1, keepdim=True).values, torch.arange(cfg.card, device="cuda"), cfg.card).amin(-1)
            assert torch.equal(tg[q], first)
            same &= tg[q] == tw[q]
    assert compared >= B


@torch.no_grad()
def test_two_streams_of_different_sizes_side_by_side():
    """Sixteen sessions of one model and nine of another, step by step in turn: each as it is alone."""
    from moshi_b200.models import LMGen
    cfg = LMConfig(**dict(BASE, depformer_dim=512, depformer_num_heads=8, depformer_dim_feedforward=2112, depformer_num_layers=2, card=2048))
    models = [_model(cfg, synth_lm_state_dict(cfg, seed=s, device="cuda")) for s in (1, 2)]
    sizes, steps = (16, 9), 3
    codes = [torch.randint(0, cfg.card, (steps, B, 8, 1), generator=torch.Generator().manual_seed(B)).cuda() for B in sizes]

    def tokens(gen, B):
        return gen.read_buffer("audio_tokens", torch.int64, (cfg.dep_q, B))

    def gens():
        made = [LMGen(m, use_sampling=False) for m in models]
        for g in made:
            g.use_graph = False
        return made

    alone = []
    for gen, B, c in zip(gens(), sizes, codes):
        with gen.streaming(B):
            alone.append([(gen.step(x), tokens(gen, B))[1] for x in c])
    a, b = gens()
    with a.streaming(sizes[0]), b.streaming(sizes[1]):
        for i in range(steps):
            for gen, B, c, want in zip((a, b), sizes, codes, alone):
                gen.step(c[i])
                assert torch.equal(tokens(gen, B), want[i])
        assert a.error_flags() == 0 and b.error_flags() == 0

"""GPU: attention of long prompt portions (csrc/dlm_flash.cu) against the softmax in fp32, alone and inside a model."""
import ctypes as C

import pytest
import torch

from .util import cptr

pytestmark = pytest.mark.gpu


def _want(q, k, v, sink, pos0, scale):
    T, H, _ = q.shape
    s = torch.einsum("thd,nhd->htn", q.float(), k.float()) * scale
    n = torch.arange(k.shape[0], device=q.device)
    s = s.masked_fill(n[None, None, :] > (pos0 + torch.arange(T, device=q.device))[None, :, None], -torch.inf)
    if sink is not None:
        s = torch.cat([s, sink.view(-1, 1, 1).expand(-1, T, 1)], -1)
    return torch.einsum("htn,nhd->thd", torch.softmax(s, -1)[..., :k.shape[0]], v.float())


@pytest.mark.parametrize("T,pos0,H,spread", [(1, 0, 1, 1.0), (127, 0, 2, 1.0), (128, 0, 3, 4.0), (129, 1, 2, 1.0), (300, 77, 2, 8.0), (640, 129, 1, 1.0), (1000, 0, 16, 2.0)])
@pytest.mark.parametrize("with_sink", [True, False])
def test_attention_of_a_portion(T, pos0, H, spread, with_sink):
    """Tiles that end before, on and behind their edge, one key to many tiles, scores whose maximum keeps moving (spread)."""
    from moshi_b200 import _lib
    lib = _lib.lib()
    g = torch.Generator().manual_seed(T + pos0)
    ctx, ld = pos0 + T, (pos0 + T + 15) // 8 * 8
    q, k, v = (torch.randn(n, H, 128, generator=g).bfloat16().cuda() for n in (T, ctx, ctx))
    k *= (1 + spread * torch.arange(ctx, device="cuda") / ctx).bfloat16()[:, None, None]
    vt = torch.full((H * 128, ld), float("nan"), dtype=torch.bfloat16, device="cuda")
    vt[:, :ctx] = v.reshape(ctx, -1).t()
    sink = torch.randn(H, generator=g).cuda() if with_sink else None
    out = torch.full((T, H, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    _lib.check(lib.b200_op_prefill_attention(cptr(q), cptr(k), cptr(vt), cptr(sink), cptr(out), T, H, pos0, ld, 128 ** -0.5,
                                             C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    want = _want(q, k, v, sink, pos0, 128 ** -0.5)
    assert not torch.isnan(out.float()).any()
    # the weights and the result are each rounded to bf16, eight significant bits: half a unit is up to 2^-8 of the value, so 2^-7 of the
    # weighted sum of |v| (which bounds the result) in all, plus fp32 order
    bound = 2.0 ** -7 * _want(q, k, v.abs(), sink, pos0, 128 ** -0.5) + 1e-4
    assert ((out.float() - want).abs() <= bound).all(), float(((out.float() - want).abs() - bound).max())


@pytest.fixture(scope="module")
def model():
    from moshi_b200.config import DecoderLMConfig
    from moshi_b200.models import loaders
    lay = {"type": "latent_attention", "mixer": {"heads": 2, "dim": 128, "vdim": 128, "kv_rank": 64, "scale": 128 ** -0.5}, "mlp": {"kind": "dense", "ff": 512}}
    cfg = DecoderLMConfig.from_dict({"architecture": "Likosun", "vocab": 320, "width": 256, "embedding": {"scale": 1.0}, "residual_mult": 0.5,
                                     "norm": {"eps": 1e-6}, "layers": [lay] * 2})
    return loaders.get_decoder_lm(None, cfg, device="cuda:0", synth_seed=5)


ALL, RULE, NONE = 2, 1, 0        # "attn_expand"


def test_long_portions_agree_with_short_ones(model):
    """A request taken as one portion, as portions on both sides of the line between the two kernels, and beside another long one."""
    from moshi_b200.models import DecoderLMGen
    g = torch.Generator().manual_seed(3)
    toks = torch.randint(0, 320, (300,), generator=g).tolist()
    other = torch.randint(0, 320, (150,), generator=g).tolist()

    def run(cuts, beside=False, expand=ALL):
        with DecoderLMGen(model, slots=2, capacity=320, max_step_tokens=512) as gen:
            gen.set_option("attn_expand", expand)
            out, at = [], 0
            for n in cuts:
                entries = [(1, toks[at:at + n])] + ([(0, other)] if beside else [])
                out.append(gen.step(entries, range(n)))
                at += n
            assert gen.error_flags() == 0
            gen.set_option("attn_expand", RULE)
            return torch.cat(out)

    whole = run([300], expand=NONE)
    for cuts, beside in (([300], False), ([128, 172], False), ([100, 100, 100], False), ([127, 173], False), ([300], True)):
        got = run(cuts, beside)
        # two bf16 layers: what the model tests allow between ways of cutting a prompt
        assert ((got - whole).norm() / whole.norm()) < 1e-2, cuts


# (tokens held before the step, new tokens) per request, in the order of the step
MIXES = [[(0, 300), (40, 1)], [(40, 1), (0, 300)], [(3, 1), (0, 128), (0, 7), (17, 1), (130, 200), (9, 2)], [(0, 129), (0, 255), (64, 128)],
         [(250, 1), (0, 127), (5, 130)]]


@pytest.mark.parametrize("mix", MIXES)
def test_long_portions_beside_short_ones(model, mix):
    """Prompts beside decoding requests, between them, several of them, behind contexts of odd lengths: long ones on expanded keys and values
    (each three launches a layer) and the rest in the latent space give what the latent space gives for all, and leave the same cache behind."""
    from moshi_b200 import _lib
    from moshi_b200.models import DecoderLMGen
    lib = _lib.lib()

    def run(expand):
        g = torch.Generator().manual_seed(len(mix))
        toks = lambda n: torch.randint(0, 320, (n,), generator=g).tolist()
        with DecoderLMGen(model, slots=len(mix) + 1, capacity=448, max_step_tokens=640) as gen:
            gen.set_option("attn_expand", NONE)
            for slot, (held, _) in enumerate(mix):
                if held:
                    gen.step([(slot + 1, toks(held))], [0])
            step, later = [(slot + 1, toks(n)) for slot, (_, n) in enumerate(mix)], [(slot + 1, toks(1)) for slot in range(len(mix))]
            gen.set_option("attn_expand", expand)
            before = lib.b200_launch_count()
            out = gen.step(step, range(sum(n for _, n in mix)))
            launches = lib.b200_launch_count() - before
            gen.set_option("attn_expand", RULE)
            after = gen.step(later, range(len(mix)))
            torch.cuda.synchronize()
            assert gen.error_flags() == 0
            return out, after, launches

    want, want_after, plain = run(NONE)
    long_ones = sum(n >= 128 for _, n in mix)
    for expand in (ALL, RULE):
        got, after, launches = run(expand)
        assert ((got - want).norm() / want.norm()) < 1e-2
        at = 0
        for _, n in mix:                      # a short request's rows must not drown in a long one's
            assert ((got[at:at + n] - want[at:at + n]).norm() / want[at:at + n].norm()) < 1e-2
            at += n
        assert ((after - want_after).norm() / want_after.norm()) < 1e-2
        if expand == ALL and long_ones < len(mix):
            # three launches per long portion and layer; the folds run once per stretch of short ones
            runs = sum(n < 128 and (i == 0 or mix[i - 1][1] >= 128) for i, (_, n) in enumerate(mix))
            assert abs(launches - plain - 2 * (3 * long_ones + 2 * (runs - 1))) <= 2      # the merge of key ranges may come or go
        elif expand == RULE:
            assert launches == plain          # two heads: a portion's own launches never pay


def test_room_for_long_portions_only_where_they_can_come():
    """16 heads over 16384 tokens make 134 MB of keys and values: a cache whose steps bring fewer than 128 tokens has none of it, one with room in
    the buffers of a latent step borrows that, and both answer alike."""
    import gc
    from moshi_b200.config import DecoderLMConfig
    from moshi_b200.models import DecoderLMGen, loaders
    lay = {"type": "latent_attention", "mixer": {"heads": 16, "dim": 128, "vdim": 128, "kv_rank": 64, "scale": 128 ** -0.5}, "mlp": {"kind": "dense", "ff": 512}}
    cfg = DecoderLMConfig.from_dict({"architecture": "Likosun", "vocab": 320, "width": 256, "embedding": {"scale": 1.0}, "residual_mult": 0.5,
                                     "norm": {"eps": 1e-6}, "layers": [lay]})
    model = loaders.get_decoder_lm(None, cfg, device="cuda:0", synth_seed=5)

    def used():
        gc.collect()
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free, total = torch.cuda.mem_get_info()
        return (total - free) / 2 ** 20

    toks = torch.randint(0, 320, (300,), generator=torch.Generator().manual_seed(1)).tolist()

    def run(capacity, step, cuts, expand):
        before = used()
        with DecoderLMGen(model, slots=1, capacity=capacity, max_step_tokens=step, max_want=300) as gen:
            took = used() - before
            gen.set_option("attn_expand", expand)
            out, at = [], 0
            for n in cuts:
                out.append(gen.step([(0, toks[at:at + n])], range(n)))
                at += n
            gen.set_option("attn_expand", RULE)
            assert gen.error_flags() == 0
            return torch.cat(out), took

    run(320, 320, [300], NONE)                                      # code and first workspaces
    want, plain = run(16384, 100, [100] * 3, NONE)
    _, narrow = run(16384, 127, [100] * 3, ALL)
    assert abs(narrow - plain) < 16
    for capacity, step in ((320, 320), (16384, 512), (16384, 300)):      # 320 rows fit the step's own buffers, 16384 do not
        got, took = run(capacity, step, [300], ALL)
        assert ((got - want).norm() / want.norm()) < 1e-2, (capacity, step)
        assert (took - plain > 100) == (capacity == 16384), (capacity, took, plain)
    assert abs(run(16384, 127, [100] * 3, ALL)[1] - plain) < 16      # and given back

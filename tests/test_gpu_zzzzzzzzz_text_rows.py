"""GPU: the decoder LMs' small kernels by rows: latents appended in runs of eight (ranks of 256 to 1024), projections to fp32 with four tokens to a CTA from 512 tokens on."""
import ctypes as C

import pytest
import torch

from .test_gpu_zz_decoder_lm import assert_close, build, gen_for, layer, make_cfg, tokens
from . import test_gpu_zzzzzz_megolorn as megolorn
from .util import cptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rank", [256, 264, 512, 1024])
def test_latents(rank, dtype):
    """One run a lane, two, four; a rank between that keeps single elements: the whole model at the suite's tolerance, every token's latent read by the ones behind."""
    cfg = make_cfg([layer(2, 16, 8, rank, 0.2, 64), layer(2, 16, 8, rank, 0.2, None)], vocab=80, width=64)
    model, orc = build(cfg, dtype)
    toks = tokens(14, cfg.vocab, rank)
    with gen_for(model) as gen:
        got = gen.step([(0, toks[:9])], list(range(9))).cpu()
        got = torch.cat([got, gen.step([(0, toks[9:])], list(range(5))).cpu()])
    assert_close(got, orc.forward(toks), dtype)


@pytest.mark.parametrize("n", [511, 512, 513, 515])
@pytest.mark.parametrize("experts,width", [(5, 52), (16, 96), (11, 264), (250, 52), (259, 264)])
def test_small_projections(experts, width, n):
    """Router logits of as many tokens as fill the last CTA and of one to three more; outputs of two groups of eight that are full and not, of eight and nine groups of 32 where eight tokens
    share a CTA, rows on 16 bytes and off them: in fp32 every logit of the model at the suite's tolerance."""
    cfg = megolorn.make_cfg([megolorn.attention(2, 1, 16, 16, 0.2, chunk=64, mlp=megolorn.moe(experts, 2, 24))], vocab=97, width=width)
    model, orc = megolorn.build(cfg, torch.float32)
    toks = tokens(n, cfg.vocab, n)
    with gen_for(model, capacity=1024, max_step_tokens=1024) as gen:
        got = gen.step([(0, toks)], list(range(n))).cpu()
    megolorn.assert_close(got, orc.forward(toks), torch.float32)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("off", [0, 8, 4])
@pytest.mark.parametrize("rank", [32, 250, 256, 512, 768, 1024, 1280])
def test_bits_of_latents(rank, off, dtype):
    """Runs of eight or single elements, the same bits: the squares in one order (every lane each 32nd element by fused additions, then the lanes by halves)."""
    from moshi_b200 import _lib
    T, eps = 131, 1e-5
    g = torch.Generator().manual_seed(rank + off)
    rows = torch.randn(T, off + (rank + 7) // 8 * 8 + 8, generator=g).bfloat16().to(dtype).cuda()      # squares of 16 bits: with a sum of 24 exact in 64
    weight = (1 + 0.1 * torch.randn(rank, generator=g)).cuda()
    out = torch.empty(T, rank, dtype=dtype, device="cuda")
    _lib.check(_lib.lib().b200_op_latent_append(cptr(rows), _lib.dtype_code(dtype), rows.shape[1], off, cptr(weight), cptr(out), T, rank, eps, C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    raw = rows[:, off:off + rank].float()
    lanes = torch.nn.functional.pad(raw, (0, -rank % 32)).view(T, -1, 32)
    s = torch.zeros(T, 32, device="cuda")
    for i in range(lanes.shape[1]):
        s = (lanes[:, i].double() ** 2 + s.double()).float()
    for o in (16, 8, 4, 2, 1):
        s = s + s[:, torch.arange(32, device="cuda") ^ o]
    rs = 1.0 / torch.sqrt(s[:, :1] / torch.full((T, 1), float(rank), device="cuda") + torch.tensor(eps, device="cuda"))      # by a number torch would multiply with its inverse
    assert torch.equal(out, (raw * rs * weight).to(dtype))


@pytest.mark.parametrize("experts,width,n,tok", [(16, 96, 512, 4), (270, 96, 504, 1), (270, 96, 512, 8), (100, 96, 992, 4), (100, 96, 1000, 8), (100, 3072, 1000, 8), (100, 3080, 1000, 4)])
def test_tokens_that_share_a_projection(experts, width, n, tok):
    """Eight tokens and 32 outputs to a CTA where there are many such CTAs, four and eight outputs elsewhere, one below 512 tokens."""
    from torch.profiler import ProfilerActivity, profile
    cfg = megolorn.make_cfg([megolorn.attention(2, 1, 16, 16, 0.2, chunk=64, mlp=megolorn.moe(experts, 2, 24))], vocab=97, width=width)
    model, _ = megolorn.build(cfg, torch.bfloat16)
    with gen_for(model, capacity=1024, max_step_tokens=1024) as gen, profile(activities=[ProfilerActivity.CUDA]) as prof:
        gen.step([(0, tokens(n, cfg.vocab, n))], [0])
        torch.cuda.synchronize()
    names = [e.name for e in prof.events() if "small_proj_f32_kernel" in e.name]
    assert names and all(f", {tok}>" in name for name in names), names

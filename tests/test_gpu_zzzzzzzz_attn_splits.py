"""GPU: the temporal attention step with any number of key ranges asked for."""
import ctypes as C

import pytest
import torch

from .util import cptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsplit", [1, 2, 31, 32, 33, 64, 65, 100])
@pytest.mark.parametrize("fills", [(0, 40), (99, 250), (1000, 63)])
def test_ranges_of_keys(nsplit, fills):
    """Fewer keys than ranges, ranges that fill one, two and more rounds of 32, a full ring; against 64 bits and, among themselves, one merge for all."""
    from moshi_b200 import _lib
    B, H, cap, D = len(fills), 2, 250, 128
    g = torch.Generator().manual_seed(sum(fills))
    qkv = torch.randn(B, 3, H, D, generator=g).bfloat16().cuda()
    k, v = (torch.randn(B, H, cap, D, generator=g).bfloat16().cuda() for _ in range(2))
    pos, mask = torch.tensor(fills, device="cuda"), torch.ones(B, dtype=torch.uint8, device="cuda")
    out = torch.full((B, H * D), float("nan"), dtype=torch.bfloat16, device="cuda")
    for _ in range(2):                                        # the arrival counters are left as they were found
        kk, vv = k.clone(), v.clone()
        _lib.check(_lib.lib().b200_op_attn_step(cptr(qkv), cptr(kk), cptr(vv), cptr(out), cptr(pos), cptr(mask), B, H, cap, nsplit, 10000.0,
                                                C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    freq = torch.exp(torch.arange(D // 2, device="cuda").double() * (-torch.log(torch.tensor(10000.0).double()) * 2 / D))
    for b, p in enumerate(fills):
        c, s = torch.cos(p * freq), torch.sin(p * freq)
        e, o = qkv[b, 0, :, 0::2].double(), qkv[b, 0, :, 1::2].double()
        q = torch.stack([e * c - o * s, e * s + o * c], -1).reshape(H, D)
        n = min(p + 1, cap)
        w = torch.softmax(torch.einsum("hd,hnd->hn", q, kk[b, :, :n].double()) / D ** 0.5, -1)
        want = torch.einsum("hn,hnd->hd", w, vv[b, :, :n].double()).reshape(-1)
        # the turned query and the result are rounded to bf16 once each: scores move by up to 2^-9 * sum |q k| / sqrt(D) (about 0.02 for
        # normal vectors), weights by that factor, the result by its half ulp
        tol = 0.03 * torch.einsum("hn,hnd->hd", w, vv[b, :, :n].double().abs()).reshape(-1) + 1e-3
        assert ((out[b].double() - want).abs() <= tol).all()


@pytest.mark.parametrize("pairs", [591, 592, 739, 740, 887, 888, 1183, 1184])
@pytest.mark.parametrize("held", [5, 600, 1099])
def test_the_handle_s_own_choice_of_ranges(pairs, held):
    """Both sides of every line of the rule: one range, two of 512 and of 1024 keys, some of them empty, against the softmax in fp32."""
    from moshi_b200 import _lib
    cap, D = 1100, 128
    g = torch.Generator(device="cuda").manual_seed(pairs + held)
    r = lambda *s: torch.empty(s, device="cuda", dtype=torch.bfloat16).normal_(generator=g)
    qkv, k, v = r(1, 3, pairs, D), r(pairs, cap, D), r(pairs, cap, D)
    pos, mask = torch.tensor([held], device="cuda"), torch.ones(1, dtype=torch.uint8, device="cuda")
    out = torch.full((1, pairs * D), float("nan"), dtype=torch.bfloat16, device="cuda")
    _lib.check(_lib.lib().b200_op_attn_step(cptr(qkv), cptr(k), cptr(v), cptr(out), cptr(pos), cptr(mask), 1, pairs, cap, 0, 10000.0,
                                            C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    freq = torch.exp(torch.arange(D // 2, device="cuda").double() * (-torch.log(torch.tensor(10000.0).double()) * 2 / D))
    c, s = torch.cos(held * freq), torch.sin(held * freq)
    e, o = qkv[0, 0, :, 0::2].double(), qkv[0, 0, :, 1::2].double()
    q = torch.stack([e * c - o * s, e * s + o * c], -1).reshape(pairs, D).float()
    w = torch.softmax(torch.einsum("hd,hnd->hn", q, k[:, :held + 1].float()) / D ** 0.5, -1)
    want = torch.einsum("hn,hnd->hd", w, v[:, :held + 1].float()).reshape(-1)
    tol = 0.03 * torch.einsum("hn,hnd->hd", w, v[:, :held + 1].float().abs()).reshape(-1) + 1e-3      # as above
    assert ((out[0].float() - want).abs() <= tol).all()

"""GPU: what a Mimi handle holds of its transformers' weights, and the row-major copies that small batches stream from."""
import ctypes as C
import gc

import pytest
import torch

from moshi_b200.config import MimiConfig
from moshi_b200.synth import synth_mimi_state_dict

from .util import cptr

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.mark.parametrize("N,K", [(16, 512), (112, 1024), (128, 512), (1536, 512), (512, 2048)])
def test_rows_come_back_bit_for_bit(N, K):
    """Weights of many sizes, every low bit in use, remainders on both sides of a rounding, powers of two and their neighbours."""
    from moshi_b200 import _lib
    g = torch.Generator().manual_seed(N)
    w = torch.randn(N, K, generator=g) * 10.0 ** torch.randint(-12, 3, (N, K), generator=g)
    bits = w.view(-1).view(torch.int32)
    bits[0::7] |= 1                                           # odd in the last place
    bits[1::7] = (bits[1::7] & ~0x1fff) | 0x1000              # halfway between two values of 11 bits
    bits[2::7] = (bits[2::7] & ~0x1fff) | 0x0fff
    bits[3::7] |= 0x7fffff                                    # just below a power of two
    bits[4::7] &= ~0x7fffff                                   # a power of two
    w = w.cuda()
    rows = torch.full_like(w, float("nan"))
    _lib.check(_lib.lib().b200_op_tc_rows(cptr(w), cptr(rows), N, K, C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert torch.equal(rows.view(torch.int32), w.view(torch.int32))


def test_weights_are_held_once():
    """A loaded codec takes the packed hi / lo pair, 8 bytes per weight, and nothing like a second copy of its linears; the row-major weights
    are there while a batch of at most 64 tokens streams, and gone behind it."""
    from moshi_b200.models import MimiModel
    cfg = MimiConfig()
    sd = synth_mimi_state_dict(cfg, seed=5)
    rows = 4 * 2 * cfg.tr_num_layers * (4 * cfg.tr_d_model ** 2 + 2 * cfg.tr_d_model * cfg.tr_dim_feedforward)

    def used():
        gc.collect()
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free, total = torch.cuda.mem_get_info()
        return total - free

    with MimiModel(cfg, sd, device="cuda").streaming(1):      # code and workspaces that the first model brings along
        pass
    before = used()
    mimi = MimiModel(cfg, sd, device="cuda")
    loaded = used()
    assert loaded - before <= 8 * sum(t.numel() for t in sd.values()) + 64 * MB
    with mimi.streaming(32):
        few = used() - loaded
    assert abs(used() - loaded) <= 8 * MB
    with mimi.streaming(33):
        many = used() - loaded
    assert few - many > rows / 2                              # a session more is about 35 MB

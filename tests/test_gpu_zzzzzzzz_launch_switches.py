"""GPU: the switches that take programmatic dependent launches out change nothing but time."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent
PROGRAM = """
import hashlib, torch
from moshi_b200.config import LMConfig, MimiConfig
from moshi_b200.models import LMGen, LMModel, MimiModel
from moshi_b200.synth import synth_lm_state_dict, synth_mimi_state_dict
digest = hashlib.sha256()
mimi = MimiModel(MimiConfig(), synth_mimi_state_dict(MimiConfig(), seed=2), device="cuda")
for B in (1, 40):
    g = torch.Generator().manual_seed(B)
    with mimi.streaming(B):
        for _ in range(3):
            codes = mimi.encode(0.1 * torch.randn(B, 1, 1920, generator=g).cuda())
            digest.update(codes.cpu().numpy().tobytes() + mimi.decode(codes).cpu().numpy().tobytes())
cfg = LMConfig(dim=1024, num_heads=8, num_layers=2, context=64, text_card=4000, card=2048, depformer_dim=512, depformer_num_heads=8,
               depformer_dim_feedforward=2112, depformer_num_layers=2)
lm = LMModel(cfg, synth_lm_state_dict(cfg, seed=5, device="cuda"), device="cuda")
for B in (1, 5, 40):
    gen = LMGen(lm, use_sampling=False)
    with gen.streaming(B):
        for i in range(4):
            t = gen.step(torch.randint(0, cfg.card, (B, 8, 1), generator=torch.Generator().manual_seed(i)).cuda())
            if t is not None:
                digest.update(t.cpu().numpy().tobytes())
        digest.update(gen.read_buffer("text_logits", torch.bfloat16, (B, cfg.text_card)).view(torch.int16).cpu().numpy().tobytes())
print(digest.hexdigest())
"""


def test_the_same_results_without_early_launches():
    def run(**env):
        r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, env=dict(os.environ, **env), capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        return r.stdout.split()[-1]

    assert run() == run(B200_PDL="0", B200_MIMI_PDL="0")

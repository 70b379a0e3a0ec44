"""What a user of this framework has it do, as timed cases: frames of a spoken dialogue (the Mimi codec, the Moshi 7B step, and the
ring attention and linears that the step is made of), and text through the decoder LMs (prompts, scoring, generation).

Every case goes through a public entry point.  Weights and inputs are drawn on the GPU from the seed; ``exact`` restates the
arithmetic in 64 bits with plain torch."""
from __future__ import annotations

import ctypes as C
import gc
import math

import torch
import torch.nn.functional as F

from moshi_b200 import _lib, synth
from moshi_b200.config import DecoderLMConfig, LMConfig, MimiConfig
from moshi_b200.models import DecoderLMGen
from moshi_b200.models.compression import MimiModel
from moshi_b200.models.decoder_lm import DecoderLM
from moshi_b200.models.lm import LMGen, LMModel

F64 = torch.float64
DEVICE = "cuda:0"
HEADS, HEAD_DIM, CONTEXT = 32, 128, 3000            # the 7B's temporal attention
SHARED = 3.0                                        # size of the direction that all text embeddings share (their own part has rms 1/64)
STORE, RESIDUAL, GATED = 0, 1, 2                    # what a packed linear does with its sums

# the 7B's linears: (outputs, inputs, epilogue); a gated one holds gate and value rows and returns half as many outputs
LINEARS = {
    "in_proj": (12288, 4096, STORE), "out_proj": (4096, 4096, RESIDUAL), "linear_in": (22528, 4096, GATED),
    "linear_out": (4096, 11264, RESIDUAL), "text_head": (32000, 4096, STORE), "depformer_in": (8192, 4096, STORE),
    "dep_in_proj": (3072, 1024, STORE), "dep_linear_in": (5632, 1024, GATED), "dep_linear_out": (1024, 2816, RESIDUAL),
}


# ---------------------------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # one young session (10 s of history): the attention of one temporal layer, where latency counts
        {"name": "attention_1", "kind": "attention", "sessions": 1, "fill": 125},
        # a loaded server: sessions of every age up to a full ring
        {"name": "attention_48", "kind": "attention", "sessions": 48, "fill": 3000},
        # linears of one temporal layer at a small pool (gated MLP input) and at a full server (q, k, v projection)
        {"name": "linear_gated_6", "kind": "linear", "layer": "linear_in", "sessions": 6, "int8": False},
        {"name": "linear_qkv_104", "kind": "linear", "layer": "in_proj", "sessions": 104, "int8": False},
        # the q8 checkpoint's linear: activations quantised row by row, int8 product, residual add
        {"name": "linear_int8_24", "kind": "linear", "layer": "linear_out", "sessions": 24, "int8": True},
        # the codec around the model, full duplex: one user's frame in and one frame out; a pool of 40 users
        {"name": "mimi_1", "kind": "mimi", "sessions": 1, "frames": 2},
        {"name": "mimi_40", "kind": "mimi", "sessions": 40, "frames": 1},
        # one step of the 7B: a single conversation, and sixteen with full rings
        {"name": "lm_1", "kind": "lm", "sessions": 1, "fill": 750},
        {"name": "lm_16", "kind": "lm", "sessions": 16, "fill": 3000},
        # a long prompt of which the next token is wanted
        {"name": "prompt_2048", "kind": "text", "design": "latent", "width": 2048, "requests": 1, "prompt": 2048, "new": 1, "score": False},
        # scoring given texts: several ragged requests in one step, logits of every token, routed experts
        {"name": "score_moe_5x230", "kind": "text", "design": "experts", "width": 2048, "requests": 5, "prompt": 230, "new": 1, "score": True},
        # short generation for a batch of requests: prompts, then token by token
        {"name": "generate_moe_8x48", "kind": "text", "design": "experts", "width": 2048, "requests": 8, "prompt": 48, "new": 12, "score": False},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["attention", "linear", "linear", "mimi", "lm", "text", "text", "text"])
    if kind == "attention":
        return {"kind": kind, "sessions": _log_int(rng, 1, 48), "fill": _log_int(rng, 1, CONTEXT)}
    if kind == "linear":
        return {"kind": kind, "layer": rng.choice(sorted(LINEARS)), "sessions": _log_int(rng, 1, 256), "int8": rng.random() < 0.3}
    if kind == "mimi":
        sessions = _log_int(rng, 1, 40)
        return {"kind": kind, "sessions": sessions, "frames": rng.randint(1, 3)}
    if kind == "lm":
        return {"kind": kind, "sessions": _log_int(rng, 1, 16), "fill": _log_int(rng, 3, CONTEXT)}
    requests = _log_int(rng, 1, 32)
    prompt = _log_int(rng, 1, 2048 // requests)
    new = rng.choice([1, 1, rng.randint(2, 16)])
    return {"kind": kind, "design": rng.choice(["latent", "experts"]), "width": rng.choice([1024, 2048, 4096]), "requests": requests,
            "prompt": prompt, "new": new, "score": new == 1 and rng.random() < 0.4}


# ---------------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _normal(g, *shape, dtype=torch.bfloat16, scale=1.0):
    t = torch.empty(shape, device=DEVICE, dtype=dtype).normal_(generator=g)
    return t if scale == 1.0 else t.mul_(scale)


def _ints(g, lo, hi, *shape):
    return torch.randint(lo, hi, shape, device=DEVICE, generator=g)


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _fills(case):
    """Frames of history per session: the pool's oldest holds ``fill``, the others are younger."""
    n, fill = case["sessions"], case["fill"]
    return [max(0, fill - (i * 997) % max(1, fill) if i else fill) for i in range(n)]


def _attention_inputs(case, seed):
    g, B = _gen(seed), case["sessions"]
    qkv = _normal(g, B, 3 * HEADS * HEAD_DIM)
    k, v = _normal(g, B, HEADS, CONTEXT, HEAD_DIM), _normal(g, B, HEADS, CONTEXT, HEAD_DIM)
    pos = torch.tensor(_fills(case), device=DEVICE, dtype=torch.int64)
    return qkv, k, v, pos


def _linear_inputs(case, seed):
    g = _gen(seed)
    N, K, epi = LINEARS[case["layer"]]
    x = _normal(g, case["sessions"], K)
    w = _normal(g, N, K, scale=K ** -0.5)
    res = _normal(g, case["sessions"], N) if epi == RESIDUAL else None
    return x, w, res


def _mimi_inputs(case, seed):
    g, cfg = _gen(seed), MimiConfig()
    B, n = case["sessions"], case["frames"]
    pcm = _normal(g, B, 1, cfg.frame_size * n, dtype=torch.float32, scale=0.1)
    codes = _ints(g, 0, cfg.q_bins, B, cfg.num_codebooks, n)
    return cfg, pcm, codes


def _mimi_weights(cfg, seed):
    return synth.synth_mimi_state_dict(cfg, seed=seed + 1, device=DEVICE)


def _lm_weights(cfg, seed):
    """(name, tensor) of a 7B whose next tokens are as certain as a trained model's mostly are: embeddings share a direction that one
    row of every head answers to."""
    g = _gen(seed + 2)
    u = torch.where(_normal(g, cfg.dim) > 0, 1.0, -1.0).to(torch.bfloat16)
    v = torch.where(_normal(g, cfg.depformer_dim) > 0, 1.0, -1.0).to(torch.bfloat16)
    picks = _ints(g, 0, cfg.card, cfg.dep_q + 1).tolist()
    for name, t in synth.iter_synth_lm_tensors(cfg, seed=seed + 3, device=DEVICE):
        if name == "text_emb.weight":
            t += SHARED * u
        elif name == "text_linear.weight":
            t[picks[0]] += 0.03 * u
        elif name.startswith(("depformer_emb.", "depformer_text_emb.")):
            t += v
        elif name.startswith("linears."):
            t[picks[1 + int(name.split(".")[1])]] += 0.03 * v
        yield name, t


def _lm_inputs(cfg, case, seed):
    """Ring of recent tokens, this frame's user codes, and the keys and values of every layer as a generator of its own."""
    g, B = _gen(seed), case["sessions"]
    user = cfg.n_q - cfg.dep_q
    cache = _ints(g, 0, cfg.card, B, cfg.n_q + 1, cfg.max_delay + 2)
    codes = _ints(g, 0, cfg.card, B, user, 1)
    return cache, codes, g


def _lm_ring(cfg, case, g):
    shape = (case["sessions"], cfg.num_heads, cfg.context, cfg.dim // cfg.num_heads)
    for _ in range(cfg.num_layers):
        yield _normal(g, *shape), _normal(g, *shape)


def _text_config(case):
    W = case["width"]
    L, H = (2 if W == 4096 else 4), W // 128
    if case["design"] == "latent":
        layer = {"type": "latent_attention", "mixer": {"heads": H, "dim": 128, "vdim": 128, "kv_rank": 512, "scale": 128 ** -0.5},
                 "mlp": {"kind": "dense", "ff": 4 * W}}
        return DecoderLMConfig.from_dict({"architecture": "Likosun", "vocab": 32000, "width": W, "embedding": {"scale": 1.0},
                                          "residual_mult": 0.5, "norm": {"eps": 1e-6}, "layers": [layer] * L})
    mixer = {"diff": 0.5, "dim": 64, "heads": H, "kv_heads": 4, "mask": {"size": 1024}, "rot": {"base": 5e5, "dims": 64, "scaling": {"factor": 8.0}},
             "scale": 64 ** -0.5, "vdim": 128}
    moe = {"expert": {"ff": 2 * W}, "kind": "moe", "router": {"experts": 16, "groups": {"count": 4, "keep": 2}, "identity": 0, "top": 2},
           "shared": {"ff": 2 * W}}
    dense = {"ff": 4 * W, "kind": "dense", "limit": 7.0}
    return DecoderLMConfig.from_dict({"architecture": "Megolorn", "embedding": {"scale": 1.0}, "norm": {"eps": 1e-6}, "vocab": 32000, "width": W,
                                      "layers": [{"type": "attention", "mixer": dict(mixer, kv_from=i - 1) if i % 2 else mixer, "mlp": moe if i % 2 else dense}
                                                 for i in range(L)]})


def _text_weights(cfg, seed):
    """(name, tensor).  Routers are as sure as trained ones: a token's embedding holds the directions of two experts, a strong and a weak
    one, which the routers answer to."""
    n = max(L.experts for L in cfg.layers)
    u = torch.where(_normal(_gen(seed + 2), max(n, 1), cfg.width) > 0, 1.0, -1.0).to(torch.bfloat16)
    for name, t in synth.iter_synth_decoder_tensors(cfg, seed=seed + 1, device=DEVICE):
        if n and name == "embed":
            first = torch.arange(cfg.vocab, device=DEVICE) % n
            t += 0.5 * u[first] + 0.35 * u[(first + 1 + torch.arange(cfg.vocab, device=DEVICE) // n % (n - 1)) % n]
        elif name.endswith("mlp.router"):
            t.mul_(0.3).add_(12.0 / cfg.width * u)
        elif name.endswith("mlp.correction"):
            t.mul_(0.05)                   # settled: beside scores that are sure, the balancing term is small
        yield name, t


def _prompt_lengths(case):
    P = case["prompt"]
    return [P if i == 0 else max(1, P - (i * 37) % max(1, P // 2)) for i in range(case["requests"])]


def _texts(cfg, case, seed):
    g = torch.Generator().manual_seed(int(seed))
    return [torch.randint(0, cfg.vocab, (n + case["new"] - 1,), generator=g).tolist() for n in _prompt_lengths(case)]


# ---------------------------------------------------------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    lib, kind, s = _lib.lib(), case["kind"], {"case": case}
    if kind == "attention":
        qkv, k, v, pos = _attention_inputs(case, seed)
        s.update(lib=lib, qkv=qkv, k=k, v=v, pos=pos, mask=torch.ones(case["sessions"], dtype=torch.uint8, device=DEVICE))
    elif kind == "linear":
        x, w, res = _linear_inputs(case, seed)
        N, K, epi = LINEARS[case["layer"]]
        gate_rows = N // 2 if epi == GATED else 0
        s.update(lib=lib, x=x, res=res, dims=(case["sessions"], N, K, epi, gate_rows))
        if case["int8"]:
            s["w"] = torch.empty(lib.b200_op_packed_bytes_i8(N, K, epi, gate_rows), dtype=torch.uint8, device=DEVICE)
            s["sw"] = torch.empty(N, dtype=torch.float32, device=DEVICE)
            _lib.check(lib.b200_op_quant_pack_tiles(_lib.ptr(w), _lib.ptr(s["w"]), _lib.ptr(s["sw"]), N, K, epi, gate_rows, _stream()))
            s["xq"] = torch.empty(case["sessions"], K, dtype=torch.int8, device=DEVICE)
            s["sa"] = torch.empty(case["sessions"], dtype=torch.float32, device=DEVICE)
        else:
            s["w"] = torch.empty(lib.b200_op_packed_bytes(N, K, epi, gate_rows), dtype=torch.uint8, device=DEVICE)
            _lib.check(lib.b200_op_pack_tiles(_lib.ptr(w), _lib.ptr(s["w"]), N, K, epi, gate_rows, _stream()))
        torch.cuda.synchronize()
    elif kind == "mimi":
        cfg, pcm, codes = _mimi_inputs(case, seed)
        mimi = MimiModel(cfg, _mimi_weights(cfg, seed), device=DEVICE)
        mimi.set_num_codebooks(cfg.num_codebooks)
        mimi.streaming_forever(case["sessions"])
        s.update(mimi=mimi, pcm=pcm, codes=codes, frame=cfg.frame_size)
    elif kind == "lm":
        cfg = LMConfig()
        gc.collect()                        # a streaming LMGen refers to itself: earlier 15 GB models go now and not some time later
        gen = LMGen(LMModel(cfg, _lm_weights(cfg, seed), device=DEVICE), use_sampling=False)
        gen.streaming_forever(case["sessions"])
        cache, codes, g = _lm_inputs(cfg, case, seed)
        for i, (k, v) in enumerate(_lm_ring(cfg, case, g)):
            gen._write_state(f"layers.{i}.k", k)
            gen._write_state(f"layers.{i}.v", v)
        torch.cuda.synchronize()
        s.update(lib=lib, cfg=cfg, gen=gen, cache=cache, codes=codes, pos=torch.tensor(_lm_fills(case), device=DEVICE, dtype=torch.int64),
                 offset=case["fill"])
    else:
        cfg = _text_config(case)
        model = DecoderLM(cfg, _text_weights(cfg, seed), device=DEVICE)
        R, P, N = case["requests"], case["prompt"], case["new"]
        lengths, texts = _prompt_lengths(case), _texts(cfg, case, seed)
        gen = DecoderLMGen(model, slots=R, capacity=P + N, max_step_tokens=max(2048, R), max_want=sum(lengths) if case["score"] else R)
        ends = [sum(lengths[:i + 1]) - 1 for i in range(R)]
        s.update(gen=gen, requests=R, prompts=[(i, t[:n]) for i, (t, n) in enumerate(zip(texts, lengths))],
                 want=list(range(sum(lengths))) if case["score"] else ends,
                 later=[[(i, [t[n + j]]) for i, (t, n) in enumerate(zip(texts, lengths))] for j in range(N - 1)])
    return s


def _lm_fills(case):
    return [max(3, f) for f in _fills(case)]           # past the first frames, where a step has no output yet


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "attention":
        out = torch.empty(case["sessions"], HEADS * HEAD_DIM, dtype=torch.bfloat16, device=DEVICE)
        _lib.check(s["lib"].b200_op_attn_step(_lib.ptr(s["qkv"]), _lib.ptr(s["k"]), _lib.ptr(s["v"]), _lib.ptr(out), _lib.ptr(s["pos"]),
                                              _lib.ptr(s["mask"]), case["sessions"], HEADS, CONTEXT, 0, 10000.0, _stream()))
        return {"out": out, "keys": s["k"], "values": s["v"]}
    if kind == "linear":
        M, N, K, epi, gate_rows = s["dims"]
        y = torch.empty(M, gate_rows or N, dtype=torch.bfloat16, device=DEVICE)
        if case["int8"]:
            _lib.check(s["lib"].b200_op_quantize_rows(_lib.ptr(s["x"]), _lib.ptr(s["xq"]), _lib.ptr(s["sa"]), M, K, _stream()))
            _lib.check(s["lib"].b200_op_linear_i8(_lib.ptr(s["xq"]), _lib.ptr(s["sa"]), _lib.ptr(s["w"]), _lib.ptr(s["sw"]), _lib.ptr(y),
                                                  _lib.ptr(s["res"]), M, N, K, epi, gate_rows, _stream()))
        else:
            _lib.check(s["lib"].b200_op_linear_sk(_lib.ptr(s["x"]), _lib.ptr(s["w"]), _lib.ptr(y), _lib.ptr(s["res"]), M, N, K, epi, gate_rows,
                                                  0, 0, 0, _stream()))
        return y
    if kind == "mimi":
        # a conversation's first frames, as they arrive: what the user said is encoded, what the model answers is decoded
        mimi, fs = s["mimi"], s["frame"]
        mimi.reset_streaming()
        codes, pcm = [], []
        for f in range(case["frames"]):
            codes.append(mimi.encode(s["pcm"][:, :, f * fs:(f + 1) * fs]))
            pcm.append(mimi.decode(s["codes"][:, :, f:f + 1]))
        return {"codes": codes, "pcm": pcm}
    if kind == "lm":
        # the sessions' positions and recent tokens are put back as they were, so that every pass is the same frame
        gen, h, lib, cfg = s["gen"], s["gen"]._h, s["lib"], s["cfg"]
        B = case["sessions"]
        for name, t in (("cache", s["cache"]), ("offsets", s["pos"]), ("model.offset", s["pos"])):
            _lib.check(lib.b200_lm_state_write(h, name.encode(), _lib.ptr(t), t.numel() * 8))
        _lib.check(lib.b200_lm_set_offset_cpu(h, s["offset"] if s["offset"] > cfg.max_delay else cfg.max_delay + 1))
        tokens = gen.step(s["codes"])
        return {"tokens": tokens, "hidden": gen.read_buffer("transformer_out", torch.bfloat16, (B, cfg.dim)),
                "text_logits": gen.read_buffer("text_logits", torch.bfloat16, (B, cfg.text_card)),
                "audio_logits": gen.read_buffer("dep_logits", torch.bfloat16, (cfg.dep_q, B, cfg.card))}
    gen = s["gen"]
    for i in range(s["requests"]):
        gen.release(i)
    logits = [gen.step(s["prompts"], s["want"])]
    for entries in s["later"]:
        logits.append(gen.step(entries, range(s["requests"])))
    return logits


# ---------------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "attention":
        B, keys = case["sessions"], sum(min(f + 1, CONTEXT) for f in _fills(case))
        row = HEADS * HEAD_DIM
        return {"bytes": 2 * (2 * keys * row + B * (3 * row + row)), "flops": 4 * keys * row}
    if kind == "linear":
        N, K, epi = LINEARS[case["layer"]]
        M, cols = case["sessions"], N // 2 if epi == GATED else N
        return {"bytes": N * K * (1 if case["int8"] else 2) + 2 * M * (K + cols + (cols if epi == RESIDUAL else 0)), "flops": 2 * M * N * K}
    if kind == "mimi":
        B, n = case["sessions"], case["frames"]
        # 317 MB of weights and codebooks in 32 bits; 0.9 GFLOP, sound and carried state per session and frame
        return {"bytes": n * (317e6 + B * (2 * 1920 * 4 + 2 * 97e3)), "flops": n * B * 0.9e9}
    if kind == "lm":
        c, B = LMConfig(), case["sessions"]
        temporal = c.num_layers * (4 * c.dim ** 2 + 3 * c.dim * c.ffn_hidden) + c.text_card * c.dim
        dd = c.depformer_dim
        dep = c.dep_q * (c.depformer_num_layers * (4 * dd ** 2 + 3 * dd * c.depformer_ffn_hidden) + c.dim * dd + c.card * dd)
        keys = sum(min(f + 1, c.context) for f in _lm_fills(case)) * c.num_layers * c.dim
        return {"bytes": 2 * (temporal + dep) + 4 * keys + B * 2 * (c.text_card + c.dep_q * c.card + 26 * c.dim), "flops": 2 * B * (temporal + dep) + 4 * keys}
    cfg, lengths = _text_config(case), _prompt_lengths(case)
    W, R = cfg.width, case["requests"]
    steps = [(lengths, [0] * R, sum(lengths) if case["score"] else R)] + [([1] * R, [n + j for n in lengths], R) for j in range(case["new"] - 1)]
    total_bytes = total_flops = 0
    for counts, start, want in steps:
        T = sum(counts)
        seen = sum(sum(range(a + 1, a + n + 1)) if n < 2 else n * a + n * (n + 1) // 2 for n, a in zip(counts, start))
        read = want * cfg.vocab * 4 + cfg.vocab * W * 2 + T * W * 2
        flops = 2 * want * cfg.vocab * W
        for L in cfg.layers:
            if case["design"] == "latent":
                p = W * L.heads * L.dim + L.kv_rank * (W + L.heads * (L.dim + L.vdim)) + L.heads * L.vdim * W + 2 * W * W + 2 * W * L.ff
                read += 2 * p + 2 * L.kv_rank * sum(a + n for n, a in zip(counts, start))
                flops += 2 * T * p + 2 * seen * L.heads * (L.dim + L.vdim)
                continue
            a = L.a
            p = W * a.heads * (2 * a.dim + a.vdim + 1) + (W * a.kv_heads * (2 * a.dim + a.vdim) if a.kv_from < 0 else 0)
            if L.mlp_kind == "clamped_glu":
                p += 3 * W * L.ff
                used = p
            else:
                p += 3 * W * L.shared_ff + W * L.experts
                used, p = p + 3 * W * L.ff * min(L.experts, T * L.top), p + 3 * W * L.ff * L.top
            read += 2 * used + 2 * a.kv_heads * (2 * a.dim + a.vdim) * sum(s0 + n for n, s0 in zip(counts, start))
            flops += 2 * T * p + 2 * seen * a.heads * (4 * a.dim + 2 * 2 * a.vdim) // 2
        total_bytes += read
        total_flops += flops
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    kind = case["kind"]
    if kind == "attention":
        return {"rel": 1e-2, "max": 0.2}
    if kind == "linear":
        return {"rel": 1e-2, "max": 0.1}
    if kind == "mimi":
        return {"rel": 1e-4, "max": 1e-2, "differ": 0.01}
    if kind == "lm":
        return {"rel": 3e-2, "max": 0.5, "differ": 0.01}
    return {"rel": 2e-2, "max": 0.3}


# ---------------------------------------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------------------------------------
def exact(case, seed):
    return {"attention": _exact_attention, "linear": _exact_linear, "mimi": _exact_mimi, "lm": _exact_lm, "text": _exact_text}[case["kind"]](case, seed)


def _rope_pairs(x, pos, period=10000.0):
    """x [..., D] turned by pos (broadcastable against the leading axes): dimension 2i with 2i + 1."""
    D = x.shape[-1]
    ang = pos[..., None].to(F64) * torch.exp(torch.arange(D // 2, device=x.device, dtype=F64) * (-math.log(period) * 2 / D))
    a, b, c, s = x[..., 0::2], x[..., 1::2], torch.cos(ang), torch.sin(ang)
    return torch.stack([a * c - b * s, a * s + b * c], -1).reshape(x.shape)


def _ring_attention(qkv, k, v, pos, cap):
    """One session: qkv [3, H, D] in 64 bits, its rings [H, cap, D], its position -> [H, D]."""
    p = torch.tensor(float(pos), device=qkv.device, dtype=F64)
    q, new_k = _rope_pairs(qkv[0], p), _rope_pairs(qkv[1], p)
    n, slot = min(pos + 1, cap), pos % cap
    kk, vv = k[:, :n].to(F64), v[:, :n].to(F64)
    kk[:, slot], vv[:, slot] = new_k, qkv[2]
    w = torch.softmax(torch.einsum("hd,hnd->hn", q, kk) / math.sqrt(q.shape[-1]), -1)
    return torch.einsum("hn,hnd->hd", w, vv)


def _exact_attention(case, seed):
    qkv, k, v, pos = _attention_inputs(case, seed)
    out = [_ring_attention(qkv[b].to(F64).view(3, HEADS, HEAD_DIM), k[b], v[b], int(pos[b]), CONTEXT).reshape(-1) for b in range(case["sessions"])]
    return {"out": torch.stack(out), "keys": None, "values": None}


def _quantised(t):
    """Rows as 8-bit whole numbers times their largest magnitude / 127."""
    top = t.abs().amax(-1, keepdim=True)
    return torch.round(t * (127.0 / top)) * (top / 127.0)


def _exact_linear(case, seed):
    x, w, res = _linear_inputs(case, seed)
    _, _, epi = LINEARS[case["layer"]]
    w = _quantised(w.to(torch.float16).to(F64)) if case["int8"] else w.to(F64)
    x = _quantised(x.to(F64)) if case["int8"] else x.to(F64)
    y = x @ w.T
    if epi == GATED:
        gate, value = y.chunk(2, -1)
        return F.silu(gate) * value
    return y + res.to(F64) if epi == RESIDUAL else y


def _exact_mimi(case, seed):
    cfg, pcm, codes = _mimi_inputs(case, seed)
    sd = {k: t.to(F64) for k, t in _mimi_weights(cfg, seed).items()}
    n = case["frames"]

    def conv(x, name, stride=1, dilation=1, replicate=False):
        w, b = sd[name + ".weight"], sd.get(name + ".bias")
        pad = (w.shape[-1] - 1) * dilation + 1 - stride
        x = F.pad(x, (pad, 0), mode="replicate") if replicate else F.pad(x, (pad, 0))
        return F.conv1d(x, w, b, stride=stride, dilation=dilation)

    def convtr(x, name, stride, groups=1):
        w, b = sd[name + ".weight"], sd.get(name + ".bias")
        return F.conv_transpose1d(x, w, b, stride=stride, groups=groups)[..., :x.shape[-1] * stride]

    def residual(x, base, dilation):
        h = conv(F.elu(x), base + ".block.1.conv.conv", dilation=dilation)
        return x + conv(F.elu(h), base + ".block.3.conv.conv")

    def seanet(x, side, layout):
        for i, (kind, idx, _, _, _, stride, dilation) in enumerate(layout):
            base = f"{side}.model.{idx}"
            if kind == "res":
                x = residual(x, base, dilation)
            else:
                x = F.elu(x) if i else x
                x = conv(x, base + ".conv.conv", stride, dilation) if kind == "conv" else convtr(x, base + ".convtr.convtr", stride)
        return x

    def transformer(x, name):
        x = x.transpose(1, 2)
        B, T, d = x.shape
        H, pos = cfg.tr_num_heads, torch.arange(T, device=x.device)
        back = pos[:, None] - pos[None, :]
        seen = (back >= 0) & (back < cfg.tr_context)
        for i in range(cfg.tr_num_layers):
            p = f"{name}.transformer.layers.{i}."
            h = F.layer_norm(x, (d,), sd[p + "norm1.weight"], sd[p + "norm1.bias"], 1e-5)
            q, k, v = (h @ sd[p + "self_attn.in_projs.0.weight"].T).view(B, T, 3, H, d // H).permute(2, 0, 3, 1, 4)
            q, k = _rope_pairs(q, pos, cfg.tr_max_period), _rope_pairs(k, pos, cfg.tr_max_period)
            sc = (q @ k.transpose(-1, -2) / math.sqrt(d // H)).masked_fill(~seen, -math.inf)
            y = (torch.softmax(sc, -1) @ v).transpose(1, 2).reshape(B, T, d) @ sd[p + "self_attn.out_projs.0.weight"].T
            x = x + sd[p + "layer_scale_1.scale"] * y
            h = F.layer_norm(x, (d,), sd[p + "norm2.weight"], sd[p + "norm2.bias"], 1e-5)
            x = x + sd[p + "layer_scale_2.scale"] * (F.gelu(h @ sd[p + "linear1.weight"].T) @ sd[p + "linear2.weight"].T)
        return x.transpose(1, 2)

    def book(name, level):
        p = f"quantizer.{name}.vq.layers.{level}._codebook."
        return sd[p + "embedding_sum"] / sd[p + "cluster_usage"].clamp(min=1e-5)[:, None]

    halves = (("rvq_first", 0, cfg.q_n_semantic), ("rvq_rest", cfg.q_n_semantic, cfg.num_codebooks))
    enc_layout, dec_layout = synth.seanet_layout(cfg)
    s = cfg.resample_stride
    latent = conv(transformer(seanet(pcm.to(F64), "encoder", enc_layout), "encoder_transformer"), "downsample.conv.conv.conv", s, replicate=True)
    found = []
    for name, lo, hi in halves:
        rest = F.conv1d(latent, sd[f"quantizer.{name}.input_proj.weight"]).transpose(1, 2)
        for level in range(hi - lo):
            cb = book(name, level)
            idx = torch.cdist(rest, cb.expand(rest.shape[0], -1, -1)).argmin(-1)
            rest = rest - cb[idx]
            found.append(idx)
    found = torch.stack(found, 1)
    quantised = 0
    for name, lo, hi in halves:
        e = sum(book(name, level)[codes[:, lo + level]] for level in range(hi - lo)).transpose(1, 2)
        quantised = quantised + F.conv1d(e, sd[f"quantizer.{name}.output_proj.weight"])
    up = convtr(quantised, "upsample.convtr.convtr.convtr", s, groups=cfg.dimension)
    sound = seanet(transformer(up, "decoder_transformer"), "decoder", dec_layout)
    return {"codes": [found[:, :, f:f + 1] for f in range(n)], "pcm": list(sound.split(cfg.frame_size, -1))}


def _exact_lm(case, seed):
    """The temporal transformer; the depformer's logits hang on the tokens chosen on the way and are left out."""
    cfg, B, fills = LMConfig(), case["sessions"], _lm_fills(case)
    cache, codes, g = _lm_inputs(cfg, case, seed)
    ring = _lm_ring(cfg, case, g)
    CT = cfg.max_delay + 2
    tokens = torch.empty(B, cfg.n_q + 1, dtype=torch.int64, device=DEVICE)
    for b, f in enumerate(fills):
        for q in range(cfg.n_q + 1):
            fresh = q > cfg.dep_q and cfg.delays[q] == 0
            tokens[b, q] = codes[b, q - cfg.dep_q - 1, 0] if fresh else cache[b, q, f % CT]
    held, x = {}, None

    def norm(x, w):
        return x * w * torch.rsqrt(1e-8 + (x * x).mean(-1, keepdim=True))

    layer, parts = 0, {}
    for name, t in _lm_weights(cfg, seed):
        if name.startswith("emb.") or name == "text_emb.weight":
            q = 0 if name.startswith("text") else 1 + int(name.split(".")[1])
            e = t[tokens[:, q]].to(F64)
            x = e if x is None else x + e
        elif name in ("text_linear.weight", "out_norm.alpha"):
            held[name] = t
        elif name.startswith("transformer.layers."):
            parts[name.split(".", 3)[3]] = t
            if len(parts) < 6:
                continue
            w = {k: v.to(F64) for k, v in parts.items()}
            parts = {}
            k, v = next(ring)
            qkv = (norm(x, w["norm1.alpha"].view(-1)) @ w["self_attn.in_projs.0.weight"].T).view(B, 3, cfg.num_heads, -1)
            o = torch.stack([_ring_attention(qkv[b], k[b], v[b], fills[b], cfg.context).reshape(-1) for b in range(B)])
            x = x + o @ w["self_attn.out_projs.0.weight"].T
            gate, value = (norm(x, w["norm2.alpha"].view(-1)) @ w["gating.linear_in.weight"].T).chunk(2, -1)
            x = x + (F.silu(gate) * value) @ w["gating.linear_out.weight"].T
            layer += 1
            if layer == cfg.num_layers:
                break
    hidden = norm(x, held["out_norm.alpha"].to(F64).view(-1))
    logits = hidden @ held["text_linear.weight"].to(F64).T
    return {"tokens": None, "hidden": hidden, "text_logits": logits, "audio_logits": None}


def _exact_text(case, seed):
    cfg = _text_config(case)
    w = {k: t.to(F64) for k, t in _text_weights(cfg, seed)}
    logits = [[] for _ in range(case["new"])]
    for text, n in zip(_texts(cfg, case, seed), _prompt_lengths(case)):
        tok = torch.tensor(text, device=DEVICE)
        lg = (_latent_stack if case["design"] == "latent" else _experts_stack)(cfg, w, tok, 0 if case["score"] else n - 1)
        logits[0].append(lg[:n] if case["score"] else lg[:1])
        for j in range(1, case["new"]):
            logits[j].append(lg[j:j + 1])
    return [torch.cat(step) for step in logits]


def _causal(T, chunk=0):
    pos = torch.arange(T, device=DEVICE)
    seen = pos[None, :] <= pos[:, None]
    return seen & (pos[None, :] // chunk == pos[:, None] // chunk) if chunk else seen


def _layer_norm(x, w, b, eps):
    return F.layer_norm(x, (x.shape[-1],), w, b, eps)


def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _latent_stack(cfg, w, tok, first):
    """Logits of the positions from ``first`` on: latent attention and squared-ReLU MLP side by side, gated, depth-averaged."""
    x = w["embed"][tok] * cfg.embedding_scale
    T, results = tok.shape[0], [x]
    for i, L in enumerate(cfg.layers):
        p = f"l{i}."
        h = _layer_norm(x, w[p + "norm1"], w[p + "norm1.b"], cfg.norm_eps)
        c = _rms(h @ w[p + "mix.dkv"].T, w[p + "mix.dkv.norm"], cfg.norm_eps)
        q = (h @ w[p + "mix.q"].T).view(T, L.heads, L.dim).transpose(0, 1)
        k = (c @ w[p + "mix.uk"].T).view(T, L.heads, L.dim).transpose(0, 1)
        v = (c @ w[p + "mix.uv"].T).view(T, L.heads, L.vdim).transpose(0, 1)
        s = (q @ k.transpose(1, 2) * L.scale).masked_fill(~_causal(T), -math.inf)
        s = torch.cat([s, w[p + "mix.sink"].view(-1, 1, 1).expand(-1, T, 1)], -1)
        o = (torch.softmax(s, -1)[..., :T] @ v).transpose(0, 1).reshape(T, -1) @ w[p + "mix.o"].T
        y = o * torch.sigmoid(h @ w[p + "rg1"].T + w[p + "rg1.b"])
        y = y + (torch.relu(h @ w[p + "mlp.up"].T) ** 2 @ w[p + "mlp.down"].T) * torch.sigmoid(h @ w[p + "rg2"].T + w[p + "rg2.b"])
        results.append(x + cfg.residual_mult * y)
        x = sum(a * r for a, r in zip(w[p + "dwa"], results))
    return _layer_norm(x[first:], w["final.norm"], w["final.norm.b"], cfg.norm_eps) @ w["head"].T


def _experts_stack(cfg, w, tok, first):
    """Differential attention on chunks of positions beside a bounded gated unit or routed experts."""
    x, eps, T = w["embed"][tok] * cfg.embedding_scale, cfg.norm_eps, tok.shape[0]
    pos, kept = torch.arange(T, device=DEVICE), {}

    def glu(h, p, q, act):
        return act(h @ w[p + q + "gate"].T, h @ w[p + q + "up"].T) @ w[p + q + "down"].T

    for i, L in enumerate(cfg.layers):
        p, m, a = f"l{i}.", f"l{i}.mix.", L.a
        factor = float((a.rot_scaling or {}).get("factor", 1.0))
        ang = pos[:, None].to(F64) * (a.rot_base ** (-2.0 * torch.arange(a.rot_dims // 2, device=DEVICE, dtype=F64) / a.rot_dims) / factor)
        cos, sin = torch.cos(ang)[:, None, None], torch.sin(ang)[:, None, None]

        def turn(u):
            e, o = u[..., 0:a.rot_dims:2], u[..., 1:a.rot_dims:2]
            return torch.cat([torch.stack([e * cos - o * sin, o * cos + e * sin], -1).flatten(-2), u[..., a.rot_dims:]], -1)

        def heads(h, nm, n):
            u = (h @ w[m + nm].T + w[m + nm + ".b"]).view(T, n, 2, a.dim)
            return turn(_rms(u, w[m + nm + ".norm"], eps)).permute(2, 1, 0, 3)

        h = F.layer_norm(x, (cfg.width,), w[p + "norm1"], None, eps)
        q = heads(h, "q", a.heads)
        if a.kv_from < 0:
            kept[i] = heads(h, "k", a.kv_heads), (h @ w[m + "v"].T + w[m + "v.b"]).view(T, a.kv_heads, a.vdim).transpose(0, 1)
        k, v = (u.repeat_interleave(a.heads // a.kv_heads, -3) for u in kept[a.kv_from if a.kv_from >= 0 else i])
        at = torch.softmax((q @ k.transpose(-1, -2) * a.scale).masked_fill(~_causal(T, a.chunk), -math.inf), -1) @ v
        lam = math.exp(float(w[m + "lq1"] @ w[m + "lk1"])) - math.exp(float(w[m + "lq2"] @ w[m + "lk2"])) + a.diff
        o = _rms(at[0] - lam * at[1], 1.0, eps) * (1.0 - a.diff) * torch.sigmoid(h @ w[m + "g"].T).T[..., None]
        y = o.transpose(0, 1).reshape(T, -1) @ w[m + "o"].T
        if L.mlp_kind == "clamped_glu":
            def act(g, u):
                g, u = g.clamp(max=L.expert_limit), u.clamp(-L.expert_limit, L.expert_limit)
                return g * torch.sigmoid(1.702 * g) * (u + 1.0)
            y = y + glu(h, p, "mlp.", act)
        else:
            def act(g, u):
                return F.silu(g) * u
            score = torch.softmax(h @ w[p + "mlp.router"].T, -1)
            choice = score + w[p + "mlp.correction"]
            grouped = choice.view(T, L.groups, -1)
            keep = torch.zeros(T, L.groups, dtype=torch.bool, device=DEVICE).scatter_(1, grouped.amax(-1).topk(L.groups_keep, -1).indices, True)
            idx = grouped.masked_fill(~keep[..., None], -math.inf).view(T, -1).topk(L.top, -1).indices
            for e in range(L.experts):
                rows = (idx == e).any(-1).nonzero().view(-1)
                if rows.numel():
                    y[rows] += score[rows, e, None] * glu(h[rows], p, f"mlp.e{e}.", act)
            y = y + glu(h, p, "mlp.shared.", act)
        x = x + y
    return F.layer_norm(x[first:], (cfg.width,), w["final.norm"], None, eps) @ w["head"].T

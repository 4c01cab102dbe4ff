"""Serving steps whose speed matters, as one list: what a step of the engine takes for the batches that a server meets.

A case is one planned step of the engine over a batch: sequences that bring several new tokens (whole prompts, or the next
turn of a conversation whose history is cached) and sequences that bring one (decoding). ``prepare`` loads the model through
``LLM``, leaves the histories in the paged cache and plans the step with the scheduler; ``run`` has the engine execute the plan
and returns the logits and the cache that the step wrote to.

Models are a few layers of the architectures that the benchmarks use, at full width and with the whole vocabulary. Weights are
random; the projections that end a sublayer are smaller than the others, as trained models have them, so that the residual
stream dominates what a sublayer adds. Quantised weights are drawn on the lattice of their format, as a checkpoint holds them.
"""
import math
import os
import random
import zlib

import numpy as np
import torch

os.environ.setdefault("DISABLE_WARMUP", "1")     # the warm-up request is start-up time, prepare() runs the step itself once

BLOCK_TOKENS = 16
MODELS = {
    "llama-8b": dict(model_type="llama", hidden_size=4096, num_heads=32, num_kv_heads=8, head_dim=128, intermediate_size=14336,
                     vocab_size=128256, rms_norm_eps=1e-5, rope_theta=500000.0, eos_token_ids=[128001]),
    "llama-70b": dict(model_type="llama", hidden_size=8192, num_heads=64, num_kv_heads=8, head_dim=128, intermediate_size=28672,
                      vocab_size=128256, rms_norm_eps=1e-5, rope_theta=500000.0, eos_token_ids=[128001]),
    "qwen-72b": dict(model_type="qwen", hidden_size=8192, num_heads=64, num_kv_heads=8, head_dim=128, intermediate_size=29568,
                     vocab_size=152064, rms_norm_eps=1e-6, rope_theta=1000000.0, qkv_bias=True, eos_token_ids=[151643]),
    "deepseek": dict(model_type="deepseek_v3", hidden_size=7168, num_heads=128, num_kv_heads=128, head_dim=192,
                     intermediate_size=18432, vocab_size=129280, rms_norm_eps=1e-6, rope_theta=10000.0, rope_neox=False,
                     num_experts=32, num_experts_per_tok=8, moe_intermediate_size=2048, shared_expert_intermediate_size=2048,
                     num_shared_experts=1, moe_scoring="sigmoid", routed_scaling_factor=2.5, n_group=8, topk_group=4,
                     first_k_dense_replace=1, q_lora_rank=1536, kv_lora_rank=512, qk_nope_head_dim=128, qk_rope_head_dim=64,
                     v_head_dim=128, eos_token_ids=[1]),
}
QUANT = {"bf16": "auto", "fp8": "fp8_block", "w4": "w4a16", "nvfp4": "nvfp4"}
BITS = {"bf16": 16.0, "fp8": 8.0, "w4": 4.25, "nvfp4": 4.5}


def _case(name, model, weights, layers, limit, prompts=0, prompt_lo=0, prompt_hi=0, history_lo=0, history_hi=0, decodes=0,
          context_lo=0, context_hi=0, kv="bf16", mix=1):
    """``prompts`` sequences bring prompt_lo..prompt_hi tokens to history_lo..history_hi cached ones, ``decodes`` sequences bring
    one token to context_lo..context_hi cached ones (lengths spread over their logarithm, by ``mix``). ``limit``: longest
    sequence that the server admits."""
    case = {"model": model, "weights": weights, "kv": kv, "layers": layers, "limit": limit, "prompts": prompts, "prompt_lo": prompt_lo,
            "prompt_hi": prompt_hi, "history_lo": history_lo, "history_hi": history_hi, "decodes": decodes, "context_lo": context_lo,
            "context_hi": context_hi, "mix": mix}
    return dict(case, name=name) if name else case


def listed():
    return [
        # one user at the keyboard: the smallest step there is
        _case("decode_8b_bf16_1", "llama-8b", "bf16", 8, 4096, decodes=1, context_lo=517, context_hi=517),
        # a busy chat server: every sequence at another length
        _case("decode_8b_bf16_64", "llama-8b", "bf16", 8, 4096, decodes=64, context_lo=100, context_hi=3000),
        # long documents held in an 8-bit cache
        _case("decode_8b_kv8_12", "llama-8b", "bf16", 4, 16384, decodes=12, context_lo=4000, context_hi=15000, kv="fp8"),
        # a 4-bit checkpoint on a small server
        _case("decode_8b_w4_16", "llama-8b", "w4", 8, 4096, decodes=16, context_lo=300, context_hi=2500),
        # the offline benchmark's decode step: 64 sequences of 2048 prompt tokens and 256 to come
        _case("decode_70b_fp8_64", "llama-70b", "fp8", 4, 2320, decodes=64, context_lo=2175, context_hi=2175),
        # latent attention and experts, decoding
        _case("decode_deepseek_fp8_64", "deepseek", "fp8", 4, 4096, decodes=64, context_lo=900, context_hi=1300),
        # continuous batching: new prompts of all lengths beside sequences that decode
        _case("mixed_8b_bf16", "llama-8b", "bf16", 4, 4096, prompts=13, prompt_lo=17, prompt_hi=1024, decodes=51, context_lo=100,
              context_hi=2000),
        # one long document
        _case("prefill_8b_bf16_16k", "llama-8b", "bf16", 4, 16640, prompts=1, prompt_lo=16384, prompt_hi=16384),
        # prompts through 4-bit floating-point products (one layer: every further one would round its operands to 4 bits again)
        _case("prefill_8b_nvfp4", "llama-8b", "nvfp4", 1, 4096, prompts=5, prompt_lo=1000, prompt_hi=3000),
        # the next turn of conversations whose earlier turns are cached
        _case("turn_72b_fp8", "qwen-72b", "fp8", 2, 4096, prompts=32, prompt_lo=60, prompt_hi=250, history_lo=1000, history_hi=3500),
        # latent attention and experts, prompts
        _case("prefill_deepseek_fp8", "deepseek", "fp8", 3, 4096, prompts=8, prompt_lo=700, prompt_hi=1500),
        # the offline benchmark's prefill step: 8 prompts of 2048 tokens
        _case("prefill_70b_fp8", "llama-70b", "fp8", 4, 2320, prompts=8, prompt_lo=2048, prompt_hi=2048),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another step of these kinds: any batch size, any lengths."""
    model, weights = rng.choice([("llama-8b", "bf16"), ("llama-8b", "bf16"), ("llama-8b", "w4"), ("llama-8b", "nvfp4"), ("llama-70b", "fp8"),
                                 ("qwen-72b", "fp8"), ("deepseek", "fp8")])
    kind = rng.choice(["decode", "decode", "prefill", "turn", "mixed"])
    layers = 1 if weights == "nvfp4" else 2 if model in ("llama-70b", "qwen-72b") else 3
    mix = rng.randrange(1, 1 << 20)
    long_ = 12000 if model == "llama-8b" else 3800
    limit = 16640 if model == "llama-8b" else 4096
    if kind == "decode":
        n = _spread(rng, 1, 128)
        hi = _spread(rng, 64, min(long_, 400000 // n))
        kv = "fp8" if model == "llama-8b" and weights == "bf16" and rng.random() < 0.4 else "bf16"
        return _case(None, model, weights, layers, limit, decodes=n, context_lo=max(16, hi // rng.randrange(1, 9)), context_hi=hi, kv=kv,
                     mix=mix)
    tokens = _spread(rng, 150, 14000)
    hi = min(_spread(rng, 100, long_), tokens)
    lo = max(8, hi // rng.randrange(1, 12))
    n = max(1, int(tokens / ((lo + hi) / 2)))
    n = min(n, 96)
    if kind == "prefill":
        return _case(None, model, weights, layers, limit, prompts=n, prompt_lo=lo, prompt_hi=hi, mix=mix)
    if kind == "turn":
        n = min(n, 48)
        hi = min(hi, 1500)
        old = _spread(rng, 100, min(long_ - hi, 3800 - hi))
        return _case(None, model, weights, layers, limit, prompts=n, prompt_lo=min(lo, hi), prompt_hi=hi, history_lo=max(16, old // 3),
                     history_hi=old, mix=mix)
    n = min(n, 24)
    d = _spread(rng, 1, 100)
    ctx = _spread(rng, 64, 3000)
    return _case(None, model, weights, layers, limit, prompts=n, prompt_lo=lo, prompt_hi=hi, decodes=d, context_lo=max(16, ctx // 6),
                 context_hi=ctx, mix=mix)


def _sequences(case):
    """(cached tokens, new tokens) of every sequence: several-token ones first, as the engine orders a step."""
    rng = random.Random(zlib.crc32(repr(sorted((k, v) for k, v in case.items() if k != "name")).encode()))
    out = []
    for _ in range(case["prompts"]):
        new = max(2, _spread(rng, case["prompt_lo"], case["prompt_hi"]))
        out.append((_spread(rng, case["history_lo"], case["history_hi"]) if case["history_hi"] else 0, new))
    for _ in range(case["decodes"]):
        out.append((_spread(rng, case["context_lo"], case["context_hi"]), 1))
    return out


# --------------------------------------------------------------------------------------------------- weights
_E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)


class Weights:
    """Tensors of a model by name, each from the seed and its name alone. ``get`` gives what a checkpoint would."""

    def __init__(self, case, seed, device="cuda"):
        self.fmt, self.seed, self.device = case["weights"], seed, device

    def _gen(self, name):
        return torch.Generator(device=self.device).manual_seed(zlib.crc32(name.encode()) + (self.seed << 32) % (1 << 62))

    def has(self, name):
        return not any(w in name for w in ("query_key_value", "gate_up_proj", "experts.gate_up", "experts.down_proj"))

    def _plain(self, name, shape, std, mean=0.0):
        return torch.empty(shape, dtype=torch.bfloat16, device=self.device).normal_(mean, std, generator=self._gen(name))

    def parts(self, name, shape):
        """The tensor of a projection in its format: (values, scales per 128 x 128 block or None)."""
        small = (2.0 ** -6 if self.fmt == "nvfp4" else 0.125) if name.endswith(("o_proj.weight", "down_proj.weight")) else 1.0
        n, k = shape
        g = self._gen(name)
        if self.fmt == "fp8":
            q = torch.empty(shape, dtype=torch.bfloat16, device=self.device).normal_(0.0, 64.0, generator=g).clamp_(-448, 448)
            e = torch.randint(0, 2, ((n + 127) // 128, (k + 127) // 128), generator=g, device=self.device)
            return q.to(torch.float8_e4m3fn), small * 2.0 ** (e.float() - 13.0)
        if self.fmt == "w4":
            # 16 levels a group of 128, all of them in use
            q = torch.randint(0, 16, (n, k // 128, 128), generator=g, device=self.device, dtype=torch.int8)
            q[..., 0], q[..., 1] = 0, 15
            s = (1.0 + torch.randint(0, 4, (n, k // 128, 1), generator=g, device=self.device) / 4.0) * 2.0 ** -9
            return ((q - 8).to(torch.bfloat16) * (small * s).to(torch.bfloat16)).view(n, k), None
        if self.fmt == "nvfp4":
            # every 16 values have one at the format's largest magnitude, and the tensor a block at the largest scale
            v = torch.tensor(_E2M1, device=self.device, dtype=torch.bfloat16)[
                torch.randint(0, 8, (n, k // 16, 16), generator=g, device=self.device, dtype=torch.int32)]
            v[..., 3] = 6.0
            v *= torch.randint(0, 2, (n, k // 16, 16), generator=g, device=self.device, dtype=torch.int8).to(v.dtype) * 2 - 1
            s = torch.randint(0x68, 0x7F, (n, k // 16, 1), generator=g, device=self.device, dtype=torch.uint8)
            s[0, 0, 0] = 0x7E                                                                   # 448
            s = s.view(torch.float8_e4m3fn).to(torch.bfloat16)
            return (v * s * (small * 2.0 ** -15)).view(n, k), None
        return self._plain(name, shape, 0.02 * small), None

    def get(self, name, shape=None, device=None, kind="normal"):
        if name.endswith("norm.weight") or name.endswith("layernorm.weight"):
            return self._plain(name, shape, 0.05, 1.0)
        if "embed_tokens" in name:
            return self._plain(name, shape, 1.0)
        if name.endswith("e_score_correction_bias"):
            return self._plain(name, shape, 0.1)
        if name.endswith("bias"):
            return self._plain(name, shape, 0.5)
        if name == "lm_head.weight" or name.endswith("mlp.gate.weight"):
            return self._plain(name, shape, 0.02)
        w, s = self.parts(name, shape)
        if s is None:
            return w
        from ksanallm_b200.models.weights import Fp8Pair
        return Fp8Pair(w, s)

    def dense(self, name, shape):
        """The same tensor in 64 bits."""
        if "proj" not in name:
            return self.get(name, shape).double()
        w, s = self.parts(name, shape)
        w = w.double()
        if s is None:
            return w
        return w * s.double().repeat_interleave(128, 0)[:shape[0]].repeat_interleave(128, 1)[:, :shape[1]]


def _tokens(case, seed):
    """New tokens of every sequence."""
    rng = np.random.default_rng([seed, 1])
    return [rng.integers(3, MODELS[case["model"]]["vocab_size"], new).tolist() for _, new in _sequences(case)]


def _history(case, seed, layer, device="cuda"):
    """What earlier steps left in a layer's cache, all sequences' tokens one after the other: [tokens, 2 * heads, size] keys then
    values, or [tokens, latent + rotary] rows."""
    m = MODELS[case["model"]]
    n = sum(old for old, _ in _sequences(case))
    g = torch.Generator(device=device).manual_seed((seed << 20) + 7 * layer + 3)
    if "kv_lora_rank" in m:
        shape = (n, m["kv_lora_rank"] + m["qk_rope_head_dim"])
    else:
        shape = (n, 2 * m["num_kv_heads"], m["head_dim"])
    x = torch.empty(shape, dtype=torch.bfloat16, device=device).normal_(0.0, 1.25, generator=g)
    return x.to(torch.float8_e4m3fn) if case["kv"] == "fp8" else x


def _blocks(case):
    return max(sum(-(-(old + new) // BLOCK_TOKENS) for old, new in _sequences(case)), case["limit"] // BLOCK_TOKENS) + 8


def _fill(cache, layer, rows, slots):
    """Rows of a layer into the paged cache [blocks, layers, 2, heads, tokens, size] or [blocks, layers, tokens, size]."""
    b, t = slots // BLOCK_TOKENS, slots % BLOCK_TOKENS
    cache = cache.view(torch.uint8) if cache.dtype == torch.float8_e4m3fn else cache
    rows = rows.view(torch.uint8) if rows.dtype == torch.float8_e4m3fn else rows
    if cache.dim() == 4:
        cache[b, layer, t] = rows
    else:
        h = cache.shape[3]
        cache[b, layer, 0, :, t] = rows[:, :h]
        cache[b, layer, 1, :, t] = rows[:, h:]


def _old_slots(case, table):
    """Cache slots of the histories' tokens by the step's block table [sequences, blocks]."""
    out = []
    for i, (old, _) in enumerate(_sequences(case)):
        p = torch.arange(old)
        out.append(table[i].long()[p // BLOCK_TOKENS] * BLOCK_TOKENS + p % BLOCK_TOKENS)
    return torch.cat(out)


# --------------------------------------------------------------------------------------------------- the step
def prepare(case, seed):
    from ksanallm_b200.config import EngineConfig, ModelConfig
    from ksanallm_b200.llm import LLM
    mc = ModelConfig(num_layers=case["layers"], max_position_embeddings=case["limit"], max_token_len=case["limit"], **MODELS[case["model"]])
    seqs = _sequences(case)
    ec = EngineConfig()
    ec.global_.enable_cuda_graph = True
    ec.batch_scheduler.max_batch_size = max(8, len(seqs))
    ec.batch_scheduler.max_token_len = case["limit"]
    ec.batch_scheduler.max_step_tokens = 16384
    ec.batch_scheduler.preempt_mode = 1
    ec.block_manager.block_token_num = BLOCK_TOKENS
    ec.block_manager.device_blocks_num = _blocks(case)
    ec.quantization.weight_quant_method = QUANT[case["weights"]]
    ec.quantization.kv_cache_dtype = "fp8_e4m3" if case["kv"] == "fp8" else "auto"
    llm = LLM(ec, mc, weights=Weights(case, seed), dtype=torch.bfloat16, max_positions=case["limit"])
    engine, scheduler = llm.engine, llm.engine.scheduler
    ids = [engine.open_given() for _ in seqs]
    old = [(i, [3] * n, []) for i, (n, _) in zip(ids, seqs) if n]
    if old:                                                      # the histories' blocks; their contents are written below
        code, message, plan, _ = scheduler.plan_given(old)
        assert code == 0, message
        scheduler.advance(plan)
    code, message, plan, _ = scheduler.plan_given([(i, t, [len(t) - 1]) for i, t in zip(ids, _tokens(case, seed))])
    assert code == 0, message
    cache = engine.model.kv_cache
    if old:
        table = torch.from_numpy(np.asarray(plan.block_table).reshape(len(seqs), -1).copy())
        slots = _old_slots(case, table).to(cache.device)
        for layer in range(case["layers"]):
            _fill(cache, layer, _history(case, seed, layer), slots)
    state = {"llm": llm, "engine": engine, "plan": plan, "cache": cache}
    engine.runner.execute(plan)                                  # a decode step's graph is captured once, as a server does
    return state


def run(state):
    logits = state["engine"].runner.execute(state["plan"])
    return {"logits": logits, "cache": state["cache"]}


# --------------------------------------------------------------------------------------------------- costs
def _layer_sizes(case, layer):
    """(parameters that every token uses, parameters of routed experts, of them used by one token) of a layer."""
    m = MODELS[case["model"]]
    H = m["hidden_size"]
    if "kv_lora_rank" in m:
        hq, r = m["num_heads"], m["kv_lora_rank"]
        n, p, v = m["qk_nope_head_dim"], m["qk_rope_head_dim"], m["v_head_dim"]
        attn = H * m["q_lora_rank"] + m["q_lora_rank"] * hq * (n + p) + H * (r + p) + hq * v * H + r * hq * (n + v)
        if layer < m["first_k_dense_replace"]:
            return attn + 3 * H * m["intermediate_size"], 0, 0
        one = 3 * H * m["moe_intermediate_size"]
        return attn + one + H * m["num_experts"], one * m["num_experts"], one * m["num_experts_per_tok"]
    q, kv = m["num_heads"] * m["head_dim"], m["num_kv_heads"] * m["head_dim"]
    return H * (q + 2 * kv) + q * H + 3 * H * m["intermediate_size"], 0, 0


def work(case):
    m = MODELS[case["model"]]
    seqs = _sequences(case)
    tokens, rows = sum(n for _, n in seqs), len(seqs)
    H, V, bits = m["hidden_size"], m["vocab_size"], BITS[case["weights"]]
    if "kv_lora_rank" in m:
        row = (m["kv_lora_rank"] + m["qk_rope_head_dim"]) * 2
        pair = 2 * m["num_heads"] * (m["qk_nope_head_dim"] + m["qk_rope_head_dim"] + m["v_head_dim"])
    else:
        row = 2 * m["num_kv_heads"] * m["head_dim"] * (1 if case["kv"] == "fp8" else 2)
        pair = 4 * m["num_heads"] * m["head_dim"]
    pairs = sum(n * old + n * (n + 1) // 2 for old, n in seqs)
    weights = flops = 0
    for layer in range(case["layers"]):
        every, routed, used = _layer_sizes(case, layer)
        weights += (every + min(routed, used * tokens)) * bits / 8
        flops += 2 * (every + used) * tokens + pair * pairs
    cached = case["layers"] * row * (sum(old for old, _ in seqs) + tokens)
    return {"bytes": weights + H * V * 2 + tokens * H * 2 + cached + rows * V * 4, "flops": flops + 2 * H * V * rows}


def tolerance(case):
    """Two correct implementations differ by the rounding of intermediate results to bf16 (seen between two splits of the attention and
    after a change of its results by one rounding step: rel 0.003 to 0.008, max 0.04), and where activations are quantised by the
    values that fall to the other side of a rounding step of the narrow format (rel 0.004 to 0.019, max 0.16)."""
    return {"rel": 0.03, "max": 0.2 if case["weights"] in ("bf16", "w4") else 0.7}


# --------------------------------------------------------------------------------------------------- the same in 64 bits
def _norm(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rotate(x, pos, theta, neox):
    """x [tokens, heads, size]: pairs (i, i + size / 2), or neighbours."""
    d = x.shape[-1]
    f = 1.0 / theta ** (torch.arange(0, d, 2, dtype=torch.float64, device=x.device) / d)
    a = pos.double()[:, None, None] * f
    c, s = a.cos(), a.sin()
    x0, x1 = (x[..., :d // 2], x[..., d // 2:]) if neox else (x[..., 0::2], x[..., 1::2])
    y0, y1 = x0 * c - x1 * s, x1 * c + x0 * s
    return torch.cat([y0, y1], -1) if neox else torch.stack([y0, y1], -1).flatten(-2)


def _attend(q, k, v, scale):
    """Causal attention of the last tokens: q [n, heads, d], k [tokens, kv heads, d], v [tokens, kv heads, dv] -> [n, heads, dv]."""
    n, hq, _ = q.shape
    hk, total = k.shape[1], k.shape[0]
    out = torch.empty(n, hq, v.shape[2], dtype=torch.float64, device=q.device)
    step = max(1, (1 << 28) // total)
    for h in range(hq):
        kh, vh = k[:, h * hk // hq], v[:, h * hk // hq]
        for a in range(0, n, step):
            b = min(n, a + step)
            s = q[a:b, h] @ kh.t() * scale
            s.masked_fill_(torch.arange(total, device=q.device) > torch.arange(total - n + a, total - n + b, device=q.device)[:, None],
                           float("-inf"))
            out[a:b, h] = torch.softmax(s, -1) @ vh
    return out


def _experts(m, W, p, x):
    """Routed experts (sigmoid scores, the choice corrected by a bias and limited to groups) and the shared one."""
    E, K, H, inter = m["num_experts"], m["num_experts_per_tok"], m["hidden_size"], m["moe_intermediate_size"]
    score = torch.sigmoid(x @ W.dense(p + "gate.weight", (E, H)).t())
    pick = score + W.get(p + "gate.e_score_correction_bias", (E,)).double()
    group = pick.unflatten(-1, (m["n_group"], -1))
    top = group.topk(2, dim=-1).values.sum(-1).topk(m["topk_group"], dim=-1).indices
    keep = torch.zeros(group.shape[:2], dtype=torch.bool, device=x.device).scatter_(1, top, True)
    ids = group.masked_fill(~keep.unsqueeze(-1), float("-inf")).flatten(-2).topk(K, dim=-1).indices
    w = score.gather(1, ids)
    w = w / w.sum(-1, keepdim=True) * m["routed_scaling_factor"]
    out = _gated(W, p + "shared_expert.", x, H, m["shared_expert_intermediate_size"])
    for e in range(E):
        row, k = (ids == e).nonzero(as_tuple=True)
        if row.numel():
            out.index_add_(0, row, _gated(W, p + f"experts.{e}.", x[row], H, inter) * w[row, k, None])
    return out


def _gated(W, p, x, H, inter):
    a = torch.nn.functional.silu(x @ W.dense(p + "gate_proj.weight", (inter, H)).t())
    a *= x @ W.dense(p + "up_proj.weight", (inter, H)).t()
    return a @ W.dense(p + "down_proj.weight", (H, inter)).t()


def _plan_slots(case):
    """Cache slots of the cached and of the new tokens, all sequences' one after the other: blocks are taken in order, by the histories
    first and by the new tokens after them."""
    seqs, taken, tables = _sequences(case), 0, []
    for old, _ in seqs:
        n = -(-old // BLOCK_TOKENS)
        tables.append(list(range(taken, taken + n)))
        taken += n
    for (old, new), table in zip(seqs, tables):
        n = -(-(old + new) // BLOCK_TOKENS) - len(table)
        table += range(taken, taken + n)
        taken += n
    spans = [(np.asarray(t)[np.arange(old + new) // BLOCK_TOKENS] * BLOCK_TOKENS + np.arange(old + new) % BLOCK_TOKENS, old)
             for t, (old, new) in zip(tables, seqs)]
    return [torch.from_numpy(np.concatenate(part)) for part in ([s[:old] for s, old in spans], [s[old:] for s, old in spans])]


def exact(case, seed):
    """Logits and cache in 64 bits, from unrounded activations. No cache where activations are rounded to 4 bits: keys and values then are
    a tenth off, and the figure would say nothing."""
    m, seqs, W = MODELS[case["model"]], _sequences(case), Weights(case, seed)
    dev, H, V, eps = "cuda", m["hidden_size"], m["vocab_size"], m["rms_norm_eps"]
    latent = "kv_lora_rank" in m
    ids = torch.tensor(sum(_tokens(case, seed), []), device=dev)
    pos = torch.cat([torch.arange(old, old + new) for old, new in seqs]).to(dev)
    x = W.get("model.embed_tokens.weight", (V, H))[ids].double()
    ends = np.cumsum([new for _, new in seqs])
    cached = np.cumsum([0] + [old for old, _ in seqs])
    row = (m["kv_lora_rank"] + m["qk_rope_head_dim"],) if latent else (2, m["num_kv_heads"])
    row = (BLOCK_TOKENS,) + row if latent else row + (BLOCK_TOKENS, m["head_dim"])
    cache = torch.zeros((_blocks(case), case["layers"]) + row, dtype=torch.float64, device=dev)
    old_slots, new_slots = (s.to(dev) for s in _plan_slots(case))
    for layer in range(case["layers"]):
        p = f"model.layers.{layer}."
        y = _norm(x, W.get(p + "input_layernorm.weight", (H,)).double(), eps)
        old = _history(case, seed, layer).double()
        if latent:
            hq, r, n_, p_, v_ = m["num_heads"], m["kv_lora_rank"], m["qk_nope_head_dim"], m["qk_rope_head_dim"], m["v_head_dim"]
            qa = y @ W.dense(p + "self_attn.q_a_proj.weight", (m["q_lora_rank"], H)).t()
            qa = _norm(qa, W.get(p + "self_attn.q_a_layernorm.weight", (m["q_lora_rank"],)).double(), eps)
            q = (qa @ W.dense(p + "self_attn.q_b_proj.weight", (hq * (n_ + p_), m["q_lora_rank"])).t()).view(-1, hq, n_ + p_)
            q = torch.cat([q[..., :n_], _rotate(q[..., n_:], pos, m["rope_theta"], False)], -1)
            kv = y @ W.dense(p + "self_attn.kv_a_proj_with_mqa.weight", (r + p_, H)).t()
            new = torch.cat([_norm(kv[:, :r], W.get(p + "self_attn.kv_a_layernorm.weight", (r,)).double(), eps),
                             _rotate(kv[:, None, r:], pos, m["rope_theta"], False)[:, 0]], -1)
            kv_b = W.dense(p + "self_attn.kv_b_proj.weight", (hq * (n_ + v_), r)).view(hq, n_ + v_, r)
            scale = 1.0 / math.sqrt(n_ + p_)
        else:
            hq, hk, d = m["num_heads"], m["num_kv_heads"], m["head_dim"]
            def proj(name, heads):
                z = y @ W.dense(p + f"self_attn.{name}_proj.weight", (heads * d, H)).t()
                if m.get("qkv_bias"):
                    z += W.get(p + f"self_attn.{name}_proj.bias", (heads * d,)).double()
                return z.view(-1, heads, d)
            q = _rotate(proj("q", hq), pos, m["rope_theta"], True)
            new = torch.cat([_rotate(proj("k", hk), pos, m["rope_theta"], True), proj("v", hk)], 1)
            scale = 1.0 / math.sqrt(d)
        _fill(cache, layer, old, old_slots)
        _fill(cache, layer, new, new_slots)
        out = []
        for i, (_, n) in enumerate(seqs):
            a, b = int(ends[i]) - n, int(ends[i])
            rows = torch.cat([old[cached[i]:cached[i + 1]], new[a:b]])
            if latent:
                k = torch.cat([torch.einsum("tr,hnr->thn", rows[:, :r], kv_b[:, :n_]),
                               rows[:, None, r:].expand(-1, hq, -1)], -1)
                v = torch.einsum("tr,hvr->thv", rows[:, :r], kv_b[:, n_:])
            else:
                k, v = rows[:, :hk], rows[:, hk:]
            out.append(_attend(q[a:b], k, v, scale).flatten(1))
        o = torch.cat(out)
        x = x + o @ W.dense(p + "self_attn.o_proj.weight", (H, o.shape[1])).t()
        y = _norm(x, W.get(p + "post_attention_layernorm.weight", (H,)).double(), eps)
        if latent and layer >= m["first_k_dense_replace"]:
            x = x + _experts(m, W, p + "mlp.", y)
        else:
            x = x + _gated(W, p + "mlp.", y, H, m["intermediate_size"])
    x = _norm(x[torch.from_numpy(ends - 1).to(dev)], W.get("model.norm.weight", (H,)).double(), eps)
    return {"logits": x @ W.dense("lm_head.weight", (V, H)).t(), "cache": None if case["weights"] == "nvfp4" else cache}

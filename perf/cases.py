"""What the speed of this framework is measured on: its public entry points over the sizes that its users meet.

  layer_f32      the drop-in fp32 attention layer, collapsed or per-head
  prefill_attn   RoPE + causal grouped-query attention over a prompt, bf16
  decode_attn    one new token per sequence over a paged bf16 cache
  llama, soluzen, duponex
                 the model families: a prompt pass (caches filled from nothing, in one portion or two), or one step of every
                 sequence replayed from the captured graph that a serving loop keeps

Widths are those of the benchmark's configurations; batch, lengths, layers and dtype vary.  Weights are random at the scale of
trained ones, drawn on the GPU from the seed."""
import math

import torch

from baranet_bdml_b200 import layers, ops, registry
from baranet_bdml_b200.checkpoint import Weights
from baranet_bdml_b200.kv_cache import PAGE_TOKENS, PagedKVCache
from baranet_bdml_b200.tensor import AGTensor, TensorF

WIDTH, VOCAB, EPS, THETA = 2048, 32000, 1e-5, 10000.0
HEADS, KV_HEADS, DIM = 32, 4, 64
LLAMA_FF, SOLUZEN_FF, DUPONEX_FF = 5632, 5632, 7424
LATENT = dict(heads=16, dim=128, rot_dim=64, vdim=128, q_rank=1536, kv_rank=512, rot={"base": THETA, "dims": 64}, scale=192 ** -0.5)
MAMBA = dict(heads=64, vdim=64, state=128, groups=1, conv=4, norm_groups=1)
SIDE, STREAMS = 256, 2


def listed():
    return [
        # one attention layer called from the reference's fp32 model
        {"name": "layer_f32_128", "path": "layer_f32", "seq": 128, "mode": "collapsed"},
        # attention inside somebody else's model: a batch of long prompts, and one short prompt of no particular length
        {"name": "prefill_attn_8x2048", "path": "prefill_attn", "batch": 8, "seq": 2048},
        {"name": "prefill_attn_1x333", "path": "prefill_attn", "batch": 1, "seq": 333},
        # a serving batch of unequal sequences, and a few very long ones
        {"name": "decode_attn_64", "path": "decode_attn", "batch": 64, "shortest": 1024, "longest": 4096},
        {"name": "decode_attn_4_long", "path": "decode_attn", "batch": 4, "shortest": 262144, "longest": 262144},
        # prompts and decode steps of each family: a batch of prompts, a long document, a document that arrives in portions;
        # a small batch, a single user, a large batch
        {"name": "llama_prompt_16x512", "path": "llama", "call": "prompt", "batch": 16, "seq": 512, "layers": 4},
        {"name": "llama_step_16", "path": "llama", "call": "step", "batch": 16, "seq": 512, "layers": 6},
        {"name": "soluzen_prompt_8x2048", "path": "soluzen", "call": "prompt", "batch": 8, "seq": 2048, "window": 1024, "portions": 1,
         "dtype": "bfloat16"},
        {"name": "soluzen_step_1", "path": "soluzen", "call": "step", "batch": 1, "seq": 1100, "window": 1024, "portions": 1,
         "dtype": "bfloat16"},
        {"name": "duponex_prompt_3x1371", "path": "duponex", "call": "prompt", "batch": 3, "seq": 1371, "chunk": 2048, "layers": 4,
         "portions": 2, "dtype": "bfloat16"},
        {"name": "duponex_step_64", "path": "duponex", "call": "step", "batch": 64, "seq": 512, "chunk": 2048, "layers": 4, "portions": 1,
         "dtype": "bfloat16"},
        # the same model in true fp32
        {"name": "duponex_f32_4x200", "path": "duponex", "call": "prompt", "batch": 4, "seq": 200, "chunk": 2048, "layers": 2, "portions": 1,
         "dtype": "float32"},
    ]


def draw(rng):
    def log_int(lo, hi):
        return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))

    def even_tiles(batch, seq):
        # A prompt whose 128-token tiles are odd in number, in a batch of more work than the GPU has multiprocessors for, is
        # left out of the causal prefill's range: attention gave up a wait there (BN_ERR_TIMEOUT) when this file was written
        tiles = -(-seq // 128)
        if tiles % 2 == 0 or batch * HEADS * ((tiles + 1) // 2) <= 148:
            return seq
        return seq + 128 if seq <= 1024 else seq - 128

    path = rng.choice(["layer_f32", "prefill_attn", "decode_attn", "llama", "soluzen", "duponex", "llama", "soluzen", "duponex"])
    if path == "layer_f32":
        return {"path": path, "seq": log_int(16, 512), "mode": rng.choice(["collapsed", "per_head"])}
    if path == "prefill_attn":
        seq = log_int(32, 4096)
        batch = log_int(1, max(1, 16384 // (seq + 128)))
        return {"path": path, "batch": batch, "seq": even_tiles(batch, seq)}
    if path == "decode_attn":
        longest = log_int(64, 65536)
        return {"path": path, "batch": log_int(1, min(256, 1048576 // longest)), "shortest": max(1, longest // rng.randint(1, 8)), "longest": longest}
    case = {"path": path, "call": rng.choice(["prompt", "step"])}
    f32 = path != "llama" and rng.random() < 0.25
    if case["call"] == "prompt":
        seq = log_int(16, 2048)
        if f32:
            seq = min(seq, 512)
        case.update(batch=log_int(1, max(1, 512 // seq if f32 else 16384 // (seq + 128))), seq=seq)
    else:
        batch = log_int(1, 64)
        case.update(batch=batch, seq=log_int(16, 2048 // batch if f32 else min(2048, 32768 // batch)))
    if path == "llama":
        case["seq"] = even_tiles(case["batch"], case["seq"])
    if path == "soluzen":
        case.update(window=rng.choice([256, 1024]), portions=rng.choice([1, 2]), dtype="float32" if f32 else "bfloat16")
    else:
        case.update(layers=rng.randint(2, 4))
    if path == "duponex":
        case.update(chunk=rng.choice([2048, 4096]), portions=rng.choice([1, 2]), dtype="float32" if f32 else "bfloat16")
    return case


# ------------------------------------------------------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(gen, *shape, std=1.0, dtype=torch.float32):
    return (torch.randn(shape, generator=gen, device="cuda") * std).to(dtype)


def _layer_inputs(case, seed):
    g, kv = _generator(seed), KV_HEADS * DIM
    x = _normal(g, case["seq"], WIDTH)
    return [x] + [_normal(g, WIDTH, n, std=0.02) for n in (WIDTH, kv, kv, WIDTH)]


def _prefill_inputs(case, seed):
    g, B, S = _generator(seed), case["batch"], case["seq"]
    return [_normal(g, B, S, h, DIM, dtype=torch.bfloat16) for h in (HEADS, KV_HEADS, KV_HEADS)]


def _lengths(case):
    B, lo, hi = case["batch"], case["shortest"], case["longest"]
    return [hi] + [lo + (hi - lo) * i // B for i in range(1, B)]


def _decode_inputs(case, seed):
    """q, the pool of pages, the page table (pages of a sequence anywhere in the pool) and the lengths"""
    g, B = _generator(seed), case["batch"]
    order = torch.randperm(B, generator=g, device="cuda").tolist()
    lens = [_lengths(case)[i] for i in order]
    pages = [-(-n // PAGE_TOKENS) for n in lens]
    pool = torch.empty((sum(pages), KV_HEADS, 2, PAGE_TOKENS, DIM), dtype=torch.bfloat16, device="cuda").normal_(generator=g)
    shuffled = torch.randperm(sum(pages), generator=g, device="cuda").to(torch.int32)
    table = torch.zeros((B, max(pages)), dtype=torch.int32, device="cuda")
    at = 0
    for b, n in enumerate(pages):
        table[b, :n] = shuffled[at:at + n]
        at += n
    q = _normal(g, B, HEADS, DIM, dtype=torch.bfloat16)
    return q, pool, table, lens


def _config(case):
    if case["path"] == "llama":
        return {"architecture": "LLaMA", "vocab_size": VOCAB, "hidden_size": WIDTH, "intermediate_size": LLAMA_FF,
                "num_hidden_layers": case["layers"], "num_attention_heads": HEADS, "num_key_value_heads": KV_HEADS, "rms_norm_eps": EPS,
                "rope_theta": THETA}
    if case["path"] == "soluzen":
        entries = [{"type": "latent_attention", "mixer": dict(LATENT, mask={"size": case["window"]}), "mlp": {"kind": "dense", "ff": SOLUZEN_FF}}]
        entries += [{"type": "mamba2", "mixer": MAMBA, "mlp": None}] * 3
        return {"architecture": "Soluzen", "layers": entries, "loop": {"start": 2, "stop": 4, "times": 2}, "norm": {"eps": EPS},
                "token_side": {"dim": SIDE}, "vocab": VOCAB, "width": WIDTH}
    mixer = dict(heads=HEADS, kv_heads=KV_HEADS, dim=DIM, vdim=DIM, mask={"size": case["chunk"]}, scale=DIM ** -0.5, v_mix=True)
    return {"architecture": "Duponex", "embedding": {"scale": 1.0}, "layers": [{"type": "attention", "mixer": mixer, "mlp": {"kind": "dense", "ff": DUPONEX_FF}}] * case["layers"],
            "norm": {"eps": EPS}, "residual_mult": 0.7, "streams": STREAMS, "vocab": VOCAB, "width": WIDTH}


def _shapes(case):
    W, s = WIDTH, {}
    if case["path"] == "llama":
        s.update({"embed_tokens": (VOCAB, W), "norm": (W,), "lm_head": (VOCAB, W)})
        kv = KV_HEADS * DIM
        for i in range(case["layers"]):
            p = f"layers.{i}."
            s.update({p + "self_attn.q_proj": (W, W), p + "self_attn.k_proj": (kv, W), p + "self_attn.v_proj": (kv, W), p + "self_attn.o_proj": (W, W),
                      p + "mlp.gate_proj": (LLAMA_FF, W), p + "mlp.up_proj": (LLAMA_FF, W), p + "mlp.down_proj": (W, LLAMA_FF),
                      p + "input_layernorm": (W,), p + "post_attention_layernorm": (W,)})
        return s
    c = _config(case)
    n = len(c["layers"])
    s.update({"embed": (VOCAB, W), "final.norm": (W,), "head": (VOCAB, W)})
    if case["path"] == "soluzen":
        s.update({"side.embed": (VOCAB, n * SIDE), "final.norm.b": (W,), "loop.in": (W, 2 * W), "loop.step": (c["loop"]["times"], W)})
    for i, lay in enumerate(c["layers"]):
        p, m = f"l{i}.", lay["mixer"]
        if case["path"] == "duponex":
            for q in "12":
                s.update({p + "norm" + q: (W,), p + "ls" + q: (W,), f"{p}hc{q}.in": (STREAMS,), f"{p}hc{q}.out": (STREAMS,), f"{p}hc{q}.mix": (STREAMS, STREAMS)})
            s.update({p + "mlp.up": (DUPONEX_FF, W), p + "mlp.down": (W, DUPONEX_FF), p + "mix.vmix": (), p + "mix.o": (W, HEADS * DIM), p + "mix.o.b": (W,),
                      p + "mix.g": (HEADS * DIM, W)})
            for k, h in (("q", HEADS), ("k", KV_HEADS), ("v", KV_HEADS)):
                s.update({p + "mix." + k: (h * DIM, W), f"{p}mix.{k}.b": (h * DIM,)})
            continue
        s.update({p + "norm1": (W,), p + "norm1.b": (W,), p + "side.gate": (SIDE, W), p + "side.proj": (W, SIDE), p + "side.norm": (W,)})
        if lay["mlp"] is not None:
            s.update({p + "norm2": (W,), p + "norm2.b": (W,), p + "mlp.gate": (SOLUZEN_FF, W), p + "mlp.up": (SOLUZEN_FF, W), p + "mlp.down": (W, SOLUZEN_FF)})
        p += "mix."
        if lay["type"] == "latent_attention":
            H, d, r, v, qr, kr = (m[k] for k in ("heads", "dim", "rot_dim", "vdim", "q_rank", "kv_rank"))
            s.update({p + "dq": (qr, W), p + "dq.norm": (qr,), p + "uq": (H * (d + r), qr), p + "dkv": (kr + r, W), p + "dkv.norm": (kr,),
                      p + "uk": (H * d, kr), p + "uv": (H * v, kr), p + "o": (W, H * v)})
        else:
            H, v, N, G = (m[k] for k in ("heads", "vdim", "state", "groups"))
            C = H * v + 2 * G * N
            s.update({p + "in": (H * v + C + H, W), p + "conv": (C, m["conv"]), p + "conv.b": (C,), p + "dt_bias": (H,), p + "A_log": (H,), p + "D": (H,),
                      p + "norm": (H * v,), p + "o": (W, H * v)})
    return s


def _weights(case, gen):
    """bf16 numbers, whatever the model's dtype: matrices N(0, 0.02), norms near 1, the recurrence's constants over the ranges
    that Mamba-2 is initialised to"""
    out = {}
    for name, shape in _shapes(case).items():
        leaf = name.rsplit(".", 1)[-1]
        x = torch.randn(shape, generator=gen, device="cuda")
        if "norm" in leaf or leaf in ("D", "ls1", "ls2"):
            x = (0.5 if leaf.startswith("ls") or name.endswith("side.norm") else 1.0) * (1.0 + 0.1 * x)
        elif leaf in ("in", "out", "vmix") and "hc" in name or leaf == "vmix":
            x = 0.5 + 0.05 * x
        elif leaf == "mix":
            x = torch.eye(*shape, device="cuda") + 0.05 * x
        elif leaf == "A_log":
            x = torch.log(1.0 + 15.0 * torch.rand(shape, generator=gen, device="cuda"))
        elif leaf == "dt_bias":
            x = torch.log(torch.expm1(torch.exp(math.log(1e-3) + math.log(1e2) * torch.rand(shape, generator=gen, device="cuda"))))
        elif leaf == "conv":
            x = 0.3 * x
        elif name == "loop.in":
            x = 0.02 * x + torch.eye(*shape, device="cuda")
        elif name not in ("embed", "side.embed"):
            x = 0.02 * x
        out[name] = x.to(torch.bfloat16)
    return out


def _tokens(case, gen):
    """prompt ids (batch, seq), and one more id per sequence for a step"""
    ids = torch.randint(0, VOCAB, (case["batch"], case["seq"] + 1), generator=gen, device="cuda", dtype=torch.int32)
    return ids[:, :-1].contiguous(), ids[:, -1].contiguous()


def _prompt(model, ids, portions):
    """A prompt pass from empty caches; returns the logits of every sequence's last position."""
    B, S = ids.shape
    if portions == 1 or S < 2:
        return model.prefill(ids, S + 1)
    model.allocate(B, S + 1)
    slots = [model.slots.acquire() for _ in range(B)]
    first = S * 5 // 8
    model.extend(ids[:, :first], slots, torch.empty(0, dtype=torch.int64, device="cuda"))
    return model.extend(ids[:, first:], slots)


def _caches(model, case):
    if case["path"] == "llama":
        return [c.pool for c in model.caches]
    return [t for s in model.states for t in s.tensors()]


def prepare(case, seed):
    if case["path"] == "layer_f32":
        x, *w = _layer_inputs(case, seed)
        layer = layers.GroupedQueryAttention(layers.LLaMAConfig(), heads_mode=case["mode"])
        layer.q_proj, layer.k_proj, layer.v_proj, layer.o_proj = (AGTensor(TensorF.from_torch(t)) for t in w)
        return {"case": case, "layer": layer, "x": AGTensor(TensorF.from_torch(x))}
    if case["path"] == "prefill_attn":
        q, k, v = _prefill_inputs(case, seed)
        return {"case": case, "q": q, "k": k, "v": v, "ws": ops.prefill_workspace(case["batch"], case["seq"], HEADS, KV_HEADS, DIM)}
    if case["path"] == "decode_attn":
        q, pool, table, lens = _decode_inputs(case, seed)
        cache = PagedKVCache(1, case["batch"], table.shape[1], KV_HEADS, DIM, THETA)
        cache.pool, cache.num_pages = pool, pool.shape[0]
        cache.page_table.copy_(table)
        cache.seq_lens.copy_(torch.tensor(lens, dtype=torch.int32))
        return {"case": case, "q": q, "cache": cache}
    gen = _generator(seed)
    weights = _weights(case, gen)
    ids, token = _tokens(case, gen)
    with layers.device_init(0.02):
        model = registry.build_model(_config(case), Weights(weights), getattr(torch, case.get("dtype", "bfloat16")))
    state = {"case": case, "model": model, "ids": ids, "token": token}
    if case["call"] == "step":
        _prompt(model, ids, case.get("portions", 1))
        state["lens"] = model.seq_lens.clone()
        state["step"] = model.capture_decode_step()
    return state


def run(state):
    case = state["case"]
    if case["path"] == "layer_f32":
        return state["layer"](state["x"]).data.torch_view()
    if case["path"] == "prefill_attn":
        return ops.attn_prefill_bf16(state["q"], state["k"], state["v"], workspace=state["ws"])
    if case["path"] == "decode_attn":
        return state["cache"].decode(state["q"], num_heads=HEADS)
    model = state["model"]
    if case["call"] == "prompt":
        logits = _prompt(model, state["ids"], case.get("portions", 1))
    else:
        # the next token of every sequence; where a step only writes the row of its position, the position is set back, so
        # that every pass is the same step (a recurrent state goes on instead, at a cost that does not depend on the length).
        # The greedy choice is made inside the step, too; the logits say all that it says, without ties
        if case["path"] != "soluzen":
            model.seq_lens.copy_(state["lens"])
        logits, _ = state["step"](state["token"])
    return [logits] + _caches(model, case)


# --------------------------------------------------------------------------------------------------------------------- work
def _product_weights(case):
    """elements of the matrices that every token is multiplied with, each as often as it is run"""
    runs = {}
    if case["path"] == "soluzen":
        runs = {2: 2, 3: 2}
    total = 0
    for name, shape in _shapes(case).items():
        if len(shape) == 2 and min(shape) > 8 and name not in ("embed", "side.embed", "embed_tokens", "head", "lm_head"):
            times = runs.get(int(name[1]), 1) if name[0] == "l" and name[1].isdigit() else 2 if name == "loop.in" else 1
            total += times * shape[0] * shape[1]
    return total


def work(case):
    if case["path"] == "layer_f32":
        S, kv = case["seq"], KV_HEADS * DIM
        scores = S * (S + 1) // 2
        return {"bytes": 4.0 * (2 * S * WIDTH + 2 * WIDTH * (WIDTH + kv)), "flops": 4.0 * S * WIDTH * (WIDTH + kv) + 4.0 * scores * WIDTH}
    if case["path"] == "prefill_attn":
        B, S = case["batch"], case["seq"]
        return {"bytes": 4.0 * B * S * (HEADS + KV_HEADS) * DIM, "flops": 4.0 * B * HEADS * DIM * (S * (S + 1) // 2)}
    if case["path"] == "decode_attn":
        n = sum(_lengths(case))
        return {"bytes": 4.0 * n * KV_HEADS * DIM + 4.0 * case["batch"] * HEADS * DIM, "flops": 4.0 * n * HEADS * DIM}
    B, S, step = case["batch"], case["seq"], case["call"] == "step"
    size = 4 if case.get("dtype") == "float32" else 2
    tokens = B if step else B * S
    params = sum(math.prod(s) for n, s in _shapes(case).items() if n not in ("embed", "side.embed", "embed_tokens"))
    flops = 2.0 * tokens * _product_weights(case) + 2.0 * B * VOCAB * WIDTH
    nbytes = float(size * params + tokens * WIDTH * size + 4 * B * VOCAB)

    def pairs(span):                          # (query, key) pairs that a sequence's new tokens see
        if step:
            return min(S + 1, span)
        return sum(min(i + 1, span) for i in range(S))

    if case["path"] == "soluzen":
        m, c = MAMBA, LATENT
        flops += 2.0 * B * pairs(case["window"]) * c["heads"] * (c["dim"] + c["rot_dim"] + c["vdim"])
        flops += 5 * 6.0 * tokens * m["heads"] * m["vdim"] * m["state"]
        state = 4 * B * m["heads"] * m["vdim"] * m["state"]
        nbytes += 5 * state * (2 if step else 1) + B * (c["kv_rank"] + c["rot_dim"]) * size * min(case["window"], S + 1)
    else:
        flops += 4.0 * case["layers"] * B * pairs(case.get("chunk", 1 << 30)) * HEADS * DIM
        nbytes += 2.0 * case["layers"] * B * KV_HEADS * DIM * size * (S + 1)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["path"] == "layer_f32":
        return {"rel": 1.5e-5, "max": 1e-3}
    if case["path"] in ("prefill_attn", "decode_attn"):
        return {"rel": 1e-2, "max": 0.2}
    if case.get("dtype") == "float32":
        return {"rel": 4e-5, "max": 4e-3}
    return {"rel": 2.5e-2, "max": 0.8}


# ------------------------------------------------------------------------------------------------------------- in 64 bits
def _turn(x, positions):
    """Adjacent pairs of the last dimension turned by fp32(position) * fp32(frequency), as the operator is defined; x (..., T, heads, D)"""
    i = torch.arange(0, x.shape[-1], 2, device=x.device, dtype=torch.float32) / x.shape[-1]
    freq = (1.0 / torch.pow(torch.tensor(THETA, device=x.device, dtype=torch.float64), i.double()).float().double()).float()
    a = (positions.float()[..., None] * freq).double()[..., None, :]
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * torch.cos(a) - v * torch.sin(a), u * torch.sin(a) + v * torch.cos(a)], dim=-1).flatten(-2)


def _turn_exact(x, positions):
    """The same with angles in 64 bits"""
    freq = THETA ** (-torch.arange(0, x.shape[-1], 2, device=x.device, dtype=torch.float64) / x.shape[-1])
    a = (positions.double()[..., None] * freq)[..., None, :]
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * torch.cos(a) - v * torch.sin(a), u * torch.sin(a) + v * torch.cos(a)], dim=-1).flatten(-2)


def _attention(q, k, v, scale, visible):
    """q (T, H, E), k (T, G, E), v (T, G, V) of one sequence -> (T, H, V)"""
    T, H, _ = q.shape
    G = k.shape[1]
    s = torch.einsum("tgre,sge->grts", q.reshape(T, G, H // G, -1), k) * scale
    s.masked_fill_(~visible, -math.inf)
    return torch.einsum("grts,sgv->tgrv", torch.softmax(s, dim=-1), v).reshape(T, H, -1)


def _causal(T, span=None, chunk=None):
    i = torch.arange(T, device="cuda")
    see = i[:, None] >= i[None, :]
    if span is not None:
        see &= i[:, None] - i[None, :] < span
    if chunk is not None:
        see &= i[:, None] // chunk == i[None, :] // chunk
    return see


def _rms(x, eps=EPS):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _exact_llama(case, w, ids):
    B, T = ids.shape
    x = w["embed_tokens"][ids.long()].double()
    pos, see = torch.arange(T, device="cuda"), _causal(T)
    pages = -(-(case["seq"] + 1) // PAGE_TOKENS)
    pools = []
    for i in range(case["layers"]):
        W = lambda n: w[f"layers.{i}." + n].double()                                              # noqa: E731
        h = _rms(x) * W("input_layernorm")
        q = _turn((h @ W("self_attn.q_proj").T).view(B, T, HEADS, DIM), pos)
        k = _turn((h @ W("self_attn.k_proj").T).view(B, T, KV_HEADS, DIM), pos)
        v = (h @ W("self_attn.v_proj").T).view(B, T, KV_HEADS, DIM)
        rows = torch.zeros((2, B, pages * PAGE_TOKENS, KV_HEADS, DIM), dtype=torch.float64, device="cuda")
        rows[0, :, :T], rows[1, :, :T] = k, v
        pools.append(rows.view(2, B * pages, PAGE_TOKENS, KV_HEADS, DIM).permute(1, 3, 0, 2, 4).contiguous())
        a = torch.stack([_attention(q[b], k[b], v[b], DIM ** -0.5, see) for b in range(B)]).reshape(B, T, -1)
        x = x + a @ W("self_attn.o_proj").T
        h = _rms(x) * W("post_attention_layernorm")
        x = x + (torch.nn.functional.silu(h @ W("mlp.gate_proj").T) * (h @ W("mlp.up_proj").T)) @ W("mlp.down_proj").T
    return [(_rms(x[:, -1]) * w["norm"].double()) @ w["lm_head"].double().T] + pools


def _last_rows(x, rows, skip):
    """(B, T, n) laid out by position % rows; `skip`: a shorter ring than the sequence keeps rows that nobody may read"""
    B, T = x.shape[:2]
    if T > rows and skip:
        return None
    out = torch.zeros((B, rows) + tuple(x.shape[2:]), dtype=torch.float64, device="cuda")
    at = torch.arange(max(0, T - rows), T, device="cuda")
    out[:, at % rows] = x[:, at]
    return out


def _gelu(z):
    return torch.nn.functional.gelu(z, approximate="tanh")


def _exact_soluzen(case, w, ids):
    cfg, (B, T) = _config(case), ids.shape
    pos, window = torch.arange(T, device="cuda"), case["window"]
    x = x0 = w["embed"][ids.long()].double()
    side = w["side.embed"][ids.long()].double()
    states = []

    def layer_norm(name, v):
        return torch.nn.functional.layer_norm(v, (WIDTH,), w[name].double(), w[name + ".b"].double(), EPS)

    def latent(h, W):
        m = LATENT
        q = (_rms(h @ W("dq").T) * W("dq.norm") @ W("uq").T).view(B, T, m["heads"], -1)
        q = torch.cat([q[..., :m["dim"]], _turn_exact(q[..., m["dim"]:], pos)], -1)
        down = h @ W("dkv").T
        c = _rms(down[..., :m["kv_rank"]]) * W("dkv.norm")
        kr = _turn_exact(down[..., None, m["kv_rank"]:], pos)
        states.append(_last_rows(torch.cat([c, kr[:, :, 0]], -1), -(-window // PAGE_TOKENS) * PAGE_TOKENS, False))
        k = torch.cat([(c @ W("uk").T).view(B, T, m["heads"], -1), kr.expand(B, T, m["heads"], -1)], -1)
        v, see = (c @ W("uv").T).view(B, T, m["heads"], -1), _causal(T, window)
        return torch.stack([_attention(q[b], k[b], v[b], m["scale"], see) for b in range(B)]).reshape(B, T, -1) @ W("o").T

    def mamba(h, W):
        m = MAMBA
        H, P, N, K = m["heads"], m["vdim"], m["state"], m["conv"]
        inner = H * P
        proj = h @ W("in").T
        z, raw, dt = proj[..., :inner], proj[..., inner:-H], torch.nn.functional.softplus(proj[..., -H:] + W("dt_bias"))
        past = torch.cat([torch.zeros_like(raw[:, :1]).expand(-1, K - 1, -1), raw], 1)
        conv = torch.nn.functional.silu(W("conv.b") + sum(past[:, k:k + T] * W("conv")[:, k] for k in range(K)))
        xs, b, c = conv[..., :inner].view(B, T, H, P), conv[..., inner:inner + N], conv[..., inner + N:]
        decay = torch.exp(-torch.exp(W("A_log")) * dt)
        S, y = torch.zeros((B, H, P, N), dtype=torch.float64, device="cuda"), torch.empty_like(xs)
        for t in range(T):
            S = torch.addcmul(S * decay[:, t, :, None, None], (dt[:, t, :, None] * xs[:, t])[..., None], b[:, t, None, None, :])
            y[:, t] = torch.matmul(S.view(B, H * P, N), c[:, t, :, None]).view(B, H, P)
        y = (y + W("D")[:, None] * xs).reshape(B, T, inner) * torch.nn.functional.silu(z)
        states.extend([S, _last_rows(raw, K, False)])
        return (_rms(y) * W("norm")) @ W("o").T

    order = [(0, None), (1, None), (2, 0), (3, None), (2, 1), (3, None)]
    for i, start in order:
        if start is not None:
            x = torch.cat([x, x0], -1) @ w["loop.in"].double().T + w["loop.step"][start].double()
        W = lambda n: w[f"l{i}." + n].double()                                                    # noqa: E731
        mixer = latent if cfg["layers"][i]["type"] == "latent_attention" else mamba
        x = x + mixer(layer_norm(f"l{i}.norm1", x), lambda n: W("mix." + n))
        if cfg["layers"][i]["mlp"] is not None:
            h = layer_norm(f"l{i}.norm2", x)
            x = x + (_gelu(h @ W("mlp.gate").T) * (h @ W("mlp.up").T)) @ W("mlp.down").T
        y = (_gelu(x @ W("side.gate").T) * side[..., i * SIDE:(i + 1) * SIDE]) @ W("side.proj").T
        x = x + _rms(y) * W("side.norm")
    return [layer_norm("final.norm", x[:, -1]) @ w["head"].double().T] + states


def _exact_duponex(case, w, ids):
    (B, T), n = ids.shape, STREAMS
    streams = w["embed"][ids.long()].double()[None].expand(n, -1, -1, -1)
    see, v_first, states = _causal(T, chunk=case["chunk"]), None, []
    ring = min(case["chunk"], case["seq"] + 1)
    for i in range(case["layers"]):
        W = lambda k: w[f"l{i}." + k].double()                                                    # noqa: E731

        def sublayer(q, f):
            h = _rms(torch.einsum("s,sbtw->btw", W(f"hc{q}.in"), streams)) * W(f"norm{q}")
            y = f(h) * W(f"ls{q}")
            return torch.einsum("su,sbtw->ubtw", W(f"hc{q}.mix"), streams) + 0.7 * W(f"hc{q}.out")[:, None, None, None] * y

        def attend(h):
            nonlocal v_first
            q, k, v = ((h @ W(f"mix.{c}").T + W(f"mix.{c}.b")).view(B, T, -1, DIM) for c in "qkv")
            q, k = _rms(q), _rms(k)
            if v_first is None:
                v_first = v
            else:
                v = (1.0 - W("mix.vmix")) * v + W("mix.vmix") * v_first
            for t in (k, v):
                rows = _last_rows(t, ring, True)
                states.append(None if rows is None else rows.transpose(1, 2).contiguous())
            a = torch.stack([_attention(q[b], k[b], v[b], DIM ** -0.5, see) for b in range(B)]).reshape(B, T, -1)
            return (a * torch.sigmoid(h @ W("mix.g").T)) @ W("mix.o").T + W("mix.o.b")

        streams = sublayer(1, attend)
        streams = sublayer(2, lambda h: torch.relu(h @ W("mlp.up").T).square() @ W("mlp.down").T)
    return [(_rms(streams.sum(0)[:, -1]) * w["final.norm"].double()) @ w["head"].double().T] + states


def exact(case, seed):
    if case["path"] == "layer_f32":
        x, wq, wk, wv, wo = (t.double() for t in _layer_inputs(case, seed))
        T, rep = case["seq"], HEADS // KV_HEADS
        pos = torch.arange(T, device="cuda")
        q, k, v = _turn((x @ wq).view(T, HEADS, DIM), pos), _turn((x @ wk).view(T, KV_HEADS, DIM), pos), (x @ wv).view(T, KV_HEADS, DIM)
        if case["mode"] == "collapsed":       # one softmax over the scores summed over the heads
            wide = lambda t: t.repeat_interleave(rep, dim=1).reshape(T, 1, WIDTH)                 # noqa: E731
            q, k, v = q.reshape(T, 1, WIDTH), wide(k), wide(v)
        return _attention(q, k, v, DIM ** -0.5, _causal(T)).reshape(T, WIDTH) @ wo
    if case["path"] == "prefill_attn":
        q, k, v = _prefill_inputs(case, seed)
        pos, see = torch.arange(case["seq"], device="cuda"), _causal(case["seq"])
        one = lambda b: _attention(_turn(q[b].double(), pos), _turn(k[b].double(), pos), v[b].double(), DIM ** -0.5, see)      # noqa: E731
        return torch.stack([one(b) for b in range(case["batch"])])
    if case["path"] == "decode_attn":
        q, pool, table, lens = _decode_inputs(case, seed)
        out = []
        for b, n in enumerate(lens):
            rows = pool[table[b, :-(-n // PAGE_TOKENS)].long()].permute(2, 0, 3, 1, 4).reshape(2, -1, KV_HEADS, DIM)[:, :n]
            turned = _turn(q[b:b + 1].double(), torch.tensor([n - 1], device="cuda"))
            out.append(_attention(turned.view(1, HEADS, DIM), rows[0].double(), rows[1].double(), DIM ** -0.5,
                                  torch.ones((1, n), dtype=torch.bool, device="cuda"))[0])
        return torch.stack(out)
    gen = _generator(seed)
    w = _weights(case, gen)
    ids, token = _tokens(case, gen)
    if case["call"] == "step":
        ids = torch.cat([ids, token[:, None]], 1)
    return {"llama": _exact_llama, "soluzen": _exact_soluzen, "duponex": _exact_duponex}[case["path"]](case, w, ids)

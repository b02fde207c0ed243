"""The work that a program has this library do, as timed cases.

A case is one pass through the public interface: ``Engine.step`` over whole prompts, over single tokens in the middle of a
generation, or a whole generation.  The models have the sizes of this repository's configurations and benchmark: Gemma 2
2B and 9B, the two tiny Gemma 2 configurations, and Papusun at the benchmark's size s; all with random weights.

Kinds of pass:

* ``prompts``: open a slot per prompt, run all prompts in one step, take the logits of each last token, give the slots
  back.  What every request begins with; no token is decoded.
* ``decode``: one token more for each of a batch of sequences whose keys and values are in the cache, as in the middle of a
  generation.  The sequences are put back by that one token afterwards, so that a pass can be repeated: the next pass
  writes the same place of the cache again.  The captured step exists before the pass, as it does in a running program.
* ``answers``: open slots, run the prompts, then a number of given tokens one step at a time, as a program does that
  scores given continuations or replays a trace; logits of every step.
* ``generate``: ``brolm_b200.generate`` from prompts to new tokens, with the logits of every draw.

The lengths of a case's sequences are a function of the case alone; token ids and weights come from the seed.
"""
from __future__ import annotations

import math

import torch

import brolm_b200 as bb

DEV = "cuda:0"
F64 = torch.float64
TYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}

# --- the models ------------------------------------------------------------------------------------------------------
GEMMA_2B = dict(vocab_size=256000, hidden_size=2304, intermediate_size=9216, num_hidden_layers=26, num_attention_heads=8,
                num_key_value_heads=4, head_dim=256, rope_theta=10000.0, sliding_window=4096, attn_logit_softcapping=50.0,
                final_logit_softcapping=30.0, query_pre_attn_scalar=256.0, rms_norm_eps=1e-6)
MODELS = {
    "gemma2-2b": GEMMA_2B,
    "gemma2-9b": dict(GEMMA_2B, num_hidden_layers=42, hidden_size=3584, num_attention_heads=16, num_key_value_heads=8,
                      intermediate_size=14336),
    "gemma2-tiny-a": dict(vocab_size=256, hidden_size=64, intermediate_size=128, num_hidden_layers=2, num_attention_heads=4,
                          num_key_value_heads=2, head_dim=16, rope_theta=10000.0, sliding_window=8,
                          attn_logit_softcapping=50.0, final_logit_softcapping=30.0, query_pre_attn_scalar=16.0,
                          rms_norm_eps=1e-6),
    "gemma2-tiny-b": dict(vocab_size=512, hidden_size=96, intermediate_size=320, num_hidden_layers=3, num_attention_heads=6,
                          num_key_value_heads=1, head_dim=32, rope_theta=1000.0, sliding_window=16,
                          attn_logit_softcapping=20.0, final_logit_softcapping=15.0, query_pre_attn_scalar=24.0,
                          rms_norm_eps=1e-5),
}
_LEFT = dict(heads=16, kv_heads=4, dim=128, vdim=128, scale=128 ** -0.5, softcap=30.0,
             rot=dict(base=10000.0, dims=128, scaling=dict(factor=8.0, low=1.0, high=4.0, original=1024)))
_RIGHT = dict(heads=16, kv_heads=16, dim=128, vdim=128, conv=4)
_PAIR = dict(left=_LEFT, right=_RIGHT, left_scale=1.0, right_scale=1.0)
_LATENT = dict(heads=16, dim=64, rot_dim=64, vdim=64, q_rank=768, kv_rank=192, scale=128 ** -0.5, mask=dict(size=1024),
               rot=dict(base=10000.0, dims=64))
_MLP = dict(kind="dense", ff=4096)
MODELS["papusun-s"] = dict(
    architecture="Papusun", vocab=32768, width=2048, norm=dict(eps=1e-5), token_side=dict(dim=128), logit_scale=0.25,
    layers=[dict(type="parallel", mixer=_PAIR, mlp=_MLP), dict(type="latent_attention", mixer=_LATENT, mlp=_MLP),
            dict(type="parallel", mixer=_PAIR, mlp=_MLP),
            dict(type="latent_attention", mixer=dict(_LATENT, kv_from=1), mlp=_MLP)])


def is_gemma(case) -> bool:
    return case["model"].startswith("gemma2")


def vocab_of(case) -> int:
    m = MODELS[case["model"]]
    return m["vocab_size"] if is_gemma(case) else m["vocab"]


def _gemma_shapes(m: dict):
    """(name, shape, mean, deviation) of every tensor; the gains are stored around zero."""
    H, F, d = m["hidden_size"], m["intermediate_size"], m["head_dim"]
    q, kv = m["num_attention_heads"] * d, m["num_key_value_heads"] * d
    std = 0.05 if H == 96 else 0.02
    out = [("model.embed_tokens.weight", (m["vocab_size"], H), 0.0, std), ("model.norm.weight", (H,), 0.0, 0.1)]
    for i in range(m["num_hidden_layers"]):
        p = f"model.layers.{i}."
        for n, shape in (("self_attn.q_proj", (q, H)), ("self_attn.k_proj", (kv, H)), ("self_attn.v_proj", (kv, H)),
                         ("self_attn.o_proj", (H, q)), ("mlp.gate_proj", (F, H)), ("mlp.up_proj", (F, H)),
                         ("mlp.down_proj", (H, F))):
            out.append((p + n + ".weight", shape, 0.0, std))
        for n in ("input_layernorm", "post_attention_layernorm", "pre_feedforward_layernorm", "post_feedforward_layernorm"):
            out.append((p + n + ".weight", (H,), 0.0, 0.1))
    return out


def _papusun_shapes(c: dict):
    W, V, D = c["width"], c["vocab"], c["token_side"]["dim"]
    out = [("embed", (V, W), 0.0, 1.0), ("side.embed", (V, D * len(c["layers"])), 0.0, 1.0), ("final.norm", (W,), 1.0, 0.1),
           ("head", (V, W), 0.0, 0.02)]

    def mat(name, rows, cols):
        out.append((name, (rows, cols), 0.0, 0.02))

    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        out += [(p + "norm1", (W,), 1.0, 0.1), (p + "norm2", (W,), 1.0, 0.1), (p + "side.norm", (W,), 1.0, 0.1)]
        if layer["type"] == "parallel":
            a, r = m["left"], m["right"]
            for n, rows in (("q", a["heads"] * a["dim"]), ("k", a["kv_heads"] * a["dim"]), ("v", a["kv_heads"] * a["vdim"])):
                mat(p + "mix.left." + n, rows, W)
                out.append((p + f"mix.left.{n}.b", (rows,), 0.0, 0.02))
            mat(p + "mix.left.o", W, a["heads"] * a["vdim"])
            q, v = r["kv_heads"] * r["dim"], r["heads"] * r["vdim"]
            for n, rows in (("q", q), ("k", q), ("v", v)):
                mat(p + "mix.right." + n, rows, W)
                out.append((p + f"mix.right.{n}.conv", (rows, r["conv"]), 0.0, 0.5))
            for n in ("b", "a"):
                mat(p + "mix.right." + n, r["heads"], W)
            # exp(A_log) softplus(a + dt_bias) between about 0.005 and 0.5: memories of a few to a few hundred tokens
            out += [(p + "mix.right.A_log", (r["heads"],), 0.0, 0.5), (p + "mix.right.dt_bias", (r["heads"],), -3.0, 0.7),
                    (p + "mix.right.norm", (r["vdim"],), 1.0, 0.1)]
            mat(p + "mix.right.g", v, W)
            mat(p + "mix.right.o", W, v)
        else:
            H, dn, dr, dv, Q, R = (m[k] for k in ("heads", "dim", "rot_dim", "vdim", "q_rank", "kv_rank"))
            mat(p + "mix.dq", Q, W)
            out.append((p + "mix.dq.norm", (Q,), 1.0, 0.1))
            mat(p + "mix.uq", H * (dn + dr), Q)
            if m.get("kv_from") is None:
                mat(p + "mix.dkv", R + dr, W)
                out.append((p + "mix.dkv.norm", (R,), 1.0, 0.1))
            mat(p + "mix.uk", H * dn, R)
            mat(p + "mix.uv", H * dv, R)
            mat(p + "mix.g", H, W)
            mat(p + "mix.o", W, H * dv)
        F = layer["mlp"]["ff"]
        mat(p + "mlp.gate", F, W)
        mat(p + "mlp.up", F, W)
        mat(p + "mlp.down", W, F)
        mat(p + "side.gate", D, W)
        mat(p + "side.proj", W, D)
    return out


def _shapes(case):
    m = MODELS[case["model"]]
    return _gemma_shapes(m) if is_gemma(case) else _papusun_shapes(m)


def _weights(case, seed: int) -> dict:
    """The checkpoint's tensors, made on the device."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    dt = TYPES[case["dtype"]]
    return {n: torch.empty(s, dtype=dt, device=DEV).normal_(mean, std, generator=g) for n, s, mean, std in _shapes(case)}


def lengths_of(case) -> list:
    """Prompt lengths, spread evenly from ``shortest`` to ``longest`` and dealt out of order."""
    B, a, b = case["batch"], case["shortest"], case["longest"]
    if B == 1:
        return [b]
    even = [a + (b - a) * i // (B - 1) for i in range(B)]
    step = next(s for s in (7, 5, 3, 1) if math.gcd(s, B) == 1)
    return [even[i * step % B] for i in range(B)]


def _ids(case, seed: int) -> list:
    """Token ids per sequence: the prompt and the tokens that follow it."""
    g = torch.Generator().manual_seed(seed + 1)
    more = {"decode": 2, "answers": case.get("steps", 0)}.get(case["kind"], 0)
    return [torch.randint(0, vocab_of(case), (n + more,), generator=g).tolist() for n in lengths_of(case)]


def _case(name, kind, model, dtype, batch, shortest, longest, **more):
    c = dict(kind=kind, model=model, dtype=dtype, batch=batch, shortest=shortest, longest=longest, **more)
    return dict(c, name=name) if name else c


def listed() -> list:
    return [
        # the smallest call: a tiny float32 model answers four short prompts with drawn tokens; all launches and latency
        _case("tiny_generate", "generate", "gemma2-tiny-b", "float32", 4, 1, 40, steps=12, sampled=True),
        # the first token of a chat turn: one short prompt
        _case("prompt_37", "prompts", "gemma2-2b", "bfloat16", 1, 37, 37),
        # the first token of a question with a document: the benchmark's prompt
        _case("prompt_2048", "prompts", "gemma2-2b", "bfloat16", 1, 2048, 2048),
        # a batch of requests of unequal lengths that arrive together
        _case("prompts_mixed", "prompts", "gemma2-2b", "bfloat16", 12, 103, 2615),
        # one user's generation, the benchmark's shortest context
        _case("decode_b1", "decode", "gemma2-2b", "bfloat16", 1, 1280, 1280),
        # the benchmark's headline: eight long sequences
        _case("decode_b8_long", "decode", "gemma2-2b", "bfloat16", 8, 8190, 8190),
        # a full batch at the benchmark's shorter context
        _case("decode_b64", "decode", "gemma2-2b", "bfloat16", 64, 1280, 1280),
        # the larger model with sequences of very unequal lengths, some beyond the sliding window
        _case("decode_9b_ragged", "decode", "gemma2-9b", "bfloat16", 16, 128, 6144),
        # the true float32 path over a prompt, as used to check a checkpoint
        _case("f32_prompt_300", "prompts", "gemma2-2b", "float32", 1, 300, 300),
        # the float32 path's decode step
        _case("f32_decode", "decode", "gemma2-2b", "float32", 3, 150, 420),
        # another architecture on the same parts: delta rule beside attention, latent attention, a side input per token
        _case("papusun_prompt", "prompts", "papusun-s", "bfloat16", 1, 2048, 2048),
        # the same model over short prompts and given continuations, where decode steps dominate
        _case("papusun_answers", "answers", "papusun-s", "bfloat16", 8, 61, 389, steps=24),
    ]


def _spread(rng, low: int, high: int) -> int:
    """Spread over the logarithm, odd values as likely as even ones."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng) -> dict:
    what = rng.choice(["generate", "prompts", "prompts", "decode", "decode", "decode", "f32_prompts", "f32_decode",
                       "papusun_prompts", "papusun_answers"])
    if what == "generate":
        model = rng.choice(["gemma2-tiny-a", "gemma2-tiny-b"])
        longest = _spread(rng, 4, 48 if model == "gemma2-tiny-a" else 100)
        return _case(None, "generate", model, "float32", rng.randint(1, 8), rng.randint(1, longest), longest,
                     steps=rng.randint(4, 16), sampled=rng.random() < 0.5)
    if what in ("prompts", "papusun_prompts"):
        most, total = (6144, 16000) if what == "prompts" else (4096, 4096)
        longest = _spread(rng, 5, most)
        batch = rng.randint(1, max(1, min(12, total // longest)))
        return _case(None, "prompts", "gemma2-2b" if what == "prompts" else "papusun-s", "bfloat16", batch,
                     rng.randint(1 + longest // 8, longest), longest)
    if what == "f32_prompts":
        longest = _spread(rng, 5, 300)
        batch = rng.randint(1, max(1, min(4, 300 // longest)))
        return _case(None, "prompts", "gemma2-2b", "float32", batch, rng.randint(1 + longest // 8, longest), longest)
    if what == "f32_decode":
        longest = _spread(rng, 20, 1024)
        return _case(None, "decode", "gemma2-2b", "float32", _spread(rng, 1, 8), rng.randint(1 + longest // 8, longest), longest)
    if what == "papusun_answers":
        longest = _spread(rng, 20, 700)
        return _case(None, "answers", "papusun-s", "bfloat16", _spread(rng, 1, 16), rng.randint(1 + longest // 8, longest),
                     longest, steps=rng.randint(8, 24))
    longest = _spread(rng, 60, 8190)
    batch = _spread(rng, 1, min(64, 8 * 8190 // longest))
    # half of the batches in step (equal lengths), the others ragged
    shortest = longest if rng.random() < 0.5 else rng.randint(1 + longest // 40, longest)
    model = "gemma2-9b" if batch * longest <= 16 * 3000 and rng.random() < 0.25 else "gemma2-2b"
    return _case(None, "decode", model, "bfloat16", batch, shortest, longest)


# --- what a program has in hand, and one pass ------------------------------------------------------------------------
class _Keeping(bb.Sampler):
    """The library's sampler for a program that keeps the logits it drew from."""

    def __init__(self, params):
        super().__init__(params)
        self.kept = []

    def __call__(self, logits, streams, counter):
        self.kept.append(logits.clone())
        return super().__call__(logits, streams, counter)


def _sampling(case):
    if case["sampled"]:
        return bb.SamplingParams(temperature=0.8, top_k=40, top_p=0.95, seed=7)
    return bb.SamplingParams(temperature=0.0)


def prepare(case, seed: int) -> dict:
    c = MODELS[case["model"]]
    cfg = bb.Gemma2Config(**c) if is_gemma(case) else bb.PapusunConfig.from_dict(c)
    model = bb.Model(cfg, dtype=case["dtype"], device=DEV).load_weights(_weights(case, seed))
    seqs, lengths = _ids(case, seed), lengths_of(case)
    longest = max(len(s) for s in seqs) + case.get("steps", 0) + 1
    room = sum((len(s) + case.get("steps", 0) + 1 + 63) // 64 * 64 for s in seqs)
    engine = bb.Engine(model, max_tokens=room, max_slots=len(seqs), max_seq_len=longest)
    state = dict(case=case, engine=engine, seqs=seqs, lengths=lengths)
    if case["kind"] == "decode":
        state["slots"] = slots = engine.open(len(seqs))
        engine.step(slots, [s[:n] for s, n in zip(seqs, lengths)])
        engine.step(slots, [[s[n]] for s, n in zip(seqs, lengths)])       # the step before the pass
        state["held"] = {s: n + 1 for s, n in zip(slots, lengths)}
        state["next"] = [[s[n + 1]] for s, n in zip(seqs, lengths)]
    elif case["kind"] == "generate":
        state["opts"] = bb.GenerateOptions(max_new_tokens=case["steps"], sampling=_sampling(case), stop_on_eos=False)
        bb.generate(engine, seqs, eos_id=-1, opts=state["opts"])          # a program that has answered before
    elif case["kind"] == "answers":
        run(state)                                                         # likewise
    return state


def run(state):
    case, engine, seqs = state["case"], state["engine"], state["seqs"]
    if case["kind"] == "decode":
        logits = engine.step(state["slots"], state["next"])
        engine.cache.commit(state["held"])
        return {"logits": logits}
    if case["kind"] == "generate":
        sampler = _Keeping(state["opts"].sampling)
        ids = bb.generate(engine, seqs, eos_id=-1, opts=state["opts"], sampler=sampler)
        return {"ids": [x for r in ids for x in r], "logits": sampler.kept}
    lengths = state["lengths"]
    slots = engine.open(len(seqs))
    logits = engine.step(slots, [s[:n] for s, n in zip(seqs, lengths)])
    if case["kind"] == "prompts":
        engine.close(slots)
        return {"logits": logits}
    kept = [logits]
    for i in range(case["steps"]):
        kept.append(engine.step(slots, [[s[n + i]] for s, n in zip(seqs, lengths)]).clone())
    engine.close(slots)
    return {"logits": kept}


# --- what a pass cannot do without -----------------------------------------------------------------------------------
def _layers(case):
    """Per layer: (weights used by every token, visible keys' limit or None, numbers of a cached token that is read,
    operations per (query, key) pair, numbers of a state that is read and written)."""
    m = MODELS[case["model"]]
    if is_gemma(case):
        H, F, d = m["hidden_size"], m["intermediate_size"], m["head_dim"]
        q, kv = m["num_attention_heads"] * d, m["num_key_value_heads"] * d
        w = H * (q + 2 * kv) + q * H + 3 * F * H
        return [(w, m["sliding_window"] if i % 2 == 0 else None, 2 * kv, 4 * q, 0) for i in range(m["num_hidden_layers"])]
    out = []
    W, D = m["width"], m["token_side"]["dim"]
    for layer in m["layers"]:
        x, F = layer["mixer"], layer["mlp"]["ff"]
        w = 3 * F * W + 2 * D * W
        if layer["type"] == "parallel":
            a, r = x["left"], x["right"]
            q, kv, v = a["heads"] * a["dim"], a["kv_heads"] * (a["dim"] + a["vdim"]), r["heads"] * r["vdim"]
            w += W * (q + kv) + a["heads"] * a["vdim"] * W + W * (2 * r["kv_heads"] * r["dim"] + v + 2 * r["heads"]) + 2 * W * v
            out.append((w, None, kv, 2 * a["heads"] * (a["dim"] + a["vdim"]), r["heads"] * r["dim"] * r["vdim"]))
        else:
            h, dn, dr, dv, Q, R = (x[k] for k in ("heads", "dim", "rot_dim", "vdim", "q_rank", "kv_rank"))
            own = x.get("kv_from") is None
            w += W * Q + Q * h * (dn + dr) + (W * (R + dr) if own else 0) + R * h * (dn + dv) + W * h + h * dv * W
            out.append((w, x["mask"]["size"], R + dr, 2 * h * (dn + dr + dv), 0))
    return out


def work(case) -> dict:
    m, item = MODELS[case["model"]], 4 if case["dtype"] == "float32" else 2
    layers = _layers(case)
    width, vocab = (m["hidden_size"] if is_gemma(case) else m["width"]), vocab_of(case)
    params = sum(w for w, *_ in layers)
    head = vocab * width
    B, steps = case["batch"], case.get("steps", 0)
    total = dict(bytes=0.0, flops=0.0)

    def prompts(lengths):
        T = sum(lengths)
        total["bytes"] += (params + head + T * width) * item + B * vocab * 4
        total["flops"] += 2.0 * T * params + 2.0 * B * head
        for w, window, kv, ops, state in layers:
            total["bytes"] += T * kv * item + B * state * 4              # keys and values, or the state, written once
            total["flops"] += 4.0 * T * state                            # the state's update and its reading
            for n in lengths:
                full = min(n, window or n)
                total["flops"] += ops * (full * (full + 1) // 2 + (n - full) * full)

    def decode(held):                                                    # tokens in the cache before the step
        total["bytes"] += (params + head + B * width) * item + B * vocab * 4
        total["flops"] += 2.0 * B * (params + head)
        for w, window, kv, ops, state in layers:
            keys = sum(min(n + 1, window or n + 1) for n in held)
            total["bytes"] += keys * kv * item + 2 * B * state * 4
            total["flops"] += keys * ops + 4.0 * B * state

    lengths = lengths_of(case)
    if case["kind"] == "decode":
        decode([n + 1 for n in lengths])
    else:
        prompts(lengths)
        for i in range(steps - 1 if case["kind"] == "generate" else steps):
            decode([n + i for n in lengths])
    return total


def tolerance(case):
    # the differences that rounding in another order leaves after all layers, measured against ``exact``
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 5e-4}
    return {"rel": 0.03, "max": 0.3}


# --- the same in 64 bits, with plain torch alone ---------------------------------------------------------------------
def _capped(x, cap):
    return cap * torch.tanh(x / cap) if cap else x


def _attend(q, k, v, scale, cap, window):
    """One sequence: q (T, H, d), k (T, G, d), v (T, G, dv) -> (T, H, dv)."""
    T, H, _ = q.shape
    G = k.shape[1]
    out = torch.empty((T, H, v.shape[2]), dtype=F64, device=q.device)
    step = 1024
    for a in range(0, T, step):
        b = min(T, a + step)
        first = max(0, a - window + 1) if window else 0
        back = torch.arange(a, b, device=q.device)[:, None] - torch.arange(first, b, device=q.device)[None, :]
        hidden = (back < 0) | (back >= window) if window else back < 0
        for h in range(H):
            g = h // (H // G)
            s = _capped((q[a:b, h] @ k[first:b, g].T) * scale, cap).masked_fill_(hidden, float("-inf"))
            out[a:b, h] = torch.softmax(s, dim=-1) @ v[first:b, g]
    return out


def _turn(x, freq, interleaved):
    """Rotate the pairs of every head of x (T, heads, d) by position times frequency."""
    n = freq.numel()
    ang = torch.arange(x.shape[0], dtype=F64, device=x.device)[:, None] * freq
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    out = x.clone()
    a, b = (slice(0, 2 * n, 2), slice(1, 2 * n, 2)) if interleaved else (slice(0, n), slice(n, 2 * n))
    out[..., a], out[..., b] = x[..., a] * c - x[..., b] * s, x[..., a] * s + x[..., b] * c
    return out


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _pieces(fn, x, rows=8192):
    return torch.cat([fn(x[i:i + rows]) for i in range(0, x.shape[0], rows)])


def _gemma_hidden(m, w, seqs):
    """The rows after the final norm of whole sequences, one tensor per sequence."""
    H, d, nq, nkv = m["hidden_size"], m["head_dim"], m["num_attention_heads"], m["num_key_value_heads"]
    eps, sizes = m["rms_norm_eps"], [len(s) for s in seqs]
    flat = torch.tensor([t for s in seqs for t in s], device=DEV)
    h = w["model.embed_tokens.weight"][flat].double() * float(torch.tensor(float(H)).sqrt())
    freq = m["rope_theta"] ** (-2.0 * torch.arange(d // 2, dtype=F64, device=DEV) / d)
    for i in range(m["num_hidden_layers"]):
        t = {k[len(f"model.layers.{i}."):]: v.double() for k, v in w.items() if k.startswith(f"model.layers.{i}.")}

        def norm(x, name):
            return _rms(x, eps) * (1.0 + t[name + ".weight"])

        x = norm(h, "input_layernorm")
        q, k, v = ((x @ t[f"self_attn.{n}_proj.weight"].T) for n in "qkv")
        rows = []
        for qs, ks, vs in zip(q.split(sizes), k.split(sizes), v.split(sizes)):
            n = qs.shape[0]
            rows.append(_attend(_turn(qs.view(n, nq, d), freq, False), _turn(ks.view(n, nkv, d), freq, False),
                                vs.view(n, nkv, d), m["query_pre_attn_scalar"] ** -0.5, m["attn_logit_softcapping"],
                                m["sliding_window"] if i % 2 == 0 else 0).reshape(n, nq * d))
        h = h + norm(torch.cat(rows) @ t["self_attn.o_proj.weight"].T, "post_attention_layernorm")
        x = norm(h, "pre_feedforward_layernorm")
        y = _pieces(lambda z: (_gelu(z @ t["mlp.gate_proj.weight"].T) * (z @ t["mlp.up_proj.weight"].T))
                    @ t["mlp.down_proj.weight"].T, x)
        h = h + norm(y, "post_feedforward_layernorm")
    return (_rms(h, eps) * (1.0 + w["model.norm.weight"].double())).split(sizes)


def _gemma_head(m, w, rows):
    table = w["model.embed_tokens.weight"]
    out = [rows @ table[i:i + 32768].double().T for i in range(0, table.shape[0], 32768)]
    return _capped(torch.cat(out, dim=1), m["final_logit_softcapping"])


def _wavelengths(rot):
    """Angle per position of each pair, stretched by wavelength where the rotation says so."""
    out = []
    for i in range(rot["dims"] // 2):
        f = rot["base"] ** (-2.0 * i / rot["dims"])
        sc = rot.get("scaling")
        if sc:
            turn = 2.0 * math.pi / f
            keep = min(1.0, max(0.0, (sc["original"] / turn - sc["low"]) / (sc["high"] - sc["low"])))
            f = keep * f + (1.0 - keep) * f / sc["factor"]
        out.append(f)
    return torch.tensor(out, dtype=F64, device=DEV)


def _papusun_delta(n, t, r, eps):
    T, H, G, d, dv = n.shape[0], r["heads"], r["kv_heads"], r["dim"], r["vdim"]
    silu = torch.nn.functional.silu

    def conv(name):
        u, taps = n @ t[name].T, t[name + ".conv"]
        u = torch.cat([torch.zeros((taps.shape[1] - 1, u.shape[1]), dtype=F64, device=DEV), u])
        return silu(sum(u[j:j + T] * taps[:, j] for j in range(taps.shape[1])))

    def unit(x):
        return x * torch.rsqrt((x * x).sum(dim=-1, keepdim=True) + 1e-6)

    own = torch.arange(H, device=DEV) // (H // G)
    q, k = (unit(conv(name).view(T, G, d))[:, own] for name in "qk")
    q, v, beta = q * d ** -0.5, conv("v").view(T, H, dv), torch.sigmoid(n @ t["b"].T)
    decay = torch.exp(-torch.exp(t["A_log"]) * torch.nn.functional.softplus(n @ t["a"].T + t["dt_bias"], threshold=100.0))
    S, out = torch.zeros((H, d, dv), dtype=F64, device=DEV), torch.empty((T, H, dv), dtype=F64, device=DEV)
    for i in range(T):
        S = S * decay[i, :, None, None]
        u = beta[i, :, None] * (v[i] - torch.bmm(k[i, :, None], S)[:, 0])
        S = torch.baddbmm(S, k[i, :, :, None], u[:, None])
        out[i] = torch.bmm(q[i, :, None], S)[:, 0]
    o = _rms(out, eps) * t["norm"]
    return (o.reshape(T, H * dv) * silu(n @ t["g"].T)) @ t["o"].T


def _papusun_logits(c, w, ids, first):
    """Logits of one sequence from position ``first`` on."""
    eps, D, T = c["norm"]["eps"], c["token_side"]["dim"], len(ids)
    ids = torch.tensor(ids, device=DEV)
    x, latents = w["embed"][ids].double(), {}
    silu = torch.nn.functional.silu

    def norm(z, gain):
        z = z - z.mean(dim=-1, keepdim=True)
        return _rms(z, eps) * gain

    for i, layer in enumerate(c["layers"]):
        m = layer["mixer"]
        t = {k[len(f"l{i}."):]: v.double() for k, v in w.items() if k.startswith(f"l{i}.")}
        n = norm(x, t["norm1"])
        if layer["type"] == "parallel":
            a = m["left"]
            s = {k[len("mix.left."):]: v for k, v in t.items() if k.startswith("mix.left.")}
            f = _wavelengths(a["rot"])
            q, k, v = (n @ s[z].T + s[z + ".b"] for z in "qkv")
            o = _attend(_turn(q.view(T, a["heads"], -1), f, True), _turn(k.view(T, a["kv_heads"], -1), f, True),
                        v.view(T, a["kv_heads"], -1), a["scale"], a["softcap"], 0)
            y = m["left_scale"] * (o.reshape(T, -1) @ s["o"].T)
            right = {k[len("mix.right."):]: v for k, v in t.items() if k.startswith("mix.right.")}
            y = y + m["right_scale"] * _papusun_delta(n, right, m["right"], eps)
        else:
            H, dn, dr, R = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
            f = _wavelengths(m["rot"])
            q = ((_rms(n @ t["mix.dq"].T, eps) * t["mix.dq.norm"]) @ t["mix.uq"].T).view(T, H, dn + dr)
            q = torch.cat([q[..., :dn], _turn(q[..., dn:], f, True)], dim=-1)
            if m.get("kv_from") is None:
                row = n @ t["mix.dkv"].T
                latents[i] = (_rms(row[:, :R], eps) * t["mix.dkv.norm"], _turn(row[:, None, R:], f, True))
            lat, shared = latents[m.get("kv_from") if m.get("kv_from") is not None else i]
            k = torch.cat([(lat @ t["mix.uk"].T).view(T, H, dn), shared.expand(T, H, dr)], dim=-1)
            o = _attend(q, k, (lat @ t["mix.uv"].T).view(T, H, -1), m["scale"], 0.0, m["mask"]["size"])
            y = (o * torch.sigmoid(n @ t["mix.g"].T)[:, :, None]).reshape(T, -1) @ t["mix.o"].T
        x = x + y
        n = norm(x, t["norm2"])
        x = x + (silu(n @ t["mlp.gate"].T) * (n @ t["mlp.up"].T)) @ t["mlp.down"].T
        e = w["side.embed"][ids][:, i * D:(i + 1) * D].double()
        x = x + _rms((_gelu(x @ t["side.gate"].T) * e) @ t["side.proj"].T, eps) * t["side.norm"]
    return (norm(x[first:], w["final.norm"].double()) @ w["head"].double().T) * c["logit_scale"]


def exact(case, seed: int):
    m = MODELS[case["model"]]
    if case["kind"] == "generate" and case["sampled"]:
        return None                                   # the draws hang on the library's own random numbers
    if 2.0 * sum(lengths_of(case)) * sum(w for w, *_ in _layers(case)) > 4e14:
        return None                                   # too long in 64 bits
    w, seqs = _weights(case, seed), _ids(case, seed)
    if not is_gemma(case):
        steps = case.get("steps", 0)
        rows = [_papusun_logits(m, w, s, n - 1) for s, n in zip(seqs, lengths_of(case))]
        kept = [torch.stack([r[i] for r in rows]) for i in range(steps + 1)]
        return {"logits": kept if case["kind"] == "answers" else kept[0]}
    if case["kind"] != "generate":
        last = torch.stack([h[-1] for h in _gemma_hidden(m, w, seqs)])
        return {"logits": _gemma_head(m, w, last)}
    grown, kept = [list(s) for s in seqs], []
    for _ in range(case["steps"]):
        kept.append(_gemma_head(m, w, torch.stack([h[-1] for h in _gemma_hidden(m, w, grown)])))
        for s, t in zip(grown, kept[-1].argmax(dim=1).tolist()):
            s.append(t)
    return {"ids": [t for s, n in zip(grown, lengths_of(case)) for t in s[n:]], "logits": kept}

"""Measured cases: what programs that use xotorch_b200 have it do, over the range they use it in.

Two kinds of case, one per native engine:

  llama    a shard of a Llama-style decoder behind `NativeShard` — a middle shard whose hidden state stays on the device
           (`forward_device`, one call per shard and step of a peer ring), or a whole model called with token ids that returns
           logits (`forward`).  `pos` tokens are in the cache already, `rows` new ones come in one call.
  layered  a model given as a list of layers behind `LayeredShard`.  A pass serves `requests` requests from their first token on:
           prompts (whole, or in portions of `portion` rows), then `steps` more tokens each, one per step, given in advance as a
           token trace gives them.  Request r joins at step r * stagger.  Every step returns the logits of each request's last row.

Weights and inputs are random (no checkpoints are to be had), scaled so that every sublayer adds to the stream what the stream
holds, and the experts' router knows its tokens the way a trained one does (a token has experts well ahead of the others)."""
import math

import numpy as np
import torch

DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64

# ---- sizes: the model shapes of xotorch_b200/synth.py and xotorch_b200/bench_layered.py ----------------------------------------
LLAMA = {
  "1b": dict(dim=2048, ffn=8192, heads=32, kv_heads=8, head_dim=64, vocab=128256, scaled=True),
  "8b": dict(dim=4096, ffn=14336, heads=32, kv_heads=8, head_dim=128, vocab=128256, scaled=False),
}
ROPE_THETA, ROPE_SCALING = 500000.0, {"factor": 32.0, "high_freq_factor": 4.0, "low_freq_factor": 1.0, "original_max_position_embeddings": 8192,
                                      "rope_type": "llama3"}
LLAMA_EPS = 1e-5

LAYERED = {
  "small": dict(width=1024, ff=4096, heads=8, dim=64, rot_dim=32, vdim=64, kv_rank=256, q_rank=384, gheads=16, gkv=4, gdim=64, dheads=16, dkv=8, ddim=64),
  "medium": dict(width=2048, ff=8192, heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=512, q_rank=768, gheads=16, gkv=4, gdim=128, dheads=32, dkv=16, ddim=64),
  "large": dict(width=4096, ff=14336, heads=32, dim=128, rot_dim=64, vdim=128, kv_rank=512, q_rank=1536, gheads=32, gkv=8, gdim=128, dheads=32, dkv=16, ddim=128),
}
VOCAB, WINDOW, DECAY_RANK, NORM_GROUPS, EXPERTS, TOP, GROUPS, KEEP, TAPS, SOFTCAP = 32000, 1024, 64, 4, 16, 4, 8, 4, 4, 30.0
LAYERED_EPS, POSITIONS = {"Zokuvik": 1e-6, "Bufulorn": 1e-5}, 8192


def _llama(name, size, rows, pos=0, layers=2, dtype="bfloat16", whole=False):
  return {"name": name, "kind": "llama", "size": size, "dtype": dtype, "layers": layers, "pos": pos, "rows": rows, "whole": whole}


def _layered(name, family, size, layers, requests=1, prompt_min=1, prompt_max=1, steps=0, portion=0, stagger=0, dtype="bfloat16"):
  return {"name": name, "kind": "layered", "family": family, "size": size, "layers": layers, "dtype": dtype, "requests": requests, "prompt_min": prompt_min,
          "prompt_max": prompt_max, "steps": steps, "portion": portion, "stagger": stagger}


ZOKUVIK, BUFULORN = "latent,window,delta", "delta,attention+moe,borrow"


def listed():
  return [
    # one decoded token of a small model through the host call: ids in, logits out — what a single-GPU chat program does per token
    _llama("llama-1b-token", "1b", 1, pos=255, whole=True),
    # one decoded token on a middle shard of a peer ring: the hidden state comes from the neighbour and goes on, all on the device
    _llama("llama-8b-token", "8b", 1, pos=1500),
    # the next turn of a chat: a handful of new tokens behind a cached conversation
    _llama("llama-8b-turn", "8b", 6, pos=300),
    # a short prompt (the length of the headline benchmark's) on one shard
    _llama("llama-8b-prompt", "8b", 128),
    # a long document on one shard in the other 16-bit type, an odd number of tokens
    _llama("llama-8b-f16-document", "8b", 2701, dtype="float16"),
    # a prompt of a latent-attention / delta-rule model at the layer sizes of a real one
    _layered("zokuvik-large-prompt", "Zokuvik", "large", ZOKUVIK, 1, 1024, 1024),
    # one user's chat with a small model: a short prompt, then token after token
    _layered("zokuvik-small-chat", "Zokuvik", "small", ZOKUVIK, 1, 37, 37, steps=24),
    # sixteen requests decoded together, as a server under load runs them
    _layered("zokuvik-large-batch", "Zokuvik", "large", ZOKUVIK, 16, 6, 30, steps=12),
    # the all-32-bit mode: checks and small research models
    _layered("zokuvik-small-f32", "Zokuvik", "small", ZOKUVIK, 2, 20, 51, steps=8, dtype="float32"),
    # a long document for a model of gated delta rule, grouped-query attention and experts
    _layered("bufulorn-medium-document", "Bufulorn", "medium", BUFULORN, 1, 3500, 3500),
    # eight requests decoded together, with experts
    _layered("bufulorn-medium-batch", "Bufulorn", "medium", BUFULORN, 8, 9, 41, steps=16),
    # requests that arrive one after the other: prompts read in portions beside requests that decode already
    _layered("bufulorn-medium-arrivals", "Bufulorn", "medium", BUFULORN, 5, 70, 230, steps=6, portion=64, stagger=3),
  ]


def _spread(rng, lo, hi):
  """an integer of [lo, hi], spread over its logarithm"""
  return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))))))


def _cost(c):
  w = work(c)
  return w["bytes"] / 6.5e12 + w["flops"] / 1.6e15


def draw(rng):
  most = max(_cost(c) for c in listed())
  while True:
    c = _draw(rng)
    if _cost(c) <= most:
      return c


def _draw(rng):
  if rng.random() < 0.4:
    size = rng.choice(["1b", "8b"])
    rows = 1 if rng.random() < 0.3 else _spread(rng, 2, 2600)
    pos = 0 if rng.random() < 0.3 else _spread(rng, 1, 2600)
    c = _llama("", size, rows, min(pos, 2701 - rows) if rows > 1 else pos, layers=rng.choice([1, 2]), dtype=rng.choice(["bfloat16", "bfloat16", "float16"]),
               whole=size == "1b" and rng.random() < 0.4)
  else:
    family = rng.choice(["Zokuvik", "Bufulorn"])
    size = rng.choice(["small", "medium", "medium", "large"] if family == "Zokuvik" else ["small", "medium", "medium"])
    pool = ["latent", "window", "delta"] if family == "Zokuvik" else ["delta", "attention", "delta+moe", "attention+moe"]
    layers = [rng.choice(pool) for _ in range(rng.choice([1, 2, 3]))]
    if family == "Bufulorn" and len(layers) < 3 and layers[-1].startswith("attention") and rng.random() < 0.5:
      layers.append("borrow")
    f32 = size == "small" and rng.random() < 0.3
    how = rng.choice(["prompt", "decode", "decode", "arrivals"])
    if how == "prompt":
      n = _spread(rng, 3, 400 if f32 else 3400)
      requests = rng.choice([1, 1, 2]) if n < 1500 else 1
      c = _layered("", family, size, ",".join(layers), requests, max(1, n - rng.randrange(0, 1 + n // 3)), n, steps=rng.choice([0, 1]), dtype="float32" if f32 else "bfloat16")
    elif how == "decode":
      lo = rng.randrange(1, 20)
      c = _layered("", family, size, ",".join(layers), _spread(rng, 1, 4 if f32 else 24), lo, lo + rng.randrange(0, 40), steps=rng.randrange(3, 13),
                   dtype="float32" if f32 else "bfloat16")
    else:
      lo = rng.randrange(20, 120)
      c = _layered("", family, size, ",".join(layers), rng.randrange(2, 6), lo, lo + rng.randrange(0, 120), steps=rng.randrange(2, 7), portion=rng.choice([16, 50, 64, 128]),
                   stagger=rng.randrange(1, 5), dtype="float32" if f32 else "bfloat16")
  del c["name"]
  return c


# ---- what a case says of its requests -------------------------------------------------------------------------------------------
def _prompts(c):
  span = c["prompt_max"] - c["prompt_min"] + 1
  return [c["prompt_min"] + (r * 7919 + span - 1) % span for r in range(c["requests"])]


def _schedule(c):
  """[(slots, first rows, row counts)] of every step"""
  need = [p + c["steps"] for p in _prompts(c)]
  prompts, at, out, s = _prompts(c), [0] * c["requests"], [], 0
  while any(a < n for a, n in zip(at, need)):
    slots, first, count = [], [], []
    for r in range(c["requests"]):
      if s >= r * c["stagger"] and at[r] < need[r]:
        left = prompts[r] - at[r]
        n = 1 if left <= 0 else min(left, c["portion"]) if c["portion"] else left
        slots.append(r), first.append(at[r]), count.append(n)
        at[r] += n
    if slots:
      out.append((slots, first, count))
    s += 1
  return out


# ---- models: configurations and tensors -------------------------------------------------------------------------------------------
def _llama_config(c):
  z = LLAMA[c["size"]]
  n = c["layers"] if c["whole"] else c["layers"] + 2
  return {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "hidden_act": "silu", "hidden_size": z["dim"], "intermediate_size": z["ffn"],
          "num_hidden_layers": n, "num_attention_heads": z["heads"], "num_key_value_heads": z["kv_heads"], "head_dim": z["head_dim"], "vocab_size": z["vocab"],
          "rms_norm_eps": LLAMA_EPS, "rope_theta": ROPE_THETA, "rope_scaling": dict(ROPE_SCALING) if z["scaled"] else None, "max_position_embeddings": 131072,
          "tie_word_embeddings": True, "torch_dtype": c["dtype"], "attention_bias": False}


def _llama_specs(c):
  """(name, shape, mean, standard deviation) of the shard's tensors"""
  z = LLAMA[c["size"]]
  D, F, q, kv = z["dim"], z["ffn"], z["heads"] * z["head_dim"], z["kv_heads"] * z["head_dim"]
  out = [("model.embed_tokens.weight", (z["vocab"], D), 0.0, 1.0), ("model.norm.weight", (D,), 1.0, 0.1)] if c["whole"] else []
  for i in range(c["layers"]):
    p = f"model.layers.{i if c['whole'] else i + 1}."
    out += [(p + "input_layernorm.weight", (D,), 1.0, 0.1), (p + "post_attention_layernorm.weight", (D,), 1.0, 0.1)]
    out += [(p + n + ".weight", s, 0.0, s[1] ** -0.5) for n, s in (
      ("self_attn.q_proj", (q, D)), ("self_attn.k_proj", (kv, D)), ("self_attn.v_proj", (kv, D)), ("self_attn.o_proj", (D, q)),
      ("mlp.gate_proj", (F, D)), ("mlp.up_proj", (F, D)), ("mlp.down_proj", (D, F)))]
  return out


def _layered_config(c):
  z, fam, layers = LAYERED[c["size"]], c["family"], []
  for i, text in enumerate(c["layers"].split(",")):
    kind, _, ff = text.partition("+")
    if fam == "Zokuvik":
      if kind == "delta":
        layers.append({"type": "general_delta", "mixer": {"heads": z["dheads"], "dim": z["ddim"]}})
      else:
        m = {"heads": z["heads"], "dim": z["dim"], "rot_dim": z["rot_dim"], "vdim": z["vdim"], "kv_rank": z["kv_rank"],
             "rot": {"base": 10000.0, "dims": z["rot_dim"]}, "scale": float((z["dim"] + z["rot_dim"]) ** -0.5)}
        m.update({"q_rank": z["q_rank"]} if kind == "latent" else {"mask": {"size": WINDOW}})
        layers.append({"type": "latent_attention" if kind == "latent" else "latent_attention_2", "mixer": m})
    elif kind == "delta":
      layers.append({"type": "delta", "mixer": {"heads": z["dheads"], "kv_heads": z["dkv"], "dim": z["ddim"], "vdim": z["ddim"], "conv": TAPS}})
    else:
      m = {"heads": z["gheads"], "kv_heads": z["gkv"], "dim": z["gdim"], "vdim": z["gdim"], "scale": float(z["gdim"] ** -0.5), "softcap": SOFTCAP, "mask": {"size": WINDOW}}
      if kind == "borrow":
        m["kv_from"] = max(j for j in range(i) if layers[j]["type"] == "attention" and "kv_from" not in layers[j]["mixer"])
      layers.append({"type": "attention", "mixer": m})
    layers[-1]["mlp"] = {"kind": "moe", "router": {"experts": EXPERTS, "top": TOP, "groups": {"count": GROUPS, "keep": KEEP}}, "expert": {"ff": z["ff"] // 4}} if ff \
      else {"kind": "dense", "ff": z["ff"]}
  cfg = {"architecture": fam, "width": z["width"], "vocab": VOCAB, "norm": {"eps": LAYERED_EPS[fam]}, "layers": layers}
  cfg.update({"max_positions": POSITIONS} if fam == "Bufulorn" else {})
  if fam == "Zokuvik":
    cfg["norm"]["groups"] = NORM_GROUPS
  return cfg


def _layered_specs(c):
  """(name, shape, mean, standard deviation) of the model's tensors"""
  cfg = _layered_config(c)
  D, out = cfg["width"], []
  vec = lambda n, k, mean=0.0, dev=0.3: out.append((n, (k,), mean, dev))           # noqa: E731
  mat = lambda n, r, k, gain=1.0: out.append((n, (r, k), 0.0, gain * k ** -0.5))   # noqa: E731
  norm = lambda n, k: vec(n, k, 1.0, 0.1)                                          # noqa: E731
  out += [("embed", (VOCAB, D), 0.0, 1.0)]
  mat("head", VOCAB, D)
  norm("final.norm", D)
  zok = c["family"] == "Zokuvik"
  if not zok:
    out.append(("pos", (POSITIONS, D), 0.0, 0.3))
    vec("final.norm.b", D)
  for i, layer in enumerate(cfg["layers"]):
    p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
    for n in ("norm1", "norm2"):
      norm(p + n, D)
      norm(p + n + "b", D) if zok else vec(p + n + ".b", D)
    x = p + "mix."
    if layer["type"].startswith("latent"):
      H, dn, dr, dv, R = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
      if "q_rank" in m:
        mat(x + "dq", m["q_rank"], D), norm(x + "dq.norm", m["q_rank"]), mat(x + "uq", H * (dn + dr), m["q_rank"]), mat(x + "g", H, D)
      else:
        mat(x + "q", H * (dn + dr), D)
      mat(x + "dkv", R + dr, D), norm(x + "dkv.norm", R), mat(x + "uk", H * dn, R), mat(x + "uv", H * dv, R), mat(x + "o", D, H * dv)
    elif layer["type"] == "general_delta":
      n = m["heads"] * m["dim"]
      for t in ("r", "k", "v", "g", "a"):
        mat(x + t, n, D, 0.3 if t in "kv" else 1.0)
      vec(x + "a.b", n), vec(x + "w0", n), norm(x + "norm", n)
      mat(x + "w1", DECAY_RANK, D), mat(x + "w2", n, DECAY_RANK), mat(x + "o", D, n)
    elif layer["type"] == "delta":
      H, G, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
      for t, n in (("q", G * dk), ("k", G * dk), ("v", H * dv)):
        mat(x + t, n, D), mat(x + t + ".conv", n, TAPS)
      mat(x + "b", H, D), mat(x + "a", H, D), vec(x + "A_log", H, 0.0, 0.5), vec(x + "dt_bias", H, -2.0, 0.5), norm(x + "norm", dv)
      mat(x + "g", H * dv, D), mat(x + "o", D, H * dv)
    else:
      H, G, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
      mat(x + "q", H * dk, D), vec(x + "q.b", H * dk), norm(x + "q.norm", dk)
      if "kv_from" not in m:
        mat(x + "k", G * dk, D), vec(x + "k.b", G * dk), norm(x + "k.norm", dk), mat(x + "v", G * dv, D), vec(x + "v.b", G * dv)
      vec(x + "r1", H, 0.15, 0.03), vec(x + "r2", H, 1.0, 0.1), mat(x + "g", H * dv, D), mat(x + "o", D, H * dv)
    y = p + "mlp."
    if mlp["kind"] == "dense":
      mat(y + "up", mlp["ff"], D), mat(y + "down", D, mlp["ff"])
      if not zok:
        vec(y + "act", 2)
    else:
      mat(y + "router", EXPERTS, D, 0.05)
      for e in range(EXPERTS):
        f = mlp["expert"]["ff"]
        mat(y + f"e{e}.gate", f, D), mat(y + f"e{e}.up", f, D), mat(y + f"e{e}.down", D, f)
  return out


def _tensors(c, seed):
  """(name, 16-bit tensor) one after the other, made from the seed alone"""
  g = torch.Generator(device=DEV).manual_seed(int(seed) * 1000003 + 17)
  dt = torch.float16 if c["dtype"] == "float16" else torch.bfloat16
  specs = _llama_specs(c) if c["kind"] == "llama" else _layered_specs(c)
  D = (LLAMA if c["kind"] == "llama" else LAYERED)[c["size"]]["dim" if c["kind"] == "llama" else "width"]
  # every token belongs to one of EXPERTS kinds, told by a direction in its embedding; each kind has TOP experts of its own
  kinds = torch.randint(0, 2, (EXPERTS, D), generator=g, device=DEV).to(torch.float32) * 2 - 1
  for name, shape, mean, dev in specs:
    t = torch.randn(shape, generator=g, device=DEV, dtype=torch.float32).mul_(dev).add_(mean) if len(shape) == 1 or shape[1] <= TAPS else \
      torch.randn(shape, generator=g, device=DEV, dtype=dt).mul_(dev)
    if c["kind"] == "layered" and "+moe" in c["layers"]:
      if name == "embed":
        t.add_(kinds.to(dt)[torch.arange(VOCAB, device=DEV) % EXPERTS] * 1.5)
      elif name.endswith("router"):
        order = torch.rand(EXPERTS, EXPERTS, generator=g, device=DEV).argsort(dim=1)              # [kind, rank] -> expert
        fond = torch.cat([torch.linspace(3.0, 1.8, TOP), torch.linspace(0.0, -1.5, EXPERTS - TOP)]).to(DEV)
        strength = torch.zeros(EXPERTS, EXPERTS, device=DEV).scatter_(1, order, fond.repeat(EXPERTS, 1))   # [kind, expert]
        t = t.to(torch.float32) + strength.T @ kinds / D
    yield name, t.to(dt)


def _ids(c, seed, vocab, n):
  return np.random.default_rng([int(seed), 5]).integers(0, vocab, size=n).astype(np.int32)


def _hidden(c, seed):
  """the hidden state of every row a middle shard sees, cached ones first"""
  g = torch.Generator(device=DEV).manual_seed(int(seed) * 1000003 + 29)
  return torch.randn(c["pos"] + c["rows"], LLAMA[c["size"]]["dim"], generator=g, device=DEV).to(torch.float16 if c["dtype"] == "float16" else torch.bfloat16)


def _load(shard, c, seed):
  for name, t in _tensors(c, seed):
    shard.load_tensor(name, t.view(torch.int16).cpu().numpy())
  shard.check_loaded()


# ---- the case itself -----------------------------------------------------------------------------------------------------------------
def prepare(c, seed):
  if c["kind"] == "llama":
    from xotorch_b200.native import NativeShard
    shard = NativeShard(_llama_config(c), 0)
    shard.set_shard(*((0, c["layers"] - 1) if c["whole"] else (1, c["layers"])))
    _load(shard, c, seed)
    shard.begin_request(c["pos"] + c["rows"] + 1)
    if c["whole"]:
      ids = _ids(c, seed, LLAMA[c["size"]]["vocab"], c["pos"] + c["rows"]).reshape(1, -1)
      if c["pos"]:
        shard.forward(ids[:, :c["pos"]], 0)
      return {"case": c, "shard": shard, "ids": np.ascontiguousarray(ids[:, c["pos"]:])}
    hidden = _hidden(c, seed)
    out = torch.empty(max(c["pos"], c["rows"]), hidden.shape[1], dtype=hidden.dtype, device=DEV)
    torch.cuda.synchronize()
    if c["pos"]:
      shard.forward_device(None, hidden.data_ptr(), c["pos"], 0, out.data_ptr())
    return {"case": c, "shard": shard, "hidden": hidden[c["pos"]:].clone(), "out": out[:c["rows"]].clone()}
  from xotorch_b200.layered import LayeredShard
  shard = LayeredShard(_layered_config(c), 0, c["dtype"])
  shard.set_shard(0, len(c["layers"].split(",")) - 1, {n: s for n, s, _, _ in _layered_specs(c)})
  _load(shard, c, seed)
  need = [p + c["steps"] for p in _prompts(c)]
  shard.begin_pool(max(need) * c["requests"], c["requests"])
  tokens = _requests_tokens(c, seed)
  steps = [(slots, [tokens[r][a:a + n] for r, a, n in zip(slots, first, count)]) for slots, first, count in _schedule(c)]
  return {"case": c, "shard": shard, "steps": steps}


def _requests_tokens(c, seed):
  return [np.random.default_rng([int(seed), 7, r]).integers(0, VOCAB, size=p + c["steps"]).astype(np.int32) for r, p in enumerate(_prompts(c))]


def run(state):
  c, shard = state["case"], state["shard"]
  if c["kind"] == "llama":
    if c["whole"]:
      return shard.forward(state["ids"], c["pos"])
    shard.forward_device(None, state["hidden"].data_ptr(), c["rows"], c["pos"], state["out"].data_ptr())
    return state["out"]
  for slot in range(c["requests"]):
    shard.clear_request(slot)
  return [shard.step(slots, rows)[0] for slots, rows in state["steps"]]


def tolerance(c):
  # about four times the error of a pass against 64 bits (one evaluation's rounding: products' inputs, caches and, in a Llama shard, the
  # stream in 16 bits; the order of the sums in 32)
  if c["dtype"] == "float32":
    return {"rel": 8e-6}
  if c["kind"] == "llama":
    return {"rel": 0.02 if c["dtype"] == "bfloat16" else 0.0025}
  return {"rel": 0.02 if c["family"] == "Zokuvik" else 0.012}


# ---- the least work of a pass ----------------------------------------------------------------------------------------------------------
def work(c):
  if c["kind"] == "llama":
    z, n, L = LLAMA[c["size"]], c["rows"], c["layers"]
    q, kv = z["heads"] * z["head_dim"], z["kv_heads"] * z["head_dim"]
    weights = 2 * z["dim"] * q + 2 * z["dim"] * kv + 3 * z["dim"] * z["ffn"]
    keys = sum(c["pos"] + i + 1 for i in range(n))
    flops = L * (2 * weights * n + 4 * q * keys)
    bytes_ = L * (2 * weights + 4 * kv * (c["pos"] + n))
    if c["whole"]:
      head = z["vocab"] * z["dim"]
      return {"bytes": bytes_ + 2 * head + 2 * z["dim"] * n + 4 * z["vocab"], "flops": flops + 2 * head}
    return {"bytes": bytes_ + 4 * z["dim"] * n, "flops": flops}
  cfg, size = _layered_config(c), 4 if c["dtype"] == "float32" else 2
  D, specs = cfg["width"], {n: s for n, s, _, _ in _layered_specs(c)}
  count = lambda p: sum(int(np.prod(s)) for n, s in specs.items() if n.startswith(p))   # noqa: E731
  flops = bytes_ = 0.0
  for slots, first, counts in _schedule(c):
    rows = sum(counts)
    bytes_ += size * (VOCAB * D + rows * D) + 4 * VOCAB * len(slots)
    flops += 2.0 * VOCAB * D * len(slots)
    for i, layer in enumerate(cfg["layers"]):
      m, moe = layer["mixer"], layer["mlp"]["kind"] == "moe"
      mix, ff = count(f"l{i}.mix."), count(f"l{i}.mlp.")
      used = 1 - (1 - TOP / EXPERTS) ** min(rows, EXPERTS) if moe else 1.0         # each kind of token has experts of its own
      bytes_ += size * (mix + ff * used)
      flops += 2.0 * rows * (mix + (ff * TOP / EXPERTS if moe else ff))
      for a, n in zip(first, counts):
        if "delta" in layer["type"]:
          state = m["heads"] * m["dim"] * m.get("vdim", m["dim"])
          bytes_ += 8.0 * state
          flops += 6.0 * state * n
          continue
        span = m["mask"]["size"] if "mask" in m else 1 << 30
        latent = layer["type"].startswith("latent")
        if latent:
          seen = sum(min(a + j + 1, span) for j in range(n))
          row, per_key = m["kv_rank"] + m["rot_dim"], m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
          reach = min(a + n, span + n - 1)
        else:
          seen = sum((a + j) % span + 1 for j in range(n))
          row, per_key = m["kv_heads"] * (m["dim"] + m["vdim"]), m["heads"] * (m["dim"] + m["vdim"])
          reach = a + n - a // span * span
        bytes_ += size * row * reach
        flops += 2.0 * per_key * seen
  return {"bytes": bytes_, "flops": flops}


# ---- the same in plain 64-bit torch -----------------------------------------------------------------------------------------------------
def _rms(x, eps):
  return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _turn(x, first, second, freqs, pos):
  """the entries `first` and `second` (index lists) of the last axis of x [T, H, d] turned by pos * freqs"""
  ang = pos[:, None] * freqs[None, :]
  cos, sin, out = torch.cos(ang)[:, None], torch.sin(ang)[:, None], x.clone()
  out[..., first] = x[..., first] * cos - x[..., second] * sin
  out[..., second] = x[..., second] * cos + x[..., first] * sin
  return out


def _attend(q, k, v, scale, visible, change=None):
  """q [T, H, d], k [S, G, d], v [S, G, e]; visible [T, S]; change(scores, head) before the mask"""
  out = torch.empty(q.shape[0], q.shape[1], v.shape[2], dtype=F64, device=q.device)
  rep = q.shape[1] // k.shape[1]
  for h in range(q.shape[1]):
    s = q[:, h] @ k[:, h // rep].T * scale
    s = change(s, h) if change else s
    out[:, h] = torch.softmax(s.masked_fill(~visible, float("-inf")), -1) @ v[:, h // rep]
  return out


def _exact_llama(c, seed):
  z, W = LLAMA[c["size"]], dict(_tensors(c, seed))
  H, G, d, T, P = z["heads"], z["kv_heads"], z["head_dim"], c["pos"] + c["rows"], c["pos"]
  w = lambda n: W[n].to(F64)                                                       # noqa: E731
  if c["whole"]:
    x = W["model.embed_tokens.weight"][torch.from_numpy(_ids(c, seed, z["vocab"], T)).long().to(DEV)].to(F64)
  else:
    x = _hidden(c, seed).to(F64)
  i = torch.arange(d // 2, dtype=F64, device=DEV)
  freqs = ROPE_THETA ** (-2.0 * i / d)
  if z["scaled"]:
    s, wave = ROPE_SCALING, 2 * math.pi / freqs
    old = s["original_max_position_embeddings"]
    mix = (old / wave - s["low_freq_factor"]) / (s["high_freq_factor"] - s["low_freq_factor"])
    soft = (1 - mix) * freqs / s["factor"] + mix * freqs
    freqs = torch.where(wave < old / s["high_freq_factor"], freqs, torch.where(wave > old / s["low_freq_factor"], freqs / s["factor"], soft))
  pos, lo, hi = torch.arange(T, dtype=F64, device=DEV), list(range(d // 2)), list(range(d // 2, d))
  visible = torch.arange(T, device=DEV)[:, None] >= torch.arange(T, device=DEV)[None, :]
  for layer in range(c["layers"]):
    p = f"model.layers.{layer if c['whole'] else layer + 1}."
    h = _rms(x, LLAMA_EPS) * w(p + "input_layernorm.weight")
    q, k, v = ((h @ w(p + f"self_attn.{n}_proj.weight").T).reshape(T, -1, d) for n in "qkv")
    o = _attend(_turn(q, lo, hi, freqs, pos), _turn(k, lo, hi, freqs, pos), v, d ** -0.5, visible)
    x = x + o.reshape(T, H * d) @ w(p + "self_attn.o_proj.weight").T
    h = _rms(x, LLAMA_EPS) * w(p + "post_attention_layernorm.weight")
    a = torch.nn.functional.silu(h @ w(p + "mlp.gate_proj.weight").T) * (h @ w(p + "mlp.up_proj.weight").T)
    x = x + a @ w(p + "mlp.down_proj.weight").T
  if not c["whole"]:
    return x[P:]
  return ((_rms(x[-1:], LLAMA_EPS) * w("model.norm.weight")) @ w("model.embed_tokens.weight").T).cpu().numpy()


def _grouped(x, wt, eps):
  return _rms(x.reshape(x.shape[0], NORM_GROUPS, -1), eps).reshape(x.shape) * wt


def _layer_norm(x, wt, b, eps):
  x = x - x.mean(-1, keepdim=True)
  return _rms(x, eps) * wt + b


def _latent(h, w, m, eps):
  T, H, dn, dr, R = h.shape[0], m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
  rank = "q_rank" in m
  q = (_rms(h @ w("dq").T, eps) * w("dq.norm")) @ w("uq").T if rank else h @ w("q").T
  q, down = q.reshape(T, H, dn + dr), h @ w("dkv").T
  lat, kr = _rms(down[:, :R], eps) * w("dkv.norm"), down[:, R:].reshape(T, 1, dr)
  first = list(range(0, dr, 2)) if rank else list(range(dr // 2))
  second = list(range(1, dr, 2)) if rank else list(range(dr // 2, dr))
  freqs = m["rot"]["base"] ** (-2.0 * torch.arange(dr // 2, dtype=F64, device=h.device) / dr)
  pos = torch.arange(T, dtype=F64, device=h.device)
  q = torch.cat([q[..., :dn], _turn(q[..., dn:], first, second, freqs, pos)], -1)
  k = torch.cat([(lat @ w("uk").T).reshape(T, H, dn), _turn(kr, first, second, freqs, pos).expand(T, H, dr)], -1)
  far = torch.arange(T, device=h.device)[:, None] - torch.arange(T, device=h.device)[None, :]
  visible = (far >= 0) & (far < (m["mask"]["size"] if "mask" in m else 1 << 30))
  o = _attend(q, k, (lat @ w("uv").T).reshape(T, H, -1), m["scale"], visible)
  if rank:
    o = o * torch.sigmoid(h @ w("g").T)[:, :, None]
  return o.reshape(T, -1) @ w("o").T


def _general_delta(h, w, m, eps):
  T, H, d = h.shape[0], m["heads"], m["dim"]
  r, k, v = ((h @ w(n).T).reshape(T, H, d) for n in "rkv")
  keep = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ w("w1").T) @ w("w2").T + w("w0"))).reshape(T, H, d, 1)
  u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
  au = (torch.sigmoid(h @ w("a").T + w("a.b")).reshape(T, H, d) * u)[..., None]
  S, out = torch.zeros(H, d, d, dtype=F64, device=h.device), torch.empty(T, H, d, dtype=F64, device=h.device)
  for t in range(T):
    S = keep[t] * S - au[t] @ (u[t][:, None] @ S) + k[t][..., None] @ v[t][:, None]
    out[t] = (r[t][:, None] @ S)[:, 0]
  return ((_rms(out, eps).reshape(T, -1) * w("norm")) * torch.sigmoid(h @ w("g").T)) @ w("o").T


def _gated_delta(h, w, m, eps):
  T, H, G, dk = h.shape[0], m["heads"], m["kv_heads"], m["dim"]

  def filtered(n):
    x = h @ w(n).T
    past = torch.cat([torch.zeros(TAPS - 1, x.shape[1], dtype=F64, device=x.device), x])
    return torch.nn.functional.silu(sum(past[i:i + T] * w(n + ".conv")[:, i] for i in range(TAPS)))
  unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)            # noqa: E731
  q = (unit(filtered("q").reshape(T, G, dk)) * dk ** -0.5).repeat_interleave(H // G, 1)
  k = unit(filtered("k").reshape(T, G, dk)).repeat_interleave(H // G, 1)
  v, beta = filtered("v").reshape(T, H, -1), torch.sigmoid(h @ w("b").T)[..., None]
  keep = torch.exp(-torch.exp(w("A_log")) * torch.nn.functional.softplus(h @ w("a").T + w("dt_bias")))[..., None, None]
  S, out = torch.zeros(H, dk, v.shape[2], dtype=F64, device=h.device), torch.empty_like(v)
  for t in range(T):
    S = keep[t] * S
    S = S + k[t][..., None] @ (beta[t] * (v[t] - (k[t][:, None] @ S)[:, 0]))[:, None]
    out[t] = (q[t][:, None] @ S)[:, 0]
  return ((_rms(out, eps) * w("norm")).reshape(T, -1) * torch.nn.functional.silu(h @ w("g").T)) @ w("o").T


def _gqa(h, w, m, eps, kept, i):
  T, dk = h.shape[0], m["dim"]
  q = _rms((h @ w("q").T + w("q.b")).reshape(T, -1, dk), eps) * w("q.norm")
  if "kv_from" not in m:
    kept[i] = (_rms((h @ w("k").T + w("k.b")).reshape(T, -1, dk), eps) * w("k.norm"), (h @ w("v").T + w("v.b")).reshape(T, -1, m["vdim"]))
  k, v = kept[m.get("kv_from", i)]
  at = torch.arange(T, device=h.device)
  far = (at[:, None] - at[None, :]).clamp(min=0).to(F64)
  visible = (at[:, None] >= at[None, :]) & (at[:, None] // m["mask"]["size"] == at[None, :] // m["mask"]["size"])
  r1, r2 = w("r1"), w("r2")
  o = _attend(q, k, v, m["scale"], visible, lambda s, a: SOFTCAP * torch.tanh(s / SOFTCAP) - r1[a] * torch.log1p(r2[a] * far))
  return (o.reshape(T, -1) * torch.sigmoid(h @ w("g").T)) @ w("o").T


def _experts(h, w):
  s = torch.softmax(h @ w("router").T, -1)
  best = s.reshape(-1, GROUPS, EXPERTS // GROUPS).amax(-1)
  kept = torch.zeros_like(best, dtype=torch.bool).scatter_(1, best.topk(KEEP, -1).indices, True).repeat_interleave(EXPERTS // GROUPS, 1)
  chosen = s.masked_fill(~kept, -1.0).topk(TOP, -1).indices
  y = torch.zeros_like(h)
  for e in range(EXPERTS):
    rows = (chosen == e).any(-1).nonzero()[:, 0]
    if len(rows):
      x = h[rows]
      a = torch.nn.functional.silu(x @ w(f"e{e}.gate").T) * (x @ w(f"e{e}.up").T)
      y[rows] += s[rows, e][:, None] * (a @ w(f"e{e}.down").T)
  return y


def _exact_layered(cfg, W, tokens, zok):
  """the rows' final normed stream"""
  eps, kept = cfg["norm"]["eps"], {}
  x = W["embed"][torch.from_numpy(tokens).long().to(DEV)].to(F64)
  if not zok:
    x = x + W["pos"][:len(tokens)].to(F64)
  for i, layer in enumerate(cfg["layers"]):
    g = lambda n: W[f"l{i}.{n}"].to(F64)                                           # noqa: E731
    mix, mlp, m = (lambda n: g("mix." + n)), (lambda n: g("mlp." + n)), layer["mixer"]
    h = _grouped(x, g("norm1"), eps) if zok else x
    kind = layer["type"]
    y = _latent(h, mix, m, eps) if kind.startswith("latent") else _general_delta(h, mix, m, eps) if kind == "general_delta" else \
      _gated_delta(h, mix, m, eps) if kind == "delta" else _gqa(h, mix, m, eps, kept, i)
    x = x + (_grouped(y, g("norm1b"), eps) if zok else _layer_norm(y, g("norm1"), g("norm1.b"), eps))
    h = _grouped(x, g("norm2"), eps) if zok else x
    if layer["mlp"]["kind"] == "moe":
      y = _experts(h, mlp)
    else:
      u = h @ mlp("up").T
      if zok:
        a = torch.relu(u) ** 2
      else:
        p, q = torch.nn.functional.softplus(mlp("act"))
        a = torch.where(u > 0, p * u * u, (0.5 + q) * (torch.expm1(u.clamp(max=0.0)) - u)) + 0.5 * u
      y = a @ mlp("down").T
    x = x + (_grouped(y, g("norm2b"), eps) if zok else _layer_norm(y, g("norm2"), g("norm2.b"), eps))
  return _grouped(x, W["final.norm"].to(F64), eps) if zok else _layer_norm(x, W["final.norm"].to(F64), W["final.norm.b"].to(F64), eps)


def exact(c, seed):
  with torch.no_grad():
    if c["kind"] == "llama":
      return _exact_llama(c, seed)
    cfg, W = _layered_config(c), dict(_tensors(c, seed))
    rows = [_exact_layered(cfg, W, t, c["family"] == "Zokuvik") for t in _requests_tokens(c, seed)]
    head = W["head"].to(F64).T
    return [(torch.stack([rows[r][a + n - 1] for r, a, n in zip(slots, first, count)]) @ head).cpu().numpy() for slots, first, count in _schedule(c)]

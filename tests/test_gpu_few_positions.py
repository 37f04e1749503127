"""Calls of 2 .. 7 positions of a dense shard run as GEMMs: their attention keeps the weights as wide as the decode kernel's fp32, and a position reads
no key or value behind its own."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from xotorch_b200.synth import PRESETS, hf_config

N_A, N_B, OUT = 24, 36, 5                                          # keys of two kinds; the column of a head that holds the values


def middle_shard(name: str, load: bool):
  from xotorch_b200.native import NativeShard
  shape = PRESETS[name]
  eng = NativeShard(hf_config(shape), 0)
  eng.set_shard(1, 1)
  if load:
    D, F, q, kv, hd = shape.dim, shape.ffn, shape.n_heads * shape.head_dim, shape.n_kv_heads * shape.head_dim, shape.head_dim
    slow = hd - 1                                                  # the rotation's slowest plane: cos within 1e-8 of 1 over these positions
    w = {n: torch.zeros(s) for n, s in (("self_attn.q_proj", (q, D)), ("self_attn.k_proj", (kv, D)), ("self_attn.v_proj", (kv, D)), ("mlp.gate_proj", (F, D)),
                                        ("mlp.up_proj", (F, D)), ("mlp.down_proj", (D, F)))}
    w["self_attn.q_proj"][slow::hd, 1] = 0.125
    w["self_attn.k_proj"][slow::hd, 2] = 0.1015625
    w["self_attn.v_proj"][OUT::hd, 3] = 0.0625
    w["self_attn.o_proj"] = torch.eye(D, q)
    w["input_layernorm"] = w["post_attention_layernorm"] = torch.ones(D)
    dt = torch.float16 if shape.dtype == "float16" else torch.bfloat16
    for n, t in w.items():
      eng.load_tensor(f"model.layers.1.{n}.weight", t.to(dt).contiguous().view(torch.int16).numpy())
    eng.check_loaded()
  else:
    eng.init_synthetic(11)
  return eng, shape


def run(eng, h, pos0):
  out = torch.empty_like(h)
  torch.cuda.synchronize()
  eng.forward_device(None, h.data_ptr(), h.shape[0], pos0, out.data_ptr())
  return out.float().cpu().numpy()


@pytest.mark.parametrize("name", ["tiny-llama-hd64", "tiny-llama-hd64-f16"])
@pytest.mark.parametrize("n", [2, 5, 7])
def test_attention_weights_stay_in_32_bits(name, n):
  """24 keys of weight 1 and value v, 36 of weight about 2/3 and value -v: they cancel but for some 4e-4, so an error of the weights shows undivided.  Weights
  rounded to 16 bits are off by 1e-3 (bf16) and 1e-4 (fp16); held in 32 bits only the output's own rounding is left."""
  eng, shape = middle_shard(name, True)
  rows = torch.zeros(N_A + N_B + n, shape.dim, dtype=torch.float16 if shape.dtype == "float16" else torch.bfloat16)
  rows[:N_A, 2], rows[:N_A, 3] = 1.0, 1.0                          # every row has two entries of 1: the norm makes them 16 or so
  rows[N_A:N_A + N_B, 6], rows[N_A:N_A + N_B, 3] = 1.0, -1.0
  rows[N_A + N_B:, 1], rows[N_A + N_B:, 6] = 1.0, 1.0
  rows = rows.cuda()
  eng.begin_request(N_A + N_B + n)
  run(eng, rows[:N_A + N_B].clone(), 0)
  got = run(eng, rows[N_A + N_B:].clone(), N_A + N_B)[:, OUT::shape.head_dim]
  x = (torch.tensor(2.0 / shape.dim + 1e-5, dtype=torch.float64) ** -0.5).to(rows.dtype).double()          # an entry of 1 behind the norm
  q, k, v = ((x * f).to(rows.dtype).item() for f in (0.125, 0.1015625, 0.0625))
  low = math.exp(-q * k / 8.0)
  for i in range(n):                                               # a new position's own key has score 0 and value 0
    exact = v * (N_A - N_B * low) / (N_A + (N_B + i + 1) * low)
    assert np.abs(got[i] - exact).max() <= abs(exact) * 2.0 ** -8 + 2e-6, (i, got[i], exact)
  eng.close()


@pytest.mark.parametrize("at", [1, 3])
def test_positions_in_front_of_a_non_finite_one(at):
  eng, shape = middle_shard("tiny-llama-hd128", False)
  g = torch.Generator().manual_seed(1)
  rows = torch.randn(66, shape.dim, generator=g).to(torch.bfloat16).cuda()
  eng.begin_request(66)
  run(eng, rows[:61].clone(), 0)
  ref = run(eng, rows[61:].clone(), 61)
  rows[61 + at] = float("nan")
  got = run(eng, rows[61:].clone(), 61)
  assert np.array_equal(got[:at], ref[:at]) and not np.isfinite(got[at]).any()
  eng.close()


def test_vocabularies_that_the_head_has_no_tile_for():
  from dataclasses import replace
  from xotorch_b200.native import NativeShard
  shape = replace(PRESETS["tiny-llama-hd64"], name="tiny-odd-vocab", vocab=2050)
  eng = NativeShard(hf_config(shape), 0)
  eng.set_shard(0, shape.n_layers - 1)
  eng.init_synthetic(2)
  ids = np.arange(5, dtype=np.int32).reshape(1, -1) * 401
  out = []
  for mode in (1, 0):
    eng.begin_request(8)
    eng.set_prefill_mode(mode)
    out.append(eng.forward(ids, 0))
  assert np.isfinite(out[0]).all() and np.array_equal(out[0], out[1])
  eng.close()


def test_a_long_cache_is_left_to_the_decode_kernel():
  """one launch walks the positions where spreading the keys over the chip pays, whatever the number of positions below the general rule; the GEMMs elsewhere"""
  eng, shape = middle_shard("tiny-llama-hd64", False)
  h = torch.randn(8, shape.dim, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()

  def launches(n, pos0):
    before = eng.kernel_launches()
    run(eng, h[:n].clone(), pos0)
    return eng.kernel_launches() - before
  eng.begin_request(2048)
  for n, pos0, gemms in ((2, 0, True), (2, 300, True), (2, 2040, False), (3, 2040, False), (7, 2040, True), (8, 2040, True), (1, 0, False)):
    assert (launches(n, pos0) > 1) == gemms, (n, pos0)
  eng.close()


@pytest.mark.parametrize("dims", [dict(dim=1024, ffn=3072, n_heads=16, n_kv_heads=4), dict(dim=2048, ffn=5632, n_heads=32, n_kv_heads=8)])
def test_layers_of_24_and_90_mb_behind_a_long_cache(dims):
  """both ways spread the keys, and the GEMMs are the cheaper one: few positions run as they do, close to what the decode kernel gives"""
  from dataclasses import replace
  from xotorch_b200.native import NativeShard
  shape = replace(PRESETS["tiny-llama-hd64"], name="small-llama", **dims)
  eng = NativeShard(hf_config(shape), 0)
  eng.set_shard(1, 1)
  eng.init_synthetic(11)
  eng.begin_request(2048)
  h = torch.randn(2048, shape.dim, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
  run(eng, h[:2040].clone(), 0)
  for n in (2, 3):
    before, out = eng.kernel_launches(), []
    for mode in (0, 1):
      eng.set_prefill_mode(mode)
      out.append(run(eng, h[2040:2040 + n].clone(), 2040))
      if mode == 0:
        assert eng.kernel_launches() - before > n
    assert np.linalg.norm(out[0] - out[1]) <= 2.0 ** -6 * np.linalg.norm(out[1])   # a layer's products round to 8 bits on both sides
  eng.close()


def test_without_memory_for_the_scratch_of_the_gemms():
  """the decode kernel takes the call, as it needs no scratch; once there is memory the GEMMs do"""
  from dataclasses import replace
  runtime = pytest.importorskip("cuda.bindings.runtime")
  from xotorch_b200.native import NativeShard
  shape = replace(PRESETS["llama-3-8b"], name="llama-3-8b-cut", n_layers=3)
  eng = NativeShard(hf_config(shape), 0)
  eng.set_shard(1, 1)
  eng.init_synthetic(5)
  eng.begin_request(16)
  h = torch.randn(5, shape.dim, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
  out = torch.empty_like(h)

  def call():
    before = eng.kernel_launches()
    torch.cuda.synchronize()
    eng.forward_device(None, h.data_ptr(), 5, 0, out.data_ptr())
    return eng.kernel_launches() - before
  eng.set_prefill_mode(1)
  call()
  ref = out.clone()
  eng.set_prefill_mode(0)
  held = []
  try:
    for size in (8 << 30, 1 << 30, 64 << 20, 2 << 20):
      while True:
        err, p = runtime.cudaMalloc(size)
        if err != runtime.cudaError_t.cudaSuccess:
          runtime.cudaGetLastError()
          break
        held.append(p)
    out.zero_()
    assert call() == 1 and torch.equal(out, ref)
  finally:
    for p in held:
      runtime.cudaFree(p)
  assert call() > 1
  eng.close()

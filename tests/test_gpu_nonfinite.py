"""A token whose values overflowed stays in its own request: prompt attention reads whole pieces of 64 tokens, and what a piece holds behind a request's
last token — the rest of a recycled page, the next request's keys in the packed buffer — must not reach the output, not even as 0 * Inf.  Inside a
request such a token reaches rows that do not see it only within the pieces of keys that they read."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from tests import bufulorn_oracle as bo, bufulorn_util as bu, layered_util as lu, zokuvik_oracle as zo

BAD = {"inf": float("inf"), "nan": float("nan")}
TOKEN = 69                                                       # the token with the bad embedding


def models(kind, bad):
  if kind == "paged":
    cfg = bu.config([bu.attention(heads=2, kv_heads=1, dim=64, vdim=64, chunk=None), bu.attention(heads=2, kv_heads=1, dim=64, vdim=128, chunk=None)], width=64, vocab=70)
    w = bo.random_weights(cfg, 3)
  else:
    window = 33 if kind == "window" else None
    cfg = lu.config([lu.attn("latent_attention_2" if window else "latent_attention", heads=2, dim=64, rot_dim=32, vdim=64, kv_rank=64, q_rank=24, window=window, ff=24)],
                    width=48, vocab=70)
    w = zo.random_weights(cfg, 3)
  w["embed"] = w["embed"].clone()
  w["embed"][TOKEN] = BAD[bad]
  return cfg, w


def good(n, seed=1):
  return lu.rand_tokens(TOKEN, n, seed)


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("kind", ["paged", "latent", "window"])
@pytest.mark.parametrize("n", [65, 100, 127, 129, 200])
def test_neighbour_in_the_batch_and_owner_of_the_pages_before(kind, n, bad):
  cfg, w = models(kind, bad)
  eng = lu.make_engine(cfg, w, "bfloat16", max_tokens=1024, page_size=64)
  rows = list(range(n))
  before = eng.prompt_attention_launches()
  ref = eng.step([0, 1], [good(n), good(90, 2)], want=rows)[0]
  assert eng.prompt_attention_launches() > before and np.isfinite(ref).all()
  for slot in (0, 1):
    eng.clear_request(slot)
  spoilt = eng.step([2, 3], [np.full(400, TOKEN, np.int32), np.full(400, TOKEN, np.int32)], want=[0])[0]   # every page but a few
  assert not np.isfinite(spoilt).any()
  for slot in (2, 3):
    eng.clear_request(slot)
  got = eng.step([0, 1], [good(n), np.full(90, TOKEN, np.int32)], want=rows)[0]
  assert np.array_equal(got, ref)
  eng.close()


@pytest.mark.parametrize("bad", BAD)
def test_rows_of_the_same_request_that_read_other_pieces(bad):
  for kind in ("paged", "latent"):
    cfg, w = models(kind, bad)
    eng = lu.make_engine(cfg, w, "bfloat16", max_tokens=1024, page_size=64)
    toks = good(128)
    ref = eng.step([0], [toks], want=list(range(64)))[0]
    toks[100] = TOKEN
    assert np.array_equal(eng.step([1], [toks], want=list(range(64)))[0], ref)      # keys 64 .. 127 are a piece of their own
    eng.close()
  cfg, w = models("window", bad)                                 # one layer, 33 tokens: token 10 lies in a piece that rows from 96 on do not read
  eng = lu.make_engine(cfg, w, "bfloat16", max_tokens=1024, page_size=64)
  toks = good(300)
  ref = eng.step([0], [toks], want=list(range(96, 300)))[0]
  toks[10] = TOKEN
  assert np.array_equal(eng.step([1], [toks], want=list(range(96, 300)))[0], ref)
  eng.close()


@pytest.mark.parametrize("n,at,clean", [(128, 100, 64), (200, 150, 128), (64, 63, 0)])
def test_rows_of_a_prompt_behind_a_shard(n, at, clean):
  """the shard engine: hidden rows in front of a non-finite one, in other pieces of keys"""
  from xotorch_b200.native import NativeShard
  from xotorch_b200.synth import PRESETS, hf_config
  shape = PRESETS["tiny-llama-hd128"]
  eng = NativeShard(hf_config(shape), 0)
  eng.set_shard(1, shape.n_layers - 2)
  eng.init_synthetic(7)
  eng.begin_request(n + 1)
  h = torch.randn(n, shape.dim, generator=torch.Generator().manual_seed(3)).to(torch.bfloat16).cuda()
  out = torch.empty_like(h)
  torch.cuda.synchronize()
  eng.forward_device(None, h.data_ptr(), n, 0, out.data_ptr())
  ref = out.float().cpu().numpy().copy()
  h[at] = float("nan")
  torch.cuda.synchronize()
  eng.begin_request(n + 1)
  eng.forward_device(None, h.data_ptr(), n, 0, out.data_ptr())
  got = out.float().cpu().numpy()
  assert np.array_equal(got[:clean], ref[:clean]) and not np.isfinite(got[at]).any()
  eng.close()

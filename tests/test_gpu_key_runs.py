"""The buffer of the key runs' partial sums belongs to steps whose attention leaves sums in it: prompts that go to the tensor cores, and single rows whose shares of the
keys meet in a cluster, take no memory for it.  When it, or a step's scratch, cannot be had the step is refused and smaller ones run as before."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from tests import bufulorn_oracle as bo, bufulorn_util as bu, layered_util as lu, zokuvik_oracle as zo
from xotorch_b200._lib import XotB200Error


def taken_by(step):
  torch.cuda.synchronize()
  before = torch.cuda.mem_get_info()[0]
  step()
  return before - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("latent", [True, False])
def test_a_prompt_on_the_tensor_cores_takes_none(latent):
  """1024 rows of 16 heads: 32 runs of 1024 x 16 sums would be 540 MB (latents of 256) and 277 MB (values of 128); what the step does need is 1024 rows of some 20000 floats, 80 MB"""
  if latent:
    cfg, oracle = lu.config([lu.attn(heads=16, dim=16, rot_dim=16, vdim=16, kv_rank=256)], width=48), zo
  else:
    cfg, oracle = bu.config([bu.attention(heads=16, kv_heads=4, dim=128, vdim=128, chunk=None)], width=64, max_positions=4000), bo
  eng = lu.make_engine(cfg, oracle.random_weights(cfg, 1), "bfloat16", max_tokens=4096, max_requests=2)
  toks = lu.rand_tokens(cfg["vocab"], 1024, 3)
  eng.step([0], [toks[:64]])                             # what is loaded on first use
  before = eng.prompt_attention_launches()
  assert taken_by(lambda: eng.step([1], [toks])) < 160 << 20
  assert eng.prompt_attention_launches() > before
  eng.close()


def test_captured_steps_stay_when_a_prompt_comes():
  """decode steps that were captured are replayed again behind a prompt no longer than what the scratch holds"""
  cfg = bu.config([bu.attention(heads=4, kv_heads=2, dim=64, vdim=64, chunk=None)], width=64, vocab=70, max_positions=4000)
  eng = lu.make_engine(cfg, bo.random_weights(cfg, 1), "bfloat16", max_tokens=2048, max_requests=3)
  toks = lu.rand_tokens(70, 200, 3)
  one = lambda i: eng.step([0], [toks[i:i + 1]])
  eng.step([1], [toks[:40]])
  eng.step([0], [toks[:100]])
  eng.clear_request(1)
  for i in range(4):
    one(i)
  replays = eng.graph_replays()
  assert replays >= 2
  eng.step([1], [toks[:100]])                            # no more rows than the first step of slot 0 brought
  eng.step([1], [toks[100:]])                            # the same behind a longer cache
  one(4)
  assert eng.graph_replays() == replays + 1
  eng.close()


def all_but(nbytes):
  """the device's free memory but `nbytes` of it, held by torch"""
  torch.cuda.synchronize()
  torch.cuda.empty_cache()
  return torch.empty(torch.cuda.mem_get_info()[0] - nbytes, dtype=torch.uint8, device="cuda")


@pytest.mark.parametrize("buffer", ["scratch", "key runs"])
def test_a_smaller_step_after_one_that_found_no_memory(buffer):
  cfg = lu.config([lu.attn(heads=16, dim=16, rot_dim=16, vdim=16, kv_rank=512)], width=48, vocab=70)
  w, rows = zo.random_weights(cfg, 1), 20000 if buffer == "scratch" else 60
  toks, more = lu.rand_tokens(70, 200, 3), lu.rand_tokens(70, rows, 4)

  def serve(big):
    eng = lu.make_engine(cfg, w, "float32", max_tokens=3 * 256 + rows, max_requests=2)
    for slot in (0, 1):
      eng.step([slot], [toks[:160]])
    out = [eng.step([slot], [toks[160:162]], want=[0, 1])[0] for slot in (0, 1)]   # two rows behind 160: six runs of keys
    big(eng)
    out += [eng.step([1], [toks[t:t + 2]], want=[0, 1])[0] for t in (162, 164)]
    eng.close()
    return np.stack(out)

  def refused(eng):
    # 20000 rows want 17 KB of scratch each and more; 60 rows leave 5 runs of 60 x 16 sums of 514 floats, 9.9 MB
    held = all_but((64 << 20) if buffer == "scratch" else (6 << 20))
    with pytest.raises(XotB200Error, match="memory"):
      eng.step([0], [more])
    del held
    torch.cuda.empty_cache()

  assert np.array_equal(serve(lambda eng: eng.step([0], [more[:60]])), serve(refused))

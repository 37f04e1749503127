"""The buffer of the key runs' partial sums belongs to steps whose attention leaves sums in it: prompts that go to the tensor cores, and single rows whose shares of the
keys meet in a cluster, take no memory for it."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from tests import bufulorn_oracle as bo, bufulorn_util as bu, layered_util as lu, zokuvik_oracle as zo


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

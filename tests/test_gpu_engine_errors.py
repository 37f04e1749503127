"""Errors that an engine comes back from.  A cache that does not fit leaves it without a request — steps are refused — and a smaller one can be begun afterwards;
page-locked memory that cannot be had; a prompt whose pipelines gave up a wait."""
from dataclasses import replace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from xotorch_b200._lib import XotB200Error
from xotorch_b200.synth import PRESETS, hf_config


@pytest.mark.parametrize("n_requests", [1, 8])
def test_a_smaller_cache_after_one_that_did_not_fit(n_requests):
  from xotorch_b200.native import NativeShard
  shape = replace(PRESETS["tiny-llama-hd64"], name="tiny-long", max_pos=200_000_000)
  eng = NativeShard(hf_config(shape), 0)
  eng.set_shard(0, shape.n_layers - 1)
  eng.init_synthetic(4)
  ids = np.arange(12, dtype=np.int32).reshape(1, -1) * 31
  eng.begin_batch(32, n_requests)
  ref = eng.forward(ids, 0).copy()
  for _ in range(2):
    with pytest.raises(XotB200Error, match="memory"):
      eng.begin_batch(150_000_000, n_requests)                    # 2 KB a token: 300 GB and more
    with pytest.raises(XotB200Error, match="begin_request"):
      eng.forward(ids, 0)
    eng.begin_batch(20, n_requests)
    assert np.array_equal(eng.forward(ids, 0), ref)
  eng.close()


@pytest.mark.parametrize("layered", [False, True])
def test_page_locked_memory_that_cannot_be_had(layered):
  """the pool goes on with plain arrays, and the step after it runs (the failure here: no such device)"""
  from xotorch_b200.pinned import library_pool
  if layered:
    from tests import bufulorn_oracle as bo, bufulorn_util as bu, layered_util as lu
    cfg = bu.config([bu.attention()])
    eng = lu.make_engine(cfg, bo.random_weights(cfg, 1), "bfloat16")
    step = lambda: eng.step([0], [np.arange(300, dtype=np.int32) % 80])[0]
  else:
    from xotorch_b200.native import NativeShard
    shape = PRESETS["tiny-llama-hd64"]
    eng = NativeShard(hf_config(shape), 0)
    eng.set_shard(1, 2)
    eng.init_synthetic(4)
    eng.begin_request(64)
    hidden = np.random.default_rng(1).standard_normal((1, 40, shape.dim)).astype(np.float32)
    step = lambda: eng.forward(hidden, 0)
  eng.results = library_pool(eng.lib, "xotb200_lm" if layered else "xotb200", 99)
  assert eng.results._alloc(1 << 20) is None
  assert np.isfinite(step()).all()
  eng.close()


@pytest.mark.parametrize("n", [5, 100])
def test_a_pipeline_wait_that_expired_is_reported_by_the_call_it_spoilt(n):
  """the error word is set as an expired wait would leave it; prompts whose hidden state stays on the device report it too, once"""
  import torch
  from xotorch_b200._lib import check
  from xotorch_b200.native import NativeShard
  shape = PRESETS["tiny-llama-hd64"]
  eng = NativeShard(hf_config(shape), 0)
  eng.set_shard(1, 2)
  eng.init_synthetic(4)
  eng.begin_request(128)
  h = torch.randn(n, shape.dim, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
  out = torch.empty_like(h)
  torch.cuda.synchronize()
  call = lambda: eng.forward_device(None, h.data_ptr(), n, 0, out.data_ptr())
  call()
  ref = out.clone()
  check(eng.lib.xotb200_debug_set_error(eng.h, 3))
  with pytest.raises(XotB200Error, match="pipeline wait"):
    call()
  call()
  assert torch.equal(out, ref)
  eng.close()

"""A cache that does not fit leaves the engine without a request — steps are refused — and a smaller one can be begun afterwards."""
from dataclasses import replace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from xotorch_b200._lib import XotB200Error
from xotorch_b200.synth import PRESETS, hf_config


@pytest.mark.parametrize("n_requests", [1, 8])
def test_a_smaller_cache_after_one_that_did_not_fit(n_requests):
  from xotorch_b200.native import NativeShard
  shape = replace(PRESETS["tiny-llama-hd64"], name="tiny-long", max_pos=2_000_000_000)
  eng = NativeShard(hf_config(shape), 0)
  eng.set_shard(0, shape.n_layers - 1)
  eng.init_synthetic(4)
  ids = np.arange(12, dtype=np.int32).reshape(1, -1) * 31
  eng.begin_batch(32, n_requests)
  ref = eng.forward(ids, 0).copy()
  for _ in range(2):
    with pytest.raises(XotB200Error, match="memory"):
      eng.begin_batch(1_500_000_000, n_requests)                  # 2 KB a token: 3 TB and more
    with pytest.raises(XotB200Error, match="begin_request"):
      eng.forward(ids, 0)
    eng.begin_batch(20, n_requests)
    assert np.array_equal(eng.forward(ids, 0), ref)
  eng.close()

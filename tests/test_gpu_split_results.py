"""Results of a first shard that is not the last: decode steps are replayed from a captured graph, and every step's hidden rows — large enough for
page-locked arrays — must land in the array that this step returned, whatever became of the arrays before it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tests import bufulorn_oracle as bo, bufulorn_util as bu, fekanex_oracle as fo, fekanex_util as fu, layered_util as lu
from xotorch_b200.pinned import SMALLEST, ResultPool, library_pool

REQUESTS, STEPS = 8, 10


def model(carry: bool):
  """two layers of width 2048: 8 rows are 64 KB; `carry`: the first layer's values go over the border behind each row"""
  if carry:
    cfg = fu.config([fu.attn(heads=2, kv_heads=2, dim=16, vdim=16, conv=2, rot_dims=8, v_mix=True) for _ in range(2)], width=2048, vocab=70)
    return cfg, fo.random_weights(cfg, 5)
  cfg = bu.config([bu.attention(heads=2, kv_heads=1, dim=16, vdim=16), bu.attention(heads=2, kv_heads=1, dim=16, vdim=16)], width=2048, vocab=70)
  return cfg, bo.random_weights(cfg, 5)


def serve(eng, graphs: bool, each=lambda s: None):
  """STEPS decode steps of REQUESTS requests; all returned arrays, none of them dropped before the end"""
  eng.set_graphs(graphs)
  for r in range(REQUESTS):
    eng.clear_request(r)
  out = []
  for s in range(STEPS):
    each(s)
    out.append(eng.step(list(range(REQUESTS)), [np.array([(7 * s + 3 * r) % 70], np.int32) for r in range(REQUESTS)]))
  return out


@pytest.mark.parametrize("carry", [False, True])
def test_every_step_fills_the_array_it_returns(carry):
  cfg, w = model(carry)
  eng = lu.make_engine(cfg, w, "bfloat16", max_tokens=REQUESTS * 32, max_requests=REQUESTS, end=0)
  ref = [a.copy() for a in serve(eng, False)]
  assert ref[0].nbytes >= SMALLEST and eng.hidden_out == 2048 + 32 * carry
  before = eng.graph_replays()
  got = serve(eng, True)
  assert eng.graph_replays() >= before + STEPS - 2
  for s in range(STEPS):
    assert np.array_equal(got[s], ref[s]), s
  eng.close()


def test_page_locked_and_plain_arrays_in_turn():
  """the bound of the pool is reached halfway through the replays, and later page-locked arrays come back"""
  cfg, w = model(False)
  eng = lu.make_engine(cfg, w, "bfloat16", max_tokens=REQUESTS * 32, max_requests=REQUESTS, end=0)
  ref = [a.copy() for a in serve(eng, False)]
  bounded = library_pool(eng.lib, "xotb200_lm")
  bounded.limit = 5 * SMALLEST
  plain = ResultPool(lambda *a: None, lambda *a: None)
  eng.results = bounded
  for s, a in enumerate(serve(eng, True)):                    # five page-locked arrays, then plain ones
    assert np.array_equal(a, ref[s]), s

  def turn(s):
    eng.results = plain if s % 2 else bounded
  for s, a in enumerate(serve(eng, True, turn)):
    assert np.array_equal(a, ref[s]), s
  eng.close()

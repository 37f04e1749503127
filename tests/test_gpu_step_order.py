"""Steps of one row per request in which the requests join, leave and change order from step to step: rows move between slots while the launches stay the same (and are
replayed), so whatever a kernel looks up ahead of its wait — the slot whose recurrent state it fetches — has to be this step's.  Every request must come out as if it
had been served alone: the 32-bit engine against the float64 oracle, and in both types the same bits whatever slots and rows the requests have."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tests import bufulorn_oracle as bo, bufulorn_util as bu, layered_util as lu, zokuvik_oracle as zo

SLOTS, LENGTH = 6, 40
# 40 tokens: sums over at most 300 terms a token, 2^-24 sqrt(40 x 300) = 6.5e-6 of a row if all were as large as the result; four times that
BOUND = 2.6e-5


def models():
  yield lu.config([lu.delta(heads=4, dim=64), lu.attn(), lu.delta(heads=3, dim=128)], width=48, vocab=60), zo, lu.oracle_logits
  yield bu.config([bu.delta(heads=4, kv_heads=2, dim=64, vdim=64), bu.attention(heads=4, kv_heads=2, dim=64, vdim=64)], width=64, vocab=60), bo, bu.oracle_logits


def schedule(seed):
  """steps of (slot, request) pairs: two to five requests each, in an order of its own; a slot is taken over by a new request when its own has ended or left"""
  rng = np.random.default_rng(seed)
  at, steps, seat, fresh = {}, [], [None] * SLOTS, 0
  for _ in range(90):
    for s in range(SLOTS):
      if seat[s] is None or at[seat[s]] == LENGTH or rng.random() < 0.02:
        seat[s], fresh = fresh, fresh + 1
        at[seat[s]] = 0
    step = []
    for s in rng.permutation(SLOTS)[:rng.integers(2, SLOTS)]:
      if at[seat[s]] < LENGTH:
        step.append((int(s), seat[s], at[seat[s]]))
        at[seat[s]] += 1
    if step:
      steps.append(step)
  return steps, fresh


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_every_request_as_if_alone(seed, dtype):
  for cfg, oracle, logits in models():
    w = oracle.random_weights(cfg, seed)
    eng = lu.make_engine(cfg, w, dtype, max_tokens=SLOTS * 64, max_requests=SLOTS)
    steps, n = schedule(seed)
    toks = [lu.rand_tokens(cfg["vocab"], LENGTH, 100 * seed + r) for r in range(n)]

    def serve(seats, order):
      got = [[] for _ in range(n)]
      for step in steps:
        step = step[::order]
        for s, _, t in step:
          if t == 0:
            eng.clear_request(seats[s])
        lg = eng.step([seats[s] for s, _, _ in step], [toks[r][t:t + 1] for _, r, t in step])[0]
        for row, (_, r, _) in zip(lg, step):
          got[r].append(row)
      return [np.stack(g) for g in got if g]

    one, two = serve(list(range(SLOTS)), 1), serve([3, 5, 0, 2, 1, 4], -1)   # the same requests in other slots, their rows in reverse
    eng.close()
    assert all(np.array_equal(a, b) for a, b in zip(one, two))
    if dtype == "float32":
      assert max(lu.row_err(g, logits(cfg, w, t)[0][:len(g)]) for g, t in zip(one, toks)) < BOUND

"""Prompts of the delta-rule mixers (from 160 rows on; gated 128, and 256 with heads above 64) over chunks of 32 tokens, and shorter ones beside them: head sizes at both padded ones and between, value columns that are no whole group, row counts around whole
chunks, requests of very different lengths in one step, key heads shared by value heads, filters shorter than the window registers — 32-bit engine against the
float64 oracles, and the state they leave carried on row by row.

Bound: a result is a chain of sums over at most 300 tokens x 128 key rows in 32 bits, each rounding 2^-24: 2^-24 sqrt(300 x 128) = 1.2e-5 of a row if they were all as large as
the result; twice that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tests import bufulorn_oracle as bo, bufulorn_util as bu, layered_util as lu, zokuvik_oracle as zo

BOUND = 2.4e-5


def check(cfg, w, oracle, rows, more=3):
  """requests of rows[r] tokens in one step, then `more` steps of one row each"""
  n = len(rows)
  eng = lu.make_engine(cfg, w, "float32", max_tokens=sum(rows) + 64 * n, max_requests=n)
  toks = [lu.rand_tokens(cfg["vocab"], k + more, 7 + r) for r, k in enumerate(rows)]
  want = list(range(sum(rows)))
  first = eng.step(list(range(n)), [t[:k] for t, k in zip(toks, rows)], want=want)[0]
  then = [eng.step(list(range(n)), [t[k + i:k + i + 1] for t, k in zip(toks, rows)])[0] for i in range(more)]
  eng.close()
  at = np.concatenate([[0], np.cumsum(rows)])
  for r, k in enumerate(rows):
    ref, _ = oracle(cfg, w, toks[r])
    got = np.concatenate([first[at[r]:at[r + 1]]] + [t[r:r + 1] for t in then])
    assert lu.row_err(got, ref) < BOUND, (r, k)


@pytest.mark.parametrize("rows", [[96], [127], [128], [129], [159], [160], [161], [300], [97, 1, 130, 33], [97, 1, 190, 33]])
@pytest.mark.parametrize("dim", [36, 64, 68, 128])
def test_general_rule(dim, rows):
  cfg = lu.config([lu.delta(heads=2, dim=dim)], width=48, vocab=50)
  check(cfg, zo.random_weights(cfg, dim), lu.oracle_logits, rows)


@pytest.mark.parametrize("rows", [[96], [128], [161], [2, 140, 31, 32, 1], [255], [256], [287], [2, 260, 31, 32, 1]])
@pytest.mark.parametrize("heads,dim,vdim,conv", [(4, 64, 64, 4), (6, 64, 64, 2), (2, 128, 128, 3), (10, 64, 30, 4), (4, 36, 72, 4), (4, 128, 64, 1), (4, 64, 64, 6)])
def test_gated_rule(heads, dim, vdim, conv, rows):
  cfg = bu.config([bu.delta(heads=heads, kv_heads=2, dim=dim, vdim=vdim, conv=conv)], width=48, vocab=50)
  check(cfg, bo.random_weights(cfg, dim + vdim), bu.oracle_logits, rows)


@pytest.mark.parametrize("decay", [-30.0, 30.0])
def test_gated_rule_at_the_ends_of_its_decay(decay):
  """every token forgets everything in front of it (exp of a large negative number: 0 in 32 bits), or nothing"""
  cfg = bu.config([bu.delta(heads=4, kv_heads=2, dim=64, vdim=64)], width=48, vocab=50)
  w = bo.random_weights(cfg, 4)
  w["l0.mix.A_log"] = w["l0.mix.A_log"] * 0 + (5.0 if decay > 0 else -20.0)
  w["l0.mix.dt_bias"] = w["l0.mix.dt_bias"] * 0 + decay
  check(cfg, w, bu.oracle_logits, [160])


def with_a_token_that_is_not_finite(general, n, at, bad):
  cfg = lu.config([lu.delta(heads=2, dim=64)], width=48, vocab=51) if general else bu.config([bu.delta(heads=4, kv_heads=2, dim=64, vdim=64)], width=48, vocab=51)
  w = (zo if general else bo).random_weights(cfg, 3)
  w["embed"] = w["embed"].clone()
  w["embed"][50] = bad
  eng = lu.make_engine(cfg, w, "float32", max_tokens=1024)
  toks = lu.rand_tokens(50, n, 5)
  ref = eng.step([0, 1], [toks, toks], want=list(range(2 * n)))[0]
  spoilt = toks.copy()
  spoilt[at] = 50
  got = eng.step([2, 3], [spoilt, toks], want=list(range(2 * n)))[0]
  assert np.isfinite(got[:at]).all() and lu.row_err(np.concatenate([got[:at], got[n:]]), np.concatenate([ref[:at], ref[n:]])) < BOUND
  assert not np.isfinite(got[at:n]).any()
  eng.close()


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("at", [0, 31, 40, 95, 99])
@pytest.mark.parametrize("general", [False, True])
def test_tokens_in_front_of_one_that_is_not_finite(general, at, bad):
  with_a_token_that_is_not_finite(general, 100, at, bad)


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("at", [0, 31, 40, 159, 160, 171])
@pytest.mark.parametrize("general", [False, True])
def test_tokens_of_a_prompt_in_front_of_one_that_is_not_finite(general, at, bad):
  """100 rows go token by token, these over chunks"""
  with_a_token_that_is_not_finite(general, 172, at, bad)


@pytest.mark.parametrize("others", [21, 22])
@pytest.mark.parametrize("general", [False, True])
def test_requests_beside_a_prompt_on_both_sides_of_the_line(general, others):
  """a prompt and requests of 40: four heads of 64 x 64 are 16 blocks, 148 / 16 - 1 of whose walks are free beside the prompt's chunks, and each 16 of its rows beyond the line pay for one more.
  Gated, 160 rows: 41 + 2 chunks, 21 others (42) go over chunks with it, with 22 all go token by token.  General, 192 rows: 49 + 2, 25 others and 26"""
  rows = [192] + [40] * (others + 4) if general else [160] + [40] * others
  if general:
    cfg = lu.config([lu.delta(heads=4, dim=64)], width=48, vocab=50)
    check(cfg, zo.random_weights(cfg, 1), lu.oracle_logits, rows, more=1)
  else:
    cfg = bu.config([bu.delta(heads=4, kv_heads=2, dim=64, vdim=64)], width=48, vocab=50)
    check(cfg, bo.random_weights(cfg, 2), bu.oracle_logits, rows, more=1)

"""Steps of one row per request over cached keys and values of 64 or 128 entries take a kernel of their own; steps of two rows per request keep the general one.  Both must give the
same rows, over every form of attention that the mixers have (soft cap, distance penalties, learned distance bias, blocks, windows with kept first tokens or pooled blocks, sinks,
gates, query temperature, rotation), one to eight query heads per key head, and caches from nothing to more runs of keys than a cluster holds.

Bound, 32 bits: sums over at most 2600 keys x 128 entries in another order, 2^-24 sqrt(2600 x 128) = 3.4e-5 of a row if all were as large as the result; twice that.  In 16 bits the products
around the attention round to 8 bits on both sides: 2^-8, twice."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tests import bufulorn_oracle as bo, bufulorn_util as bu, fekanex_oracle as fo, fekanex_util as fu, fubelorn_util as uu, layered_util as lu, tunavik_oracle as to, tunavik_util as tu

BOUND = {"float32": 7e-5, "bfloat16": 2 ** -7}


def forms(d):
  two = dict(dim=d, vdim=d)
  yield "blocks", bu.config([bu.attention(heads=8, kv_heads=2, chunk=100, **two), bu.attention(heads=4, kv_heads=4, chunk=None, softcap=None, **two)], max_positions=4000), bo
  yield "shared by 8, by 3", bu.config([bu.attention(heads=8, kv_heads=1, chunk=None, **two), bu.attention(heads=6, kv_heads=2, chunk=37, **two)], max_positions=4000), bo
  yield "learned bias", tu.config([tu.attention(heads=4, kv_heads=2, bias_max=40, **two)]), to
  yield "kept first tokens", fu.config([fu.attn(heads=4, kv_heads=2, size=45, keep=3, **two), fu.attn(heads=2, kv_heads=2, size=None, rot_dims=0, **two)]), fo


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 70, 400, 2600])
def test_one_row_against_two(n, d, dtype):
  for name, cfg, oracle in forms(d):
    w = oracle.random_weights(cfg, d + n)
    requests = 1 if n > 1000 else 3
    eng = lu.make_engine(cfg, w, dtype, max_tokens=2 * requests * (n + 80), max_requests=2 * requests, page_size=16)
    toks = [lu.rand_tokens(cfg["vocab"], n + 4, 3 + r) for r in range(requests)]
    pairs, singles = list(range(requests)), list(range(requests, 2 * requests))
    for slots in (pairs, singles):
      eng.step(slots, [t[:n] for t in toks])
    for at in (n, n + 2):
      ref = eng.step(pairs, [t[at:at + 2] for t in toks], want=list(range(2 * requests)))[0].reshape(requests, 2, -1)
      got = np.stack([eng.step(singles, [t[at + i:at + i + 1] for t in toks])[0] for i in range(2)], axis=1)
      assert lu.row_err(got.reshape(2 * requests, -1), ref.reshape(2 * requests, -1)) < BOUND[dtype], (name, at)
    eng.close()


@pytest.mark.parametrize("left", ["keep", "pool"])
@pytest.mark.parametrize("n", [3, 40, 130])
def test_windows_with_pooled_blocks_and_kept_tokens_against_the_oracle(left, n):
  cfg = uu.config([uu.parallel(left=uu.left_keep(heads=4, kv_heads=2, dim=64, vdim=64, size=33, keep=3)) if left == "keep" else
                   uu.parallel_2(left=uu.left_pool(heads=4, kv_heads=1, dim=64, vdim=64, size=33, pool=4))])
  w = uu.random_weights(cfg, n)
  eng = lu.make_engine(cfg, w, "float32", max_tokens=400, max_requests=2, page_size=8)
  toks = lu.rand_tokens(cfg["vocab"], n + 12, 3)
  got = [eng.step([1], [toks[:n]])[0]] + [eng.step([1], [toks[i:i + 1]])[0] for i in range(n, n + 12)]
  assert lu.row_err(np.concatenate(got), uu.oracle_logits(cfg, w, toks)[0][n - 1:]) < lu.TOL["float32"]
  eng.close()


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_values_that_no_row_sees(bad):
  """a token that is not finite lies in the cache in front of a block of keys that later rows do not read"""
  cfg = bu.config([bu.attention(heads=8, kv_heads=2, dim=64, vdim=64, chunk=16)], vocab=70)
  w = bo.random_weights(cfg, 3)
  w["embed"] = w["embed"].clone()
  w["embed"][69] = bad
  eng = lu.make_engine(cfg, w, "float32", max_tokens=256, page_size=8)
  toks = lu.rand_tokens(69, 40, 2)
  spoilt = toks.copy()
  spoilt[10] = 69
  for slot, t in ((0, toks), (1, spoilt)):
    eng.step([slot], [t[:36]])
  for i in range(36, 40):
    a, b = eng.step([0, 1], [toks[i:i + 1], spoilt[i:i + 1]])[0]
    assert np.isfinite(a).all() and np.array_equal(a, b)
  eng.close()

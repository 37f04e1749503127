"""The delta-rule recurrence over its variants: head sizes at the edges of the padded ones (4 .. 200, sizes that are no whole 16-byte pieces), row counts
around the groups of four tokens and the staged chunks, key heads shared by value heads, and batches wide enough for the variants with several
columns per thread — 32-bit engine against the float64 oracles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tests import bufulorn_oracle as bo, bufulorn_util as bu, layered_util as lu, zokuvik_oracle as zo


def check(cfg, w, oracle, n_req, rows):
  eng = lu.make_engine(cfg, w, "float32", max_tokens=n_req * 64, max_requests=n_req)
  toks = [lu.rand_tokens(cfg["vocab"], rows + 2, 7 + r) for r in range(n_req)]
  some = sorted({0, n_req // 2, n_req - 1})
  want = [r * rows + t for r in range(n_req) for t in range(rows)]
  first, _ = eng.step(list(range(n_req)), [t[:rows] for t in toks], want=want)
  then = [eng.step(list(range(n_req)), [t[rows + i:rows + i + 1] for t in toks])[0] for i in range(2)]   # the state carried on, row by row
  eng.close()
  for r in some:
    ref, _ = oracle(cfg, w, toks[r])
    got = np.concatenate([first.reshape(n_req, rows, -1)[r]] + [t[r:r + 1] for t in then])
    assert lu.row_err(got, ref) < lu.TOL["float32"], r


@pytest.mark.parametrize("dim", [4, 7, 16, 17, 32, 36, 64, 65, 128, 132, 200])
@pytest.mark.parametrize("rows", [1, 5, 21])
def test_general_rule(dim, rows):
  cfg = lu.config([lu.delta(heads=2, dim=dim)], width=48, vocab=50)
  check(cfg, zo.random_weights(cfg, dim), lu.oracle_logits, 1, rows)


@pytest.mark.parametrize("dim,vdim", [(8, 6), (16, 16), (24, 32), (64, 64), (64, 30), (128, 64), (72, 128)])
@pytest.mark.parametrize("rows", [3, 4, 34])
def test_gated_rule_with_shared_key_heads(dim, vdim, rows):
  cfg = bu.config([bu.delta(heads=6, kv_heads=2, dim=dim, vdim=vdim)], width=48, vocab=50)
  check(cfg, bo.random_weights(cfg, dim + vdim), bu.oracle_logits, 1, rows)


@pytest.mark.parametrize("dim", [32, 64, 128])
def test_many_requests(dim):
  cfg = bu.config([bu.delta(heads=12, kv_heads=3, dim=dim, vdim=dim)], width=48, vocab=50)
  check(cfg, bo.random_weights(cfg, dim), bu.oracle_logits, 12, 6)
  cfg = lu.config([lu.delta(heads=12, dim=dim)], width=48, vocab=50)
  check(cfg, zo.random_weights(cfg, dim), lu.oracle_logits, 12, 6)

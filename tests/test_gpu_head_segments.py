"""Steps of several wanted rows: the vocabulary in segments, each sent while the next is computed.  Vocabularies at the edges of a segment and of a 128-column tile, rows that give one segment
and several, rows wanted more than once, ties of the argmax across segments, results asked for and not — against the same rows taken one or two at a time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tests import bufulorn_oracle as bo, bufulorn_util as bu, layered_util as lu, zokuvik_oracle as zo


def make(family, vocab, rows):
  if family == "zokuvik":
    cfg = lu.config([lu.attn(heads=2, dim=16, rot_dim=8, vdim=16, kv_rank=24, ff=72)], width=128, vocab=vocab, groups=1)
    w = zo.random_weights(cfg, 7)
  else:
    cfg = bu.config([bu.attention(heads=2, kv_heads=1, dim=16, vdim=16, chunk=64, mlp=bu.dense(40))], width=128, vocab=vocab)
    w = bo.random_weights(cfg, 7)
  return cfg, w, lu.make_engine(cfg, w, "bfloat16", max_tokens=4 * rows + 64, max_requests=2)


@pytest.mark.parametrize("family", ["zokuvik", "bufulorn"])
@pytest.mark.parametrize("vocab,rows", [(4096, 33), (8192, 24), (16385, 9), (21333, 40), (32000, 8), (32000, 16), (65536, 3), (65537, 5)])
def test_segments(family, vocab, rows):
  cfg, w, eng = make(family, vocab, rows)
  toks = lu.rand_tokens(vocab, rows, rows)
  lg, best = eng.step([0], [toks], want=list(range(rows)))
  lg, best = lg.copy(), np.asarray(best).copy()
  ref, _ = (lu if family == "zokuvik" else bu).oracle_logits(cfg, w, toks)
  assert lu.row_err(lg, ref) < lu.TOL["bfloat16"]
  assert np.array_equal(best, lg.argmax(-1))
  want = [rows - 1, 0, rows - 1, rows // 2, 0]          # gathered, repeated
  eng.clear_request(0)
  few, few_best = eng.step([0], [toks], want=want)
  assert lu.row_err(few, lg[want]) < lu.TOL["bfloat16"] / 2 and np.array_equal(few_best, few.argmax(-1))
  eng.clear_request(0)
  only, _ = eng.step([0], [toks], want=list(range(rows)), argmax=False)
  assert np.array_equal(only, lg)
  eng.close()


def test_equal_entries_across_segments():
  """two columns of the head that are the same, in different segments and larger than all others: the lower one is taken"""
  vocab, rows = 32000, 16
  cfg, w, eng = make("zokuvik", vocab, rows)
  eng.close()
  name = "head"
  w[name] = w[name].clone()
  for a, b in ((100, 31990), (9000, 20000)):
    w[name][b] = w[name][a]
  eng = lu.make_engine(cfg, w, "bfloat16", max_tokens=128, max_requests=2)
  toks = lu.rand_tokens(vocab, rows, 1)
  lg, best = eng.step([0], [toks], want=list(range(rows)))
  assert np.array_equal(lg[:, 100], lg[:, 31990]) and np.array_equal(lg[:, 9000], lg[:, 20000])
  assert np.array_equal(best, lg.argmax(-1))
  eng.close()

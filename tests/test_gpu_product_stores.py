"""Products of many rows — 128 x 128 tiles, whole or with K cut over a cluster, and CTA pairs —, their way out through shared memory: 128 x 128 tiles and CTA pairs, row and column remainders of a warp's 32 rows and of a 128-byte
piece of a row, leading dimensions that are no whole pieces, 32-bit and 16-bit outputs, xIELU and gated epilogues — against the float64 oracles."""
import pytest

pytestmark = pytest.mark.gpu

from tests import bufulorn_oracle as bo, zokuvik_oracle as zo
from tests import bufulorn_util as bu, layered_util as lu


# down products with K = ff: 2056 and 2120 in two shares, 4168 in four (the last shares shorter)
@pytest.mark.parametrize("rows,ff", [(257, 40), (260, 1000), (289, 2056), (300, 2120), (390, 4168), (383, 136), (700, 5904), (1030, 3592)])
def test_xielu_products(rows, ff):
  """700 x 5904 and 1030 x 3592 on CTA pairs; the projections have 5 * 16 + 2 * 2 * 17 = 148 columns and more"""
  cfg = bu.config([bu.attention(heads=6, kv_heads=3, dim=16, vdim=17, chunk=64, mlp=bu.dense(ff))], width=520, vocab=331, max_positions=1200)
  w = bo.random_weights(cfg, 13)
  for n in w:
    if n.endswith("mlp.up"):
      w[n] = w[n] * 4                                        # arguments from -20 to 20: both branches of the activation's negative side
  toks = lu.rand_tokens(331, rows, 3)
  eng = lu.make_engine(cfg, w, "bfloat16", max_tokens=rows + 8)
  got, _ = eng.step([0], [toks], want=list(range(rows)), argmax=False)
  eng.close()
  ref, _ = bu.oracle_logits(cfg, w, toks)
  assert lu.row_err(got, ref) < lu.TOL["bfloat16"]


@pytest.mark.parametrize("rows,ff", [(300, 24), (300, 72), (520, 520)])
def test_gated_products(rows, ff):
  """experts of 128-row tiles: 2 ff columns, of which a 128-column tile is a third, most, or several"""
  cfg = bu.config([bu.attention(heads=4, kv_heads=2, dim=16, vdim=16, chunk=64, mlp=bu.moe(experts=4, top=2, groups=None, ff=ff))], width=136, vocab=150, max_positions=600)
  w = bo.random_weights(cfg, 5)
  toks = lu.rand_tokens(150, rows, rows + 1)
  eng = lu.make_engine(cfg, w, "bfloat16", max_tokens=rows + 8)
  got, _ = eng.step([0], [toks], want=list(range(rows)), argmax=False)
  eng.close()
  ref, _ = bu.oracle_logits(cfg, w, toks)
  err = sorted(lu.row_err(got[i:i + 1], ref[i:i + 1]) for i in range(rows))   # a tie within rounding may send a row to another expert
  assert err[int(0.9 * (rows - 1))] < lu.TOL["bfloat16"]


@pytest.mark.parametrize("rows", [258, 300])
def test_columns_that_are_no_whole_pieces(rows):
  cfg = lu.config([lu.attn(heads=3, dim=18, rot_dim=6, vdim=10, kv_rank=40, q_rank=72, ff=264)], width=200, vocab=331, groups=4)
  w = zo.random_weights(cfg, 11)
  toks = lu.rand_tokens(331, rows, rows)
  eng = lu.make_engine(cfg, w, "bfloat16", max_tokens=rows + 8)
  got, _ = eng.step([0], [toks], want=list(range(rows)), argmax=False)
  eng.close()
  ref, _ = lu.oracle_logits(cfg, w, toks)
  assert lu.row_err(got, ref) < lu.TOL["bfloat16"]

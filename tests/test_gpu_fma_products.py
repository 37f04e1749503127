"""Products of the all-32-bit mode (fp32 FMA tiles of 16 .. 96 rows, K cut over clusters): row counts at the edges of the tile heights, column and
K remainders, a K cut whose last CTA has no block, gated and closing epilogues — against the float64 oracles, with the 32-bit error bound."""
import pytest

pytestmark = pytest.mark.gpu

from tests import layered_util as lu, rinutar_oracle as ro, rinutar_util as ru, zokuvik_oracle as zo

ROWS = [9, 16, 17, 32, 33, 49, 65, 71, 80, 81, 96, 97, 130]


@pytest.mark.parametrize("rows", ROWS)
def test_dense_products_match_oracle(rows):
  # width 204: 6 3/8 K blocks; ff 2084: 65 1/8 K blocks over 8 CTAs of 9 (the last starts behind the end), 32 9/16 column tiles; vocabulary 331
  cfg = lu.config([lu.attn(heads=5, dim=16, rot_dim=8, vdim=24, kv_rank=40, q_rank=72, ff=2084), lu.attn("latent_attention_2", heads=2, dim=8, vdim=8, window=9, ff=132)],
                  width=204, vocab=331, groups=3)
  w = zo.random_weights(cfg, 12)
  toks = lu.rand_tokens(331, rows, rows)
  eng = lu.make_engine(cfg, w, "float32", max_tokens=256)
  got = lu.run_cut(eng, 0, toks, [rows])
  eng.close()
  ref, _ = lu.oracle_logits(cfg, w, toks)
  assert lu.row_err(got, ref) < lu.TOL["float32"]


@pytest.mark.parametrize("rows", [9, 40, 100])
def test_gated_and_closing_products_match_oracle(rows):
  cfg = ru.config([ru.attn(heads=4, mlp=ru.dense(72)), ru.attn(heads=2, mlp=ru.dense(76))], width=52, vocab=90)   # 76: gate and up rows not interleaved in eights
  w = ro.random_weights(cfg, 6)
  toks = lu.rand_tokens(90, rows, 2)
  eng = lu.make_engine(cfg, w, "float32", max_tokens=256)
  got = lu.run_cut(eng, 0, toks, [rows])
  eng.close()
  ref, _ = ru.oracle_logits(cfg, w, toks)
  assert lu.row_err(got, ref) < lu.TOL["float32"]

"""Products with few rows on the tensor cores (the streaming form of the layered engine's products): edges of its row tiles (16, 32,
64, 128, 256 rows), column and K remainders, K cut over clusters of up to eight CTAs (the last of them without a block of its own), experts' row
tiles — against the float64 oracles, with the error bound of the other 16-bit tests."""
import pytest

pytestmark = pytest.mark.gpu

from tests import bufulorn_oracle as bo, zokuvik_oracle as zo
from tests import bufulorn_util as bu, layered_util as lu

ROWS = [3, 15, 16, 17, 32, 33, 64, 65, 127, 128, 129, 255, 256, 257]


@pytest.mark.parametrize("rows", ROWS)
def test_dense_products_match_oracle(rows):
  # width 200: K of 3 1/8 blocks; ff 2072: 33 K blocks over 8 CTAs of 5 (the last has none), 16 1/5 column tiles; vocabulary 331: 2 3/5 column tiles
  cfg = lu.config([lu.attn(heads=5, dim=16, rot_dim=8, vdim=24, kv_rank=40, q_rank=72, ff=2072), lu.attn("latent_attention_2", heads=2, dim=8, vdim=8, window=9, ff=136)],
                  width=200, vocab=331, groups=4)
  w = zo.random_weights(cfg, 11)
  toks = lu.rand_tokens(331, rows, rows)
  eng = lu.make_engine(cfg, w, "bfloat16", max_tokens=264)
  before = eng.tensor_core_launches()
  got = lu.run_cut(eng, 0, toks, [rows])
  assert eng.tensor_core_launches() - before >= 11
  ref, _ = lu.oracle_logits(cfg, w, toks)
  assert lu.row_err(got, ref) < lu.TOL["bfloat16"]
  eng.set_gemm_mode(1)                                         # the FMA tiles on the same rows: only the order of the sums differs
  eng.clear_request(0)
  fma = lu.run_cut(eng, 0, toks, [rows])
  assert lu.row_err(got, fma) < lu.TOL["bfloat16"] / 2
  eng.close()


@pytest.mark.parametrize("rows", ROWS)
def test_expert_products_match_oracle(rows):
  cfg = bu.config([bu.attention(heads=4, kv_heads=2, dim=16, vdim=16, chunk=64, mlp=bu.moe(experts=12, top=3, groups=(4, 2), ff=72)),
                   bu.delta(heads=4, kv_heads=2, dim=16, vdim=24, mlp=bu.moe(experts=5, top=2, groups=None, ff=520))], width=136, vocab=150)
  w = bo.random_weights(cfg, 5)
  toks = lu.rand_tokens(150, rows, rows + 1)
  eng = lu.make_engine(cfg, w, "bfloat16", max_tokens=264)
  got = lu.run_cut(eng, 0, toks, [rows])
  eng.set_gemm_mode(1)
  eng.clear_request(0)
  fma = lu.run_cut(eng, 0, toks, [rows])                       # row kernels for the experts: the same choices unless two scores tie within rounding
  eng.close()
  ref, _ = bu.oracle_logits(cfg, w, toks)
  err = lambda a, b: sorted(lu.row_err(a[i:i + 1], b[i:i + 1]) for i in range(rows))   # noqa: E731
  assert err(got, ref)[int(0.9 * (rows - 1))] < lu.TOL["bfloat16"] and err(got, fma)[int(0.9 * (rows - 1))] < lu.TOL["bfloat16"] / 2


@pytest.mark.parametrize("rows,width,ff", [(129, 200, 2072), (700, 1032, 5904), (1030, 520, 3580)])
def test_many_rows_on_cta_pairs_match_oracle(rows, width, ff):
  """256 x 256 tiles of CTA pairs where they fill the GPU (700 rows x 5904: 3 x 24 tiles, the last row tile with 188 rows, the last column tile with 16
  columns; 1030 x 3580: a row tile with 6 rows), 128 x 128 tiles elsewhere; closing epilogues of both forms"""
  cfg = lu.config([lu.attn("latent_attention_2", heads=2, dim=16, rot_dim=8, vdim=16, kv_rank=24, window=40, ff=ff)], width=width, vocab=331, groups=1)
  w = zo.random_weights(cfg, 21)
  toks = lu.rand_tokens(331, rows, 4)
  eng = lu.make_engine(cfg, w, "bfloat16", max_tokens=rows + 8)
  got, _ = eng.step([0], [toks], want=list(range(rows)), argmax=False)
  eng.close()
  ref, _ = lu.oracle_logits(cfg, w, toks)
  assert lu.row_err(got, ref) < lu.TOL["bfloat16"]


@pytest.mark.parametrize("rows", [600])
def test_closing_products_on_cta_pairs_match_oracle(rows):
  from tests import rinutar_oracle as ro, rinutar_util as ru
  cfg = ru.config([ru.attn(heads=2, mlp=ru.dense(1032))], width=6136, vocab=64)   # down product: 600 x 6136 with K = 1032: 3 x 24 tiles
  w = ro.random_weights(cfg, 8)
  toks = lu.rand_tokens(64, rows, 5)
  eng = lu.make_engine(cfg, w, "bfloat16", max_tokens=rows + 8)
  got, _ = eng.step([0], [toks], want=list(range(rows)), argmax=False)
  eng.close()
  ref, _ = ru.oracle_logits(cfg, w, toks)
  assert lu.row_err(got, ref) < lu.TOL["bfloat16"]

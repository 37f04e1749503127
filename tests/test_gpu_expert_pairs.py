"""Experts of many rows on CTA pairs (256-row tiles): runs that end in a tile, experts with few rows and with none beside full ones, columns and K that are no whole tiles, gated and ungated
forms — against the float64 oracles."""
import pytest

pytestmark = pytest.mark.gpu

from tests import bufulorn_oracle as bo, bufulorn_util as bu, layered_util as lu, tunavik_oracle as to, tunavik_util as tu


def check(eng, rows, toks, ref):
  got, _ = eng.step([0], [toks], want=list(range(rows)), argmax=False)
  got = got.copy()
  eng.set_gemm_mode(1)                                        # the row kernels
  eng.clear_request(0)
  rowwise, _ = eng.step([0], [toks], want=list(range(rows)), argmax=False)
  eng.close()
  err = lambda a, b: sorted(lu.row_err(a[i:i + 1], b[i:i + 1]) for i in range(rows))   # noqa: E731
  assert err(got, ref)[int(0.9 * (rows - 1))] < lu.TOL["bfloat16"]                     # a tie within rounding may send a row to another expert
  assert err(got, rowwise)[int(0.9 * (rows - 1))] < lu.TOL["bfloat16"] / 2


# top 2: 2 rows / experts rows an expert on average, 256 and more
@pytest.mark.parametrize("rows,experts,width,ff", [(512, 4, 512, 512), (700, 4, 520, 520), (1000, 5, 776, 648), (1100, 3, 512, 1032)])
def test_gated_experts(rows, experts, width, ff):
  cfg = bu.config([bu.attention(heads=2, kv_heads=1, dim=16, vdim=16, chunk=64, mlp=bu.moe(experts=experts, top=2, groups=None, ff=ff))], width=width, vocab=90, max_positions=rows + 8)
  w = bo.random_weights(cfg, rows)
  toks = lu.rand_tokens(90, rows, 3)
  check(lu.make_engine(cfg, w, "bfloat16", max_tokens=rows + 8), rows, toks, bu.oracle_logits(cfg, w, toks)[0])


def test_experts_without_rows():
  """two tokens in turn: their rows' experts are full, the others' runs are empty"""
  rows = 900
  cfg = bu.config([bu.attention(heads=2, kv_heads=1, dim=16, vdim=16, chunk=64, mlp=bu.moe(experts=7, top=2, groups=None, ff=512))], width=512, vocab=90, max_positions=rows + 8)
  w = bo.random_weights(cfg, 2)
  toks = lu.rand_tokens(90, 2, 3).repeat(rows // 2)
  check(lu.make_engine(cfg, w, "bfloat16", max_tokens=rows + 8), rows, toks, bu.oracle_logits(cfg, w, toks)[0])


def test_ungated_experts():
  rows = 700
  cfg = tu.config([tu.attention(heads=2, kv_heads=1, dim=16, vdim=16, mlp=tu.moe(experts=4, top=2, ff=520))], width=520, vocab=90)
  w = to.random_weights(cfg, 4)
  toks = lu.rand_tokens(90, rows, 3)
  check(lu.make_engine(cfg, w, "bfloat16", max_tokens=rows + 8), rows, toks, tu.oracle_logits(cfg, w, toks)[0])

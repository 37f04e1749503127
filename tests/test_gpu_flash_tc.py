"""Prompt attention on tcgen05 (128-row tiles, heads of 64-entry chunks, 64-token pieces of pages): row counts at the edges of the tiles, portions behind
cached tokens, windows and blocks that start inside a piece, every head size it takes, soft cap, distance terms, sinks and gates — against the
float64 oracles, and against the mma.sync kernel (which pages of 8 tokens select)."""
import pytest

pytestmark = pytest.mark.gpu

from tests import bufulorn_oracle as bo, bufulorn_util as bu, layered_util as lu, rinutar_oracle as ro, rinutar_util as ru, tunavik_oracle as to, tunavik_util as tu, \
  zokuvik_oracle as zo


def check(cfg, w, oracle, cuts, n, page=64):
  toks = lu.rand_tokens(cfg["vocab"], n, n)
  eng = lu.make_engine(cfg, w, "bfloat16", max_tokens=n + 8, page_size=page)
  before = eng.prompt_attention_launches()
  got = lu.run_cut(eng, 0, toks, cuts)
  assert eng.prompt_attention_launches() > before
  eng.close()
  ref, _ = oracle(cfg, w, toks)
  err = lu.row_err(got, ref)
  assert err < lu.TOL["bfloat16"], err
  return got


@pytest.mark.parametrize("cuts,n", [([16], 16), ([64], 64), ([65], 65), ([127], 127), ([128], 128), ([129], 129), ([300], 300), ([40, 100, 17, 200], 357)])
@pytest.mark.parametrize("dim,vdim,chunk", [(64, 64, None), (128, 128, 96), (192, 128, 50), (64, 128, 64), (128, 64, 1)])
def test_cached_keys(dim, vdim, chunk, cuts, n):
  cfg = bu.config([bu.attention(heads=4, kv_heads=2, dim=dim, vdim=vdim, chunk=chunk, softcap=30.0 if chunk != 50 else None)], width=64, vocab=70)
  check(cfg, bo.random_weights(cfg, dim), bu.oracle_logits, cuts, n)


@pytest.mark.parametrize("cuts,n", [([150], 150), ([30, 129], 159)])
def test_distance_buckets_and_sinks(cuts, n):
  cfg = tu.config([tu.attention(heads=4, kv_heads=2, dim=64, vdim=64)], width=64, vocab=70)
  check(cfg, to.random_weights(cfg, 3), tu.oracle_logits, cuts, n)


@pytest.mark.parametrize("cuts,n", [([16], 16), ([130], 130), ([50, 300], 350)])
@pytest.mark.parametrize("dim,rot,vdim,window", [(64, 32, 64, None), (64, 64, 128, 100), (128, 64, 128, 33), (128, 8, 64, None)])
def test_latent_keys(dim, rot, vdim, window, cuts, n):
  kind = "latent_attention_2" if window else "latent_attention"
  cfg = lu.config([lu.attn(kind, heads=3, dim=dim, rot_dim=rot, vdim=vdim, kv_rank=64, q_rank=24, window=window, ff=24)], width=48, vocab=70)
  check(cfg, zo.random_weights(cfg, dim + rot), lu.oracle_logits, cuts, n)


def test_sink_of_the_latent_form_and_agreement_with_the_other_kernel():
  cfg = ru.config([ru.attn(heads=3, dim=64, rot_dim=32, vdim=64, kv_rank=40, mlp=ru.dense(24))])
  check(cfg, ro.random_weights(cfg, 4), ru.oracle_logits, [200], 200)
  cfg = bu.config([bu.attention(heads=4, kv_heads=2, dim=128, vdim=64, chunk=70)], width=64, vocab=70)
  w = bo.random_weights(cfg, 9)
  a, b = (check(cfg, w, bu.oracle_logits, [200], 200, page) for page in (64, 8))
  assert lu.row_err(a, b) < lu.TOL["bfloat16"] / 4              # the same operands and 16-bit pairs of weights: rounding of the outputs


def test_scores_that_rise_along_the_keys():
  """a score scale that makes late keys dominate: the running maximum grows by far more than the step at which the output is rescaled"""
  cfg = bu.config([bu.attention(heads=2, kv_heads=1, dim=64, vdim=64, chunk=None, scale=4.0, softcap=None)], width=64, vocab=70)
  check(cfg, bo.random_weights(cfg, 2), bu.oracle_logits, [400], 400)

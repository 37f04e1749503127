"""The element kernels around the mixers of a prompt in 16-byte pieces: convolution, unit vectors and decays in one pass (one to four taps; five take the kernels before), head norm and
gate, query / key / value preparation — at the head sizes that they take and beside them, with steps cut so that a filter's window is carried on from every side (portions of 128 and
more rows, of 1, 2, 3, and some that stay under the line), 32-bit engine against the float64 oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tests import bufulorn_oracle as bo, bufulorn_util as bu, layered_util as lu


@pytest.mark.parametrize("cut", [[128, 1, 2, 130], [1, 132, 3, 129], [2, 131, 128, 1], [96, 3, 127, 128], [256, 2, 240, 1]])
@pytest.mark.parametrize("dim,vdim,conv", [(64, 64, 1), (64, 64, 2), (64, 64, 3), (128, 128, 4), (64, 64, 5), (64, 128, 4), (68, 68, 4)])
def test_gated_delta_in_portions(dim, vdim, conv, cut):
  cfg = bu.config([bu.delta(heads=4, kv_heads=2, dim=dim, vdim=vdim, conv=conv)], width=48, vocab=50)
  w = bo.random_weights(cfg, dim + conv)
  cuts = [cut, [cut[0] + 1, *cut[1:]]]                 # the second request is a row ahead after the first portion
  toks = [lu.rand_tokens(50, sum(c), 3 + r) for r, c in enumerate(cuts)]
  eng = lu.make_engine(cfg, w, "float32", max_tokens=1024, max_requests=2)
  got, at = [[], []], [0, 0]
  for portion in zip(*cuts):
    rows = [t[a:a + n] for t, a, n in zip(toks, at, portion)]
    lg = eng.step([1, 0], rows, want=list(range(sum(portion))))[0]
    for g, part in zip(got, np.split(lg, [portion[0]])):
      g.append(part)
    at = [a + n for a, n in zip(at, portion)]
  eng.close()
  for t, g in zip(toks, got):
    assert lu.row_err(np.concatenate(g), bu.oracle_logits(cfg, w, t)[0]) < 2.4e-5   # as in the chunk tests


@pytest.mark.parametrize("dim,vdim", [(64, 64), (128, 128), (124, 60), (132, 64), (66, 64)])
@pytest.mark.parametrize("rows", [1, 70])
def test_queries_keys_values(dim, vdim, rows):
  cfg = bu.config([bu.attention(heads=6, kv_heads=2, dim=dim, vdim=vdim, chunk=None), bu.attention(heads=4, kv_heads=2, dim=dim, vdim=vdim, kv_from=0)], width=48, vocab=50)
  w = bo.random_weights(cfg, dim)
  t = lu.rand_tokens(50, rows, 2)
  for dtype in ("float32", "bfloat16"):
    eng = lu.make_engine(cfg, w, dtype, max_tokens=256)
    assert lu.row_err(eng.step([0], [t], want=list(range(rows)))[0], bu.oracle_logits(cfg, w, t)[0]) < lu.TOL[dtype], dtype
    eng.close()

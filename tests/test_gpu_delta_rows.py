"""Steps of one row per request, from the first token on: the one-launch form of the delta-rule mixers at the edges of what it holds — head sizes up to 128 that are whole
pieces of four, filters of 1 to 9 taps (8 are held), 1 to 9 value heads per key head (a cluster holds 8), low-rank branches of odd and of wide sizes — 32-bit engine
against the float64 oracles.  Bound: 12 tokens of sums over at most 300 terms, 2^-24 sqrt(12 x 300) = 3.6e-6 of a row if all were as large as the result; four times that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tests import bufulorn_oracle as bo, bufulorn_util as bu, layered_util as lu, zokuvik_oracle as zo

BOUND = 1.5e-5


def check(cfg, w, oracle, n_req=2, n=12):
  eng = lu.make_engine(cfg, w, "float32", max_tokens=n_req * 64, max_requests=n_req)
  toks = [lu.rand_tokens(cfg["vocab"], n, 11 + r) for r in range(n_req)]
  order = list(range(n_req))[::-1]                     # rows are not in the order of the slots
  got = np.stack([eng.step(order, [toks[r][t:t + 1] for r in order])[0] for t in range(n)])
  eng.close()
  for i, r in enumerate(order):
    assert lu.row_err(got[:, i], oracle(cfg, w, toks[r])[0]) < BOUND, r


@pytest.mark.parametrize("dim", [4, 12, 60, 64, 68, 128, 132])
@pytest.mark.parametrize("rank", [1, 7, 64, 256, 260])
def test_general_rule(dim, rank):
  cfg = lu.config([lu.delta(heads=3, dim=dim, decay_rank=rank)], width=48, vocab=50)
  check(cfg, zo.random_weights(cfg, dim), lu.oracle_logits)


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,conv", [(4, 2, 64, 64, 1), (4, 2, 64, 64, 2), (4, 2, 64, 64, 4), (4, 2, 64, 64, 8), (4, 2, 64, 64, 9), (3, 3, 4, 8, 4), (8, 1, 64, 60, 4),
                                                          (9, 1, 64, 64, 4), (6, 2, 128, 128, 4), (4, 2, 68, 128, 3), (4, 2, 128, 12, 4), (4, 2, 64, 62, 4)])
def test_gated_rule(heads, kv_heads, dim, vdim, conv):
  cfg = bu.config([bu.delta(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, conv=conv)], width=48, vocab=50)
  check(cfg, bo.random_weights(cfg, dim + vdim), bu.oracle_logits, n_req=5)

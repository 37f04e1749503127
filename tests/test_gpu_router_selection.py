"""Softmax routers with up to 32 experts choose with a warp, more with one lane: both must choose what the definition says (groups' best scores, ties to the lower index) and weigh the chosen by
their scores, for expert counts around a warp, every number of groups and of kept groups, and scores with ties.  Every expert has matrices of its own, so a choice shows in the
output; the oracle's own order among equals is not defined, which is why the first test cuts no pair of equals and the second states the order itself."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from tests import bufulorn_oracle as bo, bufulorn_util as bu, layered_util as lu


@pytest.mark.parametrize("experts,groups,keep,top", [(1, 1, 1, 1), (3, 1, 1, 2), (8, 4, 2, 2), (16, 8, 4, 4), (16, 4, 1, 3), (31, 1, 1, 5), (32, 16, 9, 6), (32, 2, 2, 4), (33, 3, 2, 4), (48, 8, 3, 6)])
@pytest.mark.parametrize("ties", [False, True])
def test_choice(experts, groups, keep, top, ties):
  if ties and experts > 1:
    top += top % 2                                     # whole pairs: the oracle's order among equals is not defined, which of a pair is cut off would be a matter of luck
  cfg = bu.config([bu.attention(mlp=bu.moe(experts=experts, top=top, groups=(groups, keep), ff=16))], width=32, vocab=60)
  w = bo.random_weights(cfg, experts + top)
  if ties:                                             # pairs of experts with the same scores, and the same matrices' results told apart by their index
    w["l0.mlp.router"] = w["l0.mlp.router"].clone()
    for e in range(0, experts - 1, 2):
      w["l0.mlp.router"][e + 1] = w["l0.mlp.router"][e]
  toks = lu.rand_tokens(60, 12, 3)
  ref = bu.oracle_logits(cfg, w, toks)[0]
  eng = lu.make_engine(cfg, w, "float32")
  whole = eng.step([0], [toks], want=list(range(12)))[0]
  single = np.concatenate([eng.step([1], [toks[i:i + 1]])[0] for i in range(12)])
  eng.close()
  ok = [lu.row_err(g, ref) < lu.TOL["float32"] for g in (whole, single)]
  assert all(ok)


def lower_index_first(h, w_router, r):
  """the definition with its order among equals: sorts that keep equals in place, and logits whose sums do not depend on where a row of the router lies"""
  E, top, gr = r["experts"], r["top"], r.get("groups")
  s = torch.softmax((h[:, None, :] * w_router[None]).sum(-1), dim=-1)
  free = torch.ones_like(s, dtype=torch.bool)
  if gr and gr["count"] > 1:
    best = s.reshape(-1, gr["count"], E // gr["count"]).amax(-1)
    kept = torch.zeros_like(best, dtype=torch.bool).scatter_(1, best.sort(dim=-1, descending=True, stable=True).indices[:, :gr["keep"]], True)
    free = kept.repeat_interleave(E // gr["count"], dim=1)
  idx = s.masked_fill(~free, -1.0).sort(dim=-1, descending=True, stable=True).indices[:, :top]
  return idx, s.gather(1, idx)


@pytest.mark.parametrize("equals", ["pairs", "groups", "all"])
@pytest.mark.parametrize("experts,groups,keep,top", [(8, 1, 1, 3), (8, 4, 2, 3), (16, 4, 2, 5), (16, 8, 3, 1), (31, 1, 1, 5), (32, 4, 3, 7), (32, 16, 5, 3), (48, 6, 2, 5), (64, 1, 1, 3)])
def test_ties_go_to_the_lower_index(experts, groups, keep, top, equals, monkeypatch):
  """equal scores: an expert and its neighbour (top cuts a pair), a group and all others (kept is less than their number), all experts"""
  cfg = bu.config([bu.attention(mlp=bu.moe(experts=experts, top=top, groups=(groups, keep), ff=16))], width=32, vocab=60)
  w = bo.random_weights(cfg, experts + top)
  own = {"pairs": torch.arange(experts) // 2 * 2, "groups": torch.arange(experts) % (experts // groups), "all": torch.zeros(experts, dtype=torch.long)}[equals]
  w["l0.mlp.router"] = w["l0.mlp.router"][own].clone()
  toks = lu.rand_tokens(60, 12, 3)
  monkeypatch.setattr(bo, "route", lower_index_first)
  ref = bu.oracle_logits(cfg, w, toks)[0]
  eng = lu.make_engine(cfg, w, "float32")
  whole = eng.step([0], [toks], want=list(range(12)))[0]
  single = np.concatenate([eng.step([1], [toks[i:i + 1]])[0] for i in range(12)])
  eng.close()
  assert lu.row_err(whole, ref) < lu.TOL["float32"] and lu.row_err(single, ref) < lu.TOL["float32"]

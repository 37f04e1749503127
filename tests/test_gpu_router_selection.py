"""Softmax routers with up to 32 experts choose with a warp, more with one lane: both must choose what the definition says (groups' best scores, ties to the lower index), bit for bit the
same weights, for expert counts around a warp, every number of groups and of kept groups, and scores with ties."""

import numpy as np
import pytest

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

"""Tokens that are not finite stay in the sums of the single-row attention kernels: a row that sees them is not finite, whichever warp, lanes or share of the keys they fall to —
also where a warp or a share sees nothing else — and however many shares there are; its neighbours in the batch are."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tests import bufulorn_oracle as bo, bufulorn_util as bu, layered_util as lu, zokuvik_oracle as zo

BAD = 69


def models(requests, dtype):
  yield bu.config([bu.attention(heads=8, kv_heads=2, dim=64, vdim=64, chunk=None)], vocab=70, max_positions=4000), bo
  wide = 64 if dtype == "bfloat16" else 32
  for heads in (8, 64):                                # more shares than a cluster holds, and a cluster's (three requests)
    yield lu.config([lu.attn(heads=heads, dim=16, rot_dim=wide, vdim=16, kv_rank=256)], vocab=70), zo


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("first,last", [(0, 4), (4, 8), (8, 9), (0, 9)])
def test_rows_that_see_them(first, last, dtype):
  for cfg, oracle in models(3, dtype):
    w = oracle.random_weights(cfg, 3)
    w["embed"] = w["embed"].clone()
    w["embed"][BAD] = float("nan")
    eng = lu.make_engine(cfg, w, dtype, max_tokens=1024, max_requests=3)
    toks = [lu.rand_tokens(BAD, 60, r) for r in range(3)]
    toks[1][first:last] = BAD
    eng.step([0, 1, 2], [t[:10] for t in toks])
    for i in range(10, 60):
      got = eng.step([0, 1, 2], [t[i:i + 1] for t in toks])[0]
      assert np.isfinite(got[[0, 2]]).all() and not np.isfinite(got[1]).any(), i
    eng.close()

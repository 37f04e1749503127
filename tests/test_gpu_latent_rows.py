"""Steps of one row per request over latents of 256 or 512 entries take a kernel of their own; steps of two rows per request keep the general one.  Both must give the same rows: gates,
windows, sinks, head counts that are no whole group of eight, rotated parts of every width that the kernel holds and one that it does not, caches from nothing to more shares of the
keys than a cluster holds.

Bound, 32 bits: sums over at most 2600 keys x 288 entries in another order, 2^-24 sqrt(2600 x 288) = 5.2e-5 of a row if all were as large as the result; twice that.  In 16 bits the products around
the attention round to 8 bits on both sides: 2^-8, twice."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tests import layered_util as lu, rinutar_oracle as ro, rinutar_util as ru, zokuvik_oracle as zo

BOUND = {"float32": 1.05e-4, "bfloat16": 2 ** -7}


def models(rank, dtype):
  wide = 64 if dtype == "bfloat16" else 32
  yield "gate and window", lu.config([lu.attn(heads=8, dim=16, rot_dim=wide, vdim=16, kv_rank=rank), lu.attn("latent_attention_2", heads=3, dim=16, rot_dim=wide // 2, vdim=16, kv_rank=rank, window=45)]), zo
  yield "11 heads, no whole pieces", lu.config([lu.attn(heads=11, dim=16, rot_dim=8, vdim=16, kv_rank=rank), lu.attn(heads=3, dim=16, rot_dim=4, vdim=16, kv_rank=rank)]), zo
  yield "sink", ru.config([ru.attn(heads=9, dim=16, rot_dim=16, vdim=16, kv_rank=rank)]), ro


@pytest.mark.parametrize("rank,dtype", [(256, "float32"), (256, "bfloat16"), (512, "bfloat16")])
@pytest.mark.parametrize("n", [1, 4, 15, 16, 17, 70, 400, 2600])
def test_one_row_against_two(n, rank, dtype):
  for name, cfg, oracle in models(rank, dtype):
    w = oracle.random_weights(cfg, rank + n)
    requests = 1 if n > 1000 else 3
    eng = lu.make_engine(cfg, w, dtype, max_tokens=2 * requests * (n + 80), max_requests=2 * requests, page_size=16)
    toks = [lu.rand_tokens(cfg["vocab"], n + 4, 3 + r) for r in range(requests)]
    pairs, singles = list(range(requests)), list(range(requests, 2 * requests))
    for slots in (pairs, singles):
      eng.step(slots, [t[:n] for t in toks])
    for at in (n, n + 2):
      ref = eng.step(pairs, [t[at:at + 2] for t in toks], want=list(range(2 * requests)))[0].reshape(requests, 2, -1)
      got = np.stack([eng.step(singles, [t[at + i:at + i + 1] for t in toks])[0] for i in range(2)], axis=1)
      assert lu.row_err(got.reshape(2 * requests, -1), ref.reshape(2 * requests, -1)) < BOUND[dtype], (name, at)
    eng.close()

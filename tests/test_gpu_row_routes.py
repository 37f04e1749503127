"""The lines at which single rows leave the row kernels for the general ones: behind 128 tokens for latents whose heads are one block a request, from blocks x keys = 3200 on for more, behind
256 tokens where many heads share a key head.  Rows on both sides of a line must be the same rows — against the general kernels, which take two rows at a time — with steps
captured and without (a captured step must be one of its own side of the line, and cuts the keys for a length rounded up); in 32 bits they must be the float64 oracle's too.

Bounds as for the row kernels themselves: sums over at most 420 keys x 288 entries in another order, 2^-24 sqrt(420 x 288) = 2.1e-5 of a row if all were as large as the result, twice
that; in 16 bits the products around the attention round to 8 bits on both sides, 2^-8, twice."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tests import bufulorn_oracle as bo, bufulorn_util as bu, layered_util as lu, zokuvik_oracle as zo

BOUND = {"float32": 4.2e-5, "bfloat16": 2 ** -7}


def model(kind, dtype):
  wide = 64 if dtype == "bfloat16" else 32
  if kind == "one block":                              # the line: 128 keys; a cluster's shares on its near side, one launch, and runs and a merge beyond
    return lu.config([lu.attn(heads=8, dim=16, rot_dim=wide, vdim=16, kv_rank=256)]), zo, 2, 128
  if kind == "blocks x keys":                          # 4 requests of 2 blocks: 400 keys; a layer with a window of 45 stays
    return lu.config([lu.attn(heads=16, dim=16, rot_dim=wide, vdim=16, kv_rank=256), lu.attn("latent_attention_2", heads=16, dim=16, rot_dim=wide, vdim=16, kv_rank=256, window=45)]), zo, 4, 400
  return bu.config([bu.attention(heads=16, kv_heads=1, dim=128, vdim=128, chunk=None), bu.attention(heads=8, kv_heads=1, dim=128, vdim=128, chunk=None)], max_positions=600), bo, 4, 256


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("kind", ["one block", "blocks x keys", "shared key heads"])
def test_rows_on_both_sides_of_a_line(kind, dtype):
  cfg, oracle, requests, line = model(kind, dtype)
  w = oracle.random_weights(cfg, line)
  eng = lu.make_engine(cfg, w, dtype, max_tokens=2 * requests * (line + 64), max_requests=2 * requests, page_size=16)
  toks = [lu.rand_tokens(cfg["vocab"], line + 8, 3 + r) for r in range(requests)]
  pairs, singles, start = list(range(requests)), list(range(requests, 2 * requests)), line - 8

  def serve(slots, rows):
    for s in slots:
      eng.clear_request(s)
    eng.step(slots, [t[:start] for t in toks])
    out, launches = [], []
    for at in range(start, line + 8, rows):
      before = eng.kernel_launches()
      lg = eng.step(slots, [t[at:at + rows] for t in toks], want=list(range(rows * requests)))[0]
      launches.append(eng.kernel_launches() - before)
      out.append(lg.reshape(requests, rows, -1))
    return np.concatenate(out, axis=1), launches

  ref, _ = serve(pairs, 2)
  eng.set_graphs(False)
  plain, launches = serve(singles, 1)
  eng.set_graphs(True)
  replays = eng.graph_replays()
  first, _ = serve(singles, 1)
  again, _ = serve(singles, 1)
  assert eng.graph_replays() > replays + 16
  eng.close()
  # the step that makes a request `line` tokens long is the last on the near side
  assert len(set(launches[:8])) == 1 and len(set(launches[8:])) == 1
  if kind != "blocks x keys":
    assert launches[8] == launches[7] + 1
  flat = lambda x: x.reshape(-1, x.shape[-1])            # noqa: E731
  for got in (plain, first, again):
    assert lu.row_err(flat(got), flat(ref)) < BOUND[dtype]
  if dtype == "float32":
    for r in range(requests):
      assert lu.row_err(plain[r], (bu if oracle is bo else lu).oracle_logits(cfg, w, toks[r])[0][start:]) < lu.TOL[dtype]

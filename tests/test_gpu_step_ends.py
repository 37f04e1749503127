"""The two ends of a step: index arrays and page table entries come in, logits, argmax and the error word go out through page-locked memory that the kernels
read and write.  Wherever the caller's logits lie — a block of the library's page-locked memory, somebody else's page-locked memory, ordinary memory, nowhere —
a step must leave the same bits there, at vocabularies that one block takes, that a cluster shares, and whose rows are not whole 16-byte pieces."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from tests import fekanex_oracle as fo, fekanex_util as fu, layered_util as lu, zokuvik_oracle as zo
from xotorch_b200 import _lib


def address(a):
  return a.__array_interface__["data"][0]


def step_into(eng, slots, rows, want, logits_at):
  """one step through the C entry: argmax"""
  ints = lambda v: np.ascontiguousarray(v, dtype=np.int32)               # noqa: E731
  sl, counts, tok, wn, am = ints(slots), ints([len(r) for r in rows]), ints(np.concatenate(rows)), ints(want), np.full(len(want), -1, np.int32)
  _lib.check_lm(eng.lib.xotb200_lm_step(eng.h, len(slots), address(sl), address(counts), address(tok), None, address(wn), len(want), logits_at, address(am), None))
  return am


@pytest.mark.parametrize("scaled", [False, True])
@pytest.mark.parametrize("vocab", [70, 4095, 4096, 5003, 32004])
def test_logits_in_every_kind_of_memory(vocab, scaled):
  if scaled:                                           # logits are changed on their way out
    cfg = fu.config([fu.attn(heads=2, kv_heads=1, dim=16, vdim=16)], width=64, vocab=vocab)
    cfg["logit_scale"] = 0.25
    eng = lu.make_engine(cfg, fo.random_weights(cfg, 3), "bfloat16", max_tokens=256, max_requests=3)
  else:
    cfg = lu.config([lu.attn()], vocab=vocab)
    eng = lu.make_engine(cfg, zo.random_weights(cfg, 3), "bfloat16", max_tokens=256, max_requests=3)
  schedule = [([0, 1, 2], [[1, 2, 3], [4, 5], [6]], [0, 2, 5])] + [([0, 1, 2], [[7 + s], [8 + s], [9 + s]], [0, 1, 2]) for s in range(4)] + [([1], [[5]], [0])]

  def serve(kind):
    for r in range(3):
      eng.clear_request(r)
    out = []
    for slots, rows, want in schedule:
      n = len(want) * vocab
      if kind == "block":
        p = C.c_void_p()
        _lib.check_lm(eng.lib.xotb200_lm_host_alloc(0, n * 4 + 64, C.byref(p)))
        buf = np.frombuffer((C.c_float * (n + 16)).from_address(p.value), dtype=np.float32)
      else:
        buf = torch.zeros(n + 16, pin_memory=kind == "foreign").numpy()
      buf[:] = 7.0
      am = step_into(eng, slots, [np.array(r) for r in rows], want, None if kind == "nowhere" else address(buf))
      got = buf[:n].copy().reshape(len(want), vocab)
      assert (buf[n if kind != "nowhere" else 0:] == 7.0).all()              # nothing beyond
      if kind == "block":
        del buf
        _lib.check_lm(eng.lib.xotb200_lm_host_free(0, p))
      out.append((got, am))
    return out

  ref = serve("plain")
  for got, am in ref:
    assert np.isfinite(got).all() and np.array_equal(am, got.argmax(axis=1))
  for kind in ("block", "foreign", "nowhere", "block"):
    for (a, ia), (b, ib) in zip(ref, serve(kind)):
      assert np.array_equal(ia, ib), kind
      assert kind == "nowhere" or np.array_equal(a, b), kind
  eng.close()


def test_pages_added_by_single_row_and_by_mixed_steps():
  """pages of 4 tokens: every few steps some of the requests start a page, in steps of one row each (replayed) and in steps of several"""
  cfg = lu.config([lu.attn(), lu.attn("latent_attention_2", window=6)])
  w = zo.random_weights(cfg, 9)
  out = []
  for page in (4, 64):
    eng = lu.make_engine(cfg, w, "float32", max_tokens=200, max_requests=3, page_size=page)
    rng, got = np.random.default_rng(1), []
    for s in range(24):
      rows = [rng.integers(0, 80, size=1 if s % 5 else 1 + 3 * r) for r in range(3)]
      got.append(eng.step([2, 0, 1], rows)[0])
    out.append(np.stack(got))
    eng.close()
  assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("short", [0, 1, 2, 3])
@pytest.mark.parametrize("extra", [1, 2])
def test_staged_arrays_that_end_where_their_buffer_does(extra, short):
  """the staged block grows to twice what a step needs, in whole 16-byte pieces, which is also what a step copies: steps that need all of it, and up to three ints less"""
  cfg = lu.config([lu.delta(heads=1, dim=8)], width=48, vocab=50)
  w, page, rows = zo.random_weights(cfg, 2), 64, 1000

  def ints(rows, want):                                # result pointers, tokens, slots and positions, wanted rows, one request, its new pages
    return 4 + 3 * rows + want + 4 + 2 * -(-rows // page)

  first = ints(rows, extra)
  size = (2 * first + 3) // 4 * 4
  long = max(m for m in range(rows, 4 * rows) if ints(m, 1) <= size - short)
  want = 1 + size - short - ints(long, 1)
  assert first > 2048 and ints(long, want) == size - short and want <= long
  toks, got = lu.rand_tokens(50, long, 5), []
  for grown in (False, True):
    eng = lu.make_engine(cfg, w, "float32", max_tokens=4 * rows, max_requests=1, page_size=page)
    if grown:
      eng.step([0], [lu.rand_tokens(50, rows, 6)], want=list(range(extra)))
      eng.clear_request(0)
    got.append(eng.step([0], [toks], want=list(range(long - want, long)))[0])
    eng.close()
  assert np.isfinite(got[0]).all() and np.array_equal(*got)


def test_more_wanted_rows_than_a_grid_is_high():
  """scoring every token of a long text: all rows of one step against the same rows in portions.  Bound: sums over 48 terms through
  a state that forgets within tens of tokens, 2^-24 sqrt(48 x 40) = 2.6e-6 of a row if all were as large as the result; four times that"""
  cfg = lu.config([lu.delta(heads=1, dim=8)], width=48, vocab=70)
  n = 70000
  eng = lu.make_engine(cfg, zo.random_weights(cfg, 4), "float32", max_tokens=2 * n + 256, max_requests=2, page_size=64)
  toks = lu.rand_tokens(70, n, 8)
  whole, best = eng.step([0], [toks], want=list(range(n)))
  assert whole.shape == (n, 70) and np.array_equal(best, whole.argmax(axis=1))
  parts = np.concatenate([eng.step([1], [p], want=list(range(len(p))))[0] for p in np.split(toks, 5)])
  eng.close()
  assert np.isfinite(whole).all() and lu.row_err(whole, parts) < 1e-5


@pytest.mark.parametrize("vocab", [4096, 5003])
def test_rows_shared_by_a_cluster_and_rows_of_one_block(vocab):
  """as many wanted rows as SMs go to clusters, more to a block each; the head's product may tile 148 and 157 rows otherwise, so 2^-24 sqrt(48) = 4.1e-7 of
  a row, twice"""
  cfg = lu.config([lu.delta(heads=1, dim=8)], width=48, vocab=vocab)
  sms = torch.cuda.get_device_properties(0).multi_processor_count
  eng = lu.make_engine(cfg, zo.random_weights(cfg, 4), "float32", max_tokens=2048, max_requests=2)
  toks, got = lu.rand_tokens(vocab, sms + 9, 8), []
  for n in (sms, sms + 1, sms + 9):
    eng.clear_request(0)
    lg, best = eng.step([0], [toks], want=list(range(n)))
    eng.clear_request(0)
    alone = eng.step([0], [toks], want=list(range(n)), logits=False)[1]
    assert np.array_equal(best, lg.argmax(axis=1)) and np.array_equal(best, alone)
    got.append(lg[:sms].copy())
  eng.close()
  assert np.isfinite(got[0]).all() and all(lu.row_err(g, got[0]) < 1e-6 for g in got)

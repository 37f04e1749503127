"""What `LayeredShard.step` hands to the native step: slots, row counts and wanted rows as 32-bit ints, the rows packed, addresses that are alive during the call."""
import ctypes as C

import numpy as np
import pytest

from xotorch_b200.layered import LayeredShard
from xotorch_b200.pinned import ResultPool


class FakeLib:
  def __init__(self, hidden_in=0):
    self.seen, self.hidden_in = None, hidden_in

  def xotb200_lm_step(self, h, n_seq, slots, counts, tokens, hidden, want, n_want, logits, argmax, hidden_out):
    ints = lambda p, n: np.frombuffer((C.c_int32 * max(n, 1)).from_address(p), np.int32, n).tolist()   # noqa: E731
    cs = ints(counts, n_seq)
    data = ints(tokens, sum(cs)) if tokens else np.frombuffer((C.c_float * (sum(cs) * self.hidden_in)).from_address(hidden), np.float32).tolist()
    self.seen = (ints(slots, n_seq), cs, data, ints(want, n_want), bool(logits), bool(argmax), bool(hidden_out))
    return 0


def shard(first=True, last=True):
  s = object.__new__(LayeredShard)
  s.lib, s.h, s.n_layers, s.globals = FakeLib(3), None, 3, {"vocab": 5, "width": 3}
  s.start, s.end = 0 if first else 1, 2 if last else 1
  s.hidden_in = s.hidden_out = 3
  s.results = ResultPool(lambda n: None, lambda p: None)
  return s


@pytest.mark.parametrize("rows", [[[1, 2, 3], [4], [5, 6]], [np.array([1, 2, 3]), np.array([[4]]), np.array([5, 6], np.int32)], [np.arange(1, 7, dtype=np.int32)[:3], (4,), np.array([9, 5, 6, 8], np.int32)[1:3]]])
@pytest.mark.parametrize("slots", [[7, 0, 3], (7, 0, 3), np.array([7, 0, 3])])
def test_tokens(rows, slots):
  s = shard()
  lg, am = s.step(slots, rows)
  assert s.lib.seen == ([7, 0, 3], [3, 1, 2], [1, 2, 3, 4, 5, 6], [2, 3, 5], True, True, False) and lg.shape == (3, 5) and am.shape == (3,) and am.dtype == np.int32
  for want in ([4, 0], np.array([4, 0]), (4, 0)):
    lg, am = s.step(slots, rows, want=want, argmax=False)
    assert s.lib.seen[3:] == ([4, 0], True, False, False) and lg.shape == (2, 5) and am is None
  one = s.step([2], [np.arange(12, dtype=np.int32)[::3]], logits=False)          # strided
  assert s.lib.seen == ([2], [4], [0, 3, 6, 9], [3], False, True, False) and one[0] is None


def test_hidden_rows_and_a_row_list_too_short():
  s = shard(first=False, last=False)
  out = s.step([1, 0], [np.arange(6).reshape(2, 3), np.ones(3, np.float64)])
  assert s.lib.seen == ([1, 0], [2, 1], [0, 1, 2, 3, 4, 5, 1, 1, 1], [], False, False, True) and out.shape == (3, 3)
  with pytest.raises(ValueError):
    s.step([1, 0], [np.ones(3)])


@pytest.mark.parametrize("want", [[[4, 0]], [[4], [0]], ((4,), (0,)), [np.int64(4), np.int32(0)], [np.array([4, 0])], np.array([[4], [0]]), [4.0, 0.0]])
def test_wanted_rows_of_any_shape(want):
  s = shard()
  lg, am = s.step([7, 0, 3], [[1, 2, 3], [4], [5, 6]], want=want)
  assert s.lib.seen[3] == [4, 0] and lg.shape == (2, 5) and am.shape == (2,)


def test_slots_in_a_column():
  s = shard()
  s.step(np.array([[7], [0]]), [[1, 2, 3], [4]])
  assert s.lib.seen[:4] == ([7, 0], [3, 1], [1, 2, 3, 4], [2, 3])


def test_rows_beyond_the_slots_are_not_served():
  s = shard()
  lg, _ = s.step([7, 0], [[1, 2, 3], [4], [5, 6]], want=[3, 2])
  assert s.lib.seen[:4] == ([7, 0], [3, 1], [1, 2, 3, 4], [3, 2]) and lg.shape == (2, 5)
  s.step([7, 0], [[1, 2, 3], [4], [5, 6]])               # the last rows of all three: the native step refuses the one that is not there
  assert s.lib.seen[3] == [2, 3, 5]
  s.step([7], [[1, 2], [4]])
  assert s.lib.seen[:3] == ([7], [2], [1, 2])
  s = shard(first=False, last=False)
  out = s.step([1], [np.arange(6).reshape(2, 3), np.ones(3)])
  assert s.lib.seen[:3] == ([1], [2], [0, 1, 2, 3, 4, 5]) and out.shape == (3, 3)

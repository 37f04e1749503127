"""The pool of page-locked result arrays, over a stand-in allocator: blocks come back when the last view of an array is gone, the bound holds, threads
take and give back side by side."""
import ctypes as C
import gc
import threading

import numpy as np

from xotorch_b200.pinned import SMALLEST, ResultPool


class Heap:
  def __init__(self):
    self.blocks, self.most = {}, 0

  def alloc(self, size):
    b = (C.c_char * size)()
    self.blocks[C.addressof(b)] = b
    self.most = max(self.most, sum(len(x) for x in self.blocks.values()))
    return C.addressof(b)

  def free(self, addr):
    del self.blocks[addr]


def test_blocks_are_reused_after_the_last_view_and_never_before():
  heap = Heap()
  pool = ResultPool(heap.alloc, heap.free, limit=8 * SMALLEST)
  a = pool.empty((2, SMALLEST // 8))
  a[:] = 1.0
  view = a[1:]
  addr = a.ctypes.data
  del a
  gc.collect()
  b = pool.empty((2, SMALLEST // 8))
  assert b.ctypes.data != addr                       # the view still holds the first block
  b[:] = 2.0
  assert (view == 1.0).all()
  del view
  gc.collect()
  assert pool.empty((2, SMALLEST // 8)).ctypes.data == addr
  assert pool.empty((4,)).size == 4 and len(heap.blocks) == 2   # small results are ordinary arrays


def test_the_bound_holds_and_blocks_of_other_sizes_make_room():
  heap = Heap()
  pool = ResultPool(heap.alloc, heap.free, limit=4 * SMALLEST)
  held = [pool.empty((SMALLEST,), np.uint8) for _ in range(6)]
  assert len(heap.blocks) == 4 and all(h.size == SMALLEST for h in held)
  del held
  gc.collect()
  big = pool.empty((4 * SMALLEST,), np.uint8)        # the four small blocks go
  assert list(len(b) for b in heap.blocks.values()) == [4 * SMALLEST] and big.size == 4 * SMALLEST
  assert pool.empty((5 * SMALLEST,), np.uint8).size == 5 * SMALLEST and heap.most <= 4 * SMALLEST
  none = ResultPool(lambda size: None, heap.free)
  assert none.empty((3, SMALLEST)).shape == (3, SMALLEST)


def test_threads_do_not_share_a_block():
  heap = Heap()
  pool = ResultPool(heap.alloc, heap.free, limit=64 * SMALLEST)
  bad = []

  def work(k):
    for i in range(200):
      a = pool.empty((SMALLEST // 4,), np.int32)
      a[:] = k * 1000 + i
      if not (a == k * 1000 + i).all():
        bad.append((k, i))
  threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
  [t.start() for t in threads], [t.join() for t in threads]
  assert not bad


def test_blocks_are_taken_and_freed_under_the_device_of_their_engine():
  """an array is asked for before the step makes the engine's device current: the allocation names it, in any thread"""
  from xotorch_b200 import _lib
  calls = []

  class Library:
    heap = Heap()

    def x_host_alloc(self, device, size, out):
      calls.append(("alloc", device.value, threading.get_ident()))
      out._obj.value = self.heap.alloc(size.value)
      return 0

    def x_host_free(self, device, p):
      calls.append(("free", device.value, threading.get_ident()))
      self.heap.free(p.value)
      return 0
  lib = Library()
  pools = [_lib.results(lib, "x", d) for d in (0, 3)]
  assert pools[0] is not pools[1] and _lib.results(lib, "x", 3) is pools[1]
  t = threading.Thread(target=lambda: pools[1].empty((SMALLEST,)))
  t.start(), t.join()
  assert [c[:2] for c in calls] == [("alloc", 3)] and calls[0][2] != threading.get_ident()
  gc.collect()
  pools[1].limit = 8 * SMALLEST
  pools[1].empty((8 * SMALLEST,), np.uint8)          # the smaller block makes room
  assert [c[:2] for c in calls] == [("alloc", 3), ("free", 3), ("alloc", 3)]
  for lm in (False, True):                           # both engines' signatures take the device first
    for name in ("host_alloc", "host_free"):
      assert (_lib._LM_SIGS if lm else _lib._SIGS)[("xotb200_lm_" if lm else "xotb200_") + name][1][0] is C.c_int

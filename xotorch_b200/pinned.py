"""Result arrays in page-locked host memory.

A step's results (logits, hidden states) reach the host over PCIe.  Into an ordinary numpy array that takes a staging buffer and a second copy on the CPU — and, for a
fresh array, the page faults of its memory; into page-locked memory they go directly: hidden states, and the shard engine's logits, by DMA, the layered engine's logits
by the stores of its last kernel, which takes blocks of this library alone (their bounds are known).  `ResultPool.empty` hands out ordinary numpy arrays over
page-locked blocks: when the last reference to an array (or a view of it) is gone, its block goes back to the pool and is handed out again.
The pool is bounded (`limit` bytes in use and kept together; beyond it, and where page-locked memory cannot be had, plain arrays are handed out),
blocks are taken and given back by any thread, and an array outlives the engine that filled it."""
from __future__ import annotations

import ctypes as C
import math
import threading
import weakref
from collections import deque
from typing import Callable, Dict, List, Optional

import numpy as np

SMALLEST = 64 * 1024          # smaller results are cheaper copied than managed


class ResultPool:
  def __init__(self, alloc: Callable[[int], Optional[int]], free: Callable[[int], None], limit: int = 64 << 20):
    self._alloc, self._free, self.limit = alloc, free, int(limit)
    self._lock = threading.Lock()
    self._kept: Dict[int, List[int]] = {}         # block size -> addresses of blocks not in use
    self._returned: deque = deque()               # (address, size) of blocks whose arrays have died: appended by finalizers, which take no lock
    self.total = 0                                # bytes of all blocks

  def _collect(self) -> None:
    while self._returned:
      addr, size = self._returned.popleft()
      self._kept.setdefault(size, []).append(addr)

  def _block(self, size: int) -> Optional[int]:
    with self._lock:
      self._collect()
      kept = self._kept.get(size)
      if kept:
        return kept.pop()
      if self.total + size > self.limit:          # make room: blocks of other sizes that nobody uses
        for other, addrs in self._kept.items():
          while addrs and self.total + size > self.limit:
            self._free(addrs.pop())
            self.total -= other
      if self.total + size > self.limit:
        return None
      addr = self._alloc(size)
      if addr:
        self.total += size
      return addr or None

  def empty(self, shape, dtype=np.float32) -> np.ndarray:
    count = math.prod(shape)
    nbytes = count * np.dtype(dtype).itemsize
    size = 1 << max(nbytes - 1, 0).bit_length()
    addr = self._block(size) if nbytes >= SMALLEST else None
    if addr is None:
      return np.empty(shape, dtype=dtype)
    block = (C.c_char * size).from_address(addr)
    weakref.finalize(block, self._returned.append, (addr, size)).atexit = False
    return np.frombuffer(block, dtype=dtype, count=count).reshape(shape)


def library_pool(lib, prefix: str, device: int = 0) -> ResultPool:
  """the pool of page-locked memory that a native library hands out through `<prefix>_host_alloc` / `<prefix>_host_free`.  An array is asked for BEFORE the
  step that fills it has made the engine's device the thread's current one, so the pool names it: memory taken under another would start a context there."""
  alloc_fn, free_fn = getattr(lib, prefix + "_host_alloc", None), getattr(lib, prefix + "_host_free", None)

  def alloc(size: int) -> Optional[int]:
    if alloc_fn is None:
      return None
    p = C.c_void_p()
    return p.value if alloc_fn(C.c_int(device), C.c_int64(size), C.byref(p)) == 0 else None

  return ResultPool(alloc, lambda addr: free_fn(C.c_int(device), C.c_void_p(addr)))

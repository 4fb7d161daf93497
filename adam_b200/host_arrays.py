"""Large result arrays in page-locked host memory.

A copy from the device into an ordinary numpy array goes through the driver's staging buffer at a few GB/s and takes a page
fault for every 4 KB of a fresh array (68 MB of logits: 15 ms and more); into page-locked memory it runs at the link's rate
(1.3 ms).  Locking pages costs as much as it saves, so blocks are kept when their array is garbage collected: at most
``LIMIT`` bytes, the rest is given back to the system.  Pages that are locked are lost to everything else on the machine, so
blocks in use and kept are ``LOCKED_LIMIT`` bytes together at most; beyond it arrays are ordinary ones."""
from __future__ import annotations

import collections
import ctypes
import math
import threading
import weakref

import numpy as np


class HostArrays:
    MIN = 1 << 16                   # smaller arrays are ordinary ones
    LARGE = 1 << 20
    SMALL_LIMIT = 16 << 20          # bytes of the blocks below LARGE, in use or kept
    LIMIT = 512 << 20               # bytes of unused blocks kept
    LOCKED_LIMIT = 1 << 30          # bytes of all blocks: seven results of scoring 128 tokens at a vocabulary of 262144

    def __init__(self, lib):
        self._lib, self._lock = lib, threading.Lock()
        # Blocks whose array is gone.  The finalizer runs wherever the garbage collector does, also inside `empty` in the
        # thread that holds the lock, so it never waits for the lock: it leaves the block here.
        self._returned = collections.deque()
        self._free = []             # (bytes, address)
        self._kept = 0
        self._small = 0             # bytes of the blocks below LARGE
        self._locked = 0            # bytes of all blocks
        self._closed = False

    def empty(self, shape, dtype) -> np.ndarray:
        dtype = np.dtype(dtype)
        n = math.prod(shape) * dtype.itemsize
        if n < self.MIN:
            return np.empty(shape, dtype)
        block = None
        with self._lock:            # the smallest block that holds it and is not half empty
            self._take_back()
            fits = [b for b in self._free if n <= b[0] <= 2 * n]
            if fits:
                block = min(fits)
                self._free.remove(block)
                self._kept -= block[0]
            step = self.LARGE if n >= self.LARGE else self.MIN
            size = (n + step - 1) // step * step
            if block is None:
                while self._free and self._locked + size > self.LOCKED_LIMIT:       # unused ones make room first
                    biggest = max(self._free)
                    self._free.remove(biggest)
                    self._kept -= biggest[0]
                    self._release(biggest)
                if self._locked + size > self.LOCKED_LIMIT or (size < self.LARGE and self._small + size > self.SMALL_LIMIT):
                    return np.empty(shape, dtype)
                self._count(size)
        if block is None:
            address = self._lib.adam_b200_host_alloc(size)
            if not address:
                with self._lock:
                    self._count(-size)
                return np.empty(shape, dtype)
            block = (size, address)
        raw = (ctypes.c_char * n).from_address(block[1])
        # `raw` lives as long as the array or a view of it; at exit the process gives everything back, arrays that live on included
        weakref.finalize(raw, self._give_back, block).atexit = False
        return np.frombuffer(raw, dtype).reshape(shape)

    def _give_back(self, block):
        self._returned.append(block)
        if self._lock.acquire(blocking=False):      # else whoever holds it, or the next call, takes the block back
            try:
                self._take_back()
            finally:
                self._lock.release()

    # ---- under the lock ----
    def _count(self, size):
        self._locked += size
        self._small += size if abs(size) < self.LARGE else 0

    def _release(self, block):
        self._count(-block[0])
        self._lib.adam_b200_host_free(block[1])

    def _take_back(self):
        while self._returned:
            block = self._returned.popleft()
            if not self._closed and self._kept + block[0] <= self.LIMIT:
                self._free.append(block)
                self._kept += block[0]
            else:
                self._release(block)

    def close(self):
        with self._lock:
            self._closed = True
            self._take_back()
            blocks, self._free, self._kept = self._free, [], 0
            for block in blocks:
                self._release(block)

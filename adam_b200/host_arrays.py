"""Large result arrays in page-locked host memory.

A copy from the device into an ordinary numpy array goes through the driver's staging buffer at a few GB/s and takes a page
fault for every 4 KB of a fresh array (68 MB of logits: 15 ms and more); into page-locked memory it runs at the link's rate
(1.3 ms).  Locking pages costs as much as it saves, so blocks are kept when their array is garbage collected: at most
``LIMIT`` bytes, the rest is given back to the system at once."""
from __future__ import annotations

import ctypes
import threading
import weakref

import numpy as np


class HostArrays:
    MIN = 1 << 20                   # smaller arrays are ordinary ones
    LIMIT = 512 << 20               # bytes of unused blocks kept

    def __init__(self, lib):
        self._lib, self._lock = lib, threading.Lock()
        self._free = []             # (bytes, address)
        self._kept = 0
        self._closed = False

    def empty(self, shape, dtype) -> np.ndarray:
        dtype = np.dtype(dtype)
        n = int(np.prod(shape)) * dtype.itemsize
        if n < self.MIN:
            return np.empty(shape, dtype)
        block = None
        with self._lock:            # the smallest block that holds it and is not half empty
            fits = [b for b in self._free if n <= b[0] <= 2 * n]
            if fits:
                block = min(fits)
                self._free.remove(block)
                self._kept -= block[0]
        if block is None:
            size = (n + self.MIN - 1) // self.MIN * self.MIN
            address = self._lib.adam_b200_host_alloc(size)
            if not address:
                return np.empty(shape, dtype)
            block = (size, address)
        raw = (ctypes.c_char * n).from_address(block[1])
        weakref.finalize(raw, self._give_back, block)        # `raw` lives as long as the array or a view of it
        return np.frombuffer(raw, dtype).reshape(shape)

    def _give_back(self, block):
        with self._lock:
            if not self._closed and self._kept + block[0] <= self.LIMIT:
                self._free.append(block)
                self._kept += block[0]
                return
        self._lib.adam_b200_host_free(block[1])

    def close(self):
        with self._lock:
            blocks, self._free, self._kept, self._closed = self._free, [], 0, True
        for _, address in blocks:
            self._lib.adam_b200_host_free(address)

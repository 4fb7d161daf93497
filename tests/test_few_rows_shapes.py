"""Launch shapes of the GEMM for a few rows, chosen on the host: no GPU needed."""
import ctypes
import os
import subprocess
import sys
import time

import pytest

from adam_b200 import _lib

GROUPS, UNITS, SLICES, PAIRS, STAGES, CTAS, SHARED, ITEM, SLOT, SMEM = range(10)


def _shape(ggml_type, n, k, rows, kind, sms=148):
    out = (ctypes.c_uint32 * 10)()
    assert _lib.load().adam_b200_few_rows_shape(ggml_type, n, k, rows, kind, sms, out) == 0
    return list(out)


# Gate / up pairs whose estimate picks shared items of more than 16 row groups, and the widths of the models that are timed.
@pytest.mark.parametrize("ggml_type,n,k", [(12, 28672, 2560), (2, 28928, 3584), (12, 28672, 3584), (2, 28672, 4864), (12, 14336, 4864), (12, 7168, 4864), (12, 7168, 5888),
                                           (2, 6912, 1152), (12, 21504, 5376)])
def test_a_shared_item_fits_its_slot(ggml_type, n, k):
    """Two CTAs that share an item leave their sums in slots side by side: one may not reach into the other."""
    for kind in range(3):
        for rows in range(3, 17):
            s = _shape(ggml_type, n, k, rows, kind)
            assert s[ITEM] <= s[SLOT] or not s[SHARED], (rows, kind, s)
            assert s[SMEM] <= 227 * 1024 - 2048 and s[STAGES] >= 1 and 1 <= s[CTAS] <= 148


def test_shared_items_of_more_than_16_row_groups_are_met():
    """The case above is not an empty one."""
    s = _shape(12, 28672, 3584, 12, 1)
    assert s[SHARED] and s[UNITS] * s[GROUPS] > 16


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_a_cta_of_several_items_has_two_stages(kind):
    """With one stage nothing is fetched while a CTA multiplies: only for CTAs that have one item."""
    for ggml_type, step in ((2, 64), (12, 256)):
        for n in (1152, 5376, 16384, 21504, 65536, 131072, 262144):
            for k in (step, 768, 1536, 2560, 5376, 21504):
                for rows in (3, 8, 12, 16):
                    s = _shape(ggml_type, n, k, rows, kind)
                    items = -(-(-(-n // 16 // (1 if kind == 1 else s[GROUPS]))) // s[UNITS])
                    assert s[STAGES] >= 2 or items <= s[CTAS], (ggml_type, n, k, rows, s)


@pytest.mark.parametrize("sms", [1, 3, 132, 148, 160])
def test_shapes_of_odd_sizes(sms):
    for ggml_type, step in ((2, 64), (12, 256)):
        for n in (16, 48, 1008, 14352, 50000):
            for k in (step, 5 * step, 7168, 32768):
                for kind in range(3):
                    for rows in (1, 4, 7, 12, 16):
                        s = _shape(ggml_type, n, k, rows, kind, sms)
                        assert s[ITEM] <= s[SLOT] or not s[SHARED], (ggml_type, n, k, rows, kind, s)
                        assert s[UNITS] * s[SLICES] <= 16 and s[SMEM] <= 227 * 1024 - 2048


@pytest.mark.parametrize("args", [(8, 128, 256, 4, 0, 148), (2, 100, 256, 4, 0, 148), (2, 128, 96, 4, 0, 148), (12, 128, 64, 4, 0, 148), (2, 128, 256, 17, 0, 148),
                                  (2, 128, 256, 0, 0, 148), (2, 0, 256, 4, 0, 148), (2, 128, 256, 4, 3, 148), (2, 128, 256, 4, 0, 0)])
def test_problems_it_does_not_take(args):
    assert _lib.load().adam_b200_few_rows_shape(*args, (ctypes.c_uint32 * 10)()) < 0


def test_a_shape_is_searched_once():
    """A call that has been made before does not search again: a small part of the time of first calls, with a margin for noise."""
    f, out = _lib.load().adam_b200_few_rows_shape, (ctypes.c_uint32 * 10)()

    def seconds(sizes):
        t = time.perf_counter()
        for n in sizes:
            assert f(12, n, 5376, 8, 0, 148, out) == 0
        return time.perf_counter() - t

    first = min(seconds(range(20000 + 16000 * i, 30000 + 16000 * i, 16)) for i in range(3))
    again = min(seconds([21504] * 625) for _ in range(3))
    assert again < first / 3


# 0 and negative units, slices and tile pairs; products of two that are in range though neither is; more than shared memory holds.
@pytest.mark.parametrize("force", ["1,0,1,1,0", "1,1,0,1,0", "1,1,1,0,1", "1,-2,-3,1,0", "1,1,1,-1,0", "0,1,1,1,0", "3,1,1,1,0", "1,16,1,8,1", "2,16,1,1,1", "1,4,4,2,1"])
def test_a_forced_shape_is_taken_where_it_can_be(force):
    code = ("import ctypes; from adam_b200 import _lib; o = (ctypes.c_uint32 * 10)(); f = _lib.load().adam_b200_few_rows_shape\n"
            "for a in ((2, 1152, 1152, 8, 0, 148), (12, 28672, 2560, 13, 1, 148), (2, 48, 64, 3, 2, 148)):\n"
            "    assert f(*a, o) == 0; s = list(o); print(s)\n"
            "    assert s[1] >= 1 and s[2] >= 1 and s[1] * s[2] <= 16 and 1 <= s[3] <= 8 and s[4] >= 1 and 1 <= s[5] <= 148 and (not s[6] or s[7] <= s[8]) and s[9] <= 230000")
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, ADAM_B200_GM_SHAPE=force), capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr

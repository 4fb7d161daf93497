"""Launch shapes of the decode attention, chosen on the host: no GPU needed."""
import ctypes

import pytest

from adam_b200 import _lib

SMEM = 220 * 1024              # what the kernel's launches may ask for


def _shape(n_head, n_kv, head_dim, kv_dtype, batch, reach):
    out = (ctypes.c_uint32 * 6)()
    assert _lib.load().adam_b200_attention_shape(n_head, n_kv, head_dim, kv_dtype, batch, reach, out) == 0
    return list(out)


@pytest.mark.parametrize("kv_dtype", [0, 1])
@pytest.mark.parametrize("head_dim", [32, 64, 128, 256])
def test_every_head_is_there_and_every_cluster_fits(head_dim, kv_dtype):
    for group in range(1, 9):
        for n_kv in (1, 2, 4, 16):
            for batch in range(1, 80):
                heads, pairs, cluster, slots, smem, smem_splits = _shape(group * n_kv, n_kv, head_dim, kv_dtype, batch, 2048)
                assert heads * pairs == group * n_kv * batch
                # clusters of splits: one CTA per SM, whatever the cache's type
                assert cluster == (8 if pairs <= 16 else 4 if pairs <= 32 else 2 if 56 <= pairs <= 64 else 0)
                assert smem <= SMEM and 8 <= slots <= 16
                row = head_dim * (2 if kv_dtype else 4)
                assert smem_splits == 8 * 16 * row + (heads + 2) * head_dim * 4 <= SMEM          # eight slots beside the queries
                assert not cluster or smem == slots * 16 * row + (heads + 2) * head_dim * 4 + cluster * heads * (head_dim + 4) * 4


def test_longer_reach_takes_independent_splits():
    assert _shape(4, 1, 256, 1, 1, 2048)[2] == 8 and _shape(4, 1, 256, 1, 1, 2049)[2] == 0


@pytest.mark.parametrize("args", [(4, 0, 64, 0, 1, 64), (3, 2, 64, 0, 1, 64), (9, 1, 64, 0, 1, 64), (4, 1, 48, 0, 1, 64), (4, 1, 64, 2, 1, 64), (4, 1, 64, 0, 0, 64)])
def test_shapes_that_no_decoder_has(args):
    assert _lib.load().adam_b200_attention_shape(*args, (ctypes.c_uint32 * 6)()) < 0

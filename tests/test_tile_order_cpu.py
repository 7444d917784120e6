"""Tile order of ordinary products (csrc/tile_order.h, compiled for the host): every output tile
once, and as few bytes from DRAM as the order promises."""
import ctypes

import pytest


def _walk(M, N, K, rows=256, cols=256, pairs=74):
    from terapipe_b200.ops.lib import host_lib
    num_m, num_n = -(-M // rows), -(-N // cols)
    order, coords = (ctypes.c_int * 8)(), (ctypes.c_int * (2 * num_m * num_n))()
    n = host_lib().tp_tile_order_walk(3, M, N, K, rows, cols, 0, M, pairs, order, coords)
    assert n == num_m * num_n
    return [(coords[2 * i], coords[2 * i + 1]) for i in range(n)], order


@pytest.mark.parametrize("M,N,K", [(16384, 15360, 5120), (16384, 2048, 8192), (20480, 5120, 16384),
                                   (1024, 6144, 2048), (257, 8200, 128), (12288, 49152, 4096),
                                   (8, 8, 8), (18433, 2305, 768)])
@pytest.mark.parametrize("cols", [128, 256])
def test_every_tile_once_and_operands_few_times(M, N, K, cols):
    tiles, order = _walk(M, N, K, cols=cols)
    # distinct row and column blocks of a wave, against a square wave and against walking columns
    def read(seq):
        waves = [seq[i:i + 74] for i in range(0, len(seq), 74)]
        return sum(len({m for m, _ in w}) * 256 + len({n for _, n in w}) * cols for w in waves)
    num_m, num_n = -(-M // 256), -(-N // cols)
    plain = [(i % num_m, i // num_m) for i in range(num_m * num_n)]
    if order[2] == 0:
        assert tiles == plain
    elif order[5] * K * 2 * (cols if order[2] == 2 else 256) > 40 << 20:
        assert read(tiles) < 0.6 * read(plain)      # nothing stays in L2: the waves are near square
    else:
        # the cut dimension's blocks come back only inside their own group
        key = 1 if order[2] == 2 else 0
        seen = [t[key] // order[5] for t in tiles]
        assert seen == sorted(seen)

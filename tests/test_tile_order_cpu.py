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
@pytest.mark.parametrize("cols", [128, 192, 224, 256])
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


def _tile(M, N, K, b_mn=0, cut=1, second=0):
    from terapipe_b200.ops.lib import host_lib
    return host_lib().tp_choose_tile(M, N, K, b_mn, second, cut, 148)


@pytest.mark.parametrize("M,N,K,b_mn,code", [
    # an odd number of 128-row blocks, few of them: a pair's second CTA would have no rows
    (16, 15360, 5120, 1, 128), (77, 12288, 4096, 0, 128), (77, 12288, 4096, 1, 128), (128, 10240, 2560, 0, 128),
    (300, 12288, 3072, 1, 256), (600, 6912, 2304, 0, 256), (800, 2560, 10240, 1, 128),
    # N contiguous and more than four waves, which cost more than with K contiguous
    (10240, 3840, 1280, 1, 1256), (8192, 4800, 1600, 1, 1256), (8192, 3072, 768, 1, 1256),
    # few waves, the last one nearly empty at full width
    (2048, 5120, 10240, 0, 1192), (2048, 5120, 10240, 1, 1192), (2048, 7680, 5120, 0, 1224),
    # full widths where they fit, small products on small tiles
    (1024, 2048, 8192, 0, 1128), (16384, 8192, 2048, 1, 1256), (256, 256, 256, 0, 64)])
def test_tile_choice(M, N, K, b_mn, code):
    assert _tile(M, N, K, b_mn) == code


@pytest.mark.parametrize("M,N,K,code", [(8192, 3072, 768, 1192), (5120, 4096, 1024, 1192), (5120, 4096, 2048, 1256)])
def test_a_second_matrix_bounds_the_waves_of_a_short_product(M, N, K, code):
    assert _tile(M, N, K, b_mn=1, second=1) == code and _tile(M, N, K, b_mn=1) == 1256


@pytest.mark.parametrize("M,N,K,b_mn", [(2048, 5120, 10240, 0), (2048, 5120, 10240, 1), (2048, 7680, 5120, 0),
                                        (1024, 6144, 2048, 0)])
def test_all_gather_products_keep_full_widths(M, N, K, b_mn):
    assert _tile(M, N, K, b_mn) in (1192, 1224)
    assert _tile(M, N, K, b_mn, cut=0) in (1128, 1256)


@pytest.mark.parametrize("M,N,K,code", [
    # few tiles and a long K: two to eight parts
    (77, 768, 3072, 80064), (16, 768, 768, 40064), (128, 2048, 8192, 40064), (16, 2048, 8192, 40064),
    (64, 4096, 16384, 40128), (16, 8192, 2048, 20128), (256, 256, 4096, 80064),
    # clusters that would not all run at once: fewer parts
    (32, 1024, 4096, 40064), (300, 768, 3072, 20064),
    # 32 columns where these tiles run at once
    (256, 256, 256, 32), (77, 768, 768, 32), (77, 3072, 768, 32), (128, 4096, 1024, 32), (154, 3072, 768, 64),
    # enough tiles, or operands that take longer to fetch twice
    (128, 15360, 5120, 128), (1024, 2048, 8192, 1128), (640, 768, 3072, 20064), (16384, 2048, 8192, 1256)])
def test_small_products(M, N, K, code):
    from terapipe_b200.ops.lib import host_lib
    assert host_lib().tp_choose_small(M, N, K, 0, 0, 148) == code


def test_a_split_runs_at_once():
    """Every part has a stage of K, and the clusters fit on the chip together."""
    from terapipe_b200.ops.lib import host_lib
    for M in (1, 16, 77, 128, 129, 300, 1000):
        for N in (8, 64, 256, 768, 2048, 5120, 12288):
            for K in (8, 128, 256, 1000, 4096, 49152):
                code = host_lib().tp_choose_small(M, N, K, 0, 0, 148)
                parts, bn = divmod(code, 10000)
                if code == 32:
                    assert -(-M // 128) * -(-N // 32) <= 148
                if parts:
                    assert parts in (2, 4, 8) and bn in (64, 128) and parts <= -(-K // 128)
                    assert -(-M // 128) * -(-N // bn) * parts <= {2: 148, 4: 128, 8: 96}[parts]

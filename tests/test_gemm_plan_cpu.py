"""The rule that picks the kernel and the split of a dense GEMM is host code: checked without a GPU, for a chip of 148 SMs."""
import os

import pytest

from surogate_b200.ops import _build

if not os.path.exists(_build._so_path()):
    pytest.skip("the CUDA extension is not built", allow_module_level=True)


@pytest.fixture(scope="module")
def plan():
    from surogate_b200.ops import ext

    return lambda M, N, K, elem=2, a_mn=False, b_mn=False, fp32=False, acc=False, tile_n=0: ext().gemm_plan(M, N, K, elem, a_mn, b_mn, fp32, acc, tile_n, 148)


# measured on a B200, us: the other choice -> this one
@pytest.mark.parametrize("args,pair,split", [
    (dict(M=64, N=151936, K=64, fp32=True, acc=True), True, False),            # single CTAs 94 -> 34
    (dict(M=16, N=151936, K=512, elem=1, fp32=True, acc=True), True, False),   # single CTAs 91 -> 36
    (dict(M=64, N=24576, K=1024, fp32=True, acc=True), True, False),           # single CTAs 27 -> 19
    (dict(M=64, N=24576, K=64), False, False),
    (dict(M=2048, N=1024, K=8192), False, False),                              # pairs in two pieces 45 -> 37
    (dict(M=4096, N=512, K=16384, elem=1), False, False),                      # pairs in two pieces 46 -> 38
    (dict(M=16, N=12288, K=16384, elem=1), False, False),                      # three pieces 47 -> 41
    (dict(M=1, N=4096, K=4096), False, False),                                 # four pieces 18.7 -> 17.9
    (dict(M=1, N=4096, K=12288), False, True),                                 # whole 58 -> 31
    (dict(M=8192, N=16, K=8192, elem=1, b_mn=True), False, False),             # two pieces 27 -> 25
    (dict(M=16, N=6144, K=8192, elem=1, a_mn=True, b_mn=True), False, False),  # three pieces 27 -> 24
    (dict(M=16, N=151936, K=512, elem=1, a_mn=True, b_mn=True), True, False),  # single CTAs 98 -> 78
    (dict(M=6144, N=1024, K=16384, a_mn=True, b_mn=True), True, True),         # whole 204 -> 157
    (dict(M=4096, N=16, K=17408, b_mn=True), False, True),                     # whole 91 -> 45
    (dict(M=8192, N=4096, K=4096), True, False),
    (dict(M=16, N=4096, K=17408), False, True)])
def test_measured_choices(plan, args, pair, split):
    p = plan(**args)
    assert p[0] == pair and (p[1] > 1) == split, p


def test_every_plan_can_run(plan):
    """Pieces of at least four 128-byte blocks, cut tiles behind whole waves only, a workspace that holds every piece and stays below 64 MB;
    narrow outputs never on pairs; forced kernels as asked."""
    sizes = [1, 8, 16, 100, 128, 129, 256, 520, 1000, 2048, 3000, 8192, 16384, 151936]
    up = lambda a, b: -(-a // b)
    for M in sizes:
        for N in (8, 16, 128, 136, 512, 1000, 4096, 24576, 151936):
            for K in (8, 64, 200, 1024, 4104, 16384, 151936):
                for elem in (1, 2):
                    for fp32, acc in ((False, False), (False, True), (True, False), (True, True)):
                        for tile_n in (0, 128, 256, 512):
                            pair, pieces, first, ws = plan(M, N, K, elem, fp32=fp32, acc=acc, tile_n=tile_n)
                            assert pair == (tile_n == 512) if tile_n else not (pair and N <= 128)
                            tile, slots = (256, 74) if pair else (128, 148)
                            tiles = up(M, tile) * up(N, tile)
                            if pieces == 1:
                                assert ws == 0
                                continue
                            assert tile_n in (0, 512) and 2 <= pieces <= 8 and up(K * elem, 128) // pieces >= 4
                            assert first % slots == 0 and 0 < tiles - first < slots
                            assert ws == 4 * (tiles - first) * (pieces * tile * tile + (8 if pair else 4)) and ws < 64 << 20

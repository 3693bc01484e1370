"""The rules that choose a kernel's launch from the sizes (CPU): called in the built library by their
C++ names, they launch nothing."""
import ctypes

import pytest

import eigen_b200 as eb

I64 = ctypes.c_int64


def _rule(symbol, restype, *argtypes):
    f = eb.load()[symbol]
    f.restype, f.argtypes = restype, argtypes
    return f


@pytest.mark.parametrize("rounds,k,small", [(1, 1200, True), (1, 1201, False), (2, 600, True), (2, 601, False),
                                            (10, 1, True), (11, 1, False), (10, 64, True), (11, 64, False),
                                            (11, 65, True), (12, 65, False), (12, 100, False), (60, 4, False),
                                            (1200, 1, False)])
def test_small_sgemm_pays_whole_k_tiles(rounds, k, small):
    # a round of 148 tiles costs a whole 64-deep K tile however short K is, so shallow products take
    # the kernel for few rounds only
    applies = _rule("_ZN3eb219sgemm_small_appliesElll", ctypes.c_bool, I64, I64, I64)
    assert applies(148 * 32, 32 * rounds, k) == small
    assert applies(32 * rounds, 148 * 32, k) == small


@pytest.mark.parametrize("m,n,k,aligned,unaligned", [
    (2048, 2048, 32, 128, 128), (2500, 2500, 16, 128, 128), (3000, 3000, 20, 128, 128), (1300, 1300, 16, 128, 128),
    (7000, 7000, 4, 128, 64), (1700, 1700, 32, 64, 64), (1000, 1000, 16, 64, 64), (3500, 1000, 24, 64, 64),
    (2048, 2048, 128, 64, 64), (128, 128, 128, 32, 32), (4096, 4096, 1024, 128, 128)])
def test_native_tile_of_shallow_products(m, n, k, aligned, unaligned):
    # few K tiles: the wave's fixed cost decides, as timed
    tile = _rule("_ZN3eb29dmma_tileElllb", ctypes.c_int, I64, I64, I64, ctypes.c_bool)
    assert tile(m, n, k, True) == aligned
    assert tile(m, n, k, False) == unaligned


def test_reconstruction_rounds_of_blocks():
    # 592 resident blocks; a round costs its run and one group: never much above an even split
    run_of = _rule("_ZN3eb211crt_rec_runEllb", I64, I64, I64, ctypes.c_bool)
    for row_blocks in [*range(1, 40), 100, 148, 157, 199, 297, 313, 400, 591, 592, 593, 594, 625, 1000, 3000]:
        for groups in (1, 2, 7, 32, 125, 225, 250, 500, 512, 2048):
            run = run_of(row_blocks, groups, False)
            assert 1 <= run <= groups
            used = -(-groups // run)
            cost = -(-row_blocks * used // 592) * (run + 1)
            even = row_blocks * groups / 592
            assert cost <= 1.3 * even + 6, (row_blocks, groups, run, cost, even)
            # the blocks with work fill the chip, unless a run is down to one group
            tri = run_of(row_blocks, groups, True)
            assert tri == 1 or row_blocks * (-(-groups // tri)) / 2 >= 592, (row_blocks, groups, tri)

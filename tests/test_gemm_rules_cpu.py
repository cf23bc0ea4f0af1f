"""Which kernel a product goes to, on both sides of each line of the rules."""
import ctypes
import re

import pytest

from hetu_galvatron_b200.csrc import build
from hetu_galvatron_b200.ops import _lib
from hetu_galvatron_b200.ops.gemm import OUT_BF16, OUT_F32, OUT_F32_ACC, _use_grouped_pair, _use_skinny


# the last two: as many columns as the few-row kernel's grid has tiles for, and one more
@pytest.mark.parametrize("M,N,K,few_rows", [(64, 512, 512, True), (65, 512, 512, False), (128, 4096, 1535, False),
                                            (128, 4096, 1536, True), (128, 8192, 3064, False), (128, 8192, 3072, True),
                                            (128, 8200, 4096, False), (129, 512, 4096, False), (1, 65535 * 128, 64, True),
                                            (1, 65535 * 128 + 1, 64, False)])
def test_rule_of_the_few_row_kernel(M, N, K, few_rows):
    assert _use_skinny(M, N, K, False, OUT_BF16, 0, None) is few_rows


@pytest.mark.parametrize("rows,N,K,G,pair", [(4096, 4096, 2560, 8, True), (4095, 4096, 2560, 8, False), (4096, 4096, 2552, 8, False),
                                             (4096, 255, 4096, 8, False), (512, 256, 4096, 1, True)])
def test_rule_of_the_grouped_pair_kernel(rows, N, K, G, pair):
    assert _use_grouped_pair(rows, N, K, G) is pair


def test_shared_tiles_wait_for_no_other_pair():
    """Nothing says in which order the device starts the pairs that share a tile: no warp of one may wait for another."""
    text = (build.CSRC / "sm100" / "gemm2_core.cuh").read_text()
    body = text.split("void epilogue2(", 1)[1]
    for name in ("split_arrive", "add"):
        body += text.split(" %s(" % name, 1)[1].split("\n}\n", 1)[0]
    body = re.sub(r"//.*", "", body)
    assert "split_token" in body and not re.findall(r"\bwhile\b|ld_acquire|__nanosleep", body)


def test_parts_of_shared_tiles_are_dealt_in_the_blocks_of_the_stores():
    """A warp that adds parts has counted the arrivals of the warps of its own number alone: both deals have one block size."""
    text = re.sub(r"//.*", "", (build.CSRC / "sm100" / "gemm2_core.cuh").read_text())
    store = text.split("void store_tile_tma(", 1)[1].split("\n}\n", 1)[0]
    parts = text.split("void epilogue2(", 1)[1].split("split_arrive(", 1)[0]
    assert "kBlock = block_columns(true," in store and "cols = block_columns(p.c_tma != 0, p.out_mode)" in parts
    assert "c = w.h * kBlock;" in store and "c += w.H * kBlock" in store
    assert "c0 = share.h * cols;" in parts and "c0 += H * cols" in parts


def test_nothing_throws_at_the_entry_points():
    """They are called from C: std::random_device raises where the system has no source of entropy."""
    for path in (build.CSRC / "sm100").glob("*.cu*"):
        assert not re.search(r"random_device|\bthrow\b|\.at\(", re.sub(r"//.*", "", path.read_text())), path.name


# 74 pairs.  Narrower tiles that promise more than a twentieth, less, and turned ones that promise less; a last wave that is shared
@pytest.mark.parametrize("M,N,K,mode,bn,turned,shared", [
    (1531, 3584, 3584, OUT_BF16, 192, 0, False), (4608, 2304, 1248, OUT_BF16, 192, 0, False), (12288, 1600, 808, OUT_BF16, 256, 0, False),
    (12288, 1600, 1168, OUT_F32, 256, 0, False), (11008, 2304, 784, OUT_F32, 256, 0, False), (6400, 1600, 4160, OUT_F32, 224, 0, False),
    (345, 32000, 1600, OUT_BF16, 192, 1, False), (320, 4096, 22016, OUT_BF16, 160, 1, True), (200, 3584, 8192, OUT_F32, 160, 0, True)])
def test_plans_of_products(M, N, K, mode, bn, turned, shared):
    plan = (ctypes.c_int * 5)()
    _lib.load().hg_gemm2_plan(M, N, K, mode, 1, 0, 74, plan)
    assert plan[:2] == [bn, turned] and (plan[2] > 1) is shared


# K-blocks of 512 cycles in tiles of 256 columns: the last with two epilogue warps per 32 rows and the first with one
@pytest.mark.parametrize("mode,mn,blocks", [(OUT_BF16, 0, 15), (OUT_BF16, 1, 10), (OUT_F32, 0, 15), (OUT_F32, 1, 15), (OUT_F32_ACC, 1, 39)])
def test_rule_of_the_epilogue_warps(mode, mn, blocks):
    for n, warps in ((blocks, 2), (blocks + 1, 1)):
        plan = (ctypes.c_int * 5)()
        _lib.load().hg_gemm2_plan(256 * 74, 256, 64 * n, mode, 0, mn, 74, plan)
        assert plan[0] == 256 and plan[4] == warps


def test_tiles_of_every_width_are_tested():
    """What the cases of the GPU test are cut into: narrower and turned tiles, alone and shared."""
    from tests.test_gemm_epilogue_gpu import test_tiles_of_every_width as tested

    shapes = next(m.args[1] for m in tested.pytestmark if m.name == "parametrize" and m.args[0] == "M,N,K")
    found = set()
    for mode, may_turn in ((OUT_BF16, 1), (OUT_BF16, 0), (OUT_F32, 0)):
        for shape in shapes:
            plan = (ctypes.c_int * 5)()
            _lib.load().hg_gemm2_plan(*shape, mode, may_turn, 0, 74, plan)
            found.add((mode, plan[0] < 256, bool(plan[1]), plan[2] > 1))
    assert found >= {(OUT_BF16, True, True, True), (OUT_BF16, True, False, False), (OUT_BF16, True, False, True),
                     (OUT_BF16, False, False, False), (OUT_F32, True, False, False), (OUT_F32, True, False, True)}

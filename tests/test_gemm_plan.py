"""The rules that choose a GEMM's kernel, order of tiles and work items (``csrc/gemm.cu``), asked on the host for a GPU of 148
SMs, which is what the library assumes without one."""
import ctypes

import pytest

from distdl_b200 import _native

pytestmark = pytest.mark.skipif(not _native.available(), reason="native library not built")
SINGLE, PAIR, PAIR_HALF, WIDE = range(4)
F_OUT_F32 = 1


def plan(M, N, K, batch=1, flags=0, max_ctas=0, rows=0, bound_k=0):
    out = (ctypes.c_int * 7)()
    assert _native.lib().dd_gemm_plan(M, N, K, batch, flags, max_ctas, rows, bound_k, out) == 0
    return dict(zip(("kernel", "ctas", "group", "full", "items", "parts", "ahead"), out))


@pytest.fixture(autouse=True)
def on_148_sms():
    if plan(4096, 4096, 64)["ctas"] != 148:
        pytest.skip("figures for 148 SMs")


@pytest.mark.parametrize("M,N,K,batch,items", [
    (1, 4096, 4096, 1, 32), (4, 4096, 4096, 1, 32), (15, 4096, 4096, 1, 32), (16, 4096, 4096, 1, 64),  # 16 tiles: halves, then quarters
    (1, 8192, 4096, 1, 32), (33, 8192, 4096, 1, 128), (1, 14336, 4096, 1, 56), (16, 14336, 4096, 1, 112),
    (1, 2048, 4096, 1, 32), (1, 4096, 8192, 1, 32), (8, 4096, 8192, 1, 64), (32, 8192, 1024, 1, 32), (64, 8192, 1024, 1, 128),
    (1, 4096, 4096, 2, 32), (16, 4096, 4096, 2, 128), (1, 2048, 2048, 4, 32)])
def test_few_rows_that_lie_close_together_are_read_by_few_ctas(M, N, K, batch, items):
    """An A of less than 128 KB in no more than 32 parts of tiles: in more, the CTAs wait for one another's reads of it."""
    p = plan(M, N, K, batch)
    assert p["kernel"] == SINGLE and p["items"] == items


@pytest.mark.parametrize("M,N,K,max_ctas,ahead", [
    (1, 14336, 4096, 0, 0), (8, 24576, 4096, 0, 0), (1, 4096, 4096, 0, 1), (1, 12288, 4096, 0, 1), (33, 14336, 4096, 0, 1),
    (4096, 4096, 4096, 0, 1), (33, 14336, 4096, 64, 0), (4096, 4096, 4096, 64, 0), (8192, 8192, 8192, 64, 0),
    (4096, 4096, 4096, 148, 1)])
def test_products_that_are_launched_ahead(M, N, K, max_ctas, ahead):
    """Not those that are limited to some SMs, nor many CTAs that read an A of less than 128 KB."""
    assert plan(M, N, K, max_ctas=max_ctas)["ahead"] == ahead


@pytest.mark.parametrize("M,N,K,group", [(7582, 9272, 64, 4), (9272, 7584, 512, 4), (8192, 28672, 4096, 17), (4096, 50304, 1600, 16),
                                         (28672, 8192, 4096, -17), (2304, 2816, 1024, 9), (16384, 16384, 16384, 8)])
def test_order_of_tiles(M, N, K, group):
    """Rows of D for short contractions, else a panel of up to 36 MB of the smaller operand."""
    p = plan(M, N, K)
    assert p["group"] == group and p["kernel"] in (PAIR, WIDE)


@pytest.mark.parametrize("M,N,K,batch,kernel", [
    (320, 28672, 4096, 8, WIDE), (320, 14336, 4096, 8, WIDE), (960, 16384, 3072, 8, WIDE),       # dead blocks on every other pair
    (320, 4096, 8192, 8, PAIR), (640, 4096, 14336, 8, PAIR),                                     # ... in too few waves, or few of them
    (320, 4096, 14336, 8, PAIR), (320, 4096, 28672, 8, PAIR),                                    # ... once a block is live in part
    (1280, 28672, 4096, 8, WIDE), (1280, 4096, 14336, 8, WIDE),                                  # at the power limit
    (1280, 11264, 2048, 8, PAIR), (1000, 28672, 4096, 8, PAIR), (2560, 2048, 5632, 4, PAIR),    # an odd number of blocks, or all live
    (1000, 2824, 512, 8, WIDE), (1000, 2824, 512, 4, PAIR)])
def test_entries_with_live_rows_take_wide_tiles_only_where_those_are_faster(M, N, K, batch, kernel):
    assert plan(M, N, K, batch, rows=1)["kernel"] == kernel


def test_live_rows_of_narrow_products_by_rows():
    """By columns, the tiles without live rows would follow one another on the same pairs."""
    assert plan(1698, 576, 10496, 16, rows=1)["group"] == 4 and plan(1698, 576, 10496, 16)["group"] < 0

"""The rules by which the kernel wrappers size their grids and choose a product: pure
functions of the sizes, checked without a GPU."""
import pytest
import torch

from tiny_llm_infer_b200 import ops


def test_decode_splits_give_enough_blocks_with_enough_keys_each():
    assert ops.decode_splits(8, 8, 4096) == 4            # about a thousand keys per block
    assert ops.decode_splits(1, 8, 4096) == 16           # few rows: at least 128 blocks in all
    assert ops.decode_splits(64, 8, 4096) == 4
    assert ops.decode_splits(1, 1, 100) == 1             # never less than 128 keys a block
    assert ops.decode_splits(1, 1, 1 << 20) == 64        # and never more than 64 blocks a row
    for rows in (1, 3, 8, 64):
        for ctx in (1, 17, 300, 5000):
            s = ops.decode_splits(rows, 2, ctx)
            assert 1 <= s <= 64 and (s == 1 or ctx / s >= 64)


def test_prefill_splits_fill_the_gpu_only_when_runs_stay_long():
    assert ops.prefill_splits(32, 256) == 1 and ops.prefill_splits(32, 1024) == 2
    assert ops.prefill_splits(32, 4096) == 4 and ops.prefill_splits(16, 8192) == 8
    assert ops.prefill_splits(64, 4096) == 2 and ops.prefill_splits(128, 65536) == 1
    for blocks in (1, 3, 40, 200):
        for ctx in (64, 1000, 40000):
            s = ops.prefill_splits(blocks, ctx)
            assert s in (1, 2, 4, 8) and (s == 1 or (blocks * s <= ops.SM_COUNT and -(-ctx // 64) // s >= 8))


def test_the_tcgen05_product_is_chosen_where_its_tiles_fill_the_gpu():
    bf = torch.bfloat16
    assert ops.tcgen05_pays(2048, 4096, 4096, bf) and ops.tcgen05_pays(2048, 12288, 4096, bf, col_tile=128)
    assert not ops.tcgen05_pays(2048, 6144, 4096, bf)            # 8 x 24 tiles: a ragged second round
    assert not ops.tcgen05_pays(64, 4096, 4096, bf) and not ops.tcgen05_pays(2048, 4096, 4096, torch.float32)
    assert not ops.tcgen05_pays(2048, 4096, 4100, bf)            # K no multiple of 8


@pytest.mark.parametrize("mode,segments,each,heads,dk,cols,chunks", [
    # (recurrence, portions, tokens of each, heads, key elements, value columns): measured to be faster by chunks, or not
    ("delta", 1, 2048, 32, 128, 128, True), ("delta", 8, 256, 64, 128, 128, True), ("delta", 1, 2048, 32, 64, 128, True),
    ("delta", 3, 701, 32, 64, 128, True), ("delta", 4, 256, 32, 64, 128, False), ("delta", 12, 701, 64, 64, 64, False),
    ("delta", 6, 256, 64, 128, 16, False), ("delta", 4, 256, 16, 64, 256, False), ("plain", 8, 256, 64, 64, 16, False),
    ("plain", 8, 256, 32, 64, 64, False), ("plain", 8, 256, 32, 128, 64, True), ("plain", 8, 256, 32, 64, 128, True),
    ("head", 8, 256, 64, 64, 64, True), ("head", 12, 256, 64, 64, 16, False), ("head", 1, 1023, 64, 128, 64, True),
    ("fixed", 3, 701, 32, 128, 128, True), ("fixed", 8, 160, 32, 64, 64, False), ("fixed", 4, 90, 16, 64, 128, False),
    ("delta", 1, 64, 32, 128, 128, False), ("delta", 8, 64, 32, 128, 128, True), ("delta", 64, 2, 32, 128, 128, False),
])
def test_recurrences_go_by_chunks_where_that_is_faster(mode, segments, each, heads, dk, cols, chunks):
    code = {"delta": ops.SCAN_DELTA, "plain": ops.SCAN_PLAIN, "head": ops.SCAN_HEAD_DECAY, "fixed": ops.SCAN_FIXED_DECAY}[mode]
    assert ops.chunks_pay(code, segments, segments * each, heads, dk, cols) == chunks


def test_runs_of_keys_of_one_token_attention():
    runs = ops.biased_decode_splits
    assert runs(8, 8, 2000) == 4 and runs(16, 8, 4000) == 2 and runs(40, 8, 4000) == 3 and runs(64, 8, 2000) == 1
    assert runs(80, 2, 1000) == 3 and runs(40, 4, 1000) == 3 and runs(20, 8, 1000) == 3      # whole rounds alone would take one
    assert runs(1, 1, 100) == 1 and runs(1, 1, 1 << 20) == 64
    for rows in (1, 3, 8, 64, 300):
        for reach in (1, 200, 611, 5000):
            assert 1 <= runs(rows, 8, reach) <= max(1, min(reach // 192, 64))
    before = runs.cache_info().hits                      # a step asks once per layer: the search is not made again
    assert runs(8, 8, 2000) == 4 and runs.cache_info().hits == before + 1 and runs.cache_info().maxsize

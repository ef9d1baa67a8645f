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


@pytest.mark.parametrize("rows,columns,k,plain,gated", [
    # 9 to 16 rows: measured to be faster than the library (plain), than it and the activation's kernel (gated)
    (8, 4096, 12288, True, True), (9, 4096, 1024, True, True), (16, 4096, 1024, True, True), (17, 4096, 1024, False, False),
    (16, 4736, 1536, True, True), (16, 4752, 1536, False, True), (16, 4736, 1544, False, True), (16, 1184, 4096, True, True),
    (16, 1200, 4096, False, True), (16, 1184, 4104, False, True), (16, 2560, 9728, False, False), (16, 4096, 12288, False, False),
    (9, 2048, 2048, False, True), (16, 7104, 1536, False, True), (16, 7120, 1536, False, False), (16, 7104, 1544, False, False),
    (16, 4096, 8192, False, True), (16, 512, 8200, False, False), (16, 64, 2048, True, True), (16, 64, 2052, False, False), (8, 64, 2052, False, False),
])
def test_products_of_few_rows(rows, columns, k, plain, gated):
    x, w = torch.empty(rows, k, dtype=torch.bfloat16), torch.empty(columns, k, dtype=torch.bfloat16)
    assert ops.skinny_pays(x, w) == plain and ops.skinny_pays(x, w, gated=True) == gated


def test_products_of_few_rows_want_whole_rows_on_16_bytes():
    base = torch.empty(16 * 64 + 8, dtype=torch.bfloat16)
    w = torch.empty(64, 64, dtype=torch.bfloat16)
    for rows, off, pays in ((16, 0, True), (16, 8, True), (16, 1, False), (16, 4, False), (9, 1, False)):
        assert ops.skinny_pays(base[off:off + rows * 64].view(rows, 64), w) == pays
    assert not ops.skinny_pays(torch.empty(64, 16, dtype=torch.bfloat16).t(), w)
    assert not ops.skinny_pays(torch.empty(16, 64, dtype=torch.bfloat16), torch.empty(64, 64, dtype=torch.bfloat16).t())


@pytest.mark.parametrize("rows,columns,k,pays", [
    (64, 8192, 1024, True), (64, 8188, 1024, False), (512, 1024, 1024, True), (595, 4096, 1024, True), (63, 16384, 1024, False),
    (64, 2048, 1028, True), (64, 2036, 1028, False), (128, 832, 1280, True), (64, 1408, 1536, True), (64, 1024, 2048, True),
    (64, 1020, 2048, False), (595, 1024, 2048, True), (595, 96, 64, False), (64, 4096, 4098, False), (64, 4098, 4096, False), (9, 8192, 8192, False),
])
def test_large_float32_products_run_on_the_tensor_cores(rows, columns, k, pays):
    assert ops.f32_tcgen05_pays(torch.empty(rows, k), torch.empty(columns, k)) == pays


def test_float32_operands_off_the_grid_stay_with_the_library():
    w = torch.empty(2048, 2048)
    base = torch.empty(64 * 2048 + 4)
    for off, pays in ((0, True), (4, True), (1, False), (2, False)):
        assert ops.f32_tcgen05_pays(base[off:off + 64 * 2048].view(64, 2048), w) == pays
    x = torch.empty(64, 2048)
    assert not ops.f32_tcgen05_pays(torch.empty(2048, 64).t(), w) and not ops.f32_tcgen05_pays(x, torch.empty(2048, 4096)[:, ::2])
    assert not ops.f32_tcgen05_pays(x, torch.empty(2048, 2048, requires_grad=True))


def test_shares_of_float32_sums_fill_the_gpu():
    assert ops.f32_splits(595, 4096, 1024) == 2 and ops.f32_splits(2048, 24576, 4096) == 1        # 160 tiles; far more than SMs
    assert ops.f32_splits(595, 1024, 2048) == 3 and ops.f32_splits(64, 1024, 2048) > 3 and ops.f32_splits(64, 4, 64) == 1
    for rows in (64, 300, 595, 2048):
        for columns in (96, 1024, 4096):
            for k in (64, 1028, 4096, 12288):
                s, slabs, tiles = ops.f32_splits(rows, columns, k), -(-k // 64), -(-rows // 128) * -(-columns // 128)
                assert 1 <= s <= min(slabs, 16) and (s == 1 or -(-tiles * s // ops.SM_COUNT) * -(-slabs // s) < -(-tiles // ops.SM_COUNT) * slabs)
